// sor_stream.cuh -- red-black SOR on the colour-split layout, NH / 2 whole
// iterations per pass over the grid (temporal blocking in registers).
//
// What bounds the separate colour sweeps on grids too large for the resident
// launch is traffic: a sweep moves the other colour twice (with its row
// halos), its own colour, the source and the result through L2 (185 MB at
// 256^3, 7.9 TB/s), and the arrays through HBM once they outgrow L2.  Here a
// pass moves the iterate and the source in and the iterate out once for NH
// half sweeps.  Microseconds an iteration, separate sweeps -> passes of two:
//   200^3 28.4 -> 22.0   224^3 35.6 -> 29.6   256^3 47.2 -> 42.3
//   288^3 103 -> 59.7    320^3 127 -> 71.6    384^3 187 -> 130     512^3 398 -> 287
// Now bound by the halo that every window computes again (1.9 updates for one
// that counts at 256^3, 1.6 at 512^3) and by latency: 16 warps an SM (the rings
// take all registers) issue 36% of the time, waiting for loads and shared
// memory; 2 TB/s of HBM at 256^3, 2.8 at 512^3.
//
// A CTA owns a tile of rows and vectors (16 bytes, V cells of one colour) of a
// chunk of planes, plus a halo of NH rows, planes and cells on each side that
// it recomputes; a thread owns one vector of one row and streams along i.  At
// step p half sweep h updates plane p - h, so the x neighbours of every half
// sweep are the thread's own registers (rings of NR planes, indexed at compile
// time); the y neighbours and the z neighbour outside the vector come from
// shared memory, where every thread leaves, per step, the vectors the next
// step's half sweeps read (one barrier per step).  The iterate's planes are
// loaded straight into the ring, a step ahead; the source's go to shared memory
// by cp.async (as loads too they held the step up: a warp's few scoreboards are
// shared with its shared-memory reads, which then wait for the loads).
//
// Halo cells hold wrong values more and more towards the window's edge --
// after half sweep h, h + 1 cells deep -- which owned cells never read.  The
// pass is out of place, so no CTA sees another's update.  Per cell the update
// is SorCoef<T>::update with the sweeps' operands: the iterates and norms are
// theirs bit for bit.
//
// Stop rule: the norms of a pass's iterations are known when it has ended.  If
// its first iteration was the last of the solve, the caller repeats that one
// iteration (NH = 2) from the pass's input, which is still there.
#pragma once
#include "hc_internal.cuh"
#include "sor_resident.cuh"

namespace hc {

constexpr size_t STREAM_SMEM = 225 * 1024;
// 2 NH windows with room, 6 without
inline size_t stream_smem(int NH, int W, int WV)
{
    return ((size_t)(2 * NH) * (W + 2) + 6 * W) * WV * 16 + 6 * 16 + WV * 16 + 64;
}

// threads of a CTA: the rings of two iterations take all 128 registers
constexpr int STREAM_NT4 = 512, STREAM_NT2 = 768;

struct StreamArgs {
    const float *in;
    float *out;
    const float *src;
    Split sp;
    SorCoef<float> cf;
    StreamTile t;
    double *res;
    int iter0;
    int pair;              // iterations of the passes before this one (their norms are tested), 0: the first
    double thresh;
    DevScalars *sc;
    int force;             // run whatever the stop flag says
};

// The solve is over when an iteration before iter0 left the norm below
// thresh; of the last pass's iterations the first such one counts.
__device__ __forceinline__ bool stream_stop(const double *res, int iter0, int pair, double thresh, DevScalars *sc,
                                            bool mark)
{
    if (*(volatile int *)&sc->done) return true;
    for (int q = max(0, iter0 - pair); q < iter0; q++)
        if (__longlong_as_double(*reinterpret_cast<const volatile long long *>(res + q)) < thresh) {
            if (mark) {
                sc->last_iter = q + 1;
                sc->done = 1;
            }
            return true;
        }
    return false;
}

static __global__ void stream_check_kernel(const double *res, int iter0, int pair, double thresh, DevScalars *sc)
{
    stream_stop(res, iter0, pair, thresh, sc, true);
}

template <int NH, int NT, bool EVEN>
__global__ void __launch_bounds__(NT, 1) sor_stream_kernel(const StreamArgs A)
{
    using T = float;
    constexpr int V = Pack<T>::V, NR = 6;
    using P = Pack<T>;
    extern __shared__ __align__(16) unsigned char st_smem[];
    __shared__ double wmax[NH / 2][NT / 32];
    pdl_wait_and_release();
    if (!A.force && stream_stop(A.res, A.iter0, A.pair, A.thresh, A.sc, threadIdx.x == 0)) return;

    const Split sp = A.sp;
    const StreamTile tl = A.t;
    const int tid = threadIdx.x, lane = tid & 31;
    const int H = sp.H, Hv = H / V, nz = sp.nz;
    // window rows [j0, j0 + W) with owned rows [ja, jb), vectors likewise
    const int tj = blockIdx.x % tl.tj, tk = blockIdx.x / tl.tj;
    const int jhalo = NH, vhalo = (NH + V - 1) / V;
    const int ja = tj == 0 ? 1 : tl.W - jhalo + (tj - 1) * tl.BJ;
    const int jb = tj == tl.tj - 1 ? sp.ny - 1 : tl.W - jhalo + tj * tl.BJ;
    const int j0 = tj == 0 ? 0 : ja - jhalo;
    const int va = tk == 0 ? 0 : tl.WV - vhalo + (tk - 1) * tl.BV;
    const int vb = tk == tl.tk - 1 ? Hv : tl.WV - vhalo + tk * tl.BV;
    const int v0 = tk == 0 ? 0 : va - vhalo;
    const int ia = 1 + blockIdx.y * tl.L, ie = min(sp.nx - 1, ia + tl.L);
    if (ia >= ie) return;

    const int jr = rs_div(tid, A.t.magic), j = j0 + jr, v = v0 + tid - jr * tl.WV;
    const bool in = jr < tl.W && j < sp.ny && v < Hv;
    const bool inner = in && j >= 1 && j <= sp.ny - 2;
    const bool own = inner && j >= ja && j < jb && v >= va && v < vb;
    const ResCoef<T> cf(A.cf);
    const int cs = (int)sp.cs, rp = sp.ny * H;
    const int base = in ? j * H + v * V : 0;   // offset of the thread's vector in plane 0

    // shared memory, in units of the window (lev: with a row of room at both
    // ends): what half sweeps 0 .. NH - 1 read, of 2 steps, then 3 planes each
    // of the red and the black source
    const int rowb = tl.WV * 16, win = tl.W * rowb, lev = win + 2 * rowb;
    const int mine = min(tid, tl.W * tl.WV) * 16;   // threads beyond the window share the room
    const int oX = rowb + mine, oS = NH * 2 * lev + mine, oT = oS + 3 * (win + 16);
    auto at = [&](int off) -> P & { return *reinterpret_cast<P *>(st_smem + off); };
    auto one = [&](int off) -> T { return *reinterpret_cast<const T *>(st_smem + off); };
    const unsigned sm0 = (unsigned)__cvta_generic_to_shared(st_smem);
    // Plane q, whatever it is (planes and rows outside the grid fetch others,
    // which no owned cell reads: a condition would make a slot a copy of the
    // load, and the copy wait for it)
    auto where = [&](const T *f, int c, int q) { return f + (c ? cs : 0) + min(max(q, 0), sp.nx - 1) * rp + base; };
    auto fetch = [&](P &d, int c, int q) {          // of the iterate, into its slot
        uint4 u;
        asm volatile("ld.global.nc.v4.u32 {%0, %1, %2, %3}, [%4];"
                     : "=r"(u.x), "=r"(u.y), "=r"(u.z), "=r"(u.w)
                     : "l"(where(A.in, c, q)));
        memcpy(&d, &u, 16);
    };
    auto fetch_src = [&](int off, int c, int q) {   // of the source, to shared memory
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(sm0 + off), "l"(where(A.src, c, q)) : "memory");
    };
    auto commit = [&]() { asm volatile("cp.async.commit_group;" ::: "memory"); };

    P rd[NR], bl[NR], sr[NR], sb[NR];   // red, black, their sources: plane q at slot (q - a + 1) % NR
    const P zero = {};
#pragma unroll
    for (int q = 0; q < NR; q++) rd[q] = bl[q] = sr[q] = sb[q] = zero;
    const int a = max(0, ia - NH), pend = ie + NH - 2;
    T rmax[NH / 2];
#pragma unroll
    for (int q = 0; q < NH / 2; q++) rmax[q] = (T)0;

    for (int o = tid * 16; o < NH * 2 * lev + 6 * (win + 16); o += NT * 16) at(o) = zero;
    __syncthreads();
    // what the first step, p = a + 1 (slot 2), finds
    fetch(bl[1], 1, a);
    fetch(bl[2], 1, a + 1);
    fetch(bl[3], 1, a + 2);
    fetch(rd[1], 0, a);
    fetch(rd[2], 0, a + 1);
#pragma unroll
    for (int g = 0; g < 2; g++) {
        fetch_src(oS + ((2 + g) % 3) * (win + 16), 0, a + 1 + g);
        fetch_src(oT + ((1 + g) % 3) * (win + 16), 1, a + g);
        commit();
    }
    at(oX) = bl[2];
    __syncthreads();

    int p = a + 1;
    int s = (p + j) & 1;   // z parity of every half sweep of a step
    int zoff = s ? 16 : -(int)sizeof(T);   // the z neighbour outside the vector
    // whole turns of the ring: steps beyond pend only touch planes that are not owned
#pragma unroll 1
    while (p <= pend) {
#pragma unroll
        for (int k = 0; k < NR; k++) {
            constexpr int O = 2;
            const int rdb = (k & 1) * lev, wrb = ((k + 1) & 1) * lev;   // buffers read / written (NR is even)
            asm volatile("cp.async.wait_group 1;" ::: "memory");
            fetch(bl[(k + O + 2) % NR], 1, p + 2);
            fetch(rd[(k + O + 1) % NR], 0, p + 1);
            fetch_src(oS + ((k + O + 2) % 3) * (win + 16), 0, p + 2);
            fetch_src(oT + ((k + O + 1) % 3) * (win + 16), 1, p + 1);
            commit();
            sr[(k + O) % NR] = at(oS + ((k + O) % 3) * (win + 16));
            sb[(k + O + NR - 1) % NR] = at(oT + ((k + O + 2) % 3) * (win + 16));
#pragma unroll
            for (int h = 0; h < NH; h++) {
                const int q = p - h;   // its plane; slots of planes q - 1, q, q + 1
                const int m0 = (k + O - h - 1 + 2 * NR) % NR, m1 = (k + O - h + 2 * NR) % NR,
                          m2 = (k + O - h + 1 + 2 * NR) % NR;
                P &x = (h & 1) ? bl[m1] : rd[m1];
                const P &xm = (h & 1) ? rd[m0] : bl[m0], &x0 = (h & 1) ? rd[m1] : bl[m1],
                        &xp = (h & 1) ? rd[m2] : bl[m2];
                const P &r = (h & 1) ? sb[m1] : sr[m1];
                const int buf = oX + h * 2 * lev + rdb;
                if (q >= 1 && q <= sp.nx - 2) {   // uniform over the CTA
                    const P ym = at(buf - rowb), yp = at(buf + rowb);
                    const T ze = one(buf + zoff);   // of the same row, as the y neighbours
                    T m = (T)0;
                    P nw = x;
                    rs_update<T, EVEN>(nw, xm, x0, xp, ym, yp, ze, r, s, v, Hv, nz, cf, m);
                    if (inner) x = nw;
                    if (own && q >= ia && q < ie) rmax[h / 2] = m > rmax[h / 2] ? m : rmax[h / 2];
                }
                // read by the next half sweep one step on
                if (h + 1 < NH) at(oX + (h + 1) * 2 * lev + wrb) = x;
            }
            at(oX + wrb) = bl[(k + O + 1) % NR];   // the next step's black rows
            // finished planes: both colours of plane p - (NH - 1)
            {
                const int q = p - (NH - 1), m1 = (k + O - (NH - 1) + 2 * NR) % NR;
                if (own && q >= ia && q < ie) {
                    *reinterpret_cast<P *>(A.out + q * rp + base) = rd[m1];
                    *reinterpret_cast<P *>(A.out + cs + q * rp + base) = bl[m1];
                }
            }
            __syncthreads();
            p++;
            s ^= 1;
            zoff = 16 - (int)sizeof(T) - zoff;
        }
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
#pragma unroll
    for (int q = 0; q < NH / 2; q++) {
        const double m = rs_warp_max(rmax[q]);
        if (lane == 0) wmax[q][tid >> 5] = m;
    }
    __syncthreads();
    if (tid < NH / 2) {
        double b = 0.0;
        for (int w = 0; w < NT / 32; w++) b = tmax(b, wmax[tid][w]);
        unsigned long long *slot = (unsigned long long *)(A.res + A.iter0 + tid);
        if (b > 0.0 && (unsigned long long)__double_as_longlong(b) > *(volatile unsigned long long *)slot)
            atomic_max_nonneg(slot, b);
    }
}

// Tiles of a grid for passes of `its` iterations: the tiling with the least
// warp-steps per SM (waves x window x whole turns of the ring).
inline bool stream_tile(const Split &sp, int its, int sms, StreamTile *out)
{
    const int V = Pack<float>::V, NH = 2 * its, NT = its == 2 ? STREAM_NT4 : STREAM_NT2;
    if (sp.H % V || sp.nx < 3 || sp.ny < 3 || sp.nz < 3 || sp.cs + 2LL * sp.ny * sp.H >= (1LL << 30)) return false;
    const int Hv = sp.H / V, vh = (NH + V - 1) / V;
    double best = 1e300;
    for (int tk = 1; tk <= 16; tk++) {
        // tk windows: the first and last own WV - vh vectors, the others WV - 2 vh
        int WV = tk == 1 ? Hv : (Hv + 2 * vh * (tk - 1) + tk - 1) / tk;
        if (WV <= 2 * vh && tk > 1) break;
        const int W = std::min(NT / WV, sp.ny);
        if (W < 3 || stream_smem(NH, W, WV) > STREAM_SMEM) continue;
        int tj = 1;
        if (W < sp.ny) {
            if (W <= 2 * NH) continue;
            const int BJ = W - 2 * NH, rest = sp.ny - 2 - 2 * (W - NH - 1);
            tj = 2 + (rest > 0 ? (rest + BJ - 1) / BJ : 0);
        }
        for (int ch = 1; ch <= 64 && ch <= sp.nx - 2; ch++) {
            const int L = (sp.nx - 2 + ch - 1) / ch, c = (sp.nx - 2 + L - 1) / L;
            const long long ctas = (long long)tj * tk * c;
            const double cost = (double)((ctas + sms - 1) / sms) * ((L + 2 * NH - 2 + 5) / 6 * 6 + 2) * ((W * WV + 31) / 32);
            if (cost < best) {
                best = cost;
                out->W = W;
                out->WV = WV;
                out->BJ = W - 2 * NH;
                out->BV = WV - 2 * vh;
                out->tj = tj;
                out->tk = tk;
                out->L = L;
                out->ch = c;
            }
        }
    }
    if (best >= 1e300) return false;
    out->magic = out->WV > 1 ? (unsigned)((0x100000000ULL + (unsigned)out->WV - 1) / (unsigned)out->WV) : 0u;
    return true;
}

// Whether passes of two iterations over tiles t beat the separate sweeps.  A
// grid of few planes or rows, or of rows that leave few windows, is mostly halo
// (us an iteration, sweeps and passes: 6x1132x2048 28.3 and 56.2, 2119x9x512 32.4
// and 75.6, 24x946x512 31.3 and 40.6; 24x5016x128 69.8 and 39.9, 1928x40x128 47.3
// and 33.5).  Both times by fits to 206 shapes, good to 12%: the steps of the
// waves, those that update planes, their warps; the cells of inner planes, the
// sweeps' idle lanes and rows.
inline bool stream_pays(const StreamTile &t, const Split &sp, int sms)
{
    const int waves = (t.tj * t.tk * t.ch + sms - 1) / sms, steps = (t.L + 6 + 5) / 6 * 6 + 2;
    const int act = t.ch == 1 ? t.L : steps, warps = (t.W * t.WV + 31) / 32;
    const double passes = 0.33 + waves * (0.117 * steps + 0.438 * act + 0.0126 * steps * warps);
    const double lanes = (double)((sp.H + 127) / 128 * 128) / sp.H, rows = (double)((sp.ny + 7) / 8 * 8) / sp.ny;
    const double mcell = 1e-6 * (sp.nx - 2) * sp.ny * sp.nz;
    return passes <= 5.65 + mcell * (0.385 + 2.095 * lanes + 0.80 * (rows - 1.0));
}

template <int NH, int NT, bool EVEN>
cudaError_t launch_stream(const StreamArgs &a, cudaStream_t s)
{
    const size_t smem = stream_smem(NH, a.t.W, a.t.WV);
    static std::atomic<unsigned long long> attr_set{0};
    cudaError_t e = set_smem_once(attr_set, (const void *)sor_stream_kernel<NH, NT, EVEN>, STREAM_SMEM);
    if (e != cudaSuccess) return e;
    return launch_pdl_smem(sor_stream_kernel<NH, NT, EVEN>, dim3(a.t.tj * a.t.tk, a.t.ch), dim3(NT), smem, s, a);
}

// One pass of `its` (1 or 2) iterations from in to out.
inline cudaError_t run_stream(const StreamTile &t, int its, const float *in, float *out, const float *src,
                              const Split &sp, const SorCoef<float> &cf, double *res, int iter0, int pair,
                              double thresh, int force, DevScalars *sc, cudaStream_t s)
{
    if (((uintptr_t)in | (uintptr_t)out | (uintptr_t)src) % 16) return cudaErrorInvalidValue;
    const StreamArgs a = { in, out, src, sp, cf, t, res, iter0, pair, thresh, sc, force };
    if (sp.nz % 2 == 0)
        return its == 2 ? launch_stream<4, STREAM_NT4, true>(a, s) : launch_stream<2, STREAM_NT2, true>(a, s);
    return its == 2 ? launch_stream<4, STREAM_NT4, false>(a, s) : launch_stream<2, STREAM_NT2, false>(a, s);
}

}  // namespace hc
