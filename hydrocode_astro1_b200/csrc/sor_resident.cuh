// sor_resident.cuh -- red-black SOR with the iterate resident in shared memory.
//
// A grid whose colour-split iterate fits the SMs' shared memory together
// (about 7.4 M cells in FP32, 3.7 M in FP64) needs no sweep of its own per
// colour: one cooperative launch runs many iterations.  Each CTA (one per SM)
// holds a BI x BJ block of full k rows, both colours, and after every half
// sweep sends the edge rows it updated to its four neighbours through L2.
//
// What bounds it: the separate sweeps re-read five operands per update
// through L1/L2 and pay a launch per colour (192^3 FP32: 25.9 us an
// iteration, 4.4 TB/s of L2 traffic; 64^3: 7 us, all launch).  Here only the
// source is streamed (from L2, one read per update, issued ahead) and the
// rest is 16-byte shared-memory accesses, about four per 16 bytes updated.
// Microseconds an iteration, separate sweeps -> resident (400 iterations):
//   FP32  64^3 7.0 -> 5.0   96^3 9.1 -> 5.1   128^3 14.6 -> 8.2   160^3 19.7 -> 12.4   192^3 25.9 -> 15.0
//   FP64  64^3 6.7 -> 5.4   96^3 12.2 -> 8.0   128^3 16.7 -> 12.9
// Small grids are left with the flight of a message (about 1.4 us a half
// sweep: a store to L2 and a poll of it), large ones with the latency of
// their 16 warps (the registers' limit; the issue slots are half used).
//
// Messages carry their own flags: every 8-byte word is {32 bits of payload,
// sweep number}, stored and loaded as one relaxed 64-bit access, so a row
// needs no fence, no flag line and no second round trip.  A receiver polls
// the words it needs (bounded; on a timeout the kernel sets sc->lost and
// leaves, and the caller takes the solve again by the separate sweeps).  One
// buffer per colour is enough: a sender overwrites its colour's rows two
// sweeps later, after the receiver's rows of the sweep between, which the
// receiver sends after it has read the older ones.
//
// Stop rule.  The solve must end at exactly the first iteration whose update
// norm is below the threshold, but a grid-wide test per iteration would cost
// as much as the iteration.  So iterations run in groups: at the end of a
// group all CTAs meet, read the norms of its iterations, and either write
// their block back (the next group's starting point) or, when an iteration
// inside the group was the last, reload the group's start and run exactly the
// iterations up to it again.  The first group has four (an FP32 launch that
// continues a solve: half of its iterations), the next ones at most twice as
// many as the one before, and where few are left by the norms' rate just
// those: a meeting costs half an iteration (64^3) to three (150^3), a group
// that is too long its iterations twice.  (First groups of 16 made solves of 2
// to 14 iterations slower than the separate sweeps.  64^3 FP64, us a solve,
// sweeps, 16 and now: 3 iterations 226, 298 and 222; 12 iterations 266, 350 and
// 265.)  One CTA alone tests after every iteration.
//
// Per cell the update is SorCoef<T>::update with the operands of the other
// sweep kernels, and the cells of a colour are independent: the iterates, the
// norms and the iteration counts are theirs bit for bit.
#pragma once
#include <algorithm>
#include <cstdint>
#include <type_traits>

#include "hc_internal.cuh"
#include "hc_math.cuh"
#include "sor_split.cuh"

namespace hc {

constexpr int RS_NT = 512;                    // threads of a CTA
constexpr int RS_NW = RS_NT / 32;
constexpr int RS_MAXGROUP = 128;              // iterations between two meetings
constexpr int RS_TASKS = 1024;                // warp tasks of a half sweep, at most
constexpr int RS_STATIC = 3072;               // room for the kernel's static shared memory
constexpr size_t RES_EXCH_HEAD = 256;         // arrival counter, before the message rows

template <typename T>
struct ResArgs {
    T *e;                      // colour-split iterate (in / out)
    const T *src;              // colour-split source
    Split sp;
    SorCoef<T> cf;
    int gi, gj, BI, BJ, Hp;    // CTAs and largest block along i and j; padded row length
    ulonglong2 *exch;          // message rows
    unsigned *meet;            // arrivals (zero at launch)
    double *res;               // update norms by iteration
    int it0, n;                // iterations it0 .. it0 + n - 1
    int len0;                  // iterations of the first group (FP32)
    double thresh;
    DevScalars *sc;
    unsigned magic;            // ceil(2^32 / vectors per row), 0 for one
    unsigned epoch;            // sweep numbers used: epoch .. epoch + 4 n + 16
    unsigned absent;           // blocks that no meeting sees
    unsigned long long wait_ns;
};

__device__ __forceinline__ unsigned long long rs_word(unsigned v, unsigned flag)
{
    return ((unsigned long long)flag << 32) | v;
}
__device__ __forceinline__ void rs_store2(ulonglong2 *p, unsigned long long a, unsigned long long b)
{
    asm volatile("st.relaxed.gpu.global.v2.b64 [%0], {%1, %2};" ::"l"(p), "l"(a), "l"(b) : "memory");
}
__device__ __forceinline__ ulonglong2 rs_load2(const ulonglong2 *p)
{
    ulonglong2 r;
    asm volatile("ld.relaxed.gpu.global.v2.b64 {%0, %1}, [%2];" : "=l"(r.x), "=l"(r.y) : "l"(p) : "memory");
    return r;
}
__device__ __forceinline__ unsigned long long rs_now()
{
    unsigned long long t;
    asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
    return t;
}

template <typename T, bool AL>
struct ResRow {
    static constexpr int V = Pack<T>::V;
    static __device__ __forceinline__ Pack<T> load(const T *row, int v, int H)
    {
        Pack<T> r;
        if constexpr (AL) {
            r = *reinterpret_cast<const Pack<T> *>(row + v * V);
        } else {
#pragma unroll
            for (int q = 0; q < V; q++) r.v[q] = v * V + q < H ? row[v * V + q] : (T)0;
        }
        return r;
    }
    static __device__ __forceinline__ Pack<T> load_src(const T *row, int v, int H)
    {
        Pack<T> r;
        if constexpr (AL) {
            const uint4 u = __ldg(reinterpret_cast<const uint4 *>(row + v * V));
            memcpy(&r, &u, 16);
        } else {
#pragma unroll
            for (int q = 0; q < V; q++) r.v[q] = v * V + q < H ? __ldg(row + v * V + q) : (T)0;
        }
        return r;
    }
    static __device__ __forceinline__ void store(T *row, int v, int H, const Pack<T> &r)
    {
        if constexpr (AL) {
            *reinterpret_cast<Pack<T> *>(row + v * V) = r;
        } else {
#pragma unroll
            for (int q = 0; q < V; q++)
                if (v * V + q < H) row[v * V + q] = r.v[q];
        }
    }
};

// Two FP32 operations per instruction, each rounded as the scalar one.
__device__ __forceinline__ unsigned long long rs_pack(float a, float b)
{
    unsigned long long r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ void rs_unpack(unsigned long long r, float &a, float &b)
{
    asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(r));
}
__device__ __forceinline__ unsigned long long rs_add2(unsigned long long a, unsigned long long b)
{
    unsigned long long r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ unsigned long long rs_sub2(unsigned long long a, unsigned long long b)
{
    unsigned long long r;
    asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ unsigned long long rs_mul2(unsigned long long a, unsigned long long b)
{
    unsigned long long r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ unsigned long long rs_fma2(unsigned long long a, unsigned long long b,
                                                      unsigned long long c)
{
    unsigned long long r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}

// The coefficients as the cells below take them.  The FP32 pairs are made once
// (volatile: rebuilding them at every use cost more than it saved registers).
template <typename T>
struct ResCoef : SorCoef<T> {
    __device__ explicit ResCoef(const SorCoef<T> &c) : SorCoef<T>(c) {}
};
template <>
struct ResCoef<float> {
    unsigned long long cx, cy, cz, om;
    __device__ explicit ResCoef(const SorCoef<float> &c)
    {
        auto dup = [](float a) {
            unsigned long long r;
            asm volatile("mov.b64 %0, {%1, %1};" : "=l"(r) : "f"(a));
            return r;
        };
        cx = dup(c.cx);
        cy = dup(c.cy);
        cz = dup(c.cz);
        om = dup(c.om);
    }
};

// Gauss-Seidel differences d and relaxed values of V cells: x0 holds the
// other colour's cells of the same row and index, z their second z neighbour
// (zm + zp is x0 + z in either order).  SorCoef<T>::update, term by term.
__device__ __forceinline__ void rs_cells(const ResCoef<double> &cf, const Pack<double> &old, const Pack<double> &xm,
                                         const Pack<double> &xp, const Pack<double> &ym, const Pack<double> &yp,
                                         const Pack<double> &x0, const Pack<double> &z, const Pack<double> &r,
                                         Pack<double> &nw, Pack<double> &d)
{
    double x[2], g[2];
    bool far = false;
#pragma unroll
    for (int e = 0; e < 2; e++) {
        x[e] = (xm.v[e] + xp.v[e]) * cf.ix2 + (ym.v[e] + yp.v[e]) * cf.iy2 + (x0.v[e] + z.v[e]) * cf.iz2 -
               cf.fpg * r.v[e];
        far |= cf.out_of_range(x[e]);
        g[e] = cf.quotient_in_range(x[e]);
    }
    if (far) {
        g[0] = sor_divide(x[0], cf.fac);
        g[1] = sor_divide(x[1], cf.fac);
    }
#pragma unroll
    for (int e = 0; e < 2; e++) {
        d.v[e] = g[e] - old.v[e];
        nw.v[e] = old.v[e] + cf.om * d.v[e];
    }
}
__device__ __forceinline__ void rs_cells(const ResCoef<float> &cf, const Pack<float> &old, const Pack<float> &xm,
                                         const Pack<float> &xp, const Pack<float> &ym, const Pack<float> &yp,
                                         const Pack<float> &x0, const Pack<float> &z, const Pack<float> &r,
                                         Pack<float> &nw, Pack<float> &d)
{
#pragma unroll
    for (int e = 0; e < 4; e += 2) {
        auto two = [&](const Pack<float> &p) { return rs_pack(p.v[e], p.v[e + 1]); };
        const unsigned long long o = two(old);
        const unsigned long long gs =
            rs_add2(rs_fma2(rs_add2(two(x0), two(z)), cf.cz,
                            rs_fma2(rs_add2(two(ym), two(yp)), cf.cy, rs_mul2(rs_add2(two(xm), two(xp)), cf.cx))),
                    two(r));
        const unsigned long long dd = rs_sub2(gs, o);
        rs_unpack(dd, d.v[e], d.v[e + 1]);
        rs_unpack(rs_fma2(cf.om, dd, o), nw.v[e], nw.v[e + 1]);
    }
}

// V cells of a row updated where they are interior in k: k = 2 m + s, cells
// lo .. hi of the row.  EVEN (nz even, rows of whole vectors): only the first
// cell of a row (s = 0) or its last (s = 1) is not.  ze: the other colour's
// cell before (s = 0) or after (s = 1) the vector.
template <typename T, bool EVEN>
__device__ __forceinline__ void rs_update(Pack<T> &own, const Pack<T> &xm, const Pack<T> &x0, const Pack<T> &xp,
                                          const Pack<T> &ym, const Pack<T> &yp, T ze, const Pack<T> &r, int s, int v,
                                          int Hv, int nz, const ResCoef<T> &cf, T &rmax)
{
    constexpr int V = Pack<T>::V;
    Pack<T> z, nw, d;
#pragma unroll
    for (int e = 0; e < V; e++)
        z.v[e] = s ? (e == V - 1 ? ze : x0.v[e < V - 1 ? e + 1 : e]) : (e == 0 ? ze : x0.v[e > 0 ? e - 1 : 0]);
    rs_cells(cf, own, xm, xp, ym, yp, x0, z, r, nw, d);
    const int lo = s ? 0 : 1, hi = (nz - 2 - s) >> 1;
#pragma unroll
    for (int e = 0; e < V; e++) {
        bool in = true;
        if (!EVEN) in = v * V + e >= lo && v * V + e <= hi;
        else if (e == 0) in = s || v > 0;
        else if (e == V - 1) in = !s || v < Hv - 1;
        own.v[e] = in ? nw.v[e] : own.v[e];
        const T a = in ? fabs(d.v[e]) : (T)0;
        rmax = a > rmax ? a : rmax;
    }
}

// n / d for n < 2^16 with magic = ceil(2^32 / d), 0 for d = 1
__device__ __forceinline__ int rs_div(int n, unsigned magic) { return magic ? (int)__umulhi((unsigned)n, magic) : n; }

__device__ __forceinline__ double rs_warp_max(double m)
{
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) m = tmax(m, __shfl_xor_sync(0xffffffffu, m, off));
    return m;
}
__device__ __forceinline__ double rs_warp_max(float m)   // m >= 0: ordered as its bits
{
    return (double)__uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(m)));
}

template <typename T, bool AL, bool EVEN>
__global__ void __launch_bounds__(RS_NT, 1) sor_resident_kernel(const ResArgs<T> A)
{
    constexpr int V = Pack<T>::V;
    using P = Pack<T>;
    using Row = ResRow<T, AL>;
    extern __shared__ __align__(16) unsigned char rs_smem[];
    __shared__ unsigned long long bmax[2];
    __shared__ int quit, hit, glen, met;
    __shared__ double gv[2];
    __shared__ unsigned short tasks[RS_TASKS];

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const Split sp = A.sp;
    const int H = sp.H, Hp = A.Hp, Hv = Hp / V, nz = sp.nz;
    const int ncta = A.gi * A.gj, cta = blockIdx.x;
    const int ci = cta / A.gj, cj = cta - ci * A.gj;
    const int ni = sp.nx - 2, nj = sp.ny - 2;
    const int ib = 1 + (int)((long long)ni * ci / A.gi), bi = 1 + (int)((long long)ni * (ci + 1) / A.gi) - ib;
    const int jb = 1 + (int)((long long)nj * cj / A.gj), bj = 1 + (int)((long long)nj * (cj + 1) / A.gj) - jb;
    const int RS = bj * Hp, CS = bi * RS;             // plane and colour strides of the block
    T *S = reinterpret_cast<T *>(rs_smem);            // [colour][plane][row][Hp]
    T *hal = S + 2 * CS;                              // rows beyond the block: i-, i+ (bj each), j-, j+ (bi each)
    const int nh = 2 * bj + 2 * bi;
    const bool multi = ncta > 1;
    const bool im = ci > 0, ip = ci < A.gi - 1, jm = cj > 0, jp = cj < A.gj - 1;   // neighbours
    const int HR = 2 * A.BJ + 2 * A.BI;
    const ResCoef<T> cf(A.cf);
    // 32-bit offsets: a grid that fits has far fewer than 2^31 cells
    const int cs = (int)sp.cs, rp = sp.ny * H, r00 = ib * rp + jb * H;
    auto grow = [&](int c, int q, int jj) -> int {   // offset of block row (q, jj), neighbours included
        return (c ? cs : 0) + r00 + q * rp + jj * H;
    };
    auto slot = [&](int who, int c, int row, int v) -> ulonglong2 * {
        return A.exch + (((who * 2 + c) * HR + row) * Hv + v) * 2;
    };

    if (*(volatile int *)&A.sc->done) return;
    // iteration it0 - 1 (a sweep's, before the boundary values were set) may
    // have been the last
    if (A.it0 > 0 &&
        __longlong_as_double(*reinterpret_cast<const volatile long long *>(A.res + A.it0 - 1)) < A.thresh) {
        if (cta == 0 && tid == 0) {
            A.sc->last_iter = A.it0;
            A.sc->done = 1;
        }
        return;
    }
    if (tid == 0) {
        quit = met = 0;
        bmax[0] = bmax[1] = 0;
    }

    auto load_block = [&]() {
#pragma unroll 1
        for (int row = warp; row < 2 * bi * bj; row += RS_NW) {
            const int c = row >= bi * bj, r = row - c * bi * bj, q = r / bj;
            const T *g = A.e + grow(c, q, r - q * bj);
#pragma unroll 1
            for (int v = lane; v < Hv; v += 32) *reinterpret_cast<P *>(S + row * Hp + v * V) = Row::load(g, v, H);
        }
    };
    auto store_block = [&]() {
#pragma unroll 1
        for (int row = warp; row < 2 * bi * bj; row += RS_NW) {
            const int c = row >= bi * bj, r = row - c * bi * bj, q = r / bj;
            T *g = A.e + grow(c, q, r - q * bj);
#pragma unroll 1
            for (int v = lane; v < Hv; v += 32) Row::store(g, v, H, *reinterpret_cast<const P *>(S + row * Hp + v * V));
        }
    };
    // 16 bytes of shared memory to row `row` of the messages at d
    auto post = [&](int off, ulonglong2 *d, unsigned flag) {
        const uint4 u = *reinterpret_cast<const uint4 *>(rs_smem + off);
        rs_store2(d, rs_word(u.x, flag), rs_word(u.y, flag));
        rs_store2(d + 1, rs_word(u.z, flag), rs_word(u.w, flag));
    };
    // all edge rows of colour c: i-, i+ (bj rows each), j-, j+ (bi each)
    auto send_edges = [&](int c, unsigned flag) {
#pragma unroll 1
        for (int t = tid; t < nh * Hv; t += RS_NT) {
            const int hr = rs_div(t, A.magic), v = t - hr * Hv;
            const bool iside = hr < 2 * bj;
            const int r = iside ? hr : hr - 2 * bj, far = iside ? r >= bj : r >= bi;
            const int k = r - (far ? (iside ? bj : bi) : 0);   // place along the side
            const int q = iside ? (far ? bi - 1 : 0) : k, jj = iside ? k : (far ? bj - 1 : 0);
            if (!(iside ? (far ? ip : im) : (far ? jp : jm))) continue;
            const int row = iside ? far * A.BJ + k : 2 * A.BJ + far * A.BI + k;
            post((c * CS + (q * bj + jj) * Hp + v * V) * (int)sizeof(T), slot(cta, c, row, v), flag);
        }
    };
    auto give_up = [&]() {
        quit = 1;
        atomicExch(&A.sc->lost, 1);
    };
    // colour o's rows around the block, as sweep `flag` left them
    auto receive = [&](int o, unsigned flag) {
#pragma unroll 1
        for (int t = tid; t < nh * Hv; t += RS_NT) {
            const int hr = rs_div(t, A.magic), v = t - hr * Hv;
            int q, jj, who, row;
            bool far;
            if (hr < bj) { q = -1; jj = hr; far = im; who = cta - A.gj; row = A.BJ + jj; }
            else if (hr < 2 * bj) { q = bi; jj = hr - bj; far = ip; who = cta + A.gj; row = jj; }
            else if (hr < 2 * bj + bi) { q = hr - 2 * bj; jj = -1; far = jm; who = cta - 1; row = 2 * A.BJ + A.BI + q; }
            else { q = hr - 2 * bj - bi; jj = bj; far = jp; who = cta + 1; row = 2 * A.BJ + q; }
            P p;
            if (far) {
                const ulonglong2 *d = slot(who, o, row, v);
                ulonglong2 a = rs_load2(d), b = rs_load2(d + 1);
                unsigned tries = 0;
                unsigned long long t0 = 0;
                while ((unsigned)(a.x >> 32) != flag || (unsigned)(a.y >> 32) != flag ||
                       (unsigned)(b.x >> 32) != flag || (unsigned)(b.y >> 32) != flag) {
                    if ((++tries & 1023u) == 0) {
                        const unsigned long long now = rs_now();
                        if (!t0) t0 = now;
                        if (now - t0 > A.wait_ns || *(volatile int *)&A.sc->lost) {
                            give_up();
                            break;
                        }
                    }
                    a = rs_load2(d);
                    b = rs_load2(d + 1);
                }
                const uint4 u = make_uint4((unsigned)a.x, (unsigned)a.y, (unsigned)b.x, (unsigned)b.y);
                memcpy(&p, &u, 16);
            } else {
                p = Row::load(A.e + grow(o, q, jj), v, H);   // a face of the grid: fixed during the sweeps
            }
            *reinterpret_cast<P *>(hal + hr * Hp + v * V) = p;
        }
    };

    // The half sweep.  A thread takes a vector of two adjacent rows a and b
    // (each is the other's y neighbour) along a segment of the planes (the x
    // neighbours stay in registers), so an update costs 4 instead of 7 16-byte
    // shared-memory accesses; a warp takes 32 consecutive vectors of the row
    // pairs, whose first rows share their parity, so s is the same for the
    // whole warp.  The last pair of an odd bj has one row: its b is the row
    // beyond the block, read only.  Tasks that touch the block's edge come
    // first, so that their rows are on the way while the others run.
    const int pairs = (bj + 1) / 2, chunks = (pairs * Hv + 31) / 32;
    int ng = 1, sl = bi;
    {
        int best = 1 << 30;
        for (int t = 1; t <= min(bi, 8); t++) {
            const int l = (bi + t - 1) / t, cost = ((chunks * t + RS_NW - 1) / RS_NW) * (l + 2);
            if (cost < best && chunks * t <= RS_TASKS) {
                best = cost;
                ng = (bi + l - 1) / l;
                sl = l;
            }
        }
    }
    if (warp == 0) {
        const int ca = (Hv + 31) / 32, cb = (pairs - 1) * Hv / 32;   // chunks ca .. cb - 1 hold no edge row
        int at = 0;
        for (int pass = 0; pass < 2; pass++)
            for (int sg = 0; sg < ng; sg++)
                for (int ch = 0; ch < chunks; ch++)
                    if ((sg > 0 && sg < ng - 1 && ch >= ca && ch < cb) == (pass == 1)) {
                        if (lane == 0) tasks[at] = (unsigned short)(sg << 12 | ch);
                        at++;
                    }
    }
    // byte offsets in shared memory: planes, rows, the rows beyond the block
    constexpr int B = (int)sizeof(T);
    const int RSb = RS * B, Hb = Hp * B, CSb = CS * B, hb = 2 * CSb;
    auto at = [&](int off) -> P & { return *reinterpret_cast<P *>(rs_smem + off); };
    auto one = [&](int off) -> T { return *reinterpret_cast<const T *>(rs_smem + off); };

    load_block();
    __syncthreads();
    unsigned ep = A.epoch;   // number of the last sweep sent
    if (multi) send_edges(1, ep);
    int t = A.it0;
    const int tend = A.it0 + A.n;
    // (FP64 solves hardly ever need a second launch, and their loop has no register to spare)
    int len = !multi ? 1 : sizeof(T) == 4 ? A.len0 : min(4, A.n);
    int t0 = t, t1 = min(tend, t + len);   // the group of iterations
    int last = -1;                         // the iteration that converged
    bool again = false;                    // the group runs again, up to `last`
    while (true) {
#pragma unroll 1
        for (; t < t1; t++) {
            T maxa = (T)0, maxb = (T)0;
#pragma unroll 1
            for (int c = 0; c < 2; c++) {
                const int own = c ? CSb : -CSb;   // from the other colour's row to the swept colour's
                bool met_rows = false;
#pragma unroll 1
                for (int w = warp; w < chunks * ng || !met_rows; w += RS_NW) {
                    const int task = tasks[min(w, chunks * ng - 1)], sg = task >> 12, ch = task & 4095;
                    const int qa = sg * sl, qb = min(bi, qa + sl);
                    const int p0 = ch * 32 + lane;
                    const bool act = p0 < pairs * Hv;
                    const int p = act ? p0 : pairs * Hv - 1;
                    const int jr = rs_div(p, A.magic), v = p - jr * Hv, jj = 2 * jr;
                    const bool two = jj + 1 < bj, top = jj + 2 >= bj, act2 = act && two;
                    const bool fl = lane == 0 && v > 0, fr = lane == 31 && v < Hv - 1;
                    // the other colour's rows: a, b (the row beyond the block
                    // where the pair has one row), and the y neighbours beyond
                    const int hj = hb + (2 * bj + qa) * Hb + v * 16;
                    int pa = (c ? 0 : CSb) + (qa * bj + jj) * Hb + v * 16;
                    int pb = two ? pa + Hb : hj + bi * Hb, pm = jj > 0 ? pa - Hb : hj;
                    int pp = top ? hj + bi * Hb : pa + 2 * Hb;
                    const int tb = two ? RSb : Hb, tm = jj > 0 ? RSb : Hb, tp = top ? Hb : RSb, nb = two ? Hb : 0;
                    const int rb = two ? H : 0;
                    int ra = grow(c, qa, jj);   // next source rows to fetch
                    P r0a = Row::load_src(A.src + ra, v, H), r0b = Row::load_src(A.src + ra + rb, v, H);
                    P r1a = r0a, r1b = r0b;
                    ra += rp;
                    if (qa + 1 < qb) {
                        r1a = Row::load_src(A.src + ra, v, H);
                        r1b = Row::load_src(A.src + ra + rb, v, H);
                    }
                    if (!met_rows) {
                        // the first task's sources are on their way meanwhile
                        receive(c ^ 1, ep);
                        __syncthreads();
                        if (quit) return;
                        ep++;
                        met_rows = true;
                        if (w >= chunks * ng) break;
                    }
                    P xa = at(pa), xb = at(pb);
                    const int px = qa > 0 ? pa - RSb : hb + jj * Hb + v * 16;
                    P xma = at(px), xmb = at(px + nb);
                    int s = (ib + qa + jb + c) & 1;   // of row a; row b has 1 - s
#pragma unroll 1
                    for (int q = qa; q < qb; q++) {
                        ra += rp;
                        P na = r1a, nb2 = r1b;
                        if (q + 2 < qb) {
                            na = Row::load_src(A.src + ra, v, H);
                            nb2 = Row::load_src(A.src + ra + rb, v, H);
                        }
                        const int pn = q < bi - 1 ? pa + RSb : hb + (bj + jj) * Hb + v * 16;
                        const P xpa = at(pn), ym = at(pm), yp = at(pp);
                        P xpb = at(pn + nb);
                        P owa = at(pa + own), owb = at(pa + own + nb);
                        T zu = __shfl_up_sync(0xffffffffu, s ? xb.v[V - 1] : xa.v[V - 1], 1);
                        T zd = __shfl_down_sync(0xffffffffu, s ? xa.v[0] : xb.v[0], 1);
                        if (fl) zu = one((s ? pb : pa) - B);
                        if (fr) zd = one((s ? pa : pb) + 16);
                        // a lane beyond the last vector has other z neighbours:
                        // its values are neither stored nor counted
                        T ma = maxa, mb = maxb;
                        rs_update<T, EVEN>(owa, xma, xa, xpa, ym, xb, s ? zd : zu, r0a, s, v, Hv, nz, cf, ma);
                        rs_update<T, EVEN>(owb, xmb, xb, xpb, xa, yp, s ? zu : zd, r0b, 1 - s, v, Hv, nz, cf, mb);
                        if (act) {
                            at(pa + own) = owa;
                            maxa = ma;
                        }
                        if (act2) {
                            at(pa + own + Hb) = owb;
                            maxb = mb;
                        }
                        pa += RSb;
                        pb += tb;
                        pm += tm;
                        pp += tp;
                        if (!two && q < bi - 1) xpb = at(pb);   // the row beyond the block
                        xma = xa;
                        xmb = xb;
                        xa = xpa;
                        xb = xpb;
                        r0a = r1a;
                        r0b = r1b;
                        r1a = na;
                        r1b = nb2;
                        s ^= 1;
                    }
                    // the task's edge rows to the neighbours that read them
                    // (each thread its own vectors)
                    const int po = (c ? CSb : 0) + (qa * bj + jj) * Hb + v * 16;
                    ulonglong2 *const d0 = slot(cta, c, 0, v);
                    if ((im && qa == 0) || (ip && qb == bi)) {
#pragma unroll 1
                        for (int k = 0; k < 4; k++) {
                            const int far = k >> 1, b = k & 1;
                            if ((far ? ip && qb == bi : im && qa == 0) && (b ? act2 : act))
                                post(po + b * Hb + (far ? qb - 1 - qa : 0) * RSb, d0 + (far * A.BJ + jj + b) * (Hv * 2), ep);
                        }
                    }
                    const bool pjm = act && jj == 0 && jm, pjp = act && top && jp;
                    if (pjm || pjp) {
#pragma unroll 1
                        for (int k = pjm ? 0 : 1; k < (pjp ? 2 : 1); k++) {
                            int off = po + (k && two ? Hb : 0);
                            ulonglong2 *d = d0 + (2 * A.BJ + k * A.BI + qa) * (Hv * 2);
#pragma unroll 1
                            for (int q = qa; q < qb; q++, off += RSb, d += Hv * 2) post(off, d, ep);
                        }
                    }
                }
                if (c == 1) {
                    const double m = rs_warp_max(maxa > maxb ? maxa : maxb);
                    if (lane == 0 && m > 0.0) atomic_max_nonneg(&bmax[t & 1], m);
                }
                __syncthreads();
            }
            if (tid == 0) {
                const unsigned long long m = bmax[t & 1];
                if (m && !again) atomicMax((unsigned long long *)(A.res + t), m);
                if (!multi) gv[0] = __longlong_as_double((long long)m);
                bmax[t & 1] = 0;   // its next use is two iterations away
            }
        }
        if (again) break;
        if (!multi) {
            __syncthreads();
            if (gv[0] < A.thresh) last = t1 - 1;
            __syncthreads();
            if (last >= 0 || t >= tend) break;
            t1 = t + 1;
            continue;
        }
        // all CTAs have recorded the norms of their iterations so far
        if (tid == 0) {
            hit = 1 << 30;
            met++;
            __threadfence();
            atomicAdd(A.meet, 1u);
            const unsigned want = (unsigned)met * (unsigned)ncta + A.absent;
            unsigned seen, tries = 0;
            unsigned long long w0 = 0;
            while (true) {
                asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(seen) : "l"(A.meet) : "memory");
                if (seen >= want) break;
                if ((++tries & 1023u) == 0) {
                    const unsigned long long now = rs_now();
                    if (!w0) w0 = now;
                    if (now - w0 > A.wait_ns || *(volatile int *)&A.sc->lost) {
                        give_up();
                        break;
                    }
                }
            }
            __threadfence();
        }
        __syncthreads();
        if (quit) return;
        if (tid < t1 - t0) {
            const double v = __longlong_as_double(*reinterpret_cast<const volatile long long *>(A.res + t0 + tid));
            if (v < A.thresh) atomicMin(&hit, t0 + tid);
            if (tid == max(0, t1 - t0 - 33)) gv[0] = v;
            if (tid == t1 - t0 - 1) gv[1] = v;
        }
        __syncthreads();
        if (hit < (1 << 30)) last = hit;
        if (last >= 0 && last < t1 - 1) {
            load_block();
            __syncthreads();
            send_edges(1, ++ep);
            again = true;
            t = t0;
            t1 = last + 1;
            continue;
        }
        if (last >= 0 || t >= tend) break;
        if (tid == 0) {
            // iterations left at the norms' rate over the last ones of the group,
            // seven tenths of them while they are many
            const int w = min(32, t1 - t0 - 1);
            int l = min(2 * len, RS_MAXGROUP);
            if (w >= 1 && gv[1] > 0.0 && gv[0] > gv[1]) {
                const float rate = __logf((float)(gv[0] / gv[1])) / (float)w;
                const float left = __logf((float)(gv[1] / A.thresh)) / rate;
                l = min(l, left < 10.f ? max(1, (int)left) : (int)fminf(left * 0.7f, (float)RS_MAXGROUP));
            }
            glen = l;
        }
        store_block();   // where the next group starts
        __syncthreads();
        len = glen;
        t0 = t;
        t1 = min(tend, t + len);
    }
    store_block();
    if (last >= 0 && cta == 0 && tid == 0) {
        A.sc->last_iter = last + 1;
        A.sc->done = 1;
    }
}

// Whether the plan beats the separate sweeps.  Blocks of a few long rows are
// mostly edge: every iteration polls and posts them all, 512 vectors a round, and
// that takes longer than the sweeps (us an iteration, sweeps and resident:
// FP64 4x15x4132 5.9 and 23.5, 20x20x1000 8.1 and 12.0, 64x64x600 18.6 and 25.3,
// 118x3x1059 9.4 and 6.3; FP32 23x10x5511 9.3 and 24.9, 8x8x512 5.8 and 4.8).  Both
// times by fits to 270 shapes, good to 15%: rounds and warp units of a half sweep;
// cells, with the sweeps' idle lanes.  Blocks with fewer edge rows, or rows
// below 48 vectors, are always faster resident.
inline bool res_pays(const ResPlan &p, const Geom &g, size_t elem)
{
    const int V = (int)(16 / elem), Hv = p.Hp / V, H = (g.nz + 1) / 2;
    if (Hv < 48 || p.BI * p.BJ > 3 * (p.BI + p.BJ)) return true;
    const int edge = (p.gi > 1 ? 2 : 1) * p.BJ + (p.gj > 1 ? 2 : 1) * p.BI;   // a face's rows count half
    const int rounds = (edge * Hv + RS_NT - 1) / RS_NT, chunks = ((p.BJ + 1) / 2 * Hv + 31) / 32;
    int units = 1 << 30;
    for (int t = 1; t <= std::min(p.BI, 8); t++)
        if (chunks * t <= RS_TASKS)
            units = std::min(units, (chunks * t + RS_NW - 1) / RS_NW * ((p.BI + t - 1) / t + 2));
    const double res = p.gi * p.gj > 1 ? 1.38 * rounds + 1.83 * units - 1.75 : 1.85 * rounds + 0.62 * units + 0.36;
    const int lanes = elem == 4 && H % V == 0 ? 32 * V : 32;
    const double mcell = 1e-6 * (double)g.n / H * ((H + lanes - 1) / lanes * lanes);
    const double sweeps = elem == 8 ? 5.1 + 5.4 * mcell : 5.9 + (lanes > 32 ? 2.0 : 2.77) * mcell;
    return res <= sweeps;
}

// Blocks of a grid (ResPlan): the split into gi x gj CTAs (at most one per SM) with the
// least work per CTA that fits shared memory; one CTA alone when its work is
// below the cost of the exchange (about 300 vectors).
inline bool res_plan(const Geom &g, size_t elem, int sms, size_t smem_max, ResPlan *out)
{
    if (g.nx < 3 || g.ny < 3 || g.nz < 3) return false;
    const int V = (int)(16 / elem), H = (g.nz + 1) / 2, Hp = (H + V - 1) / V * V, Hv = Hp / V;
    const int ni = g.nx - 2, nj = g.ny - 2;
    double best = 1e300;
    ResPlan p;
    for (int gi = 1; gi <= std::min(ni, sms); gi++) {
        const int BI = (ni + gi - 1) / gi;
        for (int gj = 1; gj <= std::min(nj, sms / gi); gj++) {
            const int BJ = (nj + gj - 1) / gj;
            const long long rows = 2LL * BI * BJ + 2LL * (BI + BJ);
            const size_t smem = (size_t)rows * Hp * elem;
            if (smem > smem_max) continue;
            const double cost = (double)Hv * ((double)BI * BJ + 0.7 * (BI + BJ)) + (gi * gj > 1 ? 300.0 : 0.0);
            if (cost < best) {
                best = cost;
                p.gi = gi;
                p.gj = gj;
                p.BI = BI;
                p.BJ = BJ;
                p.Hp = Hp;
                p.smem = smem;
                p.exch_bytes = RES_EXCH_HEAD + (size_t)gi * gj * 2 * (2 * BI + 2 * BJ) * Hv * 32;
            }
        }
    }
    if (best >= 1e300 || !res_pays(p, g, elem)) return false;
    *out = p;
    return true;
}

template <typename T, bool AL, bool EVEN>
cudaError_t launch_resident(const ResArgs<T> &a, size_t smem, cudaStream_t s)
{
    // the limit is raised once per device to the most a plan may ask for
    int dev = 0, optin = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
    if (e != cudaSuccess) return e;
    static std::atomic<unsigned long long> attr_set{0};
    e = set_smem_once(attr_set, (const void *)sor_resident_kernel<T, AL, EVEN>, optin - RS_STATIC);
    if (e != cudaSuccess) return e;
    e = cudaMemsetAsync(a.meet, 0, sizeof(unsigned), s);
    if (e != cudaSuccess) return e;
    ResArgs<T> v = a;
    void *args[] = { &v };
    return cudaLaunchCooperativeKernel((const void *)sor_resident_kernel<T, AL, EVEN>, dim3(a.gi * a.gj), dim3(RS_NT), args,
                                       smem, s);
}

template <typename T>
cudaError_t run_resident(const ResPlan &p, T *e, const T *src, const Split &sp, const SorCoef<T> &cf, void *exch,
                         unsigned epoch, double *res, int it0, int n, double thresh, DevScalars *sc, cudaStream_t s)
{
    ResArgs<T> a;
    a.e = e;
    a.src = src;
    a.sp = sp;
    a.cf = cf;
    a.gi = p.gi;
    a.gj = p.gj;
    a.BI = p.BI;
    a.BJ = p.BJ;
    a.Hp = p.Hp;
    a.meet = reinterpret_cast<unsigned *>(exch);
    a.exch = reinterpret_cast<ulonglong2 *>(static_cast<char *>(exch) + RES_EXCH_HEAD);
    a.res = res;
    a.it0 = it0;
    a.n = n;
    // a launch that continues a solve has been given the iterations left and a tenth more
    a.len0 = it0 > 1 ? std::max(4, std::min(n / 2, RS_MAXGROUP)) : 4;
    a.thresh = thresh;
    a.sc = sc;
    a.magic = (unsigned)((0x100000000ULL + (unsigned)(p.Hp / Pack<T>::V) - 1) / (unsigned)(p.Hp / Pack<T>::V));
    a.epoch = epoch;
    a.absent = p.absent;
    a.wait_ns = p.wait_ns;
    const bool al = sp.H % Pack<T>::V == 0 && ((uintptr_t)e | (uintptr_t)src) % 16 == 0 && sp.cs % Pack<T>::V == 0;
    if (!al) return launch_resident<T, false, false>(a, p.smem, s);
    return sp.nz % 2 == 0 ? launch_resident<T, true, true>(a, p.smem, s) : launch_resident<T, true, false>(a, p.smem, s);
}

}  // namespace hc
