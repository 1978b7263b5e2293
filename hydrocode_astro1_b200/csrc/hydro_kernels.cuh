// hydro_kernels.cuh -- the godunov step as CUDA kernels, templated on the
// state type.  Included by hydro_fp64.cu (T = double, compiled -fmad=false so
// that results are bit-identical to the reference) and hydro_fp32.cu.
//
// One step (godunov_step_3d, hydro_solver_3d.c:637-811) is:
//   dt kernel          dt = cfl*min(d/smax) from the max signal speed that
//                      the previous step's kernels reduced (compute_dt_3d,
//                      :422-450, evaluated on the same final state)
//   interior kernel    per interior cell: three HLLC face fluxes per axis
//                      shared through shared memory, flux difference update
//                      (:729-764), floors (:765-768), gravity source (:597-631)
//                      with g = -grad(phi) formed in place, next-step CFL max
//   boundary kernel    the six faces (never flux-updated, :729-731): gravity
//                      source with g copied from the nearest interior cell
//                      (gravity_solver_3d.c:842-897), periodic copies and
//                      boundary conditions (hydro_solver_3d.c:779-807 then
//                      :456-552, axis by axis), max signal speed
// The state is double-buffered: every kernel reads step-n values and writes
// the step-(n+1) buffer, which is what the reference's separate flux arrays
// give it.
#pragma once
#include <algorithm>
#include <atomic>

#include "hc_internal.cuh"
#include "hc_math.cuh"

namespace hc {

template <typename T>
__device__ __forceinline__ Cons<T> ld_cons(const T *const *q, long long c)
{
    Cons<T> r;
    r.d = q[0][c]; r.m[0] = q[1][c]; r.m[1] = q[2][c]; r.m[2] = q[3][c]; r.e = q[4][c];
    return r;
}
template <typename T>
__device__ __forceinline__ void st_cons(T *const *q, long long c, const Cons<T> &r)
{
    q[0][c] = r.d; q[1][c] = r.m[0]; q[2][c] = r.m[1]; q[3][c] = r.m[2]; q[4][c] = r.e;
}

template <typename T> struct AccT { typedef double type; };

template <typename T>
__device__ __forceinline__ void block_max_to(T v, unsigned long long *slot64, unsigned int *slot32)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = tmax(v, __shfl_xor_sync(0xffffffffu, v, o));
    __shared__ T wmax[32];
    const int nt = blockDim.x * blockDim.y;
    const int tid = threadIdx.y * blockDim.x + threadIdx.x;
    if ((tid & 31) == 0) wmax[tid >> 5] = v;
    __syncthreads();
    if (tid < 32) {
        T m = (tid < (nt + 31) / 32) ? wmax[tid] : (T)0;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) m = tmax(m, __shfl_xor_sync(0xffffffffu, m, o));
        if (tid == 0) {
            if (sizeof(T) == 8) atomic_max_nonneg(slot64, (double)m);
            else atomic_max_nonneg(slot32, (float)m);
        }
    }
}

// Per-cell values a face flux needs: conserved state, primitives, sound speed.
template <typename T> struct CellS {
    Cons<T> q;
    Prim<T> w;
    T c;
};

template <typename T>
__device__ __forceinline__ CellS<T> make_cell(const Cons<T> &q, T gm1, T gam)
{
    CellS<T> s;
    s.q = q;
    s.w = to_prim(q, gm1);
    s.c = csound(s.w, gam);
    return s;
}

// --------------------------------------------------------------------------
// interior kernel
// --------------------------------------------------------------------------
// In FP64 the chains of divisions and square roots of the primitives and the
// faces bound it (about 29 divisions per cell), so no cell of a tile is turned
// into primitives twice: the thread that owns it keeps it for the x face and
// posts it, and a halo cell has a thread of its own.  Its loads run during the
// y and z faces.  Two blocks to an SM (128 registers): at 138 one fits, three
// spill.  256^3 1550 -> 1063 us against forming tile and halo from a staged raw
// plane, 128^3 220 -> 155, 90 x 101 x 97 115 -> 77, 64^3 39 -> 31; tiles of 4
// rows 5 % and of 16 rows 1 % slower at 256^3.
template <typename T, int TK, int TJ>
__global__ void __launch_bounds__(TK * TJ, 2)
interior_kernel(HydroArgs a, int ilen, int k00, int j00)   // k00, j00: first cell of the tiles
{
    constexpr int SK = TK + 2, SJ = TJ + 2, NS = SK * SJ;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    CellS<T> *P = reinterpret_cast<CellS<T> *>(smem_raw);            // plane i, tile+halo
    Cons<T> *FY = reinterpret_cast<Cons<T> *>(P + NS);                 // (TJ+1) x TK
    Cons<T> *FZ = FY + (TJ + 1) * TK;                                   // TJ x (TK+1)

    const int nx = a.g.nx, ny = a.g.ny, nz = a.g.nz;
    const long long sI = (long long)ny * nz, sJ = nz;
    const int tx = threadIdx.x, ty = threadIdx.y, tid = ty * TK + tx;
    const int k0 = k00 + blockIdx.x * TK, j0 = j00 + blockIdx.y * TJ;
    const int k = k0 + tx, j = j0 + ty;
    const int ib = 1 + blockIdx.z * ilen;
    const int ie = min(nx - 1, ib + ilen);   // exclusive; interior is [1, nx-2]
    if (ib >= ie) return;

    const T *const *qin = reinterpret_cast<const T *const *>(a.qin);
    T *const *qout = reinterpret_cast<T *const *>(a.qout);
    const T gam = (T)a.gamma, gm1 = (T)(a.gamma - 1.0);
    const T dt = (T)a.sc->dt;
    const T dtdx = dt / (T)a.g.dx, dtdy = dt / (T)a.g.dy, dtdz = dt / (T)a.g.dz;
    const double idx2 = 2.0 * a.g.dx, idy2 = 2.0 * a.g.dy, idz2 = 2.0 * a.g.dz;
    const bool own_in = (j < ny) && (k < nz);
    const bool own_int = (j >= 1) && (j <= ny - 2) && (k >= 1) && (k <= nz - 2);

    // state of cell (gj, gk) of plane i; a harmless one outside the grid
    auto load = [&](int i, int gj, int gk) {
        Cons<T> q;
        if (gj >= 0 && gj < ny && gk >= 0 && gk < nz) {
            q = ld_cons(qin, (long long)i * sI + gj * sJ + gk);
        } else {
            q.d = (T)1; q.m[0] = q.m[1] = q.m[2] = (T)0; q.e = (T)1;
        }
        return q;
    };
    // One of the NH halo cells around the tile, for the last NH threads (the
    // first two rows of threads form the faces behind the tile).
    constexpr int NH = 2 * SK + 2 * TJ;
    static_assert(NH <= TK * TJ, "a thread per halo cell");
    const int h = tid - (TK * TJ - NH);
    int hj = 0, hk = 0;
    if (h >= 2 * SK) {
        hj = 1 + ((h - 2 * SK) >> 1);
        hk = (h & 1) ? SK - 1 : 0;
    } else if (h >= 0) {
        hj = h < SK ? 0 : SJ - 1;
        hk = h % SK;
    }
    const int own = (ty + 1) * SK + tx + 1;

    // prologue: plane ib-1 (own cell only) and plane ib (tile + halo)
    const CellS<T> me_prev = make_cell(load(ib - 1, j, k), gm1, gam);
    CellS<T> me = make_cell(load(ib, j, k), gm1, gam);
    P[own] = me;
    if (h >= 0) P[hj * SK + hk] = make_cell(load(ib, j0 - 1 + hj, k0 - 1 + hk), gm1, gam);
    Cons<T> fxm = hllc<0>(me_prev.q, me_prev.w, me_prev.c, me.q, me.w, me.c);
    __syncthreads();

    T smax = (T)0;
    for (int i = ib; i < ie; i++) {
        // plane i+1: this thread's cell and its halo cell, on their way during
        // the faces of plane i
        const Cons<T> qn = load(i + 1, j, k);
        Cons<T> qh;
        if (h >= 0) qh = load(i + 1, j0 - 1 + hj, k0 - 1 + hk);
        {
            const CellS<T> &ay = P[(ty + 2) * SK + tx + 1];
            const CellS<T> &az = P[(ty + 1) * SK + tx + 2];
            FY[(ty + 1) * TK + tx] = hllc<1>(me.q, me.w, me.c, ay.q, ay.w, ay.c);
            FZ[ty * (TK + 1) + tx + 1] = hllc<2>(me.q, me.w, me.c, az.q, az.w, az.c);
            if (ty == 0) {
                const CellS<T> &b0 = P[tx + 1];
                FY[tx] = hllc<1>(b0.q, b0.w, b0.c, me.q, me.w, me.c);
            } else if (ty == 1 && tx < TJ) {
                const CellS<T> &c0 = P[(tx + 1) * SK];
                const CellS<T> &c1 = P[(tx + 1) * SK + 1];
                FZ[tx * (TK + 1)] = hllc<2>(c0.q, c0.w, c0.c, c1.q, c1.w, c1.c);
            }
        }
        const CellS<T> nx1 = make_cell(qn, gm1, gam);
        const Cons<T> fxp = hllc<0>(me.q, me.w, me.c, nx1.q, nx1.w, nx1.c);
        __syncthreads();
        // P is free again: plane i+1 for the next iteration
        P[own] = nx1;
        if (h >= 0) P[hj * SK + hk] = make_cell(qh, gm1, gam);

        if (own_in && own_int) {
            const Cons<T> &yp = FY[(ty + 1) * TK + tx], &ym = FY[ty * TK + tx];
            const Cons<T> &zp = FZ[ty * (TK + 1) + tx + 1], &zm = FZ[ty * (TK + 1) + tx];
            Cons<T> q = me.q;
            q.d = q.d + (-dtdx * (fxp.d - fxm.d) - dtdy * (yp.d - ym.d) - dtdz * (zp.d - zm.d));
#pragma unroll
            for (int c = 0; c < 3; c++)
                q.m[c] = q.m[c] + (-dtdx * (fxp.m[c] - fxm.m[c]) - dtdy * (yp.m[c] - ym.m[c]) -
                                   dtdz * (zp.m[c] - zm.m[c]));
            q.e = q.e + (-dtdx * (fxp.e - fxm.e) - dtdy * (yp.e - ym.e) - dtdz * (zp.e - zm.e));
            // floors: rho floor, then a prim round trip (hydro_solver_3d.c:765-768)
            q.d = tmax(q.d, (T)HC_RHO_FLOOR);
            Prim<T> w = to_prim(q, gm1);
            w.p = tmax(w.p, (T)HC_P_FLOOR);
            q = to_cons(w, gm1);
            const long long c = (long long)i * sI + j * sJ + k;
            if (a.gravity) {
                const double *ph = a.phig;
                double ax = -(__ldg(ph + c + sI) - __ldg(ph + c - sI)) / idx2;
                double ay = -(__ldg(ph + c + sJ) - __ldg(ph + c - sJ)) / idy2;
                double az = -(__ldg(ph + c + 1) - __ldg(ph + c - 1)) / idz2;
                gravity_source(q, ax, ay, az, dt);
            }
            st_cons(qout, c, q);
            smax = tmax(smax, signal_speed(to_prim(q, gm1), gam));
        }
        __syncthreads();
        fxm = fxp;
        me = nx1;
    }
    block_max_to(smax, &a.sc->smax[a.step_parity ^ 1],
                 reinterpret_cast<unsigned int *>(&a.sc->smax[a.step_parity ^ 1]));
}

template <typename T, int TK, int TJ>
constexpr size_t interior_smem()
{
    return sizeof(CellS<T>) * (TK + 2) * (TJ + 2) + sizeof(Cons<T>) * ((TJ + 1) * TK + TJ * (TK + 1));
}

// Planes of a chunk along i: the fewest waves x (planes + the prologue's one)
// over the CTAs that run at once.  (A fixed four waves of at least 8 planes
// left most SMs idle on small grids.  FP64, by this rule alone: 16^3 107 -> 19 us,
// 64^3 66 -> 40, 128^3 246 -> 220, 256^3 1664 -> 1550.)
inline int chunk_planes(long long tiles, int nint, long long slots)
{
    int best = nint;
    long long cost = -1;
    for (int l = 1; l <= nint; l++) {
        const long long ctas = tiles * ((nint + l - 1) / l), c = (ctas + slots - 1) / slots * (l + 1);
        if (cost < 0 || c <= cost) {
            cost = c;
            best = l;
        }
    }
    return best;
}

// One launch of interior_kernel.
template <typename T, int TK, int TJ>
cudaError_t launch_interior(const HydroArgs &a, cudaStream_t s)
{
    constexpr size_t sm = interior_smem<T, TK, TJ>();
    static std::atomic<unsigned long long> attr_set{0};
    cudaError_t e = set_smem_once(attr_set, (const void *)interior_kernel<T, TK, TJ>, (int)sm);
    if (e != cudaSuccess) return e;
    static std::atomic<int> slots_dev[64];
    int dev = 0;
    e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    int slots = (dev >= 0 && dev < 64) ? slots_dev[dev].load() : 0;
    if (!slots) {
        int per_sm = 0, sms = 0;
        e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, interior_kernel<T, TK, TJ>, TK * TJ, sm);
        if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        if (e != cudaSuccess) return e;
        slots = std::max(1, per_sm) * sms;
        if (dev >= 0 && dev < 64) slots_dev[dev].store(slots);
    }
    // tiles from cell 0 (aligned rows) or, where that saves a tile, from the
    // first interior cell (101 x 99 x 97 FP64: 146 -> 117 us)
    auto tiles = [](int n, int t, int &o) {
        o = (n - 2 + t - 1) / t < (n - 1 + t - 1) / t ? 1 : 0;
        return (n - 1 - o + t - 1) / t;
    };
    int k00, j00;
    const int tk = tiles(a.g.nz, TK, k00), tj = tiles(a.g.ny, TJ, j00), nint = a.g.nx - 2;
    const int ilen = chunk_planes((long long)tk * tj, nint, slots);
    interior_kernel<T, TK, TJ><<<dim3(tk, tj, (nint + ilen - 1) / ilen), dim3(TK, TJ), sm, s>>>(a, ilen, k00, j00);
    return cudaGetLastError();
}

// --------------------------------------------------------------------------
// small kernels
// --------------------------------------------------------------------------
template <typename T>
__global__ void dt_kernel(HydroArgs a)
{
    unsigned long long *slots = a.sc->smax;
    T smax;
    if (sizeof(T) == 8) smax = (T)__longlong_as_double((long long)slots[a.step_parity]);
    else smax = (T)__uint_as_float((unsigned int)slots[a.step_parity]);
    T tx = (T)a.g.dx / smax, ty = (T)a.g.dy / smax, tz = (T)a.g.dz / smax;
    T dtv = (T)a.cfl * tmin(tx, tmin(ty, tz));
    a.sc->dt = (double)dtv;
    // for the host at its next synchronisation; a copy of 8 bytes per step
    // stood between two steps' kernels (64^3: 72.8 -> 64.4 us per step)
    *a.dt_host = (double)dtv;
    // initial max speed of compute_dt_3d (hydro_solver_3d.c:423)
    if (sizeof(T) == 8) slots[a.step_parity ^ 1] = (unsigned long long)__double_as_longlong(1.0e-10);
    else slots[a.step_parity ^ 1] = (unsigned long long)__float_as_uint(1.0e-10f);
}

template <typename T>
__global__ void cfl_full_kernel(HydroArgs a)
{
    const T *const *q = reinterpret_cast<const T *const *>(a.qin);
    const T gam = (T)a.gamma, gm1 = (T)(a.gamma - 1.0);
    T m = (T)0;
    for (long long c = blockIdx.x * (long long)blockDim.x + threadIdx.x; c < a.g.n;
         c += (long long)gridDim.x * blockDim.x)
        m = tmax(m, signal_speed(to_prim(ld_cons(q, c), gm1), gam));
    block_max_to(m, &a.sc->smax[a.step_parity],
                 reinterpret_cast<unsigned int *>(&a.sc->smax[a.step_parity]));
}

// The face cells, in one launch: gravity source, periodic copies, boundary
// conditions and their signal speed.  The reference applies these one after
// the other to whole faces (source :612-628, periodic x, y, z :779-807, then
// conditions x, y, z :456-552); each step either leaves a cell, copies the
// value another cell has before it, or flips the cell's own velocity.  So a
// cell's final value is one cell's value after the source -- found by walking
// the steps backwards -- with the flips on the way applied in order; nothing
// is read that this launch writes.  (One launch per step read and wrote the
// faces up to six times, the z faces a sector per cell.  With the dt kernel, per
// step: 256^3 FP32 109 -> 46 us, 16^3 FP64 35 -> 17 us.)
template <typename T>
__device__ __forceinline__ Cons<T> boundary_value(const HydroArgs &a, int i, int j, int k)
{
    const int n[3] = { a.g.nx, a.g.ny, a.g.nz };
    const T gm1 = (T)(a.gamma - 1.0);
    int x[3] = { i, j, k };
    bool flip[3] = { false, false, false };
#pragma unroll
    for (int ax = 2; ax >= 0; ax--) {
        const bool lo = x[ax] == 0, hi = x[ax] == n[ax] - 1;
        if (!lo && !hi) continue;
        const int type = a.bc[2 * ax + (hi ? 1 : 0)];
        if (type == 2) x[ax] = hi ? n[ax] - 2 : 1;   // BC_OUTFLOW: the neighbour
        else if (type == 1) flip[ax] = true;         // BC_REFLECTIVE: negate own normal velocity
    }
#pragma unroll
    for (int ax = 2; ax >= 0; ax--)
        if (x[ax] == 0 && a.bc[2 * ax] == 0 && a.bc[2 * ax + 1] == 0) x[ax] = n[ax] - 1;   // periodic
    const long long sI = (long long)n[1] * n[2], sJ = n[2];
    const long long c = x[0] * sI + x[1] * sJ + x[2];
    bool face = false;
#pragma unroll
    for (int ax = 0; ax < 3; ax++) face = face || x[ax] == 0 || x[ax] == n[ax] - 1;
    Cons<T> q;
    if (face) {
        q = ld_cons(reinterpret_cast<const T *const *>(a.qin), c);
        if (a.gravity) {
            // g on a boundary cell equals g of the nearest interior cell after the
            // x, y, z copy passes of gravity_compute_acceleration (:842-897)
            const int ci = min(max(x[0], 1), n[0] - 2), cj = min(max(x[1], 1), n[1] - 2), ck = min(max(x[2], 1), n[2] - 2);
            const long long cc = ci * sI + cj * sJ + ck;
            const double *ph = a.phig;
            double ax = -(ph[cc + sI] - ph[cc - sI]) / (2.0 * a.g.dx);
            double ay = -(ph[cc + sJ] - ph[cc - sJ]) / (2.0 * a.g.dy);
            double az = -(ph[cc + 1] - ph[cc - 1]) / (2.0 * a.g.dz);
            gravity_source(q, ax, ay, az, (T)a.sc->dt);
        }
    } else {
        q = ld_cons(reinterpret_cast<const T *const *>(a.qout), c);
    }
#pragma unroll
    for (int ax = 0; ax < 3; ax++)
        if (flip[ax]) {
            Prim<T> w = to_prim(q, gm1);
            w.v[ax] = -w.v[ax];
            q = to_cons(w, gm1);
        }
    return q;
}

template <typename T>
__global__ void __launch_bounds__(256) boundary_kernel(HydroArgs a)
{
    const int nx = a.g.nx, ny = a.g.ny, nz = a.g.nz;
    const long long nb = boundary_count(nx, ny, nz, true);
    const long long t = blockIdx.x * 256LL + threadIdx.x;
    const T gam = (T)a.gamma, gm1 = (T)(a.gamma - 1.0);
    T m = (T)0;
    if (t < nb) {
        int i, j, k;
        boundary_cell(t, nx, ny, nz, true, i, j, k);
        const Cons<T> q = boundary_value<T>(a, i, j, k);
        st_cons(reinterpret_cast<T *const *>(a.qout), ((long long)i * ny + j) * nz + k, q);
        m = signal_speed(to_prim(q, gm1), gam);
    }
    block_max_to(m, &a.sc->smax[a.step_parity ^ 1],
                 reinterpret_cast<unsigned int *>(&a.sc->smax[a.step_parity ^ 1]));
}

}  // namespace hc
