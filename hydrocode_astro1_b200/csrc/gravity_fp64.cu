// gravity_fp64.cu -- FP64 Poisson solve of the reference gravity solver.
// Built with -fmad=false so that every value keeps the reference's rounding
// (gravity_solver_3d.c:164-911).
//
//   moments      M, centre of mass and the Cartesian quadrupole Q_ij over
//                cells with rho > 0 (:164-262).  HC_MOMENTS_SEQUENTIAL sums in
//                the reference's (i,j,k) order -- bit-exact (seq_* below);
//                HC_MOMENTS_TREE is a fixed-shape (deterministic) tree.
//   boundary     monopole + quadrupole potential on the six faces (:302-498),
//                each face cell given the value of the face loop that writes
//                it last (x, then y, then z); periodic copies (:273-301).
//   SOR          red-black sweeps (:642-708, :577-633 for nz == 1); the
//                per-iteration max |phi_GS - phi_old| is reduced with a warp
//                max and one atomic per block into a per-iteration slot, and
//                the next iteration's first kernel stops the solve when the
//                slot is below tol (:715) -- no host round trip per iteration.
//   acceleration g = -grad phi with the boundary copies (:753-899).
#include <algorithm>

#include "hc_internal.cuh"
#include "hc_math.cuh"

namespace hc {

namespace {

__device__ __forceinline__ double slot_val(const double *res, int it)
{
    return __longlong_as_double(*reinterpret_cast<const long long *>(res + it));
}

template <int NT>
__device__ __forceinline__ double block_max_d(double v)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = tmax(v, __shfl_xor_sync(0xffffffffu, v, o));
    __shared__ double w[NT / 32];
    const int tid = threadIdx.x + blockDim.x * (threadIdx.y + blockDim.y * threadIdx.z);
    if ((tid & 31) == 0) w[tid >> 5] = v;
    __syncthreads();
    double m = 0.0;
    if (tid == 0) {
        for (int t = 0; t < NT / 32; t++) m = tmax(m, w[t]);
    }
    return m;   // valid in thread 0
}

// ---------------------------------------------------------------- moments
// The terms of a cell of density r: pass 0 (dm, dm x, dm y, dm z), pass 1 the
// quadrupole terms about com (gravity_solver_3d.c:181-190, :236-255); zero
// where r <= 0.
__device__ __forceinline__ void seq_terms(const Geom &g, int pass, double r, int i, int j, int k, const double *com,
                                          double *t)
{
    if (!(r > 0.0)) return;
    const double dm = r * (g.dx * g.dy * g.dz);
    if (pass == 0) {
        double x = g.xmin + (i + g.ioff + 0.5) * g.dx;
        double y = g.ymin + (j + 0.5) * g.dy;
        double z = g.zmin + (k + 0.5) * g.dz;
        t[0] = dm; t[1] = dm * x; t[2] = dm * y; t[3] = dm * z;
    } else {
        double x = g.xmin + (i + g.ioff + 0.5) * g.dx - com[0];
        double y = g.ymin + (j + 0.5) * g.dy - com[1];
        double z = g.zmin + (k + 0.5) * g.dz - com[2];
        double r2 = x * x + y * y + z * z;
        t[0] = dm * (3.0 * x * x - r2);
        t[1] = dm * (3.0 * x * y);
        t[2] = dm * (3.0 * x * z);
        t[3] = dm * (3.0 * y * x);
        t[4] = dm * (3.0 * y * y - r2);
        t[5] = dm * (3.0 * y * z);
        t[6] = dm * (3.0 * z * x);
        t[7] = dm * (3.0 * z * y);
        t[8] = dm * (3.0 * z * z - r2);
    }
}

__device__ __forceinline__ double seq_density(const GravArgs &a, long long c)
{
    return a.rho ? a.rho[c] : (double)a.rho32[c];
}

__device__ __forceinline__ void centre_of_mass(const Geom &g, const double *acc, double *out)
{
    const double M = acc[0];
    out[0] = M;
    if (M > 0.0) {
        out[1] = acc[1] / M; out[2] = acc[2] / M; out[3] = acc[3] / M;
    } else {
        out[1] = 0.5 * (g.xmin + g.xmax);
        out[2] = 0.5 * (g.ymin + g.ymax);
        out[3] = 0.5 * (g.zmin + g.zmax);
    }
}

// The sums in the reference's cell order, bit for bit, in parallel.
//
// Let r_i = RN(r_(i-1) + t_i) be the partial sums of a run of cells from a
// start g, u_i the unit in the last place of r_i and U the largest of them.
// From g + d, d a multiple of 2 U, every partial sum is r_i + d, as long as
// r_i and r_i + d lie in the same binade throughout: d is a multiple of every
// u_i, an even one, so it passes through each rounding, halves included.  So
// a run that was added up from a guess gives the result for any start that
// differs from it by such a d, smaller than the least distance of an r_i to
// the ends of its binade (the margin).
//   seq_totals   plain sums of the runs (32 .. 256 cells), added up by
//                seq_prefix to estimates of the sum at each run's start
//   seq_first    every run added up from its estimate
//   seq_second   again from g = (the result of the run before) + the multiple
//                of U nearest to the estimate, and from g + U: a run forgets
//                its start's bits below its own U, so the result before has
//                the right low bits although its high ones are a guess
//   seq_groups   the same twice for groups of 32 runs (first, then second), a
//                run taken by its record where that holds, else cell by cell
//   seq_walk     from the true sum over the groups; a group whose record does
//                not hold is taken run by run, a run cell by cell
// A guess only decides whether a record can be used; what is used is checked
// against the sum itself.  The records hold for sums that keep their sign as
// for those that return to zero in every row (z and the mixed moments of a
// centred box), where the binade changes every few cells, and where symmetry
// leaves rounding errors alone (a star without noise in a centred box, whole
// solve of one iteration at 128^3: 35 ms cell by cell, 80 with the binade's
// margins alone, 2.1 with those of exact additions).  Sums below 2^-963 are
// taken cell by cell (1.4 to 4 times the one CTA's time).
// Bound: a chain of dependent FP64 additions.  One CTA adding cell by cell (17
// cycles a cell) took 4.65 ms at 64^3, 35.8 ms at 128^3 and 317 ms at 256^3 for both
// passes; this takes 0.45-0.54, 1.3-1.8 and 7-17 ms, the last walk and, at
// 256^3, the terms' arithmetic being the most of it.
constexpr int SEQ_GRP = 32;        // runs of a group
constexpr int SEQ_RUN = 256;       // cells of a run, at most
constexpr int SEQ_DIRECT = 20000;  // cells below which the sums are added cell by cell: a whole solve of one
                                   // iteration takes 0.30 ms at 23^3 and 0.37 at 26^3, with the records'
                                   // sixteen launches 0.35 to 0.55 ms on either
constexpr double SEQ_ALL = 1e300;  // the margin before the first term

struct SeqRecs {
    double *g, *out, *margin;   // [variant][sum][record]
    int *ue;                    // exponent of U
    long long n;                // records per sum
};
struct SeqWork {
    double *pre;                // per run: plain total, then the estimate at its start
    double *out1[2];            // first results of runs / groups
    int *ue1[2];
    SeqRecs lev[2];             // runs, groups
    int G;                      // cells of a run
};

// The margin of acc = was + t without rounding error (0 for others): acc is a
// multiple of w, the lesser of its lowest bit and 2 U, and stays a double when
// moved by a multiple of 2 U as long as it is below 2^53 w.  Out of line: few
// additions need it.
__device__ __noinline__ double seq_exact(double was, double t, double acc, int ue)
{
    const double bb = acc - was, err = (was - (acc - bb)) + (t - bb);
    const int e = (__double2hiint(acc) >> 20) & 0x7ff;
    if (err != 0.0 || ue <= 60 || ue >= 1900 || (e <= 110 && acc != 0.0)) return 0.0;
    int w = ue - 51;   // biased exponent of 2 U
    if (acc != 0.0) w = min(w, e - 53 + __ffsll((__double_as_longlong(acc) & ((1LL << 52) - 1)) | (1LL << 52)));
    return __hiloint2double((w + 53) << 20, 0) - fabs(acc);
}

// Partial sums: the sum, the largest unit and the margin.
struct SeqSum {
    double acc, margin;
    int ue;                     // biased exponent of the largest partial sum
    template <bool MARGIN = true>
    __device__ __forceinline__ void add(double t)
    {
        if (t == 0.0) return;   // acc + 0 is acc
        const double was = acc;
        acc += t;
        const int hi = __double2hiint(acc) & 0x7fffffff, e = hi >> 20;
        if (!MARGIN) {
            ue = max(ue, e);
            return;
        }
        const double m = fabs(acc), bin = __hiloint2double(e << 20, 0);
        double mi = e > 60 && e < 2000 ? fmin(m - bin, 2.0 * bin - m) : 0.0;
        ue = max(ue, e);
        // only where the binade is so close that a start may well be past it
        // (2^-22 of the largest partial sum): a random term's rounded sums
        // hardly ever are
        if (mi < margin && (__double2hiint(mi) >> 20) < ue - 22) mi = fmax(mi, seq_exact(was, t, acc, ue));
        margin = fmin(margin, mi);
    }
};
__device__ __forceinline__ double seq_unit(int ue) { return __hiloint2double((ue - 52) << 20, 0); }

// The sum after a record, from s: exactly the start, or 2 U-multiples away
// from it within the margin.
__device__ __forceinline__ bool seq_use(SeqSum &s, double g, double out, double margin, int ue)
{
    if (margin >= SEQ_ALL) return true;   // no term but zeros
    const double d = s.acc - g;
    if (d != 0.0) {
        if (!(fabs(d) < margin)) return false;
        // d exact (two-sum), and a multiple of 2 U
        const double bb = s.acc - d;
        if (((s.acc - (d + bb)) + (bb - g)) != 0.0) return false;
        const double q = d * __hiloint2double((2097 - ue) << 20, 0);   // d / (2 U), 2 U = 2^(ue - 1074)
        if (!(fabs(q) < 0x1p50) || q != rint(q)) return false;
    }
    s.acc = out + d;
    s.margin = fmin(s.margin, margin - fabs(d));
    s.ue = max(s.ue, ue);
    return true;
}

// term q of pass PASS of cell c
template <int PASS>
__device__ __forceinline__ double seq_term(const GravArgs &a, int q, double r, int i, int j, int k, const double *com)
{
    constexpr int NV = PASS ? 9 : 4;
    double t[9] = {};
    seq_terms(a.g, PASS, r, i, j, k, com, t);
    double v = t[0];
#pragma unroll
    for (int x = 1; x < NV; x++) v = q == x ? t[x] : v;
    return v;
}

// f(term q) for the cells [c, c + n) below c1, in order
template <int PASS, typename F>
__device__ __forceinline__ void seq_cells(const GravArgs &a, int q, long long c, int n, long long c1,
                                          const double *com, F f)
{
    const Geom &g = a.g;
    const int sjk = g.ny * g.nz;
    int i = (int)(c / sjk), rest = (int)(c % sjk), j = rest / g.nz, k = rest % g.nz;
    n = (int)min((long long)n, c1 - c);
#pragma unroll 4
    for (int x = 0; x < n; x++) {
        f(seq_term<PASS>(a, q, seq_density(a, c + x), i, j, k, com));
        if (++k == g.nz) {
            k = 0;
            if (++j == g.ny) {
                j = 0;
                i++;
            }
        }
    }
}

// the plain total of every run (blockIdx.y: the sum)
template <int PASS>
__global__ void __launch_bounds__(128) seq_totals_kernel(GravArgs a, long long c0, long long c1, SeqWork w)
{
    const int q = blockIdx.y;
    const long long r = blockIdx.x * 128LL + threadIdx.x, n = w.lev[0].n;
    if (r >= n) return;
    const double com[3] = { a.sc->moments[1], a.sc->moments[2], a.sc->moments[3] };
    double s = 0.0;
    seq_cells<PASS>(a, q, c0 + r * w.G, w.G, c1, com, [&](double t) { s += t; });
    w.pre[q * n + r] = s;
}

// totals -> estimates of the sum at each run's start (CTA per sum, a stretch
// of the runs per thread)
__global__ void __launch_bounds__(1024) seq_prefix_kernel(SeqWork w, const double *acc)
{
    const int q = blockIdx.x, tid = threadIdx.x, lane = tid & 31;
    const long long n = w.lev[0].n, per = (n + 1023) / 1024, i0 = tid * per, i1 = min(n, i0 + per);
    double *p = w.pre + q * n;
    double s = 0.0;
    for (long long i = i0; i < i1; i++) s += p[i];
    __shared__ double ws[32];
    double x = s;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const double y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) ws[tid >> 5] = x;
    __syncthreads();
    double base = acc[q] + (x - s);
    for (int v = 0; v < tid >> 5; v++) base += ws[v];
    for (long long i = i0; i < i1; i++) {
        const double v = p[i];
        p[i] = base;
        base += v;
    }
}

// runs from their estimates
template <int PASS>
__global__ void __launch_bounds__(128) seq_first_kernel(GravArgs a, long long c0, long long c1, SeqWork w)
{
    const int q = blockIdx.y;
    const long long r = blockIdx.x * 128LL + threadIdx.x, n = w.lev[0].n;
    if (r >= n) return;
    const double com[3] = { a.sc->moments[1], a.sc->moments[2], a.sc->moments[3] };
    SeqSum s = { w.pre[q * n + r], SEQ_ALL, 0 };
    seq_cells<PASS>(a, q, c0 + r * w.G, w.G, c1, com, [&](double t) { s.add<false>(t); });
    w.out1[0][q * n + r] = s.acc;
    w.ue1[0][q * n + r] = s.ue;
}

// the guess for record r of a level: the low bits of the result before it,
// the high bits of the estimate; variant 1 one U further
__device__ __forceinline__ double seq_guess(const double *out1, int ue, long long at, long long r, double est,
                                            double first, int variant)
{
    const double U = ue > 60 ? seq_unit(ue) : 0.0;
    double g = first;
    if (r > 0) {
        const double p = out1[at - 1];
        g = U > 0.0 ? p + rint((est - p) / U) * U : p;
    }
    return variant ? g + U : g;
}

// runs from their guesses (blockIdx.z: the variant)
template <int PASS>
__global__ void __launch_bounds__(128) seq_second_kernel(GravArgs a, long long c0, long long c1, SeqWork w,
                                                         const double *acc)
{
    const int q = blockIdx.y, v = blockIdx.z;
    const long long r = blockIdx.x * 128LL + threadIdx.x, n = w.lev[0].n;
    if (r >= n) return;
    const double com[3] = { a.sc->moments[1], a.sc->moments[2], a.sc->moments[3] };
    const long long at = q * n + r;
    const double g = seq_guess(w.out1[0], w.ue1[0][at], at, r, w.pre[at], acc[q], v);
    SeqSum s = { g, SEQ_ALL, 0 };
    seq_cells<PASS>(a, q, c0 + r * w.G, w.G, c1, com, [&](double t) { s.add(t); });
    const SeqRecs &o = w.lev[0];
    const long long x = (long long)v * (PASS ? 9 : 4) * n + at;
    o.g[x] = g;
    o.out[x] = s.acc;
    o.margin[x] = s.margin;
    o.ue[x] = s.ue;
}

// 32 records of one sum, both variants, one per lane
struct SeqBatch {
    double g[2], out[2], margin[2];
    int ue[2];
    __device__ __forceinline__ void fetch(const SeqRecs &r, int nv, int q, long long at)
    {
#pragma unroll
        for (int v = 0; v < 2; v++) {
            const long long x = ((long long)v * nv + q) * r.n + min(at, r.n - 1);
            g[v] = r.g[x];
            out[v] = r.out[x];
            margin[v] = r.margin[x];
            ue[v] = r.ue[x];
        }
    }
    // s after lane j's record (the same in every lane)
    __device__ __forceinline__ bool use(int j, SeqSum &s) const
    {
#pragma unroll
        for (int v = 0; v < 2; v++)
            if (seq_use(s, __shfl_sync(0xffffffffu, g[v], j), __shfl_sync(0xffffffffu, out[v], j),
                        __shfl_sync(0xffffffffu, margin[v], j), __shfl_sync(0xffffffffu, ue[v], j)))
                return true;
        return false;
    }
};

// A warp takes sum q over the runs [r0, r1), at most SEQ_GRP of them, a run
// whose record does not hold cell by cell: the terms of the run in parallel
// into buf (SEQ_RUN doubles of the warp's own shared memory), then their chain.
// TRACK: with the margin, for a record.
template <int PASS, bool TRACK>
__device__ __forceinline__ void seq_runs(const GravArgs &a, long long c0, long long c1, const SeqWork &w, int q,
                                         long long r0, long long r1, const double *com, double *buf, SeqSum &s)
{
    const int lane = threadIdx.x & 31, sjk = a.g.ny * a.g.nz;
    SeqBatch b;
    b.fetch(w.lev[0], PASS ? 9 : 4, q, r0 + lane);
    for (int j = 0; j < (int)(r1 - r0); j++) {
        if (b.use(j, s)) continue;
        const long long c = c0 + (r0 + j) * w.G + lane, ce = min(c1, c - lane + w.G);
        double r[SEQ_RUN / 32];
#pragma unroll
        for (int u = 0; u < SEQ_RUN / 32; u++) r[u] = c + u * 32 < ce ? seq_density(a, c + u * 32) : 0.0;
        int ci = (int)(c / sjk), rest = (int)(c % sjk), cj = rest / a.g.nz, ck = rest % a.g.nz;
#pragma unroll
        for (int u = 0; u < SEQ_RUN / 32; u++) {
            if (u * 32 >= w.G) break;
            buf[u * 32 + lane] = seq_term<PASS>(a, q, r[u], ci, cj, ck, com);
            for (ck += 32; ck >= a.g.nz; ck -= a.g.nz)
                if (++cj == a.g.ny) {
                    cj = 0;
                    ci++;
                }
        }
        __syncwarp();
#pragma unroll 16
        for (int k = 0; k < w.G; k += 2) {
            const double2 v = *reinterpret_cast<const double2 *>(buf + k);
            if (TRACK) {
                s.add(v.x);
                s.add(v.y);
            } else {
                s.acc += v.x;
                s.acc += v.y;
            }
        }
        __syncwarp();
    }
}

// groups (warp per group, sum blockIdx.y): first from the first run's guess,
// then (second) from the guesses made of the first results, as for the runs
template <int PASS>
__global__ void __launch_bounds__(32) seq_groups_kernel(GravArgs a, long long c0, long long c1, SeqWork w,
                                                        const double *acc, int second)
{
    __shared__ __align__(16) double buf[SEQ_RUN];
    const int q = blockIdx.y, v = blockIdx.z;
    const long long h = blockIdx.x, n0 = w.lev[0].n, n = w.lev[1].n, r0 = h * SEQ_GRP;
    const double com[3] = { a.sc->moments[1], a.sc->moments[2], a.sc->moments[3] };
    const long long at = q * n + h;
    const double est = w.lev[0].g[q * n0 + r0];
    const double g = second ? seq_guess(w.out1[1], w.ue1[1][at], at, h, est, acc[q], v) : est;
    SeqSum s = { g, SEQ_ALL, 0 };
    seq_runs<PASS, true>(a, c0, c1, w, q, r0, min(n0, r0 + SEQ_GRP), com, buf, s);
    if (threadIdx.x != 0) return;
    if (!second) {
        w.out1[1][at] = s.acc;
        w.ue1[1][at] = s.ue;
        return;
    }
    const SeqRecs &o = w.lev[1];
    const long long x = (long long)v * (PASS ? 9 : 4) * n + at;
    o.g[x] = g;
    o.out[x] = s.acc;
    o.margin[x] = s.margin;
    o.ue[x] = s.ue;
}

// The cells [c0, c1) one by one, by the whole CTA: the terms of a stretch of
// cells in parallel into shared memory, then thread q < NV adds term q of each
// to acc, in order.
constexpr int SEQ_CH = 448, SEQ_ST = SEQ_CH + 1;   // an odd stride: the sums' terms lie in different banks
template <int PASS>
__device__ double seq_chain(const GravArgs &a, long long c0, long long c1, const double *com, double *term, double acc)
{
    constexpr int NV = PASS ? 9 : 4;
    const Geom &g = a.g;
    const int tid = threadIdx.x, sjk = g.ny * g.nz;
    for (long long b = c0; b < c1; b += SEQ_CH) {
        const int m = (int)min((long long)SEQ_CH, c1 - b);
        for (int e = tid; e < m; e += blockDim.x) {
            const long long c = b + e;
            const int i = (int)(c / sjk), rest = (int)(c % sjk);
            double t[9] = {};
            seq_terms(g, PASS, seq_density(a, c), i, rest / g.nz, rest % g.nz, com, t);
#pragma unroll
            for (int q = 0; q < NV; q++) term[q * SEQ_ST + e] = t[q];
        }
        __syncthreads();
        if (tid < NV) {
            const double *tt = term + tid * SEQ_ST;
#pragma unroll 16
            for (int e = 0; e < m; e++) acc += tt[e];
        }
        __syncthreads();
    }
    return acc;
}

// Both passes in one launch, cell by cell: below SEQ_DIRECT cells the chain
// is shorter than the launches of the records.
__global__ void __launch_bounds__(288) seq_direct_kernel(GravArgs a)
{
    __shared__ double term[9 * SEQ_ST], acc[9], mc[4];
    const int q = threadIdx.x;
    double v = seq_chain<0>(a, 0, a.g.n, nullptr, term, 0.0);
    if (q < 4) acc[q] = v;
    __syncthreads();
    if (q == 0) centre_of_mass(a.g, acc, mc);
    __syncthreads();
    v = seq_chain<1>(a, 0, a.g.n, mc + 1, term, 0.0);
    if (q < 9) a.sc->moments[4 + q] = v;
    if (q < 4) a.sc->moments[q] = mc[q];
}

// Warp q takes sum q over the cells [c0, c1), from acc[q] to acc[q].  Without
// work memory (w.G == 0) cell by cell.
template <int PASS>
__global__ void __launch_bounds__(PASS ? 288 : 128) seq_walk_kernel(GravArgs a, long long c0, long long c1,
                                                                    SeqWork w, double *acc)
{
    __shared__ __align__(16) double term[(PASS ? 9 : 4) * SEQ_ST];
    const int q = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const double com[3] = { a.sc->moments[1], a.sc->moments[2], a.sc->moments[3] };
    if (!w.G) {
        const int t = threadIdx.x;
        const double v = seq_chain<PASS>(a, c0, c1, com, term, t < (PASS ? 9 : 4) ? acc[t] : 0.0);
        if (t < (PASS ? 9 : 4)) acc[t] = v;
        return;
    }
    SeqSum s = { acc[q], SEQ_ALL, 0 };   // the same in every lane
    {
        SeqBatch b;
        for (long long h = 0; h < w.lev[1].n; h++) {
            const int j = (int)(h % 32);
            if (j == 0) b.fetch(w.lev[1], PASS ? 9 : 4, q, h + lane);
            if (!b.use(j, s))
                seq_runs<PASS, false>(a, c0, c1, w, q, h * SEQ_GRP, min(w.lev[0].n, (h + 1) * SEQ_GRP), com,
                                      term + q * SEQ_RUN, s);
        }
    }
    if (lane == 0) acc[q] = s.acc;
}

__global__ void moments_seq_set_kernel(GravArgs a, int pass, const double *acc)
{
    if (threadIdx.x != 0) return;
    if (pass == 0) centre_of_mass(a.g, acc, a.sc->moments);
    else
        for (int t = 0; t < 9; t++) a.sc->moments[4 + t] = acc[t];
}

// Deterministic tree: one CTA per plane (thread-strided cells, warp and
// block sums in a fixed order), then the planes' partials added in plane
// order -- a fixed order that a grid split into slabs of planes reproduces.
constexpr int TREE_NT = 256;

__global__ void __launch_bounds__(TREE_NT) moments_tree_partial(GravArgs a, int pass, double *parts)
{
    const Geom g = a.g;
    const long long sjk = (long long)g.ny * g.nz;
    const long long c0 = (long long)(g.olo + blockIdx.x) * sjk;
    const int nv = pass == 0 ? 4 : 9;
    const double *com = a.sc->moments + 1;
    double acc[9] = { 0, 0, 0, 0, 0, 0, 0, 0, 0 };
    for (long long c = c0 + threadIdx.x; c < c0 + sjk; c += TREE_NT) {
        double t[9] = { 0, 0, 0, 0, 0, 0, 0, 0, 0 };
        const int r = (int)(c - c0);
        seq_terms(g, pass, seq_density(a, c), g.olo + blockIdx.x, r / g.nz, r % g.nz, com, t);
        for (int q = 0; q < nv; q++) acc[q] += t[q];
    }
    __shared__ double red[TREE_NT / 32][9];
    for (int q = 0; q < nv; q++) {
        double v = acc[q];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
        if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5][q] = v;
    }
    __syncthreads();
    if (threadIdx.x < nv) {
        double s = 0.0;
        for (int w = 0; w < TREE_NT / 32; w++) s += red[w][threadIdx.x];
        parts[(long long)blockIdx.x * 9 + threadIdx.x] = s;
    }
}

__global__ void moments_tree_final(GravArgs a, int pass, const double *parts, int nparts)
{
    const int q = threadIdx.x;
    const int nv = pass == 0 ? 4 : 9;
    __shared__ double v[9];
    if (q < nv) {
        double s = 0.0;
        for (int b = 0; b < nparts; b++) s += parts[(long long)b * 9 + q];
        v[q] = s;
    }
    __syncthreads();
    if (q != 0) return;
    if (pass == 0) {
        centre_of_mass(a.g, v, a.sc->moments);
    } else {
        for (int t = 0; t < 9; t++) a.sc->moments[4 + t] = v[t];
    }
}

// ---------------------------------------------------------------- boundary
// gravity_solver_3d.c:327-345 for one boundary point.
__device__ __forceinline__ double mono_quad(double x, double y, double z, const double *mom,
                                            double G)
{
    double rx = x - mom[1], ry = y - mom[2], rz = z - mom[3];
    double r = sqrt(rx * rx + ry * ry + rz * rz);
    double ph = 0.0;
    if (r > 0.0) {
        const double *Q = mom + 4;
        ph = -G * mom[0] / r;
        double r5 = r * r * r * r * r;
        double Qr = Q[0] * rx * rx + Q[1] * rx * ry + Q[2] * rx * rz +
                    Q[3] * ry * rx + Q[4] * ry * ry + Q[5] * ry * rz +
                    Q[6] * rz * rx + Q[7] * rz * ry + Q[8] * rz * rz;
        double pq = -G * Qr / (2.0 * r5);
        ph += pq;
    }
    return ph;
}

// Evaluation point of a boundary cell as written by the last face loop that
// touches it: z faces (nz > 1) after y faces after x faces.
__device__ __forceinline__ void face_point(const Geom &g, int i, int j, int k, bool zb,
                                           double &x, double &y, double &z)
{
    x = g.xmin + (i + g.ioff + 0.5) * g.dx;
    y = g.ymin + (j + 0.5) * g.dy;
    z = g.zmin + (k + 0.5) * g.dz;
    if (zb && (k == 0 || k == g.nz - 1)) {
        z = (k == g.nz - 1) ? g.zmax - 0.5 * g.dz : g.zmin + 0.5 * g.dz;
    } else if (j == 0 || j == g.ny - 1) {
        y = (j == g.ny - 1) ? g.ymax - 0.5 * g.dy : g.ymin + 0.5 * g.dy;
    } else {
        x = (i + g.ioff == g.gnx - 1) ? g.xmax - 0.5 * g.dx : g.xmin + 0.5 * g.dx;
    }
}

__global__ void boundary_ref_kernel(GravArgs a)
{
    const Geom g = a.g;
    const bool zb = g.nz > 1;
    const long long nb = boundary_count(g.nx, g.ny, g.nz, zb);
    const long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (t >= nb) return;
    int i, j, k;
    boundary_cell(t, g.nx, g.ny, g.nz, zb, i, j, k);
    if (i < g.olo || i >= g.ohi) return;   // a ghost plane: the neighbour's cells
    double x, y, z;
    face_point(g, i, j, k, zb, x, y, z);
    a.phi[((long long)i * g.ny + j) * g.nz + k] = mono_quad(x, y, z, a.sc->moments, a.G);
}

__global__ void periodic_phi_kernel(GravArgs a, int axis)
{
    const Geom g = a.g;
    const int n[3] = { g.nx, g.ny, g.nz };
    const int nu = (axis == 0) ? n[1] : n[0], nv = (axis == 2) ? n[1] : n[2];
    const long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (t >= (long long)nu * nv) return;
    const int u = (int)(t / nv), v = (int)(t % nv);
    const long long sI = (long long)g.ny * g.nz, sJ = g.nz;
    long long c0, c1;
    if (axis == 0) { c0 = u * sJ + v; c1 = (n[0] - 1) * sI + u * sJ + v; }
    else if (axis == 1) { c0 = u * sI + v; c1 = u * sI + (n[1] - 1) * sJ + v; }
    else { c0 = u * sI + v * sJ; c1 = u * sI + v * sJ + n[2] - 1; }
    a.phi[c0] = a.phi[c1];
}

// ---------------------------------------------------------------- SOR
struct SorConst {
    double ix2, iy2, iz2, fpg, fac;
};

__device__ __forceinline__ SorConst sor_const(const GravArgs &a)
{
    SorConst c;
    c.ix2 = 1.0 / (a.g.dx * a.g.dx);
    c.iy2 = 1.0 / (a.g.dy * a.g.dy);
    c.iz2 = 1.0 / (a.g.dz * a.g.dz);
    c.fpg = 4.0 * M_PI * a.G;
    c.fac = (a.g.nz == 1) ? 2.0 * (c.ix2 + c.iy2) : 2.0 * (c.ix2 + c.iy2 + c.iz2);
    return c;
}

// Stop rule of gravity_solver_3d.c:715, evaluated on the device: iteration
// `iter` starts only if iteration iter-1 left the update norm >= tol.
__device__ __forceinline__ bool sor_should_stop(const GravArgs &a, int iter)
{
    if (*(volatile int *)&a.sc->done) return true;
    if (iter > 0 && slot_val(a.res, iter - 1) < a.tol) {
        if (threadIdx.x == 0 && threadIdx.y == 0) {
            a.sc->last_iter = iter;
            a.sc->done = 1;
        }
        return true;
    }
    return false;
}

constexpr int SOR_BX = 32, SOR_BY = 8;

__global__ void __launch_bounds__(SOR_BX * SOR_BY) sor_color3d(GravArgs a, int color, int iter)
{
    if (sor_should_stop(a, color == 0 ? iter : -1)) return;
    const Geom g = a.g;
    const int i = 1 + blockIdx.z;
    const int j = 1 + blockIdx.y * SOR_BY + threadIdx.y;
    const int k0 = ((i + j + 1) % 2 == color) ? 1 : 2;
    const int k = k0 + 2 * (blockIdx.x * SOR_BX + threadIdx.x);
    const SorConst sc = sor_const(a);
    double r = 0.0;
    if (j <= g.ny - 2 && k <= g.nz - 2) {
        const long long sI = (long long)g.ny * g.nz, sJ = g.nz;
        const long long c = i * sI + j * sJ + k;
        double *phi = a.phi;
        double old = phi[c];
        double lap = (phi[c - sI] + phi[c + sI]) * sc.ix2 + (phi[c - sJ] + phi[c + sJ]) * sc.iy2 +
                     (phi[c - 1] + phi[c + 1]) * sc.iz2;
        double nw = (lap - sc.fpg * a.rho[c]) / sc.fac;
        phi[c] = old + a.omega * (nw - old);
        r = fabs(nw - old);
    }
    double m = block_max_d<SOR_BX * SOR_BY>(r);
    if (threadIdx.x == 0 && threadIdx.y == 0) atomic_max_nonneg((unsigned long long *)(a.res + iter), m);
}

__global__ void __launch_bounds__(256) sor_color2d(GravArgs a, int color, int iter)
{
    if (sor_should_stop(a, color == 0 ? iter : -1)) return;
    const Geom g = a.g;
    const SorConst sc = sor_const(a);
    const long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    const long long cnt = (long long)(g.nx - 2) * (g.ny - 2);
    double r = 0.0;
    if (t < cnt) {
        int i = 1 + (int)(t / (g.ny - 2)), j = 1 + (int)(t % (g.ny - 2));
        if ((i + j) % 2 == color) {
            const long long sI = g.ny, c = (long long)i * sI + j;
            double *phi = a.phi;
            double old = phi[c];
            double lap = (phi[c - sI] + phi[c + sI]) * sc.ix2 + (phi[c - 1] + phi[c + 1]) * sc.iy2;
            double nw = (lap - sc.fpg * a.rho[c]) / sc.fac;
            phi[c] = old + a.omega * (nw - old);
            r = fabs(nw - old);
        }
    }
    double m = block_max_d<256>(r);
    if (threadIdx.x == 0) atomic_max_nonneg((unsigned long long *)(a.res + iter), m);
}

__global__ void check_kernel(GravArgs a, int iter) { sor_should_stop(a, iter); }

// ---------------------------------------------------------------- accel
__global__ void accel_kernel(GravArgs a)
{
    const Geom g = a.g;
    const long long sI = (long long)g.ny * g.nz, sJ = g.nz;
    for (long long c = blockIdx.x * (long long)blockDim.x + threadIdx.x; c < g.n;
         c += (long long)gridDim.x * blockDim.x) {
        int i = (int)(c / sI), j = (int)((c / sJ) % g.ny), k = (int)(c % sJ);
        const double *phi = a.phi;
        if (g.nz == 1) {
            if (i >= 1 && i <= g.nx - 2 && j >= 1 && j <= g.ny - 2) {
                a.gx[c] = -(phi[c + sI] - phi[c - sI]) / (2.0 * g.dx);
                a.gy[c] = -(phi[c + sJ] - phi[c - sJ]) / (2.0 * g.dy);
            } else {
                a.gx[c] = 0.0; a.gy[c] = 0.0;
            }
            a.gz[c] = 0.0;
            continue;
        }
        int ci = min(max(i, 1), g.nx - 2), cj = min(max(j, 1), g.ny - 2), ck = min(max(k, 1), g.nz - 2);
        long long cc = ci * sI + cj * sJ + ck;
        a.gx[c] = -(phi[cc + sI] - phi[cc - sI]) / (2.0 * g.dx);
        a.gy[c] = -(phi[cc + sJ] - phi[cc - sJ]) / (2.0 * g.dy);
        a.gz[c] = -(phi[cc + 1] - phi[cc - 1]) / (2.0 * g.dz);
    }
}

__global__ void residual_kernel(GravArgs a, const double *phi)
{
    const Geom g = a.g;
    const SorConst sc = sor_const(a);
    const long long sI = (long long)g.ny * g.nz, sJ = g.nz;
    double m = 0.0;
    for (long long c = blockIdx.x * (long long)blockDim.x + threadIdx.x; c < g.n;
         c += (long long)gridDim.x * blockDim.x) {
        int i = (int)(c / sI), j = (int)((c / sJ) % g.ny), k = (int)(c % sJ);
        if (i < 1 || i > g.nx - 2 || j < 1 || j > g.ny - 2 || k < 1 || k > g.nz - 2) continue;
        double lap = (phi[c - sI] + phi[c + sI]) * sc.ix2 + (phi[c - sJ] + phi[c + sJ]) * sc.iy2 +
                     (phi[c - 1] + phi[c + 1]) * sc.iz2;
        double rr = a.rho ? a.rho[c] : (double)a.rho32[c];
        double nw = (lap - sc.fpg * rr) / sc.fac;
        m = tmax(m, fabs(nw - phi[c]));
    }
    double b = block_max_d<256>(m);
    if (threadIdx.x == 0) atomic_max_nonneg((unsigned long long *)&a.sc->resnorm, b);
}

__global__ void zero_slots(double *res, int from, int count)
{
    for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < count; t += gridDim.x * blockDim.x)
        res[from + t] = 0.0;
}

inline int grid_for(long long n, int bs) { return (int)((n + bs - 1) / bs); }

}  // namespace

// Where the records of a pass over n cells lie in the work buffer.  Runs of
// 32 cells for small grids (a chain is short), up to 256 for large ones (the
// last walk is over n / (32 G) groups).
static SeqWork seq_layout(long long n0, void *buf, size_t *bytes)
{
    SeqWork w;
    w.G = 0;
    char *p = static_cast<char *>(buf);
    auto take = [&](long long items, size_t each) {
        char *r = p;
        p += (items * each + 255) / 256 * 256;
        return r;
    };
    w.pre = reinterpret_cast<double *>(take(9 * n0, 8));
    for (int l = 0; l < 2; l++) {
        const long long k = l ? (n0 + SEQ_GRP - 1) / SEQ_GRP : n0;
        w.out1[l] = reinterpret_cast<double *>(take(9 * k, 8));
        w.ue1[l] = reinterpret_cast<int *>(take(9 * k, 4));
        w.lev[l].g = reinterpret_cast<double *>(take(18 * k, 8));
        w.lev[l].out = reinterpret_cast<double *>(take(18 * k, 8));
        w.lev[l].margin = reinterpret_cast<double *>(take(18 * k, 8));
        w.lev[l].ue = reinterpret_cast<int *>(take(18 * k, 4));
        w.lev[l].n = k;
    }
    if (bytes) *bytes = (size_t)(p - static_cast<char *>(buf));
    return w;
}

static SeqWork seq_work(long long n, void *buf)
{
    int G = 32;
    while (G < SEQ_RUN && n / G > 4096) G *= 2;
    SeqWork w = seq_layout((n + G - 1) / G, buf, nullptr);
    w.G = G;
    return w;
}

bool grav_seq_records(long long cells) { return cells >= SEQ_DIRECT; }

size_t grav_seq_bytes(const Geom &g)
{
    // the most runs of any range of the grid: 4097 of fewer than SEQ_RUN cells, or n / SEQ_RUN
    size_t b = 0;
    seq_layout(std::max<long long>(g.n / SEQ_RUN + 1, std::min<long long>(g.n / 32 + 1, 4097)), nullptr, &b);
    return b;
}

template <int PASS>
static cudaError_t seq_run(const GravArgs &a, long long c0, long long c1, double *acc, cudaStream_t s,
                           long long *launched)
{
    constexpr int NV = PASS ? 9 : 4;
    SeqWork w = {};
    *launched += 1;
    if (a.seq && grav_seq_records(c1 - c0)) {
        *launched += 6;
        w = seq_work(c1 - c0, a.seq);
        const unsigned nb = (unsigned)((w.lev[0].n + 127) / 128), ng = (unsigned)w.lev[1].n;
        seq_totals_kernel<PASS><<<dim3(nb, NV), 128, 0, s>>>(a, c0, c1, w);
        seq_prefix_kernel<<<NV, 1024, 0, s>>>(w, acc);
        seq_first_kernel<PASS><<<dim3(nb, NV), 128, 0, s>>>(a, c0, c1, w);
        seq_second_kernel<PASS><<<dim3(nb, NV, 2), 128, 0, s>>>(a, c0, c1, w, acc);
        seq_groups_kernel<PASS><<<dim3(ng, NV), 32, 0, s>>>(a, c0, c1, w, acc, 0);
        seq_groups_kernel<PASS><<<dim3(ng, NV, 2), 32, 0, s>>>(a, c0, c1, w, acc, 1);
    }
    seq_walk_kernel<PASS><<<1, 32 * NV, 0, s>>>(a, c0, c1, w, acc);
    return cudaGetLastError();
}

// A slab's share of the sequential sums: the own planes, continuing acc.
cudaError_t grav_moments_seq_slab(const GravArgs &a, int pass, double *acc, cudaStream_t s, long long *launched)
{
    const long long sjk = (long long)a.g.ny * a.g.nz;
    return pass == 0 ? seq_run<0>(a, a.g.olo * sjk, a.g.ohi * sjk, acc, s, launched)
                     : seq_run<1>(a, a.g.olo * sjk, a.g.ohi * sjk, acc, s, launched);
}

cudaError_t grav_moments_sequential(const GravArgs &a, cudaStream_t s, long long *launched)
{
    if (!grav_seq_records(a.g.n)) {
        *launched += 1;
        seq_direct_kernel<<<1, 288, 0, s>>>(a);
        return cudaGetLastError();
    }
    if (a.scratch_len < 9) return cudaErrorInvalidValue;
    for (int pass = 0; pass < 2; pass++) {
        cudaError_t e = cudaMemsetAsync(a.scratch, 0, 9 * sizeof(double), s);
        if (e == cudaSuccess)
            e = pass == 0 ? seq_run<0>(a, 0, a.g.n, a.scratch, s, launched)
                          : seq_run<1>(a, 0, a.g.n, a.scratch, s, launched);
        *launched += 1;
        if (e == cudaSuccess) e = grav_moments_seq_set(a, pass, a.scratch, s);
        if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
}

cudaError_t grav_moments_seq_set(const GravArgs &a, int pass, const double *acc, cudaStream_t s)
{
    moments_seq_set_kernel<<<1, 32, 0, s>>>(a, pass, acc);
    return cudaGetLastError();
}

cudaError_t grav_moments_tree_parts(const GravArgs &a, int pass, double *parts, cudaStream_t s)
{
    if (a.g.ohi <= a.g.olo) return cudaErrorInvalidValue;
    moments_tree_partial<<<a.g.ohi - a.g.olo, TREE_NT, 0, s>>>(a, pass, parts);
    return cudaGetLastError();
}

cudaError_t grav_moments_tree_set(const GravArgs &a, int pass, const double *parts, int nparts, cudaStream_t s)
{
    moments_tree_final<<<1, 32, 0, s>>>(a, pass, parts, nparts);
    return cudaGetLastError();
}

cudaError_t grav_moments_tree(const GravArgs &a, cudaStream_t s)
{
    if (a.scratch_len < (long long)a.g.nx * 9) return cudaErrorInvalidValue;
    for (int pass = 0; pass < 2; pass++) {
        cudaError_t e = grav_moments_tree_parts(a, pass, a.scratch, s);
        if (e != cudaSuccess) return e;
        e = grav_moments_tree_set(a, pass, a.scratch, a.g.ohi - a.g.olo, s);
        if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
}

cudaError_t grav_boundary_ref(const GravArgs &a, cudaStream_t s)
{
    long long nb = boundary_count(a.g.nx, a.g.ny, a.g.nz, a.g.nz > 1);
    boundary_ref_kernel<<<grid_for(nb, 256), 256, 0, s>>>(a);
    return cudaGetLastError();
}

cudaError_t grav_boundary_periodic(const GravArgs &a, cudaStream_t s)
{
    const int n[3] = { a.g.nx, a.g.ny, a.g.nz };
    for (int axis = 0; axis < 3; axis++) {
        if (axis == 2 && a.g.nz <= 1) break;
        long long cnt = (long long)((axis == 0) ? n[1] : n[0]) * ((axis == 2) ? n[1] : n[2]);
        periodic_phi_kernel<<<grid_for(cnt, 256), 256, 0, s>>>(a, axis);
    }
    return cudaGetLastError();
}

cudaError_t grav_sor_color(const GravArgs &a, int color, int iter, cudaStream_t s)
{
    if (a.g.nz == 1) {
        long long cnt = (long long)(a.g.nx - 2) * (a.g.ny - 2);
        sor_color2d<<<grid_for(cnt, 256), 256, 0, s>>>(a, color, iter);
    } else {
        int nhalf = (a.g.nz - 1) / 2;   // cells of one colour per row, upper bound
        dim3 grid(grid_for(nhalf, SOR_BX), grid_for(a.g.ny - 2, SOR_BY), a.g.nx - 2);
        sor_color3d<<<grid, dim3(SOR_BX, SOR_BY), 0, s>>>(a, color, iter);
    }
    return cudaGetLastError();
}

cudaError_t grav_check(const GravArgs &a, int iter, cudaStream_t s)
{
    check_kernel<<<1, 1, 0, s>>>(a, iter);
    return cudaGetLastError();
}

cudaError_t grav_accel(const GravArgs &a, cudaStream_t s)
{
    accel_kernel<<<148 * 8, 256, 0, s>>>(a);
    return cudaGetLastError();
}

cudaError_t grav_residual_norm(const GravArgs &a, const double *phi, cudaStream_t s)
{
    residual_kernel<<<148 * 8, 256, 0, s>>>(a, phi);
    return cudaGetLastError();
}

cudaError_t grav_reset_slots(const GravArgs &a, int from, int count, cudaStream_t s)
{
    if (count <= 0) return cudaSuccess;
    zero_slots<<<std::min(grid_for(count, 256), 1024), 256, 0, s>>>(a.res, from, count);
    return cudaGetLastError();
}

}  // namespace hc

// ---------------------------------------------------------------------------
// One full red-black iteration per pass over HBM (wavefront, out of place).
// ---------------------------------------------------------------------------
#include "sor_wavefront.cuh"
#include "sor_wavefront_tma.cuh"
#include "tmap.cuh"

namespace hc {
namespace {
constexpr int WF64_T = 1, WF64_TJ = 16, WF64_TK = 64, WF64_NT = 256;
}

// HC_NO_TMA=1 selects the plain-load kernels (A/B comparisons).
bool wf_tma_enabled()
{
    static int on = -1;
    if (on < 0) {
        const char *e = getenv("HC_NO_TMA");
        on = (e && atoi(e) != 0) ? 0 : 1;
    }
    return on == 1;
}

cudaError_t grav_sor_pass64(const GravArgs &a, const double *in, double *out, int iter0, cudaStream_t s)
{
    constexpr size_t sm = sor_wavefront_smem<double, WF64_T, WF64_TJ, WF64_TK>();
    auto kern = sor_wavefront_kernel<double, double, WF64_T, WF64_TJ, WF64_TK, WF64_NT>;
    static std::atomic<unsigned long long> attr_set{0};
    cudaError_t e = set_smem_once(attr_set, (const void *)kern, (int)sm);
    if (e != cudaSuccess) return e;
    const SorCoef<double> cf = sor_coef64(a.g.dx, a.g.dy, a.g.dz, a.G, a.omega);
    const int tj = (a.g.ny + WF64_TJ - 1) / WF64_TJ, tk = (a.g.nz + WF64_TK - 1) / WF64_TK;
    const int nint = a.g.nx - 2;
    // about 3 waves of 4 CTAs per SM; at least 16 planes per chunk
    long long want = 148LL * 4 * 3;
    int chunks = (int)std::max(1LL, std::min((long long)nint / 16, (want + tj * tk - 1) / (tj * tk)));
    chunks = std::max(chunks, 1);
    int chunk = (nint + chunks - 1) / chunks;
    chunks = (nint + chunk - 1) / chunk;
    dim3 grid(tk, tj, chunks);
    // operands staged by TMA where the layout allows it (16-byte row stride)
    using SH = wtma::Shape<double, WF64_T, WF64_TJ, WF64_TK>;
    CUtensorMap tin, tsrc;
    if (wf_tma_enabled() && tmap3(in, 8, a.g.nx, a.g.ny, a.g.nz, SH::SK, SH::SJ, &tin) &&
        tmap3(a.rho, 8, a.g.nx, a.g.ny, a.g.nz, SH::SK, SH::SJ, &tsrc)) {
        auto kt = wtma::sor_wavefront_tma_kernel<double, double, WF64_T, WF64_TJ, WF64_TK, WF64_NT>;
        static std::atomic<unsigned long long> attr_t{0};
        e = set_smem_once(attr_t, (const void *)kt, (int)SH::SMEM);
        if (e != cudaSuccess) return e;
        kt<<<grid, WF64_NT, SH::SMEM, s>>>(tin, tsrc, out, a.g, cf, a.res, iter0, a.tol, a.sc, chunk);
        return cudaGetLastError();
    }
    kern<<<grid, WF64_NT, sm, s>>>(in, out, a.rho, a.g, cf, a.res, iter0, a.tol, a.sc, chunk);
    return cudaGetLastError();
}

}  // namespace hc

// ---------------------------------------------------------------------------
// Colour-split SOR (the default FP64 solve for nz >= 3)
// ---------------------------------------------------------------------------
#include "sor_resident.cuh"
#include "sor_split.cuh"

namespace hc {

long long split_len(const Geom &g)
{
    const Split sp = make_split(g);
    return 2 * sp.cs;
}

cudaError_t grav_split_fields(const GravArgs &a, double *phs, double *rhs, cudaStream_t s)
{
    const Split sp = make_split(a.g);
    const unsigned rows = (unsigned)((long long)a.g.nx * a.g.ny);
    const int nt = a.g.nz >= 256 ? 256 : 128;
    split_copy_kernel<double, double><<<rows, nt, 0, s>>>(a.phi, phs, sp);
    if (rhs) split_copy_kernel<double, double><<<rows, nt, 0, s>>>(a.rho, rhs, sp);
    return cudaGetLastError();
}

cudaError_t grav_split_boundary(const GravArgs &a, double *phs, cudaStream_t s)
{
    const Split sp = make_split(a.g);
    split_boundary_kernel<double><<<148 * 4, 256, 0, s>>>(a.phi, phs, sp);
    return cudaGetLastError();
}

cudaError_t grav_unsplit(const GravArgs &a, const double *phs, cudaStream_t s)
{
    const Split sp = make_split(a.g);
    const unsigned rows = (unsigned)((long long)a.g.nx * a.g.ny);
    unsplit_copy_kernel<double><<<rows, a.g.nz >= 256 ? 256 : 128, 0, s>>>(phs, a.phi, sp);
    return cudaGetLastError();
}

static SorCoef<double> sor_coef64(const GravArgs &a) { return sor_coef64(a.g.dx, a.g.dy, a.g.dz, a.G, a.omega); }

cudaError_t grav_sor_split(const GravArgs &a, double *phs, const double *rhs, int colour, int iter, cudaStream_t s)
{
    return launch_sor_split<double, double>(phs, rhs, make_split(a.g), sor_coef64(a), colour, a.res, iter, a.tol, a.sc,
                                            s);
}

bool grav_resident_plan(const Geom &g, size_t elem, ResPlan *out)
{
    int dev = 0, sms = 0, optin = 0, coop = 0;
    if (cudaGetDevice(&dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev) != cudaSuccess)
        return false;
    return coop && optin > RS_STATIC && res_plan(g, elem, sms, (size_t)(optin - RS_STATIC), out);
}

cudaError_t grav_sor_resident(const GravArgs &a, double *phs, const double *rhs, const ResPlan &p, void *exch,
                              unsigned epoch, int it0, int n, cudaStream_t s)
{
    return run_resident<double>(p, phs, rhs, make_split(a.g), sor_coef64(a), exch, epoch, a.res, it0, n, a.tol, a.sc,
                                s);
}

}  // namespace hc
