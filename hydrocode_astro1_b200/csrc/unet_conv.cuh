// unet_conv.cuh -- 3x3x3 "same" convolutions of 16-channel BF16 volumes on
// the 5th-generation tensor cores (tcgen05, TMEM accumulators).
//
// Activations: channels-last (NDHWC), 16 BF16 channels = 32 bytes per voxel,
// voxel index v = (i*ny + j)*nz + k.  Weights: W[co][tap][ci] BF16 with
// tap = (di+1)*9 + (dj+1)*3 + (dk+1), i.e. the GEMM operand B with K = tap*16+ci
// contiguous (K-major).
//
// Forward (and input gradient) as an implicit GEMM:
//   Y[v][co] = sum_{tap,ci} X[v + off(tap)][ci] * W[co][tap][ci]
//   M = 128 voxels per CTA, N = 16 output channels, K = 27*16 = 432 in seven
//   chunks of four taps (64 columns, the last zero-padded).  The four warps
//   gather each A chunk (one 16-byte vector = 8 channels of one neighbour per
//   store) into a K-major canonical tile, double-buffered; one thread issues
//   four tcgen05.mma (K = 16 each) per chunk and commits them to the chunk
//   buffer's mbarrier; the accumulator (128 lanes x 16 FP32 columns) is read
//   back with tcgen05.ld for the epilogue (bias, LeakyReLU, BF16 store).
//   The input gradient is the same GEMM with W'[ci][tap][co] = W[co][26-tap][ci].
//
// Weight gradient as a GEMM over voxels:
//   dW[co][tap][ci] = sum_v dY[v][co] * X[v + off(tap)][ci]
//   D (M = (tap, ci) rows in four 128-row tiles, N = 16) += A * B^T with
//   K = 64 voxels per chunk; A[(tap,ci)][v] and B[co][v] are gathered
//   MN-major (8 consecutive channels of one voxel = one 16-byte row), so the
//   instruction descriptor sets a_major = b_major = 1.  Each CTA accumulates
//   its voxel range in TMEM (4 x 16 columns) and writes FP32 partial sums;
//   a second kernel adds the partials in a fixed order (deterministic).
//
// Every mbarrier wait is bounded; a wait that gives up sets the error flag,
// and the CTA still frees its TMEM before returning.
#pragma once
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "tc.cuh"

namespace hc {
namespace unet {

constexpr int CH = 16;          // channels of every hidden volume
constexpr int NTAP = 27;
constexpr int TM = 128;         // voxels per CTA (GEMM M)
constexpr int KC = 64;          // K columns per chunk (4 taps x 16 channels)
constexpr int NCHUNK = 7;       // ceil(27/4)
constexpr int WELEM = CH * NTAP * CH;   // 6912 weights of one conv

struct Dims {
    int nx, ny, nz;
    long long n;                // voxels
};

__device__ __forceinline__ void voxel_ijk(const Dims &d, long long v, int &i, int &j, int &k)
{
    k = (int)(v % d.nz);
    long long t = v / d.nz;
    j = (int)(t % d.ny);
    i = (int)(t / d.ny);
}

// neighbour of (i,j,k) through tap, or -1 outside the volume
__device__ __forceinline__ long long neighbour(const Dims &d, int i, int j, int k, int tap)
{
    const int di = tap / 9 - 1, dj = (tap / 3) % 3 - 1, dk = tap % 3 - 1;
    const int a = i + di, b = j + dj, c = k + dk;
    if (a < 0 || a >= d.nx || b < 0 || b >= d.ny || c < 0 || c >= d.nz) return -1;
    return ((long long)a * d.ny + b) * d.nz + c;
}

__device__ __forceinline__ float leaky(float x) { return x > 0.f ? x : 0.1f * x; }

struct ConvSmem {
    __align__(128) unsigned char a[2][TM * KC * 2];        // 2 x 16 KB
    __align__(128) unsigned char b[NCHUNK][CH * KC * 2];   // 7 x 2 KB
    __align__(8) uint64_t bar[2];
    uint32_t tmem;
};

// out_mode: 0 = BF16 16 channels (+bias, LeakyReLU if act), 1 = BF16 16
// channels, no bias/activation (input gradient), 2 = FP32 channel 0 only
// (+bias[0], no activation: the network output), 3 = FP32 16 channels +bias
// (no rounding: the kernel's accumulators, for tests).
__global__ void __launch_bounds__(128)
conv3_kernel(const __nv_bfloat16 *__restrict__ x, const __nv_bfloat16 *__restrict__ w,
             const float *__restrict__ bias, void *__restrict__ out, Dims d, int out_mode, int act, int *err)
{
    extern __shared__ __align__(128) unsigned char smraw[];
    ConvSmem &sm = *reinterpret_cast<ConvSmem *>(smraw);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const long long v0 = (long long)blockIdx.x * TM;

    if (warp == 0) {
        tc::tmem_alloc(&sm.tmem, 32);
        tc::fence_before();
    }
    if (tid == 0) {
        tc::bar_init(&sm.bar[0], 1);
        tc::bar_init(&sm.bar[1], 1);
    }
    // weights -> B tiles (K-major canonical, 16 rows x 64 columns per chunk)
    for (int t = tid; t < NCHUNK * CH * (KC / 8); t += blockDim.x) {
        const int c = t / (CH * (KC / 8));
        const int rem = t % (CH * (KC / 8));
        const int co = rem / (KC / 8), kg = rem % (KC / 8);   // kg: 8-column group
        const int tap = c * 4 + kg / 2, half = kg & 1;
        uint4 val = make_uint4(0, 0, 0, 0);
        if (tap < NTAP) val = *reinterpret_cast<const uint4 *>(w + ((size_t)co * NTAP + tap) * CH + half * 8);
        *reinterpret_cast<uint4 *>(sm.b[c] + tc::kmajor_off(co, kg * 8, KC)) = val;
    }
    __syncthreads();
    tc::fence_after();
    const uint32_t tmem = sm.tmem;
    constexpr uint32_t IDESC = tc::idesc_bf16(TM, CH);
    bool ok = true;

    // this thread gathers row r = tid of every A chunk
    const long long v = v0 + tid;
    const bool vin = v < d.n;
    int vi = 0, vj = 0, vk = 0;
    if (vin) voxel_ijk(d, v, vi, vj, vk);

    for (int c = 0; c < NCHUNK; c++) {
        const int buf = c & 1;
        if (c >= 2) ok = tc::bar_wait(&sm.bar[buf], ((c - 2) >> 1) & 1) && ok;   // MMAs of chunk c-2 done
        unsigned char *A = sm.a[buf];
#pragma unroll
        for (int tl = 0; tl < 4; tl++) {
            const int tap = c * 4 + tl;
            long long nb = -1;
            if (vin && tap < NTAP) nb = neighbour(d, vi, vj, vk, tap);
#pragma unroll
            for (int half = 0; half < 2; half++) {
                uint4 val = make_uint4(0, 0, 0, 0);
                if (nb >= 0) val = *reinterpret_cast<const uint4 *>(x + nb * CH + half * 8);
                *reinterpret_cast<uint4 *>(A + tc::kmajor_off(tid, tl * 16 + half * 8, KC)) = val;
            }
        }
        tc::fence_smem_to_async();
        __syncthreads();
        if (tid == 0) {
            tc::fence_after();
            const uint32_t sa = tc::smem_u32(A), sb = tc::smem_u32(sm.b[c]);
#pragma unroll
            for (int s = 0; s < 4; s++) {
                const uint64_t da = tc::sdesc(sa + s * 256, 128, 16 * KC);
                const uint64_t db = tc::sdesc(sb + s * 256, 128, 16 * KC);
                tc::mma_bf16(tmem, da, db, IDESC, (c > 0 || s > 0) ? 1u : 0u);
            }
            tc::mma_commit(&sm.bar[buf]);
        }
    }
    // the last commit (chunk 6, buffer 0, its 4th phase) covers every MMA;
    // chunk 5's commit on buffer 1 is waited for too, so no arrive is pending
    ok = tc::bar_wait(&sm.bar[0], ((NCHUNK - 1) >> 1) & 1) && ok;
    ok = tc::bar_wait(&sm.bar[1], ((NCHUNK - 2) >> 1) & 1) && ok;
    tc::fence_after();
    float acc[16];
    tc::tmem_ld16(tmem + ((uint32_t)(warp * 32) << 16), acc);
    const long long vo = v0 + warp * 32 + lane;   // TMEM lane = row of D
    if (vo < d.n) {
        if (out_mode == 2) {
            reinterpret_cast<float *>(out)[vo] = acc[0] + bias[0];
        } else if (out_mode == 3) {
            float *o = reinterpret_cast<float *>(out) + vo * CH;
#pragma unroll
            for (int t = 0; t < 16; t++) o[t] = acc[t] + bias[t];
        } else {
            __align__(16) __nv_bfloat16 h[16];
#pragma unroll
            for (int t = 0; t < 16; t++) {
                float y = acc[t];
                if (out_mode == 0) {
                    y += bias[t];
                    if (act) y = leaky(y);
                }
                h[t] = __float2bfloat16(y);
            }
            uint4 *o = reinterpret_cast<uint4 *>(reinterpret_cast<__nv_bfloat16 *>(out) + vo * CH);
            o[0] = *reinterpret_cast<const uint4 *>(&h[0]);
            o[1] = *reinterpret_cast<const uint4 *>(&h[8]);
        }
    }
    tc::fence_before();
    __syncthreads();
    if (warp == 0) tc::tmem_dealloc(tmem, 32);
    if (!ok && tid == 0) atomicExch(err, -6);
}

// ---------------------------------------------------------------- weight gradient
constexpr int WG_LT = 256, WG_NT = WG_LT + 32;   // loading threads, and a warp that issues
constexpr int WG_MT = 4;                   // 128-row tiles: taps 0-7, 8-15, 16-23, 24-26
constexpr int WG_ST = 3;                   // chunks staged in shared memory
struct WgradSmem {
    __align__(128) unsigned char a[WG_ST][WG_MT][TM * KC * 2];   // 3 x 4 x 16 KB
    __align__(128) unsigned char b[WG_ST][CH * KC * 2];          // 3 x 2 KB
    __align__(8) uint64_t full[WG_ST], done[WG_ST];
    uint32_t tmem;
};

// byte offset of (mn, k) in an MN-major no-swizzle tile with KC columns:
// 8 consecutive mn = one 16-byte row, 8 rows (k) per core matrix
__host__ __device__ __forceinline__ constexpr uint32_t mnmajor_off(int mn, int k, int kc)
{
    return (uint32_t)((mn >> 3) * (16 * kc) + (k >> 3) * 128 + (k & 7) * 16 + (mn & 7) * 2);
}

// 16 bytes to shared memory without passing registers; zeros if !in
__device__ __forceinline__ void cp16(unsigned char *dst, const __nv_bfloat16 *src, bool in)
{
    asm volatile("cp.async.ca.shared.global [%0], [%1], 16, %2;" ::"r"(tc::smem_u32(dst)), "l"(src), "r"(in ? 16 : 0)
                 : "memory");
}

// Arrive on `bar` when this thread's cp.async so far have landed.  The thread
// that waits on it fences for the tensor core: a proxy fence here would wait
// for all copies in flight, a memory latency per chunk.
__device__ __forceinline__ void arrive_async(uint64_t *bar)
{
    asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(tc::smem_u32(bar)) : "memory");
}

// Taps G, G+2, ... of one voxel and channel half into the A tiles of a stage;
// the warps of G = 1 have one tap less and fetch dY instead.
template <int G>
__device__ __forceinline__ void wgrad_fetch(WgradSmem &sm, int st, const __nv_bfloat16 *__restrict__ x,
                                            const __nv_bfloat16 *__restrict__ dy, const Dims &d, long long v, int kk,
                                            int half)
{
    const bool live = v < d.n;
    int i = 0, j = 0, k = 0;
    if (d.n <= 0x7fffffffLL) {
        const unsigned u = (unsigned)v, row = u / (unsigned)d.nz;   // (the divisions of the 64-bit form cost 5x)
        k = (int)(u - row * (unsigned)d.nz);
        i = (int)(row / (unsigned)d.ny);
        j = (int)(row - (unsigned)i * (unsigned)d.ny);
    } else {
        voxel_ijk(d, v, i, j, k);
    }
    const bool ok_i[3] = { live && i > 0, live, live && i < d.nx - 1 };
    const bool ok_j[3] = { j > 0, true, j < d.ny - 1 };
    const bool ok_k[3] = { k > 0, true, k < d.nz - 1 };
    const long long plane = (long long)d.ny * d.nz;
    const __nv_bfloat16 *xh = x + half * 8;
    unsigned char *dst = sm.a[st][0] + mnmajor_off(half * 8, kk, KC);
#pragma unroll
    for (int m = 0; m < 14; m++) {
        constexpr int STEP = mnmajor_off(CH, 0, KC), TILE = TM * KC * 2;
        const int tap = G + 2 * m;
        if (tap < NTAP) {
            const int a = tap / 9, b = (tap / 3) % 3, c = tap % 3;
            const bool in = ok_i[a] && ok_j[b] && ok_k[c];
            const long long nb = v + (a - 1) * plane + (b - 1) * d.nz + (c - 1);
            cp16(dst + (tap >> 3) * TILE + (tap & 7) * STEP, in ? xh + nb * CH : x, in);
        }
    }
    if (G == 1) cp16(sm.b[st] + mnmajor_off(half * 8, kk, KC), live ? dy + v * CH + half * 8 : dy, live);
}

// partial[cta][tap][ci][co] over the CTA's voxel chunks [c0, c1).
//
// Each chunk of 64 voxels is staged as the 27 shifted copies of its x (the A
// operand of 16 MMAs of 16 voxels), and what bounds it is shared memory: 54 KB
// written and 72 KB read by the MMAs per chunk, about 1000 cycles.  Chunks are
// fetched by cp.async two ahead of the one the tensor core works on; a warp
// takes 16 voxels x 2 halves, 512 contiguous bytes.  Rows of taps past 26 are
// never written and never read back.  128^3 voxels 1650 -> 209 us, 64^3 205 ->
// 32 us against fetching through registers one chunk at a time, with a 64-bit
// division chain per 16 bytes.  One thread of a warp of its own issues, after
// the one proxy fence, and elected: with the fence in the loading threads and a
// thread-index test 128^3 stayed at 261 us.
__global__ void __launch_bounds__(WG_NT)
wgrad_kernel(const __nv_bfloat16 *__restrict__ x, const __nv_bfloat16 *__restrict__ dy, float *__restrict__ partial,
             Dims d, int chunks_per_cta, int *err)
{
    extern __shared__ __align__(128) unsigned char smraw[];
    WgradSmem &sm = *reinterpret_cast<WgradSmem *>(smraw);
    const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
    const long long nchunk = (d.n + KC - 1) / KC;
    const long long c0 = (long long)blockIdx.x * chunks_per_cta;
    const int nq = (int)(min(nchunk, c0 + chunks_per_cta) - c0);
    const int kk = (warp & 3) * 16 + (lane >> 4) * 8 + (lane & 7), half = (lane >> 3) & 1;

    if (warp == 0) {
        tc::tmem_alloc(&sm.tmem, 64);
        tc::fence_before();
    }
    if (tid == 0)
        for (int q = 0; q < WG_ST; q++) {
            tc::bar_init(&sm.full[q], WG_LT);
            tc::bar_init(&sm.done[q], 1);
        }
    __syncthreads();
    tc::fence_after();
    const uint32_t tmem = sm.tmem;
    constexpr uint32_t IDESC = tc::idesc_bf16(TM, CH) | (1u << 15) | (1u << 16);
    bool ok = true;

    if (warp < WG_LT / 32) {
        for (int q = 0; q < nq; q++) {
            const int st = q % WG_ST;
            if (q >= WG_ST) ok = tc::bar_wait(&sm.done[st], (q / WG_ST - 1) & 1) && ok;
            const long long v = (c0 + q) * KC + kk;
            if (warp < 4) wgrad_fetch<0>(sm, st, x, dy, d, v, kk, half);
            else wgrad_fetch<1>(sm, st, x, dy, d, v, kk, half);
            arrive_async(&sm.full[st]);
        }
    } else if (tc::elect_one()) {
        for (int q = 0; q < nq; q++) {
            const int st = q % WG_ST;
            ok = tc::bar_wait(&sm.full[st], (q / WG_ST) & 1) && ok;
            tc::fence_smem_to_async();
            tc::fence_after();
            const uint32_t sb = tc::smem_u32(sm.b[st]);
#pragma unroll
            for (int tile = 0; tile < WG_MT; tile++) {
                const uint32_t sa = tc::smem_u32(sm.a[st][tile]);
#pragma unroll
                for (int s = 0; s < 4; s++) {
                    const uint64_t da = tc::sdesc(sa + s * 256, 128, 16 * KC);
                    const uint64_t db = tc::sdesc(sb + s * 256, 128, 16 * KC);
                    tc::mma_bf16(tmem + tile * 16, da, db, IDESC, (q > 0 || s > 0) ? 1u : 0u);
                }
            }
            tc::mma_commit(&sm.done[st]);
        }
    }
    __syncthreads();
    float *p = partial + (size_t)blockIdx.x * (WG_MT * TM * CH);
    ok = tc::bar_wait(&sm.done[(nq - 1) % WG_ST], ((nq - 1) / WG_ST) & 1) && ok;   // the last commit covers all
    __syncwarp();
    tc::fence_after();
#pragma unroll
    for (int tile = 0; tile < WG_MT; tile++) {
        const int row = tile * TM + warp * 32 + lane;   // (tap, ci) = (row / 16, row % 16)
        if (warp < 4) {   // warps 0-3 own TMEM lanes 0-127
            float acc[16];
            tc::tmem_ld16(tmem + ((uint32_t)(warp * 32) << 16) + tile * 16, acc);
            float4 *o = reinterpret_cast<float4 *>(p + (size_t)row * CH);
            if (row < NTAP * CH) {
#pragma unroll
                for (int co = 0; co < 4; co++)
                    o[co] = make_float4(acc[4 * co], acc[4 * co + 1], acc[4 * co + 2], acc[4 * co + 3]);
            }
        }
    }
    tc::fence_before();
    __syncthreads();
    if (warp == 0) tc::tmem_dealloc(tmem, 64);
    if (!ok) atomicExch(err, -6);
}

// The sum of n values `stride` apart in their order, 16 loads in flight: with
// one add per load the chain is n memory latencies.  (37 with the last batch
// masked is slower: the masks cost more than the fewer latencies save.)
__device__ __forceinline__ float sum_in_order(const float *__restrict__ p, int n, int stride)
{
    float s = 0.f;
    int q = 0;
    for (; q + 16 <= n; q += 16) {
        float f[16];
#pragma unroll
        for (int t = 0; t < 16; t++) f[t] = p[(size_t)(q + t) * stride];
#pragma unroll
        for (int t = 0; t < 16; t++) s += f[t];
    }
    for (; q < n; q++) s += p[(size_t)q * stride];
    return s;
}

// dW[co][tap][ci] = sum over CTAs of partial[cta][tap*16+ci][co], fixed order.
// Neighbouring threads read neighbouring co (15 -> 9.5 us for 148 parts).
constexpr int WRED_NT = 64;
__global__ void __launch_bounds__(WRED_NT) wgrad_reduce_kernel(const float *__restrict__ partial, int nparts,
                                                               float *__restrict__ dw)
{
    const int e = blockIdx.x * blockDim.x + threadIdx.x;   // (tap, ci, co)
    if (e >= WELEM) return;
    dw[(size_t)(e % CH) * (NTAP * CH) + e / CH] = sum_in_order(partial + e, nparts, WG_MT * TM * CH);
}


// ---------------------------------------------------------------------------
// Halo-tile convolution (forward / input gradient) without an im2col copy.
//
// A CTA owns a 16 (j) x 8 (k) column of output voxels and marches along i.
// Each input plane of the column plus its halo (18 x 10 voxels) is fetched by
// two cp.async.bulk.tensor loads (one per 8-channel half, zero-filled outside
// the volume) into a 4-slot ring laid out [half][j][k][8 ch]: 8 consecutive k
// of one half are 128 contiguous bytes, i.e. one core matrix of a K-major
// operand.  The A operand of tap (a,b,c) for output plane i is therefore a
// descriptor into the halo of plane i+a-1 starting at row (b, c): SBO = 160
// bytes (next j), LBO = one half-plane (2944-byte stride, channels 8..15).  Each
// output plane is 27 MMAs (M=128 voxels, N=16, K=16 channels) accumulated in
// one of two TMEM buffers; the epilogue of plane p-1 runs while the MMAs of
// plane p execute, and the halo slot of plane p-2 is refilled once the MMAs
// of plane p-1 have completed.
// ---------------------------------------------------------------------------
constexpr int HT_J = 16, HT_K = 8;                  // output tile
constexpr int HH_J = HT_J + 2, HH_K = HT_K + 2;     // halo tile
constexpr int HALF_BYTES = HH_J * HH_K * 16;        // 2880 loaded per channel half
constexpr int HALF_STRIDE = 2944;                   // 128-byte aligned stride (the descriptor LBO)
constexpr int SLOT_BYTES = 2 * HALF_STRIDE;         // 5888
constexpr int NSLOT = 4;

struct HaloSmem {
    __align__(128) unsigned char slot[NSLOT][SLOT_BYTES];
    __align__(128) unsigned char w[NTAP][512];      // B per tap: 16 co x 16 ci, K-major
    __align__(8) uint64_t tbar[NSLOT];
    __align__(8) uint64_t mbar[2];
    uint32_t tmem;
};

__device__ __forceinline__ void halo_load(const CUtensorMap *tm, HaloSmem &sm, int slot, int k0, int j0, int i)
{
    uint64_t *bar = &sm.tbar[slot];
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(tc::smem_u32(bar)),
                 "r"((unsigned)(2 * HALF_BYTES))
                 : "memory");
#pragma unroll
    for (int h = 0; h < 2; h++)
        asm volatile("cp.async.bulk.tensor.4d.shared::cluster.global.mbarrier::complete_tx::bytes"
                     " [%0], [%1, {%2, %3, %4, %5}], [%6];" ::"r"(tc::smem_u32(sm.slot[slot] + h * HALF_STRIDE)),
                     "l"(reinterpret_cast<uint64_t>(tm)), "r"(8 * h), "r"(k0 - 1), "r"(j0 - 1), "r"(i),
                     "r"(tc::smem_u32(bar))
                     : "memory");
}

__global__ void __launch_bounds__(128)
conv3_halo_kernel(const __grid_constant__ CUtensorMap tmx, const __nv_bfloat16 *__restrict__ w,
                  const float *__restrict__ bias, void *__restrict__ out, Dims d, int out_mode, int act, int chunk,
                  int *err)
{
    extern __shared__ __align__(128) unsigned char smraw[];
    HaloSmem &sm = *reinterpret_cast<HaloSmem *>(smraw);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int k0 = blockIdx.x * HT_K, j0 = blockIdx.y * HT_J;
    const int i0 = blockIdx.z * chunk, i1 = min(d.nx, i0 + chunk);
    if (i0 >= i1) return;
    const int np = i1 - i0;

    if (warp == 0) {
        tc::tmem_alloc(&sm.tmem, 32);
        tc::fence_before();
    }
    if (tid == 0) {
        for (int q = 0; q < NSLOT; q++) tc::bar_init(&sm.tbar[q], 1);
        tc::bar_init(&sm.mbar[0], 1);
        tc::bar_init(&sm.mbar[1], 1);
    }
    // weights: B of tap t, row co, K = ci: (co/8)*256 + (ci/8)*128 + (co%8)*16 + (ci%8)*2
    for (int q = tid; q < NTAP * CH * 2; q += blockDim.x) {
        const int tap = q / (CH * 2), rem = q % (CH * 2), co = rem >> 1, half = rem & 1;
        const uint4 v = *reinterpret_cast<const uint4 *>(w + ((size_t)co * NTAP + tap) * CH + half * 8);
        *reinterpret_cast<uint4 *>(sm.w[tap] + (co >> 3) * 256 + half * 128 + (co & 7) * 16) = v;
    }
    tc::fence_smem_to_async();
    __syncthreads();
    tc::fence_after();
    const uint32_t tmem = sm.tmem;
    constexpr uint32_t IDESC = tc::idesc_bf16(TM, CH);
    bool ok = true;
    unsigned tph[NSLOT] = { 0, 0, 0, 0 }, mph[2] = { 0, 0 };
    auto slot_of = [](int plane) { return (plane + 4) & 3; };   // plane >= -1

    if (tid == 0) {
        halo_load(&tmx, sm, slot_of(i0 - 1), k0, j0, i0 - 1);
        halo_load(&tmx, sm, slot_of(i0), k0, j0, i0);
        halo_load(&tmx, sm, slot_of(i0 + 1), k0, j0, i0 + 1);
    }
    auto wait_plane = [&](int plane) {
        const int sl = slot_of(plane);
        ok = tc::bar_wait(&sm.tbar[sl], tph[sl] & 1) && ok;
        tph[sl]++;
    };
    auto epilogue = [&](int p) {
        const int b = p & 1;
        ok = tc::bar_wait(&sm.mbar[b], mph[b] & 1) && ok;
        mph[b]++;
        tc::fence_after();
        float acc[16];
        tc::tmem_ld16(tmem + ((uint32_t)(warp * 32) << 16) + b * 16, acc);
        const int r = warp * 32 + lane, jj = r >> 3, kk = r & 7;
        const int j = j0 + jj, k = k0 + kk, i = i0 + p;
        if (j < d.ny && k < d.nz) {
            const long long vo = ((long long)i * d.ny + j) * d.nz + k;
            if (out_mode == 2) {
                reinterpret_cast<float *>(out)[vo] = acc[0] + bias[0];
            } else if (out_mode == 3) {
                float *o = reinterpret_cast<float *>(out) + vo * CH;
#pragma unroll
                for (int t = 0; t < 16; t++) o[t] = acc[t] + bias[t];
            } else {
                __align__(16) __nv_bfloat16 h[16];
#pragma unroll
                for (int t = 0; t < 16; t++) {
                    float y = acc[t];
                    if (out_mode == 0) {
                        y += bias[t];
                        if (act) y = leaky(y);
                    }
                    h[t] = __float2bfloat16(y);
                }
                uint4 *o = reinterpret_cast<uint4 *>(reinterpret_cast<__nv_bfloat16 *>(out) + vo * CH);
                o[0] = *reinterpret_cast<const uint4 *>(&h[0]);
                o[1] = *reinterpret_cast<const uint4 *>(&h[8]);
            }
        }
    };

    wait_plane(i0 - 1);
    wait_plane(i0);
    for (int p = 0; p < np; p++) {
        const int i = i0 + p;
        wait_plane(i + 1);
        if (tid == 0) {
            tc::fence_after();
            const uint32_t wb = tc::smem_u32(sm.w[0]);
#pragma unroll 1
            for (int a = 0; a < 3; a++) {
                const uint32_t base = tc::smem_u32(sm.slot[slot_of(i + a - 1)]);
#pragma unroll
                for (int bc = 0; bc < 9; bc++) {
                    const int b = bc / 3, c = bc % 3, tap = a * 9 + bc;
                    const uint64_t da = tc::sdesc(base + (b * HH_K + c) * 16, HALF_STRIDE, HH_K * 16);
                    const uint64_t db = tc::sdesc(wb + tap * 512, 128, 256);
                    tc::mma_bf16(tmem + (p & 1) * 16, da, db, IDESC, tap > 0 ? 1u : 0u);
                }
            }
            tc::mma_commit(&sm.mbar[p & 1]);
        }
        if (p >= 1) epilogue(p - 1);   // also: the MMAs of plane p-1 are done
        if (tid == 0 && p + 2 < np + 1) halo_load(&tmx, sm, slot_of(i + 2), k0, j0, i + 2);
        tc::fence_before();
        __syncthreads();   // TMEM buffer of plane p-1 read by all before plane p+1 reuses it
    }
    epilogue(np - 1);
    // the last halo load (plane i1) was consumed by the last plane; planes past it were not issued
    tc::fence_before();
    __syncthreads();
    if (warp == 0) tc::tmem_dealloc(tmem, 32);
    if (!ok && tid == 0) atomicExch(err, -6);
}

// ---------------------------------------------------------------------------
// Weight gradient without shifted copies, for rows of a multiple of 16 voxels.
//
// A CTA walks its voxels row by row.  Rows j-1, j, j+1 of planes i-1, i, i+1
// live in a ring of slots, each {row j of three planes}, with one voxel of halo
// at both ends (zeros outside the volume), laid out [half][plane][k][8 ch]: for
// MMAs that contract over 16 voxels the 6 groups (half, plane) are rows 0-47 of
// an MN-major A operand with one stride, and the tap's shift along k is 16 bytes
// of the descriptor's start.  So 16 voxels are 9 MMAs (M = 64: three planes x 16
// channels and two groups of whatever follows, never read back; N = 16), one per
// (tap j, tap k), and stepping j loads only one new slot.  The voxels are grouped
// and added up in the order of wgrad_kernel over the same ranges: the bits are
// the same.
//
// Five warps fetch by cp.async, row by row in turn.  Three threads issue, one
// per tap j, each into accumulators of its own: one thread spends 670 cycles
// between the last MMA of a row and the first of the next, and the tensor core
// waits for it.
//
// What bounds it is the rate of these MMAs, 23 cycles each (17 of them to read
// the 64 rows of A from shared memory), 13 per voxel.  128^3 voxels 209 us
// (wgrad_kernel) -> 112, 96^3 94 -> 52, 64^3 32 -> 22.
// ---------------------------------------------------------------------------
constexpr int WR_NT = 256, WR_LW = 5;      // threads; loading warps (the last three issue, one per tap j)
constexpr int WR_MAXS = 10, WR_MINS = 4;   // slots: three in use, the rest ahead
constexpr int WR_RING = 16;                // > slots: rows between the loaders and the issuer
constexpr unsigned WR_SMEM = 227 * 1024;

struct WrowBars {
    uint64_t ready[WR_RING], done[WR_RING], fin;
    uint32_t tmem;
};

struct WrowGeom {
    int kb, slots, dys;                    // voxels of a row with its halo, ring slots, rows of dY staged
    unsigned slot_bytes, dy_bytes;
    // the two groups past the last slot's planes fall into the rows of dY
    __host__ __device__ unsigned bars_at() const { return slots * slot_bytes + dys * dy_bytes; }
    __host__ __device__ unsigned smem() const { return bars_at() + (unsigned)sizeof(WrowBars); }
};

// Whether wgrad_row_kernel takes a volume, `per_cta` chunks to a CTA.  Not rows
// of odd lengths (a group of 16 voxels would span rows), short ones (256 x 256 x
// 16: 151 us against 106; 32^3: 9.8 against 8.8; 48^3: 13.7 against 15.9), and
// CTAs of a few rows, which fetch mostly neighbours (16 x 16 x 384, two rows:
// 20 against 16; 32 x 32 x 256, seven: 24 against 31).
__host__ inline bool wrow_geom(const Dims &d, int per_cta, WrowGeom *g)
{
    if (d.nz % 16 || d.nz < 48 || d.nz > 1024 || (long long)per_cta * KC < 4LL * d.nz) return false;
    g->kb = d.nz + 2;
    g->slot_bytes = 96u * g->kb;
    g->dy_bytes = 32u * d.nz;
    for (g->slots = WR_MAXS; g->slots >= WR_MINS; g->slots--) {
        g->dys = g->slots - 2;
        if (g->smem() <= WR_SMEM) return true;
    }
    return false;                          // rows past 512 leave no room for four slots
}

// partial[cta][tap][ci][co] over the voxels of chunks [c0, c1), as wgrad_kernel
__global__ void __launch_bounds__(WR_NT)
wgrad_row_kernel(const __nv_bfloat16 *__restrict__ x, const __nv_bfloat16 *__restrict__ dy, float *__restrict__ partial,
                 Dims d, WrowGeom g, int chunks_per_cta, int *err)
{
    extern __shared__ __align__(128) unsigned char smraw[];
    WrowBars &sm = *reinterpret_cast<WrowBars *>(smraw + g.bars_at());
    const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
    const long long v0 = (long long)blockIdx.x * chunks_per_cta * KC;
    const long long v1 = min(d.n, v0 + (long long)chunks_per_cta * KC);
    const long long row0 = v0 / d.nz;
    const int nu = (int)((v1 - 1) / d.nz - row0) + 1;              // rows touched
    const int kfirst = (int)(v0 - row0 * d.nz), klast = (int)(v1 - (row0 + nu - 1) * d.nz);
    const int i0 = (int)(row0 / d.ny), j0 = (int)(row0 % d.ny);

    if (warp == 0) {
        tc::tmem_alloc(&sm.tmem, 256);
        tc::fence_before();
    }
    if (tid == 0) {
        for (int q = 0; q < WR_RING; q++) {
            tc::bar_init(&sm.ready[q], 32);
            tc::bar_init(&sm.done[q], 3);
        }
        tc::bar_init(&sm.fin, 3);
    }
    __syncthreads();
    tc::fence_after();
    const uint32_t tmem = sm.tmem, sx = tc::smem_u32(smraw), sy = sx + g.slots * g.slot_bytes;
    bool ok = true;

    if (warp < WR_LW) {
        // Row u needs loads ell(u) .. ell(u) + 2, ell stepping by 1 within a plane and by 3 into the next.  Loading
        // warps take rows in turn: one row's loads are a chain of a thousand cycles and more.
        int ld = 0, slot = 0, w = -1, wj = j0 - 1, well = -1;      // w: last row known to be done, its j and ell
        int i = i0, j = j0;
        const int half = (lane >> 3) & 1, kl = (lane >> 4) * 8 + (lane & 7);   // 8 voxels of one half, then the other
        for (int u = 0; u < nu; u++) {
            const int jfrom = (u == 0 || j == 0) ? j - 1 : j + 1, nl = j + 2 - jfrom;
            const bool mine = u % WR_LW == warp;
            if (mine) {
                // rows still reading what the new loads and the row of dY replace
                const int w0 = w;
                for (;;) {
                    const int next = w < 0 ? 0 : wj + 1 == d.ny ? well + 3 : well + 1;
                    if (w + 1 >= u || (next > ld + nl - 1 - g.slots && w + 1 > u - g.dys)) break;
                    w++;
                    well = next;
                    if (++wj == d.ny) wj = 0;
                }
                if (w > w0) ok = tc::bar_wait(&sm.done[w % WR_RING], (w / WR_RING) & 1) && ok;
                __syncwarp();
            }
            for (int jj = jfrom; jj <= j + 1; jj++) {
                if (mine) {
                    const bool in_j = jj >= 0 && jj < d.ny;
#pragma unroll
                    for (int a = 0; a < 3; a++) {
                        const int ii = i + a - 1;
                        const bool in = in_j && ii >= 0 && ii < d.nx;
                        const __nv_bfloat16 *src = in ? x + ((long long)ii * d.ny + jj) * d.nz * CH + half * 8 - CH : x;
                        unsigned char *dst = smraw + slot * g.slot_bytes + (a + 3 * half) * 16 * g.kb;
#pragma unroll 4
                        for (int k = kl; k < g.kb; k += 16) {      // k: voxel k - 1
                            const bool there = in && k > 0 && k <= d.nz;
                            cp16(dst + k * 16, there ? src + k * CH : x, there);
                        }
                    }
                }
                ld++;
                if (++slot == g.slots) slot = 0;
            }
            if (mine) {
                const __nv_bfloat16 *src = dy + ((long long)i * d.ny + j) * d.nz * CH + half * 8;
                unsigned char *dst = smraw + g.slots * g.slot_bytes + (u % g.dys) * g.dy_bytes + half * 16 * d.nz;
#pragma unroll 4
                for (int k = kl; k < d.nz; k += 16) cp16(dst + k * 16, src + k * CH, true);
                arrive_async(&sm.ready[u % WR_RING]);
            }
            if (++j == d.ny) j = 0, i++;
        }
    } else if (tc::elect_one()) {
        constexpr uint32_t IDESC = tc::idesc_bf16(64, CH) | (1u << 15) | (1u << 16);
        const int b = warp - WR_LW;        // tap j
        const uint64_t xd = tc::sdesc(sx, 128, 16 * g.kb), yd = tc::sdesc(sy, 128, 16 * d.nz);
        const uint32_t acc0 = tmem + b * 3 * 16;
        int slot = b, j = j0, dyr = 0;     // slot of load ell + b
        uint32_t acc = 0;
        for (int u = 0; u < nu; u++) {
            const uint64_t xb = xd + (slot * g.slot_bytes >> 4), yb = yd + (dyr * g.dy_bytes >> 4);
            const int ke = u == nu - 1 ? klast : d.nz;
            ok = tc::bar_wait(&sm.ready[u % WR_RING], (u / WR_RING) & 1) && ok;
            tc::fence_smem_to_async();
            tc::fence_after();
            for (int k = u == 0 ? kfirst : 0; k < ke; k += 16) {
#pragma unroll
                for (int c = 0; c < 3; c++) tc::mma_bf16(acc0 + c * 16, xb + k + c, yb + k, IDESC, acc);
                acc = 1;
            }
            tc::mma_commit(&sm.done[u % WR_RING]);
            const int step = ++j == d.ny ? 3 : 1;
            if (j == d.ny) j = 0;
            slot += step;
            if (slot >= g.slots) slot -= g.slots;
            if (++dyr == g.dys) dyr = 0;
        }
        tc::mma_commit(&sm.fin);
    }
    __syncthreads();
    ok = tc::bar_wait(&sm.fin, 0) && ok;
    __syncwarp();
    tc::fence_after();
    if (warp < 4) {
        // M = 64: row r lies in TMEM lane 32 (r / 16) + r % 16
        const int r = warp * 16 + (lane & 15), half = r / 24, a = (r % 24) >> 3, ci = half * 8 + (r & 7);
        float *p = partial + (size_t)blockIdx.x * (WG_MT * TM * CH);
#pragma unroll
        for (int bc = 0; bc < 9; bc++) {
            float v[16];
            tc::tmem_ld16(tmem + ((uint32_t)(warp * 32) << 16) + bc * 16, v);
            if (lane < 16 && r < 48) {
                float4 *o = reinterpret_cast<float4 *>(p + (size_t)((a * 9 + bc) * CH + ci) * CH);
#pragma unroll
                for (int co = 0; co < 4; co++)
                    o[co] = make_float4(v[4 * co], v[4 * co + 1], v[4 * co + 2], v[4 * co + 3]);
            }
        }
    }
    tc::fence_before();
    __syncthreads();
    if (warp == 0) tc::tmem_dealloc(tmem, 256);
    if (!ok) atomicExch(err, -6);
}

}  // namespace unet
}  // namespace hc
