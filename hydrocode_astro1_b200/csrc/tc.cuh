// tc.cuh -- 5th-generation tensor core (tcgen05) primitives for sm_100a:
// TMEM allocation, shared-memory matrix descriptors, BF16 MMA with FP32
// accumulation in TMEM, commit to an mbarrier, TMEM loads.
//
// Operand layout (K-major, no swizzle): a tile of R rows x K columns of bf16
// is stored as core matrices of 8 rows x 16 bytes (8 bf16 along K), 128
// contiguous bytes each, row r of a core matrix at +16 r.  Core matrices
// adjacent along K are LBO bytes apart, groups of 8 rows SBO bytes apart.
// With a K extent of KC elements per stage the natural packing is
// LBO = 128 and SBO = 16 KC bytes:
//     byte(r, k) = (r / 8) * 16 KC + (k / 8) * 128 + (r % 8) * 16 + (k % 8) * 2
// One MMA consumes K = 16 (two core matrices along K); the descriptor of the
// s-th K slice starts 256 s bytes further.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

namespace hc {
namespace tc {

__device__ __forceinline__ uint32_t smem_u32(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }

// byte offset of element (r, k) in a K-major no-swizzle tile with KC columns
__host__ __device__ __forceinline__ uint32_t kmajor_off(int r, int k, int KC)
{
    return (uint32_t)((r >> 3) * (16 * KC) + (k >> 3) * 128 + (r & 7) * 16 + (k & 7) * 2);
}

// True in one thread of a converged warp.  MMAs are issued under this, not
// under a test of the thread index: the compiler then knows that one thread
// runs and keeps descriptors where the instruction takes them, and a stream of
// M = 128, N = 16 MMAs runs at the tensor core's 39 cycles each (M = 64: 23)
// instead of the 45 to 53 that a thread-index branch takes to issue one.
__device__ __forceinline__ bool elect_one()
{
    uint32_t one;
    asm volatile("{\n\t.reg .pred q;\n\telect.sync _|q, 0xffffffff;\n\tselp.u32 %0, 1, 0, q;\n\t}" : "=r"(one));
    return one != 0;
}

// One full warp executes alloc and dealloc.  ncols: power of two >= 32.
__device__ __forceinline__ void tmem_alloc(uint32_t *smem_dst, uint32_t ncols)
{
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(smem_dst)),
                 "r"(ncols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t ncols)
{
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}

// Shared-memory matrix descriptor: SWIZZLE_NONE (layout type 0), version 1.
__device__ __forceinline__ uint64_t sdesc(uint32_t saddr, uint32_t lbo, uint32_t sbo)
{
    uint64_t d = 0;
    d |= (uint64_t)((saddr >> 4) & 0x3FFFu);
    d |= (uint64_t)((lbo >> 4) & 0x3FFFu) << 16;
    d |= (uint64_t)((sbo >> 4) & 0x3FFFu) << 32;
    d |= (uint64_t)1 << 46;
    return d;
}

// Instruction descriptor, kind::f16: BF16 A and B, FP32 D, both K-major.
__host__ __device__ constexpr uint32_t idesc_bf16(int M, int N)
{
    return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(N >> 3) << 17) | ((uint32_t)(M >> 4) << 24);
}

// D[tmem] (+)= A[smem] * B[smem]^T, issued by one thread.
__device__ __forceinline__ void mma_bf16(uint32_t d_tmem, uint64_t a, uint64_t b, uint32_t idesc, uint32_t acc)
{
    asm volatile("{\n\t.reg .pred p;\n\t"
                 "setp.ne.b32 p, %4, 0;\n\t"
                 "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, {%5, %6, %7, %8}, p;\n\t}\n" ::"r"(d_tmem),
                 "l"(a), "l"(b), "r"(idesc), "r"(acc), "r"(0u), "r"(0u), "r"(0u), "r"(0u)
                 : "memory");
}

// Arrive once on `bar` when every MMA this thread issued so far has completed.
__device__ __forceinline__ void mma_commit(uint64_t *bar)
{
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                     smem_u32(bar))
                 : "memory");
}

__device__ __forceinline__ void fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
// generic-proxy shared-memory writes -> visible to the tensor core (async proxy)
__device__ __forceinline__ void fence_smem_to_async() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }

__device__ __forceinline__ void bar_init(uint64_t *bar, unsigned count)
{
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}

// Bounded wait for the completion of the phase with the given parity;
// false if the limit ran out.
__device__ __forceinline__ bool bar_wait(uint64_t *bar, unsigned parity)
{
    const uint32_t a = smem_u32(bar);
    for (int it = 0; it < (1 << 22); it++) {
        uint32_t ok;
        asm volatile("{\n\t.reg .pred p;\n\t"
                     "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
                     "selp.u32 %0, 1, 0, p;\n\t}"
                     : "=r"(ok)
                     : "r"(a), "r"(parity)
                     : "memory");
        if (ok) return true;
        if (it > 64) __nanosleep(32);
    }
    return false;
}

// 32 TMEM lanes (this warp's quarter) x 16 FP32 columns.
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, float (&v)[16])
{
    uint32_t r[16];
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 "
                 "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
                   "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]),
                   "=r"(r[15])
                 : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int t = 0; t < 16; t++) v[t] = __uint_as_float(r[t]);
}

}  // namespace tc
}  // namespace hc
