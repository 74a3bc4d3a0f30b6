// tc05.cuh -- the fifth-generation tensor-core and asynchronous-copy instructions the
// kernels use, as inline PTX: mbarriers with bounded waits, the untiled bulk copy,
// tensor memory (TMEM) allocation, load and store, and tcgen05.mma with the A operand
// in TMEM.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

namespace vpm {

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(uint64_t* m, uint32_t count)
{
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(m)), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_init_fence()
{
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
__device__ __forceinline__ void mbar_arrive(uint64_t* m)
{
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(m)) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t* m, uint32_t bytes)
{
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(m)), "r"(bytes) : "memory");
}
// A wait of a whole warp for the phase of m with this parity: a look, then up to `rounds` rounds of
// try_wait (each suspends the threads for a hardware time slice; a wait in normal running ends within
// the first few), after which it gives up.  The same answer in all 32 lanes: true if every lane saw the
// phase complete.
__device__ __forceinline__ bool mbar_wait(uint64_t* m, uint32_t parity, uint32_t rounds)
{
    uint32_t done;
    asm volatile("{\n\t.reg .pred p, q;\n\t.reg .u32 n;\n\tmov.u32 n, %3;\n\t"
                 "mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n"
                 "WAIT:\n\t@p bra DONE;\n\tsetp.eq.u32 q, n, 0;\n\t@q bra DONE;\n\tsub.u32 n, n, 1;\n\t"
                 "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tbra WAIT;\n"
                 "DONE:\n\tselp.u32 %0, 1, 0, p;\n\t}"
                 : "=r"(done) : "r"(smem_u32(m)), "r"(parity), "r"(rounds) : "memory");
    return __all_sync(0xffffffffu, done != 0);
}

// one lane of a converged warp
__device__ __forceinline__ bool elect_one()
{
    uint32_t p;
    asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(p));
    return p != 0;
}

// bulk copy global -> shared of `bytes` (a multiple of 16; both addresses 16-byte aligned),
// counted on m
__device__ __forceinline__ void bulk_load(void* dst, const void* src, uint32_t bytes, uint64_t* m)
{
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                 ::"r"(smem_u32(dst)), "l"(src), "r"(bytes), "r"(smem_u32(m)) : "memory");
}

// TMEM allocation of `cols` columns (a power of two, at least 32) by one whole warp; the
// address lands in *slot (shared memory).  It waits while other blocks of the SM hold the
// columns, so a kernel's resident blocks must fit the SM's 512 columns together.
__device__ __forceinline__ void tmem_alloc(uint32_t* slot, uint32_t cols)
{
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(slot)), "r"(cols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc(uint32_t addr, uint32_t cols)
{
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(addr), "r"(cols) : "memory");
}

__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
// Waits for this warp's TMEM loads; v: the registers they fill, which no instruction may use
// before the wait.
template <int N>
__device__ __forceinline__ void tc_wait_ld(float (&v)[N])
{
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int k = 0; k < N; k++) asm volatile("" : "+f"(v[k]));
}

// 8 consecutive columns of this thread's TMEM lane (whole warp, lanes 32 (warp % 4) ...)
__device__ __forceinline__ void tmem_st8(uint32_t addr, const uint32_t (&r)[8])
{
    asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};"
                 ::"r"(addr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7])
                 : "memory");
}
__device__ __forceinline__ void tmem_st4(uint32_t addr, const uint32_t (&r)[4])
{
    asm volatile("tcgen05.st.sync.aligned.32x32b.x4.b32 [%0], {%1, %2, %3, %4};"
                 ::"r"(addr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]) : "memory");
}
__device__ __forceinline__ void tmem_ld8(uint32_t addr, float* r)
{
    uint32_t v[8];
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7])
                 : "r"(addr) : "memory");
#pragma unroll
    for (int k = 0; k < 8; k++) r[k] = __uint_as_float(v[k]);
}

// Shared-memory matrix descriptor, K-major, no swizzle: 8-row x 16-byte core matrices,
// lbo bytes apart along K and sbo bytes apart along the rows.
__device__ __forceinline__ uint64_t smem_desc(uint32_t addr, uint32_t lbo, uint32_t sbo)
{
    return (uint64_t)((addr >> 4) & 0x3FFFu) | ((uint64_t)((lbo >> 4) & 0x3FFFu) << 16) |
           ((uint64_t)((sbo >> 4) & 0x3FFFu) << 32) | (1ull << 46);
}
// Instruction descriptor of kind::f16 with f16 operands, FP32 accumulators, both K-major
__host__ __device__ constexpr uint32_t idesc_f16(uint32_t m, uint32_t n)
{
    return (1u << 4) | ((n >> 3) << 17) | ((m >> 4) << 24);
}
// D[128 x N] (TMEM) (+)= A[128 x 16] (TMEM, two f16 a column) * B[N x 16]^T (shared memory);
// one thread issues it
__device__ __forceinline__ void mma_f16_ts(uint32_t d, uint32_t a, uint64_t bdesc, uint32_t idesc, bool accumulate)
{
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
                 "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
                 ::"r"(d), "r"(a), "l"(bdesc), "r"(idesc), "r"(accumulate ? 1u : 0u) : "memory");
}
// arrive on m when every tcgen05 operation this thread has issued so far is complete
__device__ __forceinline__ void mma_commit(uint64_t* m)
{
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(m))
                 : "memory");
}

}  // namespace vpm
