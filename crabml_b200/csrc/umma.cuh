// umma.cuh -- inline PTX of the 5th-generation tensor cores that the product kernels share (prefill_gemm.cu, split_gemm.cuh): mbarriers, TMA tile
// loads, tcgen05.mma with its descriptors.  Tiles are rows of 64 16-bit numbers (128 bytes) under the 128-byte swizzle.
#pragma once
#include <stdint.h>

#define PG_BLOCK_M 128
#define PG_BLOCK_K 64                     // 64 16-bit numbers = 128 bytes = one swizzle-128B row
#define PG_UMMA_K 16

// ---- PTX helpers ------------------------------------------------------------------------------------------------------------
__device__ __forceinline__ unsigned pg_smem(const void* p) { return (unsigned)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void pg_mbar_init(unsigned bar, unsigned count) { asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory"); }
__device__ __forceinline__ void pg_mbar_expect_tx(unsigned bar, unsigned bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ void pg_mbar_wait(unsigned bar, unsigned parity) {
    unsigned done = 0;
    for (unsigned it = 0; !done; it++) {
        asm volatile("{\n.reg .pred p;\nmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\nselp.u32 %0, 1, 0, p;\n}\n" : "=r"(done) : "r"(bar), "r"(parity) : "memory");
        if (it > (1u << 26)) __trap();          // bounded: a pipeline bug must not hang the GPU
    }
}
__device__ __forceinline__ void pg_tma_load_2d(unsigned dst, const void* tmap, unsigned bar, int x, int y) {
    asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
                 ::"r"(dst), "l"(tmap), "r"(bar), "r"(x), "r"(y) : "memory");
}
__device__ __forceinline__ void pg_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void pg_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
// D[tmem] (+)= A[smem] * B[smem]^T, f16 inputs, f32 accumulate; issued by ONE thread
__device__ __forceinline__ void pg_umma_f16(unsigned tmem_d, uint64_t desc_a, uint64_t desc_b, unsigned idesc, unsigned accumulate) {
    asm volatile("{\n.reg .pred p;\nsetp.ne.b32 p, %4, 0;\ntcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n"
                 ::"r"(tmem_d), "l"(desc_a), "l"(desc_b), "r"(idesc), "r"(accumulate) : "memory");
}
// all tcgen05 operations issued so far by this thread arrive (once) on the mbarrier when they complete
__device__ __forceinline__ void pg_umma_commit(unsigned bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}
// shared-memory matrix descriptor of a K-major tile stored as rows of 128 bytes with the 128-byte swizzle (what the TMA box
// {64 x rows} with CU_TENSOR_MAP_SWIZZLE_128B writes): 8-row groups are 1024 bytes apart (stride byte offset), the leading byte
// offset is unused for swizzled K-major operands, descriptor version 1 (sm_100), layout type 2 = SWIZZLE_128B.
__device__ __forceinline__ uint64_t pg_smem_desc(unsigned smem_addr) {
    uint64_t d = 0;
    d |= (uint64_t)((smem_addr & 0x3FFFF) >> 4);                  // bits [0, 14): start address >> 4
    d |= (uint64_t)0 << 16;                                       // bits [16, 30): leading byte offset >> 4
    d |= (uint64_t)(1024 >> 4) << 32;                             // bits [32, 46): stride byte offset >> 4
    d |= (uint64_t)1 << 46;                                       // bits [46, 48): descriptor version
    d |= (uint64_t)2 << 61;                                       // bits [61, 64): SWIZZLE_128B
    return d;
}
// instruction descriptor of kind::f16: f32 accumulator, f16 A and B, both K-major, dense
__host__ __device__ constexpr unsigned pg_instr_desc(int umma_m, int umma_n, int fmt = 0) {
    return (1u << 4)                          // bits [4, 6): accumulator format, 1 = F32
           | ((unsigned)fmt << 7) | ((unsigned)fmt << 10)   // bits [7, 10) / [10, 13): A / B format, 0 = F16, 1 = BF16
           | (0u << 15) | (0u << 16)          // A / B major: 0 = K-major
           | ((unsigned)(umma_n >> 3) << 17)  // bits [17, 23): N >> 3
           | ((unsigned)(umma_m >> 4) << 24); // bits [24, 29): M >> 4
}
