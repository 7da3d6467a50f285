// Tensor-core (tcgen05) and tensor-map (TMA) instructions shared by the fused matrix-product kernels.
#pragma once
#include <cuda.h>
#include <cudaTypedefs.h>

#include "common.cuh"

namespace rptc {

// fp16 [rows][cols] with `ld` elements between rows, in boxes of `box_cols` columns (64: 128-byte swizzle, 32: 64-byte) x
// `box_rows` rows.                                                                                     gemm_tcgen05.cu
int encode_map(CUtensorMap &map, const void *base, int64_t cols, int64_t rows, int64_t ld, int box_rows, int box_cols = 64);

#ifdef __CUDACC__
__device__ __forceinline__ void tma_load_2d(uint32_t dst, const CUtensorMap *map, int x, int y, uint32_t bar) {
    asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(dst),
                 "l"(map), "r"(x), "r"(y), "r"(bar)
                 : "memory");
}
// Tile of shared memory -> global through the tensor map (clipped at the tensor's bounds), tracked by the thread's bulk group.
__device__ __forceinline__ void tma_store_2d(const CUtensorMap *map, int x, int y, uint32_t src) {
    asm volatile("cp.async.bulk.tensor.2d.global.shared::cta.bulk_group [%0, {%1, %2}], [%3];" ::"l"(map), "r"(x), "r"(y), "r"(src) : "memory");
}
__device__ __forceinline__ void fence_proxy_async_smem() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_commit(uint32_t bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}
// D[tmem] (+)= A[smem desc] * B[smem desc]^T, kind::f16, cta_group::1
__device__ __forceinline__ void tc_mma_f16(uint32_t tmem_d, uint64_t a_desc, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
        ::"r"(tmem_d), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate)
        : "memory");
}
// The same with A in tensor memory: row i in lane i, two fp16 values per 32-bit column, K = 16 in eight columns.
__device__ __forceinline__ void tc_mma_f16_ta(uint32_t tmem_d, uint32_t tmem_a, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
        ::"r"(tmem_d), "r"(tmem_a), "l"(b_desc), "r"(idesc), "r"(accumulate)
        : "memory");
}
// K-major operand tile, 128-byte swizzle, 8-row groups 1024 bytes apart; `addr` + 32 bytes per K = 16 step.
__device__ __forceinline__ uint64_t umma_desc_sw128(uint32_t addr) {
    return (uint64_t)((addr >> 4) & 0x3FFFu) | ((uint64_t)1 << 16) | ((uint64_t)(1024 >> 4) << 32) | ((uint64_t)1 << 46) |
           ((uint64_t)2 << 61);
}
// fp32 accumulate, fp16 A and B, both K-major, M = 128
__host__ __device__ constexpr uint32_t instr_desc(int n_rows) {
    return (1u << 4) | ((uint32_t)(n_rows >> 3) << 17) | ((uint32_t)(128 >> 4) << 24);
}
// 16 registers -> 16 columns of tensor memory, one lane per thread (a warp reaches lanes 32 * (warp % 4) ... only); complete behind
// tmem_store_wait.
__device__ __forceinline__ void tmem_store16_begin(uint32_t taddr, const uint32_t (&v)[16]) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};" ::"r"(taddr), "r"(v[0]),
                 "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]), "r"(v[8]), "r"(v[9]), "r"(v[10]), "r"(v[11]),
                 "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15])
                 : "memory");
}
__device__ __forceinline__ void tmem_store_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
// 8 columns of tensor memory -> 8 registers.  `v` holds the values after tmem_load_wait, which names the registers so that no use of them
// moves in front of it.
__device__ __forceinline__ void tmem_load8_begin(uint32_t taddr, uint32_t (&v)[8]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                 : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7])
                 : "r"(taddr));
}
__device__ __forceinline__ void tmem_load_wait(uint32_t (&v)[8], uint32_t (&w)[8]) {
    asm volatile("tcgen05.wait::ld.sync.aligned;"
                 : "+r"(v[0]), "+r"(v[1]), "+r"(v[2]), "+r"(v[3]), "+r"(v[4]), "+r"(v[5]), "+r"(v[6]), "+r"(v[7]), "+r"(w[0]), "+r"(w[1]),
                   "+r"(w[2]), "+r"(w[3]), "+r"(w[4]), "+r"(w[5]), "+r"(w[6]), "+r"(w[7])
                 :
                 : "memory");
}
__device__ __forceinline__ void tma_prefetch_map(const void *map) {
    asm volatile("prefetch.tensormap [%0];" ::"l"(map) : "memory");
}

// True in one lane of a warp, all of whose lanes have to come here.  Lanes of a warp that waits as a whole may run out of tries one by one (the
// barrier completes at the others' last), so a lane whose wait gave up goes on with its warp to the end of the loop: it waits no more,
// and issues nothing if it is the elected one.  Elected in front of the wait: behind it 1 % more time (4096 x 11008 HASH, 400 tokens in
// tiles of 128 x 128 69.4 us against 68.3).
__device__ __forceinline__ bool elect_one() {
    uint32_t one;
    asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xFFFFFFFF;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(one));
    return one != 0;
}

// Position in a ring of `n` stages without a division per step.
struct RingPos {
    int s;
    uint32_t phase;
    __device__ __forceinline__ void advance(int n) {
        if (++s == n) s = 0, phase ^= 1u;
    }
    __device__ __forceinline__ void advance_by(int k, int n) {
        for (int i = 0; i < k; ++i) advance(n);
    }
};
#endif  // __CUDACC__

}  // namespace rptc
