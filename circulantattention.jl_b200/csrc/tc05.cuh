// tcgen05 (5th-generation tensor core) and tensor-memory helpers for sm_100a.  Single-CTA forms only.
#pragma once
#include "tma.cuh"

namespace ca {

// One thread of the warp (the same every time): MMAs and commits are issued by one thread.
__device__ __forceinline__ bool elect_one() {
    uint32_t p;
    asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(p));
    return p != 0;
}

// Whole-warp allocation of tensor-memory columns (a power of two >= 32); the address lands in shared memory.
template <int COLS>
__device__ __forceinline__ void tmem_alloc(uint32_t* dst) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(dst)), "n"(COLS) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
}
template <int COLS>
__device__ __forceinline__ void tmem_free(uint32_t t) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(t), "n"(COLS));
}
// Arrives on the barrier when every MMA that this thread has issued is complete.
__device__ __forceinline__ void tc_commit(uint64_t* bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tmem_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void tmem_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

// D (tensor memory, FP32) = or += A (tensor memory, 16 bf16 per lane in 8 columns) * B (shared memory).
__device__ __forceinline__ void mma_ts(uint32_t d, uint32_t a, uint64_t b, uint32_t idesc, bool accumulate) {
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %4, 0;\n\t"
                 "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
                 ::"r"(d), "r"(a), "l"(b), "r"(idesc), "r"((uint32_t)accumulate) : "memory");
}

// 8 consecutive columns of this warp's 32 lanes.
__device__ __forceinline__ void tmem_ld8(uint32_t t, uint32_t* v) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                 : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]) : "r"(t) : "memory");
}
__device__ __forceinline__ void tmem_st8(uint32_t t, const uint32_t* v) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};"
                 ::"r"(t), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]) : "memory");
}

// Shared-memory operand without swizzle: 8 x 16-byte core matrices (128 contiguous bytes).  K-major operands: `lbo` steps
// along K, `sbo` along the rows; MN-major operands: `lbo` steps along K, `sbo` along M/N.
__device__ __forceinline__ uint64_t smem_operand(uint32_t addr, uint32_t lbo, uint32_t sbo) {
    return (uint64_t)((addr >> 4) & 0x3fff) | ((uint64_t)((lbo >> 4) & 0x3fff) << 16) | ((uint64_t)((sbo >> 4) & 0x3fff) << 32) | (1ull << 46);
}
// bf16 x bf16 -> FP32, M = 128, A K-major, B K-major or (mn_major) MN-major.
__host__ __device__ constexpr uint32_t mma_shape(int N, bool mn_major) {
    return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)mn_major << 16) | ((uint32_t)(N >> 3) << 17) | (8u << 24);
}

// Untiled bulk copy global -> shared (both 16-byte aligned, a multiple of 16 bytes), completing on an mbarrier.
__device__ __forceinline__ void bulk_load(uint32_t dst, const void* src, uint32_t bytes, uint64_t* bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                 ::"r"(dst), "l"(src), "r"(bytes), "r"(smem_u32(bar)) : "memory");
}

// ---------------------------------------------------------------- packed FP32 pairs and the exact split into bf16
__device__ __forceinline__ uint64_t pair(float a, float b) {
    uint64_t r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ float2 unpair(uint64_t v) {
    float2 r;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
    return r;
}
__device__ __forceinline__ uint64_t fma_pair(uint64_t a, uint64_t b, uint64_t c) {
    uint64_t r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
__device__ __forceinline__ uint64_t add_pair(uint64_t a, uint64_t b) {
    uint64_t r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ uint64_t mul_pair(uint64_t a, uint64_t b) {
    uint64_t r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ uint32_t to_bf16x2(float lo, float hi) {
    uint32_t r;
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(hi), "f"(lo));
    return r;
}
// x = hi + mid + lo to the last bit of a 24-bit significand: each step rounds to the nearest bf16 (8 bits) and the
// remainder is exact in FP32.
__device__ __forceinline__ void split3(uint64_t x, uint32_t& hi, uint32_t& mid, uint32_t& lo) {
    const uint64_t minus1 = pair(-1.f, -1.f);
    float2 f = unpair(x);
    hi = to_bf16x2(f.x, f.y);
    x = fma_pair(pair(__uint_as_float(hi << 16), __uint_as_float(hi & 0xffff0000u)), minus1, x);
    f = unpair(x);
    mid = to_bf16x2(f.x, f.y);
    x = fma_pair(pair(__uint_as_float(mid << 16), __uint_as_float(mid & 0xffff0000u)), minus1, x);
    f = unpair(x);
    lo = to_bf16x2(f.x, f.y);
}

}  // namespace ca
