// Inline PTX for the Blackwell tensor-core path shared by the kernels that use it: mbarriers with bounded
// waits, TMA tile loads (never with cluster multicast), tcgen05 fences / commit / mma / ld / st, the
// shared-memory matrix descriptors and the kind::f16 instruction descriptor.
#pragma once
#include "async_copy.cuh"
#include <cuda.h>

namespace {

__device__ __forceinline__ void tma_load_2d(uint32_t dst, const CUtensorMap* map, int c0, int c1, uint32_t bar) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
        ::"r"(dst), "l"(map), "r"(c0), "r"(c1), "r"(bar) : "memory");
}

__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

__device__ __forceinline__ void tc_commit(uint32_t bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}

__device__ __forceinline__ void tc_mma_bf16(uint32_t tmem_d, uint64_t desc_a, uint64_t desc_b, uint32_t idesc,
                                            uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, {%5, %5, %5, %5}, p;\n\t}"
        ::"r"(tmem_d), "l"(desc_a), "l"(desc_b), "r"(idesc), "r"(accumulate), "r"(0u) : "memory");
}

// 32 lanes x 32 consecutive 32-bit columns: thread i of the warp gets lane (base lane + i)
__device__ __forceinline__ void tc_ld_32x32(uint32_t taddr, uint32_t* r) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
        "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
          "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
          "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
        : "r"(taddr) : "memory");
}
// 32 lanes x 8 consecutive columns
__device__ __forceinline__ void tc_ld_32x8(uint32_t taddr, uint32_t* r) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
                 : "r"(taddr) : "memory");
}
__device__ __forceinline__ void tc_ld_wait() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }

// Shared-memory matrix descriptor of a K-major tile with 128-byte swizzle: rows of 128 bytes,
// groups of 8 rows 1024 bytes apart (SBO), LBO 1 (unused by swizzled K-major), version 1.
__device__ __forceinline__ uint64_t umma_desc_sw128(uint32_t smem_addr) {
    uint64_t d = 0;
    d |= (uint64_t)((smem_addr & 0x3FFFF) >> 4);
    d |= (uint64_t)1 << 16;
    d |= (uint64_t)(1024 >> 4) << 32;
    d |= (uint64_t)1 << 46;
    d |= (uint64_t)2 << 61;
    return d;
}

// kind::f16 instruction descriptor: D float32, A and B bfloat16, both K-major, M x N
__host__ __device__ constexpr uint32_t umma_idesc_bf16(int m, int n) {
    return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(m >> 4) << 24);
}


// A from tensor memory (K-major, two bfloat16 per 32-bit column), B from shared memory
__device__ __forceinline__ void tc_mma_bf16_ts(uint32_t tmem_d, uint32_t tmem_a, uint64_t desc_b, uint32_t idesc,
                                               uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, {%5, %5, %5, %5}, p;\n\t}"
        ::"r"(tmem_d), "r"(tmem_a), "l"(desc_b), "r"(idesc), "r"(accumulate), "r"(0u) : "memory");
}

// 32 lanes x 16 consecutive 32-bit columns, registers to tensor memory
__device__ __forceinline__ void tc_st_32x16(uint32_t taddr, const uint32_t* r) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], "
        "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};"
        ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]),
          "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]) : "memory");
}
__device__ __forceinline__ void tc_st_32x32(uint32_t taddr, const uint32_t* r) {
    tc_st_32x16(taddr, r);
    tc_st_32x16(taddr + 16, r + 16);
}
__device__ __forceinline__ void tc_st_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

// Shared-memory descriptor of an MN-major tile with 128-byte swizzle (rows of 64 bfloat16 along M or N,
// one row per K index): 8 K rows form a 1024-byte group (SBO); ``lbo_bytes`` leads to the next 64 of M/N.
__device__ __forceinline__ uint64_t umma_desc_mn_sw128(uint32_t smem_addr, uint32_t lbo_bytes) {
    uint64_t d = 0;
    d |= (uint64_t)((smem_addr & 0x3FFFF) >> 4);
    d |= (uint64_t)((lbo_bytes >> 4) & 0x3FFF) << 16;
    d |= (uint64_t)(1024 >> 4) << 32;
    d |= (uint64_t)1 << 46;
    d |= (uint64_t)2 << 61;
    return d;
}

// kind::f16 instruction descriptor with B MN-major (A K-major): D float32, A and B bfloat16
__host__ __device__ constexpr uint32_t umma_idesc_bf16_bmn(int m, int n) {
    return umma_idesc_bf16(m, n) | (1u << 16);
}

// x / d for 1 <= d <= 2^100 and finite x: the remainder of a quotient by an approximate reciprocal (two units at most off)
// corrects it to within half a unit and 2^-20 of one, with a REFINED reciprocal (a step of Newton's) to within half a unit
// (P. Markstein, "Computation of elementary functions on the IBM RISC System/6000 processor", 1990). No branch, unlike
// the general quotient. Compared with that one for every gate g that comes here: x = g and d = 1 + expf(-slope·g), |slope·g| <= 60,
// the same bits for a slope of 1 as it is, for 172 slopes from 0.013 to 200 when refined (without: up to 3 g a slope differ in
// the last bit); the tanh form of gelu, |g| <= 8.6, the same bits when refined; where g is -0 the quotient is +0.
template <bool REFINED>
__device__ __forceinline__ float tc_quotient(float x, float d) {
    float r;
    asm("rcp.approx.f32 %0, %1;" : "=f"(r) : "f"(d));
    if (REFINED) r = fmaf(fmaf(-d, r, 1.0f), r, r);
    const float q = x * r;
    return fmaf(fmaf(-d, q, x), r, q);
}
// act(gate)·up of 32 pairs of an epilogue's thread (the first ``n`` exist), each times its ``scale``, in place of the gate:
// sp_gated. Gates of ordinary size (all of them, in earnest) go through without a branch on one value, so that the 32 overlap:
// tc_mid.cu, 301 tokens x 16,384 x 2,048: 27.3 us, 32.0 with the general quotient, 40 with a branch on the activation around
// each value. In tc_gemm.cu the general quotient's way for a numerator of zero, which the rows behind the last token all take,
// held up the tiles behind them: 16,384 x 2,048 on weights from HBM, 1,408 tokens 130 us, 82 here (2,048 tokens, without
// such rows, 123 and 102; of the 8B shape, 28,672 x 4,096, 6,000 tokens 1,180 and 1,098); gelu's, on the same way until it
// had this form, 200 tokens 40.9 and 21.7, 1,024 columns of 400 tokens x 8,192 34.5 and 15.7.
// Both ways give a value the same bits, so a token's result depends neither on its neighbours in the warp nor on rows that nobody
// reads (holes among the routed experts' rows hold what the memory held). Deciding for each value by its own gate in the
// second loop as well makes that loop twice as long: 2,048 tokens x 16,384 x 2,048 by pairs 100.5 -> 103 us.
template <int KIND, typename Scale>
__device__ __forceinline__ void tc_activate(uint32_t (&rg)[32], uint32_t (&ru)[32], Scale scale, int n, SpGate ga) {
    ga.kind = KIND;
    const float slope = KIND == SP_ACT_CLAMPED ? ga.slope : 1.0f;
    constexpr float edge = KIND == SP_ACT_GELU ? 8.6f : 60.0f;   // the exponent stays within 60
    float top[4] = {0.0f, 0.0f, 0.0f, 0.0f};                     // (NaN is left out: the quotient is NaN either way)
#pragma unroll
    for (int j = 0; j < 32; ++j) {
        float g = __uint_as_float(rg[j]) * scale(j);
        if (KIND == SP_ACT_CLAMPED) g = fminf(g, ga.limit);
        top[j & 3] = fmaxf(top[j & 3], j < n ? fabsf(slope * g) : 0.0f);
        rg[j] = __float_as_uint(g);
        ru[j] = __float_as_uint(__uint_as_float(ru[j]) * scale(j));
    }
    if (__all_sync(0xffffffffu, fmaxf(fmaxf(top[0], top[1]), fmaxf(top[2], top[3])) <= edge)) {
#pragma unroll
        for (int j = 0; j < 32; ++j) {
            const float g = __uint_as_float(rg[j]);
            float u = __uint_as_float(ru[j]);
            if (KIND == SP_ACT_CLAMPED) u = fminf(fmaxf(u, -ga.limit), ga.limit) + 1.0f;
            rg[j] = __float_as_uint(tc_quotient<KIND != SP_ACT_SILU>(g, 1.0f + expf(KIND == SP_ACT_GELU ? sp_gelu_exponent(g) : -slope * g)) * u * ga.mult);
        }
        return;
    }
#pragma unroll
    for (int j = 0; j < 32; ++j) rg[j] = __float_as_uint(sp_gated(__uint_as_float(rg[j]), __uint_as_float(ru[j]), ga));
}

}  // namespace
