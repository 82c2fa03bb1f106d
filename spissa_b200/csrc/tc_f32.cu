// 32-bit product C[M,N] (+)= A[M,K] · W[N,K]ᵀ (float32 operands and result; crates/spissa-runtime/src/ops.rs:62-105) on the
// 5th-generation tensor cores, for more rows than the weight-streaming FFMA kernel takes.
//
// The FFMA tile kernel of generic_kernels.cu is bound by shared memory (0.21 of the FFMA rate, 16 TFLOP/s), and the FFMA rate
// itself (74 TFLOP/s) is a twentieth of the bfloat16 rate. A float32 has 24 significant bits, a bfloat16 8 and the same
// exponents, so x = x1 + x2 + x3 exactly, each part the leading 8 bits of what the parts before leave (cut off, not rounded:
// the differences are exact). Of the nine products of parts the six largest are computed, a1w1, a1w2, a2w1, a1w3, a2w2,
// a3w1; the three left out have the product's own sign and are together below 2^-21 of |a||w| (|a2| < 2^-7 |a|, |a3| <
// 2^-15 |a|) and 2^-24.5 of it on average. Products of 8-bit parts are exact; the tensor core adds them into a float32
// accumulator and truncates, so an accumulator holds 64 terms of K only: then it is added to a float32 sum in registers,
// rounded to nearest. Both losses are toward zero, so they add up where all terms have one sign: 1.2e-7 of the result, for
// any K. Even so the result is nearer to 64 bits than a float32 sum in order (relative error, this / in order, operands of one
// sign: K = 128 1.27e-7 / 1.64e-7, 2,048 1.28e-7 / 6.6e-7; of both signs 1.28e-7 / 2.0e-7 and 1.4e-7 / 8.1e-7;
// tests/test_f32_path_gpu.py holds it to that). Parts below 2^-126 have fewer bits: a term loses up to 2^-133 times its other
// factor, which is beyond the 24th bit of values from 2^-109 on.
// A value that is not finite has no such parts: a CTA that meets one computes its tile again with plain FFMA.
//
//   warps 0-15  split, block of 64 of K by block, 128 x 64 of W and tokens x 64 of A (fetched a block ahead into registers, 32
//               bytes a load) into three tiles each in the swizzled layout of the instruction's operands;
//   warps 16-19 add the finished accumulator of the block before (two in tensor memory, in turn) to the sums, which stand behind
//               them in tensor memory: 128 rows of W x tokens;
//   warp 20     issues tcgen05.mma: M 128 rows of W, N tokens, K 16, small products first.
// What bounds it is the path to shared memory: of a block's 1.65 us at 128 tokens 1.45 are its 128 bytes a cycle (split
// tiles in 768 cycles, the loads 512, the instructions' operands 1,536). 500 tokens x 16,384 x 2,048: 239 us = 140 TFLOP/s
// (1,640 us on FFMA tiles; 345 with 16-byte loads and all warps in step; 262 with the sums in the splitting warps' registers,
// which read every accumulator between two blocks; 219 by pairs of CTAs, M 256 and N 256 in two halves, but its other products
// 62 / 62 / 204 for 60 / 38 / 114 here: an accumulator's way through both CTAs' barriers takes longer than a block).
// Adding an accumulator only every 256 terms of K is 3 % faster and ten times as far from the exact result: the small products
// are cut off against a large sum.
// K is cut over the CTAs of a cluster where the tiles alone leave SMs idle; the pieces are added in order through
// distributed shared memory. Every wait is bounded and records a code in ``status``.
#include "tcgen05.cuh"

SP_API const char* sp_tc_f32_last_error() { return sp_error_text; }
SP_DEFINE_RANGE_API(tc_f32)

namespace {

constexpr int BW = 128;                     // rows of W per CTA
constexpr int BK = 64;                      // K per stage: 64 bf16 of a part = 128 bytes = one swizzle span
constexpr int MAX_NT = 128;                 // tokens per CTA
constexpr int STAGES = 2;                   // of split operands, and accumulators
constexpr int WARPS = 16;                   // that split operands; four that add accumulators to the sums and one that issues the products
constexpr int ISSUER = WARPS + 4;
constexpr int THREADS = 32 * (ISSUER + 1);
constexpr int PART_W = BW * BK * 2;
constexpr int MAX_PIECES = 8;

struct Args {
    const float* A;
    const float* W;
    float* C;
    int* status;
    int M, N, K, lda, ldw, ldc, accumulate, nt, pieces;
};

// Two float32 side by side
__device__ __forceinline__ uint64_t pair(uint32_t a, uint32_t b) {
    uint64_t v;
    asm("mov.b64 %0, {%1, %2};" : "=l"(v) : "r"(a), "r"(b));
    return v;
}
__device__ __forceinline__ void unpair(uint64_t v, uint32_t& a, uint32_t& b) { asm("mov.b64 {%0, %1}, %2;" : "=r"(a), "=r"(b) : "l"(v)); }
__device__ __forceinline__ uint64_t sub2(uint64_t a, uint64_t b) {
    uint64_t v;
    asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(v) : "l"(a), "l"(b));
    return v;
}
__device__ __forceinline__ uint64_t add2(uint64_t a, uint64_t b) {
    uint64_t v;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(v) : "l"(a), "l"(b));
    return v;
}
__device__ __forceinline__ uint64_t fma2(uint64_t a, uint64_t b, uint64_t c) {
    uint64_t v;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(v) : "l"(a), "l"(b), "l"(c));
    return v;
}

// Eight values of a row as three rows of eight bfloat16: the leading 8 bits, the next 8, the last 8 (all exact). ``check``
// stays zero while every value is finite: what is left of an infinity or NaN is NaN.
__device__ __forceinline__ void split8(const uint4& lo, const uint4& hi, uint4 (&part)[3], uint64_t& check) {
    uint32_t v[8] = {lo.x, lo.y, lo.z, lo.w, hi.x, hi.y, hi.z, hi.w};
#pragma unroll
    for (int p = 0; p < 3; ++p) {
        uint32_t w[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) w[e] = __byte_perm(v[2 * e], v[2 * e + 1], 0x7632);
        part[p] = make_uint4(w[0], w[1], w[2], w[3]);
        if (p == 2) break;
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const uint64_t left = sub2(pair(v[2 * e], v[2 * e + 1]), pair(v[2 * e] & 0xffff0000u, v[2 * e + 1] & 0xffff0000u));
            if (p == 0) check = fma2(left, 0ull, check);
            unpair(left, v[2 * e], v[2 * e + 1]);
        }
    }
}

__global__ void __launch_bounds__(THREADS, 1)
tc_f32_kernel(const Args a) {
    extern __shared__ uint8_t smem_raw[];
    __shared__ __align__(8) uint64_t bar_full[STAGES], bar_empty[STAGES], bar_done[2], bar_free[2];
    __shared__ uint32_t tmem_slot;
    __shared__ int odd, failed;

    const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int tile = blockIdx.x / a.pieces, piece = blockIdx.x % a.pieces;     // the cluster's rank is the piece of K
    const int row0 = tile * BW, tok0 = blockIdx.y * a.nt;
    const int count = min(a.nt, a.M - tok0);
    const int num_kb = (a.K + BK - 1) / BK, per = (num_kb + a.pieces - 1) / a.pieces;
    const int kb0 = piece * per, blocks = min(num_kb, kb0 + per) - kb0;       // the host makes every piece non-empty
    const uint32_t part_a = (uint32_t)a.nt * (BK * 2), stage_bytes = 3 * (PART_W + part_a);

    if (threadIdx.x == 0) {
        for (int s = 0; s < STAGES; ++s) {
            mbar_init(smem_u32(&bar_full[s]), WARPS);
            mbar_init(smem_u32(&bar_empty[s]), 1);
        }
        for (int b = 0; b < 2; ++b) {
            mbar_init(smem_u32(&bar_done[b]), 1);
            mbar_init(smem_u32(&bar_free[b]), 4);
        }
        odd = 0;
        failed = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    __syncwarp();
    if (warp == ISSUER) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_slot)), "r"(4u * MAX_NT) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = tmem_slot;
    const int row = (warp & 3) * 32 + lane;                       // a thread's row of W
    const uint32_t lanes = tmem_base + ((uint32_t)((warp & 3) * 32) << 16);
    // tensor memory: two accumulators, which take the blocks of K in turn, and the sums behind them
    if (warp < WARPS) {
        // eight lanes take the 64 values of a row, a warp four rows at a time; the 16-byte stores of eight lanes fall on the
        // eight swizzled places of one row: no bank conflicts
        const int c = lane & 7, r0 = warp * 4 + (lane >> 3);      // 64 rows between a thread's two tasks
        uint4 wl[2], wh[2], al[2], ah[2];
        // the loads stay where they stand (volatile): a block of K ahead of their use, which the compiler would else undo
        const float* const w_at = a.W + (size_t)(row0 + r0) * a.ldw + c * 8;
        const float* const a_at = a.A + (size_t)(tok0 + r0) * a.lda + c * 8;
        auto fetch = [&](const float* at, int ld, bool ok, int t, int kb, uint4& lo, uint4& hi) {
            const float* p = at + (size_t)(64 * t) * ld + (size_t)kb * BK;
            asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %9, 0;\n\t"
                         "mov.b32 %0, 0;\n\tmov.b32 %1, 0;\n\tmov.b32 %2, 0;\n\tmov.b32 %3, 0;\n\t"
                         "mov.b32 %4, 0;\n\tmov.b32 %5, 0;\n\tmov.b32 %6, 0;\n\tmov.b32 %7, 0;\n\t"
                         "@p ld.global.nc.L2::256B.v8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];\n\t}"
                         : "=&r"(lo.x), "=&r"(lo.y), "=&r"(lo.z), "=&r"(lo.w), "=&r"(hi.x), "=&r"(hi.y), "=&r"(hi.z), "=&r"(hi.w)
                         : "l"(p), "r"((int)(ok && kb * BK + c * 8 < a.K)));           // K is a multiple of 8
        };
        bool w_ok[2], a_ok[2];
#pragma unroll
        for (int t = 0; t < 2; ++t) {
            w_ok[t] = row0 + r0 + 64 * t < a.N;
            a_ok[t] = r0 + 64 * t < count;
            fetch(w_at, a.ldw, w_ok[t], t, kb0, wl[t], wh[t]);
            fetch(a_at, a.lda, a_ok[t], t, kb0, al[t], ah[t]);
        }
        uint64_t check = 0;
        for (int i = 0; i < blocks; ++i) {
            const int s = i & 1;
            if (!__all_sync(0xffffffffu, mbar_wait_flag(smem_u32(&bar_empty[s]), (((uint32_t)i >> 1) & 1u) ^ 1u, a.status, 143, &failed))) break;
            const uint32_t dst = smem_base + (uint32_t)s * stage_bytes;
            const bool more = i + 1 < blocks;
#pragma unroll
            for (int t = 0; t < 2; ++t) {
                const int r = r0 + 64 * t;
                const uint32_t at = (uint32_t)(r * 128 + ((c ^ (r & 7)) * 16));
                uint4 part[3];
                split8(wl[t], wh[t], part, check);
                if (more) fetch(w_at, a.ldw, w_ok[t], t, kb0 + i + 1, wl[t], wh[t]);
#pragma unroll
                for (int p = 0; p < 3; ++p)
                    asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(dst + p * PART_W + at), "r"(part[p].x), "r"(part[p].y), "r"(part[p].z), "r"(part[p].w) : "memory");
                if (r < a.nt) {
                    split8(al[t], ah[t], part, check);
                    if (more) fetch(a_at, a.lda, a_ok[t], t, kb0 + i + 1, al[t], ah[t]);
#pragma unroll
                    for (int p = 0; p < 3; ++p)
                        asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(dst + 3 * PART_W + p * part_a + at), "r"(part[p].x), "r"(part[p].y), "r"(part[p].z), "r"(part[p].w) : "memory");
                }
            }
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            __syncwarp();
            if (lane == 0) mbar_arrive(smem_u32(&bar_full[s]));
        }
        uint32_t c_lo, c_hi;
        unpair(check, c_lo, c_hi);
        if ((c_lo | c_hi) & 0x7fffffffu) odd = 1;
    } else if (warp < ISSUER) {
        // an accumulator's 32-bit values into the sums, rounded to nearest
        for (int i = 0; i < blocks; ++i) {
            const int b = i & 1;
            if (!__all_sync(0xffffffffu, mbar_wait_flag(smem_u32(&bar_done[b]), ((uint32_t)i >> 1) & 1u, a.status, 142, &failed))) break;
            tc_fence_after();
            const uint32_t from = lanes + (uint32_t)(b * MAX_NT), to = lanes + (uint32_t)(2 * MAX_NT);
            for (int c = 0; c < a.nt; c += 16) {
                uint32_t r[16], t[16];
                tc_ld_32x8(from + c, r);
                tc_ld_32x8(from + c + 8, r + 8);
                if (i > 0) {
                    tc_ld_32x8(to + c, t);
                    tc_ld_32x8(to + c + 8, t + 8);
                }
                tc_ld_wait();
                if (i > 0) {
#pragma unroll
                    for (int j = 0; j < 16; j += 2) unpair(add2(pair(t[j], t[j + 1]), pair(r[j], r[j + 1])), r[j], r[j + 1]);
                }
                tc_st_32x16(to + c, r);
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(smem_u32(&bar_free[b]));
            tc_st_wait();
        }
    } else if (lane == 0) {
        const uint32_t idesc = umma_idesc_bf16(BW, a.nt);
        for (int i = 0; i < blocks; ++i) {
            const int s = i & 1, b = i & 1;
            if (!mbar_wait_flag(smem_u32(&bar_free[b]), (((uint32_t)i >> 1) & 1u) ^ 1u, a.status, 144, &failed)) break;
            if (!mbar_wait_flag(smem_u32(&bar_full[s]), ((uint32_t)i >> 1) & 1u, a.status, 141, &failed)) break;
            tc_fence_after();
            const uint32_t src = smem_base + (uint32_t)s * stage_bytes;
            // (part of W, part of A), the smallest products first
            constexpr int PW[6] = {2, 1, 0, 1, 0, 0}, PA[6] = {0, 1, 2, 0, 1, 0};
#pragma unroll
            for (int p = 0; p < 6; ++p) {
                const uint64_t dw = umma_desc_sw128(src + PW[p] * PART_W);
                const uint64_t da = umma_desc_sw128(src + 3 * PART_W + PA[p] * part_a);
#pragma unroll
                for (int k = 0; k < BK / 16; ++k)
                    tc_mma_bf16(tmem_base + (uint32_t)(b * MAX_NT), dw + 2 * k, da + 2 * k, idesc, (p | k) != 0 ? 1u : 0u);
            }
            tc_commit(smem_u32(&bar_empty[s]));
            tc_commit(smem_u32(&bar_done[b]));
        }
    }
    tc_fence_before();
    __syncwarp();
    // all products are done (or a wait was given up), ``odd`` is known
    __syncthreads();
    tc_fence_after();
    if (warp < WARPS) {
        // the sums, [token][row of W], into shared memory, whose stages are free
        for (int c = (warp >> 2) * 8; c < a.nt; c += 32) {
            uint32_t r[8];
            tc_ld_32x8(lanes + (uint32_t)(2 * MAX_NT + c), r);
            tc_ld_wait();
            if (odd) {
                // infinities or NaN among the operands: this piece again, term by term
                const int k1 = min(a.K, (kb0 + blocks) * BK);
                const float* w = a.W + (size_t)min(row0 + row, a.N - 1) * a.ldw;
                float again[8] = {};
                for (int k = kb0 * BK; k < k1; ++k)
#pragma unroll
                    for (int j = 0; j < 8; ++j) again[j] = fmaf(__ldg(w + k), __ldg(a.A + (size_t)(tok0 + min(c + j, count - 1)) * a.lda + k), again[j]);
#pragma unroll
                for (int j = 0; j < 8; ++j) r[j] = __float_as_uint(again[j]);
            }
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                if (c + j < count) asm volatile("st.shared.b32 [%0], %1;" ::"r"(smem_base + (uint32_t)(((c + j) * BW + row) * 4)), "r"(r[j]) : "memory");
            }
        }
    }
    if (a.pieces > 1) asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
    else __syncthreads();
    if (warp < WARPS && !failed) {
        // a warp owns a token, a lane four neighbouring columns; the pieces in their order
        const int share = (count + a.pieces - 1) / a.pieces, j1 = min(count, (piece + 1) * share);
        const int col = row0 + 4 * lane, left = a.N - col;
        const bool whole = left >= 4 && (a.ldc & 3) == 0 && ((uintptr_t)a.C & 15) == 0;
        uint32_t peer[MAX_PIECES];
#pragma unroll
        for (int sp = 0; sp < MAX_PIECES; ++sp)
            asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(peer[sp]) : "r"(smem_base), "r"(sp < a.pieces ? sp : 0));
        for (int j = piece * share + warp; j < j1; j += WARPS) {
            float* out = a.C + (size_t)(tok0 + j) * a.ldc + col;
            float4 old = make_float4(0.f, 0.f, 0.f, 0.f), p[MAX_PIECES];
            if (a.accumulate && whole) old = *(const float4*)out;
#pragma unroll
            for (int sp = 0; sp < MAX_PIECES; ++sp)
                if (sp < a.pieces)
                    asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(p[sp].x), "=f"(p[sp].y), "=f"(p[sp].z), "=f"(p[sp].w) : "r"(peer[sp] + (uint32_t)((j * BW + 4 * lane) * 4)));
            float v[4] = {p[0].x, p[0].y, p[0].z, p[0].w};
#pragma unroll
            for (int sp = 1; sp < MAX_PIECES; ++sp)
                if (sp < a.pieces) { v[0] += p[sp].x; v[1] += p[sp].y; v[2] += p[sp].z; v[3] += p[sp].w; }
            if (whole) {
                *(float4*)out = make_float4(old.x + v[0], old.y + v[1], old.z + v[2], old.w + v[3]);
            } else {
                for (int e = 0; e < 4 && e < left; ++e) out[e] = a.accumulate ? out[e] + v[e] : v[e];
            }
        }
    }
    __syncwarp();
    // nobody leaves (and frees its shared memory) before every CTA has read what it needs
    tc_fence_before();
    if (a.pieces > 1) asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
    else __syncthreads();
    if (warp == ISSUER) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(4u * MAX_NT) : "memory");
    }
}

// What a CTA asks for, more than it needs at fewer tokens: it takes all of an SM's tensor memory, so nothing that takes some
// may share the SM with it (clusters that wait for one another's tensor memory on two SMs would wait for good).
constexpr int SMEM = 224 * 1024;
static_assert(2 * 3 * (PART_W + MAX_NT * BK * 2) + 1024 <= SMEM && MAX_NT * BW * 4 + 1024 <= SMEM, "two stages, or the sums");

// Tokens in equal tiles of at most 128; as many pieces of K (a power of two) as shorten the longest SM's work: a block of K
// takes about 1.3 us and 2.7 ns a token, a CTA 6 us around them; clusters leave SMs over.
void plan(int M, int N, int K, int* nt, int* token_tiles, int* pieces) {
    const int num_kb = (K + BK - 1) / BK, sms = sp_sm_count() > 0 ? sp_sm_count() : 148;
    const int tt = (M + MAX_NT - 1) / MAX_NT;
    *nt = ((M + tt - 1) / tt + 15) / 16 * 16;
    *token_tiles = (M + *nt - 1) / *nt;
    double best = 0;
    *pieces = 1;
    for (int p = 1; p <= MAX_PIECES && p <= num_kb; p *= 2) {
        const int mine = (num_kb + p - 1) / p;
        if ((p - 1) * mine >= num_kb) continue;                    // no empty piece
        const int room = p <= 2 ? sms : p == 4 ? sms * 132 / 148 : sms * 112 / 148;
        const int ctas = (N + BW - 1) / BW * *token_tiles * p;
        const double t = (double)((ctas + room - 1) / room) * (mine * (1.3 + 0.0027 * *nt) + 6.0 + (p > 1 ? 1.5 : 0.0));
        if (p == 1 || t < best) { best = t; *pieces = p; }
    }
}

}  // namespace

// Whether this kernel takes the product (0) or the FFMA kernels have to (1, the reason as the last error).
SP_API int sp_tc_f32_supported(const void* A, const void* W, int M, int N, int K, int lda, int ldw) {
    if (M <= 0 || N <= 0 || K <= 0) SP_FAIL("tc_f32: empty product");
    if ((K | lda | ldw) & 7) SP_FAIL("tc_f32: K and the leading dimensions must be multiples of 8 (32-byte loads)");
    if (((uintptr_t)A | (uintptr_t)W) & 31) SP_FAIL("tc_f32: operands must start on a 32-byte boundary");
    if ((M + MAX_NT - 1) / MAX_NT > 65535) SP_FAIL("tc_f32: M=%d is beyond this kernel's grid", M);
    return 0;
}

// C [M, N] = A [M, K] · W [N, K]ᵀ, or C += with ``accumulate``; all float32.
SP_API int sp_tc_f32(const void* A, const void* W, void* C, int M, int N, int K, int lda, int ldw, int ldc, int accumulate,
                     int* status, cudaStream_t stream) {
    if (M <= 0 || N <= 0) return 0;
    if (sp_tc_f32_supported(A, W, M, N, K, lda, ldw)) return 1;
    static SpPerDevice configured;
    if (!configured.done()) {
        cudaError_t e = cudaFuncSetAttribute(tc_f32_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM);
        if (e != cudaSuccess) SP_FAIL("tc_f32: cannot reserve %d bytes of shared memory: %s", SMEM, cudaGetErrorString(e));
        configured.mark();
    }
    Args args{(const float*)A, (const float*)W, (float*)C, status, M, N, K, lda, ldw, ldc, accumulate, 0, 0};
    int token_tiles = 1;
    plan(M, N, K, &args.nt, &token_tiles, &args.pieces);
    SP_CHECK_CALL("tc_f32", sp_launch_cluster(tc_f32_kernel, dim3((N + BW - 1) / BW * args.pieces, token_tiles), dim3(THREADS), (size_t)SMEM, stream,
                                              args.pieces, args));
    return 0;
}
