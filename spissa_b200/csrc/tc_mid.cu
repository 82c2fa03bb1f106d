// bfloat16 product for some dozens to some hundreds of tokens on the 5th-generation tensor cores:
// C[M,N] = A[M,K] · W[N,K]ᵀ (crates/spissa-runtime/src/ops.rs:62-105 states the layout and the product).
//
// What bounds it: the bytes each SM takes in from L2 (about 115 a nanosecond). The tile kernel (tc_gemm.cu) has 128 tokens
// as the instruction's M; with a few hundred tokens that leaves a third of its rows to padding and too few tiles for 148 SMs
// (72 for the QKV product of 301 tokens of the 1B shape), each of which walks all of K alone. Here 128 rows of W are the
// instruction's M and up to 256 tokens its N, in steps of 16: no padding to speak of, W passes through once per token tile,
// and the count of CTAs comes from two divisors the host chooses together (``plan_of``): token tiles (at most 256 tokens
// each) and pieces of K, whose CTAs form a cluster.
//   warp 0     one thread fetches, per stage, 128 x 64 of W (gated: gate and up rows) and tokens x 64 of A by TMA;
//   warp 1     one thread issues tcgen05.mma (M 128, N = tokens, K 16);
//   warps 2-9  the epilogue. First the accumulator goes into shared memory as [token][128 rows of W] (a thread owns a
//              row: 32 neighbouring lanes write 32 neighbouring words). Then a warp owns a TOKEN and a lane four
//              neighbouring columns: the pieces of K are added in their order through distributed shared memory, 16 bytes
//              a load, and global memory is touched in whole lines (tc_stream.cu's thread-per-column epilogue costs a
//              microsecond per four tokens, which is what keeps that kernel to a few dozen).
// Measured back to back on weights from HBM (us, this kernel / the one that ran before), 1B shape: 301 tokens QKV 11.0 / 17.2,
// output 10.5 / 17.6, gate/up 27.3 / 59.3, down 19.1 / 27.5; 64 tokens (before: tc_stream.cu) 8.1 / 8.5, 7.3 / 8.0,
// 18.7 / 20.6, 13.1 / 13.4.
// Grouped (routed experts, sp_tc_mid_grouped): A's rows lie in runs of one expert each, in equal tiles of at most 256 rows
// (moe_place_kernel cuts them), each multiplied with that expert's rows of the stacked weights; a CTA reads its tile's entry
// of the table on the device.
// 2,048 tokens, 4 of 32 experts of 2,048 x 2,048: 353 us the whole layer, 426 on tc_gemm.cu's tiles of 128 tokens, of which a
// fifth is padding. Five waves of CTAs that are alone on their SM, about half of each its bytes. (Where each CTA found its
// tile by walking its expert's entries of the table, an expert of 65,536 tokens took twice as long as on tc_gemm.cu.)
// Every mbarrier wait is bounded and records a code in ``status``; no load uses cluster multicast.
#include "tcgen05.cuh"
#include <string.h>

SP_API const char* sp_tc_mid_last_error() { return sp_error_text; }
SP_DEFINE_RANGE_API(tc_mid)

namespace {

constexpr int BW = 128;                     // rows of W per CTA (gated: of gate and of up each)
constexpr int BK = 64;                      // 64 bf16 = 128 bytes = one swizzle span
constexpr int UMMA_K = 16;
constexpr int MAX_PIECES = 8;
constexpr int MAX_STAGES = 8;
constexpr int MAX_NT = 256;
constexpr int EPI_WARPS = 8;
constexpr int THREADS = 64 + 32 * EPI_WARPS;
constexpr int SMEM_LIMIT = 220 * 1024;      // a CTA alone on its SM
constexpr int SMEM_SHARED = 112 * 1024;     // two side by side: the next launch's CTAs move in beside this one's

enum { MODE_STORE = 0, MODE_ACCUMULATE = 1, MODE_SILU_MUL = 2, MODE_QKV_ROPE = 4 };

// What the fused epilogues need beyond C; all zero for the plain ones. The layout is the one tc_gemm.cu and tc_stream.cu
// take, so that the host packs one structure for all three.
struct EpiArgs {
    const float* row_ssq;          // [M][n_ssq] partial sums of squares of the residual rows (null: no scaling)
    int n_ssq, norm_width;         // 1/rms = 1/sqrt(sum/norm_width + eps)
    float eps;
    int w_settled;                 // W may be read before the kernel in front of this one has finished: see the loader
    __nv_bfloat16* xw;             // MODE_ACCUMULATE: [M][N] new C ⊙ next_w (null: plain accumulation)
    const __nv_bfloat16* next_w;   // [N]
    float* ssq_out;                // [M][tiles of 128 columns]
    const float2* cs;              // MODE_QKV_ROPE: [M][hd / 2] (cos, sin)
    const int* tok_page;           // [M]
    const int* positions;          // [M]
    __nv_bfloat16* q_out;          // [M][nh * hd]
    __nv_bfloat16* kpool;          // [pages][nkv][page_size][hd]
    __nv_bfloat16* vpool;
    int nh, nkv, hd, page_size;
};
static_assert(sizeof(EpiArgs) == 112, "the host packs this layout");

struct Args {
    void* C;                // [M, ldc]: float32 or bfloat16
    int* status;
    int c_dt, M, N, K, ldc, mode;
    int nt, pieces, stages; // tokens per tile (a multiple of 16), pieces of K, stages of the ring
    uint32_t tmem_cols;
    EpiArgs ep;
    SpRange rg;
    SpGate ga;
    const int* tiles;       // grouped: per token tile (expert or -1, first row of A, rows: 1 to MAX_NT)
};
constexpr int GROUP_BOX = 64;               // rows of A per box of a grouped product

__device__ __forceinline__ float4 ld_cluster4(uint32_t addr) {
    float4 v;
    asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(addr));
    return v;
}
__device__ __forceinline__ uint2 pack4(const float (&v)[4]) {
    const __nv_bfloat162 lo = __floats2bfloat162_rn(v[0], v[1]), hi = __floats2bfloat162_rn(v[2], v[3]);
    return make_uint2(*(const uint32_t*)&lo, *(const uint32_t*)&hi);
}

// The second part of the epilogue: a warp owns a token at a time (``first``, then every eighth below ``end``), a lane four
// neighbouring columns of it.
struct Share { uint32_t smem_base; int tile, tok0, first, end, lane, nt; };

template <bool GATED, int PIECES>
__device__ __forceinline__ void finish(const Args& a, const Share& sh, const float* rstd_s) {
    const EpiArgs& ep = a.ep;
    const int tile = sh.tile, tok0 = sh.tok0, j1 = sh.end, lane = sh.lane;
    const int n_out = GATED ? a.N / 2 : a.N;
    const int col = tile * BW + 4 * lane;
    const bool col_ok = col < n_out;                               // columns come in fours: N is a multiple of 8
    const bool prepares_norm = !GATED && a.mode == MODE_ACCUMULATE && ep.xw != nullptr;
    const bool rope_mode = !GATED && a.mode == MODE_QKV_ROPE;
    constexpr bool two_parts = GATED && PIECES > 1;
    // MODE_QKV_ROPE: a tile holds whole heads; dims d and d + hd/2 of a head are rotation partners, hd/8 lanes apart
    int r_head = 0, r_d = 0, r_half = 4, r_kvh = 0;
    bool r_q = false, r_k = false;
    if (rope_mode) {
        r_half = ep.hd >> 1;
        r_head = col / ep.hd;
        r_d = col - r_head * ep.hd;
        r_q = r_head < ep.nh;
        r_k = !r_q && r_head < ep.nh + ep.nkv;
        r_kvh = r_k ? r_head - ep.nh : r_head - ep.nh - ep.nkv;
    }
    float4 nw = make_float4(0.f, 0.f, 0.f, 0.f);
    if (prepares_norm && col_ok) {
        const uint2 w = __ldg((const uint2*)(ep.next_w + col));
        const float2 lo = __bfloat1622float2(*(const __nv_bfloat162*)&w.x), hi = __bfloat1622float2(*(const __nv_bfloat162*)&w.y);
        nw = make_float4(lo.x, lo.y, hi.x, hi.y);
    }
    uint32_t peer[PIECES];
#pragma unroll
    for (int sp = 0; sp < PIECES; ++sp) {
        if (PIECES == 1) peer[sp] = sh.smem_base;
        else asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(peer[sp]) : "r"(sh.smem_base), "r"(sp));
    }
    constexpr int TB = PIECES >= 8 ? 1 : 2;                        // tokens of a warp whose loads are in flight together
#pragma unroll 1
    for (int jb = sh.first; jb < j1; jb += TB * EPI_WARPS) {
        float4 ea[TB], eb[TB];                                     // the old C, or the token's angles
        int page[TB], pos[TB];
#pragma unroll
        for (int t = 0; t < TB; ++t) {
            const int j = jb + t * EPI_WARPS;
            const size_t m = (size_t)(tok0 + j);
            ea[t] = eb[t] = make_float4(0.f, 0.f, 0.f, 0.f);
            page[t] = pos[t] = 0;
            if (j >= j1 || !col_ok || GATED) continue;
            if (a.mode == MODE_ACCUMULATE) ea[t] = *(const float4*)((const float*)a.C + m * a.ldc + col);
            if (rope_mode) {
                if (r_q || r_k) {
                    const float4* src = (const float4*)(ep.cs + m * r_half + (r_d < r_half ? r_d : r_d - r_half));
                    ea[t] = sp_ld_written(src);
                    eb[t] = sp_ld_written(src + 1);
                }
                if (!r_q) {
                    page[t] = sp_ld_written(ep.tok_page + m);
                    pos[t] = sp_ld_written(ep.positions + m);
                }
            }
        }
        float4 pg[TB][PIECES], pu[TB][two_parts ? PIECES : 1];
#pragma unroll
        for (int t = 0; t < TB; ++t) {
            const int j = jb + t * EPI_WARPS;
            const uint32_t at = (uint32_t)((j * BW + 4 * lane) * 4);
#pragma unroll
            for (int sp = 0; sp < PIECES; ++sp) {
                if (j < j1) {
                    pg[t][sp] = ld_cluster4(peer[sp] + at);
                    if (two_parts) pu[t][two_parts ? sp : 0] = ld_cluster4(peer[sp] + at + (uint32_t)(sh.nt * BW * 4));
                }
            }
        }
#pragma unroll
        for (int t = 0; t < TB; ++t) {
            const int j = jb + t * EPI_WARPS;
            if (j >= j1) break;                                    // uniform in the warp
            const size_t m = (size_t)(tok0 + j);
            float v[4] = {pg[t][0].x, pg[t][0].y, pg[t][0].z, pg[t][0].w};
#pragma unroll
            for (int sp = 1; sp < PIECES; ++sp) { v[0] += pg[t][sp].x; v[1] += pg[t][sp].y; v[2] += pg[t][sp].z; v[3] += pg[t][sp].w; }
            const float rs = rstd_s[j];
            if (GATED) {
                if (two_parts) {
                    float u[4] = {pu[t][0].x, pu[t][0].y, pu[t][0].z, pu[t][0].w};
#pragma unroll
                    for (int sp = 1; sp < PIECES; ++sp) { const float4 o = pu[t][two_parts ? sp : 0]; u[0] += o.x; u[1] += o.y; u[2] += o.z; u[3] += o.w; }
#pragma unroll
                    for (int e = 0; e < 4; ++e) v[e] = sp_gated(v[e] * rs, u[e] * rs, a.ga);
                }
                if (col_ok) {
                    if (a.c_dt == SP_DT_F32) *(float4*)((float*)a.C + m * a.ldc + col) = make_float4(v[0], v[1], v[2], v[3]);
                    else *(uint2*)((__nv_bfloat16*)a.C + m * a.ldc + col) = pack4(v);
                }
                continue;
            }
            if (rope_mode) {
                float o[4];
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    v[e] *= rs;
                    o[e] = __shfl_xor_sync(0xffffffffu, v[e], ep.hd >> 3);      // the partner: hd/2 columns = hd/8 lanes away
                }
                if (!col_ok) continue;
                if (r_q || r_k) {
                    const float c[4] = {ea[t].x, ea[t].z, eb[t].x, eb[t].z}, s[4] = {ea[t].y, ea[t].w, eb[t].y, eb[t].w};
#pragma unroll
                    for (int e = 0; e < 4; ++e) v[e] = r_d < r_half ? v[e] * c[e] - o[e] * s[e] : v[e] * c[e] + o[e] * s[e];
                }
                if (r_q) {
                    *(uint2*)(ep.q_out + (m * ep.nh + r_head) * ep.hd + r_d) = pack4(v);
                } else if (sp_index_ok(page[t], a.rg.n_pages, a.rg, 401)) {      // debug build: reported, not written
                    *(uint2*)((r_k ? ep.kpool : ep.vpool) + (((size_t)page[t] * ep.nkv + r_kvh) * ep.page_size + pos[t] % ep.page_size) * ep.hd + r_d) = pack4(v);
                }
                continue;
            }
            if (a.mode == MODE_ACCUMULATE) {
                v[0] += ea[t].x; v[1] += ea[t].y; v[2] += ea[t].z; v[3] += ea[t].w;
                float sq = 0.0f;
                if (col_ok) {
                    *(float4*)((float*)a.C + m * a.ldc + col) = make_float4(v[0], v[1], v[2], v[3]);
                    if (prepares_norm) {
                        sq = v[0] * v[0] + v[1] * v[1] + v[2] * v[2] + v[3] * v[3];
                        const float x[4] = {v[0] * nw.x, v[1] * nw.y, v[2] * nw.z, v[3] * nw.w};
                        *(uint2*)(ep.xw + m * a.N + col) = pack4(x);
                    }
                }
                if (prepares_norm) {
                    sq = sp_warp_sum(sq);
                    if (lane == 0) ep.ssq_out[m * ((a.N + BW - 1) / BW) + tile] = sq;
                }
                continue;
            }
#pragma unroll
            for (int e = 0; e < 4; ++e) v[e] *= rs;
            if (col_ok) {
                if (a.c_dt == SP_DT_F32) *(float4*)((float*)a.C + m * a.ldc + col) = make_float4(v[0], v[1], v[2], v[3]);
                else *(uint2*)((__nv_bfloat16*)a.C + m * a.ldc + col) = pack4(v);
            }
        }
    }
}

// GATED: two tiles of W per CTA, gate rows and the up rows 128 further on
template <bool GATED, bool GROUPED>
__global__ void __launch_bounds__(THREADS, GATED ? 1 : 2)
tc_mid_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_a, const Args a) {
    constexpr int PARTS = GATED ? 2 : 1;
    constexpr uint32_t W_BYTES = BW * BK * 2;
    extern __shared__ uint8_t smem_raw[];
    __shared__ __align__(8) uint64_t bar_full[MAX_STAGES], bar_empty[MAX_STAGES], bar_acc;
    __shared__ uint32_t tmem_slot;
    __shared__ float rstd_s[MAX_NT];
    __shared__ int unhealthy;

    const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int tile = blockIdx.x / a.pieces, piece = blockIdx.x % a.pieces;     // the cluster's rank is the piece of K
    int tok0 = blockIdx.y * a.nt, count = min(a.nt, a.M - tok0), nt = a.nt, expert = 0;      // tokens of this tile
    if (GROUPED) {
        sp_wait_for_predecessor();
        expert = a.tiles[3 * blockIdx.y];
        if (expert < 0) return;
        tok0 = a.tiles[3 * blockIdx.y + 1];
        count = a.tiles[3 * blockIdx.y + 2];
        nt = (count + 15) & ~15;
    }
    const int num_kb = (a.K + BK - 1) / BK;
    const int per = (num_kb + a.pieces - 1) / a.pieces;
    const int kb0 = piece * per, kb1 = min(num_kb, kb0 + per);                 // the host makes every piece non-empty
    const int row0 = (GROUPED ? expert * a.N : 0) + tile * BW * PARTS;
    const int boxes = GROUPED ? (nt + GROUP_BOX - 1) / GROUP_BOX : 1;          // of A, GROUP_BOX rows each
    const uint32_t stage_bytes = PARTS * W_BYTES + (uint32_t)(GROUPED ? MAX_NT : nt) * (BK * 2);
    const uint32_t load_bytes = GROUPED ? PARTS * W_BYTES + (uint32_t)boxes * (GROUP_BOX * BK * 2) : stage_bytes;
    const int ntp = (nt + 31) & ~31;                                         // columns between the two accumulators

    if (threadIdx.x == 32) {
        asm volatile("prefetch.tensormap [%0];" ::"l"(&map_w) : "memory");
        asm volatile("prefetch.tensormap [%0];" ::"l"(&map_a) : "memory");
    }
    if (threadIdx.x == 0) {
        for (int s = 0; s < a.stages; ++s) {
            mbar_init(smem_u32(&bar_full[s]), 1);
            mbar_init(smem_u32(&bar_empty[s]), 1);
        }
        mbar_init(smem_u32(&bar_acc), 1);
        unhealthy = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    __syncwarp();
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
                     ::"r"(smem_u32(&tmem_slot)), "r"(a.tmem_cols) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = tmem_slot;
    // what touches global memory below waits for the predecessor first, but for W where the caller says that it is settled

    const EpiArgs& ep = a.ep;
    const int ew = warp - 2;                                      // epilogue warp 0..7
    const int j0 = piece * ((count + a.pieces - 1) / a.pieces);   // this CTA's share of the tile's tokens in the second part
    const int j1 = min(count, j0 + (count + a.pieces - 1) / a.pieces);
    bool healthy = false;

    if (warp == 0) {
        if (lane == 0) {
            auto load_w = [&](int kb, int s) {
                const uint32_t dst = smem_base + (uint32_t)s * stage_bytes;
                mbar_expect_tx(smem_u32(&bar_full[s]), load_bytes);
                tma_load_2d(dst, &map_w, kb * BK, row0, smem_u32(&bar_full[s]));
                if (GATED) tma_load_2d(dst + W_BYTES, &map_w, kb * BK, row0 + BW, smem_u32(&bar_full[s]));
            };
            // The ring's first tiles of W are asked for while the predecessor's epilogue runs. That is for weights which were
            // complete before the predecessor began, as in a step's layers (a kernel without a signal of its own, torch's for
            // instance, lets this one in when its CTAs have left, before their writes need be visible): the caller says so. (In a
            // step norm_prepare stands in front of the first product, launched in the ordinary way: what the stream held before, a
            // copy into a weight for instance, has ended when it begins, and no kernel of a step writes a weight.)
            // A step of 40 tokens of the 1B shape 1,184 -> 1,147 us, 64: 1,236 -> 1,174, 301: 1,600 -> 1,564; a decode step of
            // 64 sequences 960 -> 945. (With the signal at the kernels' start it was 1,255 -> 1,272 for 40 tokens.)
            const int ahead = GROUPED || !ep.w_settled ? 0 : min(a.stages, kb1 - kb0);
            for (int i = 0; i < ahead; ++i) load_w(kb0 + i, i);
            sp_wait_for_predecessor();
            int s = 0;
            uint32_t ph = 1;
            for (int kb = kb0; kb < kb1; ++kb) {
                if (kb - kb0 >= ahead) {
                    if (!mbar_wait(smem_u32(&bar_empty[s]), ph, a.status, 131)) break;
                    load_w(kb, s);
                }
                const uint32_t dst = smem_base + (uint32_t)s * stage_bytes;
                for (int b = 0; b < boxes; ++b)
                    tma_load_2d(dst + PARTS * W_BYTES + (uint32_t)b * (GROUP_BOX * BK * 2), &map_a, kb * BK, tok0 + b * GROUP_BOX, smem_u32(&bar_full[s]));
                if (++s == a.stages) { s = 0; ph ^= 1u; }
            }
        }
    } else if (warp == 1) {
        if (lane == 0) {
            const uint32_t idesc = umma_idesc_bf16(BW, nt);
            int s = 0;
            uint32_t ph = 0;
            for (int kb = kb0; kb < kb1; ++kb) {
                if (!mbar_wait(smem_u32(&bar_full[s]), ph, a.status, 132)) break;
                tc_fence_after();
                const uint32_t src = smem_base + (uint32_t)s * stage_bytes;
                const uint64_t dw = umma_desc_sw128(src);
                const uint64_t du = umma_desc_sw128(src + W_BYTES);
                const uint64_t da = umma_desc_sw128(src + PARTS * W_BYTES);
#pragma unroll
                for (int k = 0; k < BK / UMMA_K; ++k) {
                    const uint32_t acc = (kb != kb0 || k != 0) ? 1u : 0u;
                    tc_mma_bf16(tmem_base, dw + 2 * k, da + 2 * k, idesc, acc);
                    if (GATED) tc_mma_bf16(tmem_base + (uint32_t)ntp, du + 2 * k, da + 2 * k, idesc, acc);
                }
                tc_commit(smem_u32(&bar_empty[s]));
                if (++s == a.stages) { s = 0; ph ^= 1u; }
            }
            tc_commit(smem_u32(&bar_acc));                         // also after a failed wait: the epilogue must not hang
        }
    } else {
        sp_wait_for_predecessor();
        // while the products run: each token's 1/rms from the partial sums, a warp per token
        for (int jb = ew; jb < count; jb += 4 * EPI_WARPS) {
            float sum[4];
#pragma unroll
            for (int t = 0; t < 4; ++t) {
                const int j = jb + t * EPI_WARPS;
                sum[t] = 0.0f;
                if (ep.row_ssq && j < count)
                    for (int i = lane; i < ep.n_ssq; i += 32) sum[t] += sp_ld_written(ep.row_ssq + (size_t)(tok0 + j) * ep.n_ssq + i);
            }
#pragma unroll
            for (int t = 0; t < 4; ++t) {
                const int j = jb + t * EPI_WARPS;
                const float total = sp_warp_sum(sum[t]);
                if (lane == 0 && j < count)
                    rstd_s[j] = ep.row_ssq ? 1.0f / sqrtf(total / (float)ep.norm_width + ep.eps) : 1.0f;
            }
        }
        const bool ok = mbar_wait(smem_u32(&bar_acc), 0, a.status, 133);
        tc_fence_after();
        // The next kernel's CTAs may come now: what they ask for ahead then falls into this one's epilogue. (Allowed from the
        // start, they sat beside its products and crowded on the SMs that were free first.)
        sp_allow_dependents();
        // the epilogue threads act together from here on: one verdict for all of them
        if (!(ok && !(a.status && *(volatile int*)a.status != 0))) unhealthy = 1;
        asm volatile("bar.sync 1, 256;" ::: "memory");
        healthy = unhealthy == 0;
        // first part: the accumulator into shared memory (the ring's stages are free by now), [part][token][row of W];
        // a gated tile that holds all of K applies its activation on the way
        const int q = warp & 3, row = q * 32 + lane;
        const uint32_t lane_base = tmem_base + ((uint32_t)(q * 32) << 16);
        const bool act_now = GATED && a.pieces == 1;
#pragma unroll 1
        for (int c0 = (ew >> 2) * 32; c0 < count; c0 += 64) {
            uint32_t rg[32], ru[32];
            tc_ld_32x32(lane_base + (uint32_t)c0, rg);
            if (GATED) tc_ld_32x32(lane_base + (uint32_t)(ntp + c0), ru);
            tc_ld_wait();
            if (GATED && act_now) {
                // (the kind is a constant to each loop, so that the 32 values are independent of one another)
                if (a.ga.kind == SP_ACT_SILU) tc_activate<SP_ACT_SILU>(rg, ru, [&](int j) { return rstd_s[c0 + j]; }, count - c0, a.ga);
                else if (a.ga.kind == SP_ACT_CLAMPED) tc_activate<SP_ACT_CLAMPED>(rg, ru, [&](int j) { return rstd_s[c0 + j]; }, count - c0, a.ga);
                else tc_activate<SP_ACT_GELU>(rg, ru, [&](int j) { return rstd_s[c0 + j]; }, count - c0, a.ga);
            }
            const uint32_t dst = smem_base + (uint32_t)((c0 * BW + row) * 4);
#pragma unroll
            for (int j = 0; j < 32; ++j) {
                if (c0 + j < count) {
                    asm volatile("st.shared.b32 [%0], %1;" ::"r"(dst + (uint32_t)(j * BW * 4)), "r"(rg[j]) : "memory");
                    if (GATED && !act_now)
                        asm volatile("st.shared.b32 [%0], %1;" ::"r"(dst + (uint32_t)((nt + j) * BW * 4)), "r"(ru[j]) : "memory");
                }
            }
        }
    }
    __syncwarp();
    // every CTA of the cluster has left its piece in its shared memory
    if (a.pieces > 1) asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
    else __syncthreads();

    if (warp >= 2 && healthy) {
        const Share sh{smem_base, tile, tok0, j0 + ew, j1, lane, nt};
        if (GROUPED) finish<GATED, 1>(a, sh, rstd_s);
        else switch (a.pieces) {
            case 1: finish<GATED, 1>(a, sh, rstd_s); break;
            case 2: finish<GATED, 2>(a, sh, rstd_s); break;
            case 4: finish<GATED, 4>(a, sh, rstd_s); break;
            default: finish<GATED, 8>(a, sh, rstd_s); break;
        }
    }
    __syncwarp();
    // nobody leaves (and frees its shared memory) before every CTA has read what it needs
    if (a.pieces > 1) asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(a.tmem_cols) : "memory");
    }
}

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiledFn encode_fn() {
    static EncodeTiledFn fn = nullptr;
    if (!fn) {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            fn = (EncodeTiledFn)p;
    }
    return fn;
}

// A [rows, K] bfloat16 matrix with leading dimension ld, fetched in boxes of box_rows x 64
int encode_map(CUtensorMap* map, const void* ptr, int rows, int K, int ld, int box_rows) {
    EncodeTiledFn fn = encode_fn();
    if (!fn) SP_FAIL("tc_mid: the driver does not offer cuTensorMapEncodeTiled");
    cuuint64_t dims[2] = {(cuuint64_t)K, (cuuint64_t)rows};
    cuuint64_t strides[1] = {(cuuint64_t)ld * 2};
    cuuint32_t box[2] = {(cuuint32_t)BK, (cuuint32_t)box_rows};
    cuuint32_t estr[2] = {1, 1};
    CUresult r = fn(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(ptr), dims, strides, box, estr,
                    CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                    CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) SP_FAIL("tc_mid: cuTensorMapEncodeTiled failed with code %d", (int)r);
    return 0;
}

int round_up(int v, int to) { return (v + to - 1) / to * to; }

struct Plan { int token_tiles, nt, pieces, stages, smem; uint32_t tmem_cols; };

int parts_of(int mode) { return mode == MODE_SILU_MUL ? 2 : 1; }

// Fills in what follows from the divisors; false where they do not fit.
bool fill_plan(Plan& p, int parts, int M, int num_kb) {
    p.nt = round_up((M + p.token_tiles - 1) / p.token_tiles, 16);
    if (p.nt > MAX_NT || (p.token_tiles - 1) * p.nt >= M) return false;
    const int mine = (num_kb + p.pieces - 1) / p.pieces;
    if ((p.pieces - 1) * mine >= num_kb) return false;                                        // no empty piece
    const int stage = parts * BW * BK * 2 + p.nt * BK * 2;
    const int held = (p.pieces > 1 ? parts : 1) * p.nt * BW * 4;                              // the sums the epilogue exchanges
    const int limit = parts == 1 && held + 1024 <= SMEM_SHARED && 3 * stage + 1024 <= SMEM_SHARED ? SMEM_SHARED : SMEM_LIMIT;
    if (held + 1024 > limit) return false;
    p.stages = (limit - 1024) / stage;
    if (p.stages > MAX_STAGES) p.stages = MAX_STAGES;
    if (p.stages > mine) p.stages = mine;
    const int ring = p.stages * stage;
    p.smem = (ring > held ? ring : held) + 1024;
    const int cols = parts == 2 ? round_up(p.nt, 32) + p.nt : p.nt;
    p.tmem_cols = 32;
    while ((int)p.tmem_cols < round_up(cols, 32)) p.tmem_cols *= 2;
    return p.stages >= 1 && p.tmem_cols <= 512;
}

// The division of a product, by an estimate of its time in nanoseconds (``estimate``) that was fitted to 1,276 measured
// divisions of the products of the 1B and 8B layer sizes at 17 to 1,000 tokens (its choices are 1.5 % slower than the best of
// them on average, 11 % at worst). A CTA takes in its blocks of K at about 115 bytes a nanosecond, two on one SM together at 136;
// every wave adds the epilogue: 42 ns a token of the tile, 12 per token of the share, a microsecond for the exchange of
// pieces and 170 ns per piece. Clusters of 4 and 8 do not find room on every SM: 136 and 128 CTAs at a time.
Plan plan_of(int mode, int M, int N, int K, double* estimate = nullptr) {
    const int parts = parts_of(mode);
    const int row_tiles = (N + BW * parts - 1) / (BW * parts), num_kb = (K + BK - 1) / BK;
    const int sms = sp_sm_count() > 0 ? sp_sm_count() : 148;
    Plan best{};
    double best_t = 0;
    for (int tt = (M + MAX_NT - 1) / MAX_NT; tt <= 16 && (tt == 1 || M >= 32 * (tt - 1)); ++tt)
        for (int pieces = 1; pieces <= MAX_PIECES; pieces *= 2) {
            Plan p{tt, 0, pieces, 0, 0, 0};
            if (!fill_plan(p, parts, M, num_kb)) continue;
            const int room = pieces <= 2 ? sms : pieces == 4 ? sms * 136 / 148 : sms * 128 / 148;
            const int side = parts == 1 && p.smem <= SMEM_SHARED ? 2 : 1;             // CTAs that fit on one SM
            const int ctas = row_tiles * tt * pieces, deep = (ctas + room - 1) / room, waves = (ctas + room * side - 1) / (room * side);
            const double bytes = (double)((num_kb + pieces - 1) / pieces) * (parts * BW + p.nt) * (BK * 2);
            const double t = 2800.0 + bytes * deep / (side == 2 && deep > 1 ? 136.0 : 115.0)
                             + waves * (42.0 * p.nt + 12.0 * p.nt / pieces + (pieces > 1 ? 1000.0 : 0.0) + 170.0 * pieces);
            if (best.nt == 0 || t < best_t) { best = p; best_t = t; }
        }
    if (estimate) *estimate = best_t;
    return best;
}

template <bool GATED, bool GROUPED>
int launch(const CUtensorMap& mw, const CUtensorMap& ma, const Args& args, const Plan& p, int row_tiles, cudaStream_t stream) {
    static SpPerDevice configured;
    if (!configured.done()) {
        cudaError_t e = cudaFuncSetAttribute(tc_mid_kernel<GATED, GROUPED>, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_LIMIT);
        if (e != cudaSuccess) SP_FAIL("tc_mid: cannot reserve %d bytes of shared memory: %s", SMEM_LIMIT, cudaGetErrorString(e));
        configured.mark();
    }
    SP_CHECK_CALL("tc_mid", sp_launch_cluster(tc_mid_kernel<GATED, GROUPED>, dim3(row_tiles * p.pieces, p.token_tiles), dim3(THREADS),
                                              (size_t)p.smem, stream, -p.pieces, mw, ma, args));
    return 0;
}

}  // namespace

// How a product is divided: token tiles, tokens per tile, pieces of K, stages (for tests and measurements).
SP_API int sp_tc_mid_plan(int mode, int M, int N, int K, int* out) {
    const Plan p = plan_of(mode, M, N, K);
    out[0] = p.token_tiles; out[1] = p.nt; out[2] = p.pieces; out[3] = p.stages;
    return p.nt ? 0 : 1;
}

// Which kernel takes a product of more than 128 tokens that both this one and the tiles by pairs of CTAs of tc_gemm.cu (256
// rows, 74 pairs on 148 SMs) could: the width of those tiles, a multiple of ``multiple``, or 0 for this kernel. By two estimates of
// time, compared with 2,902 measured products (N 512 to 32,000, K 256 to 14,336): the choice is 0.3 % slower than the better
// kernel on average for gated ones and 2.8 % for the others.
//   Pairs: a round of tiles takes 0.36 us per 64 of K at 256 columns, 0.335 at 192 and 0.31 at 128, the launch with its last
// epilogue 10 us, less where one round of narrow tiles does and K is short (512 x 512, 2,048 tokens 7.9 us, this kernel 10.8); gated
// ones 0.36 in the first round and 0.323 in the others, 3.5 for a round's epilogue and 5 for the launch.
//   This kernel: plan_of's, which was made to compare divisions and is 12 % short for gated products on average.
// Gated products are worth pairs as soon as their rounds come out full, for they have the most rows of W (us, this kernel /
// pairs: 1B 200 tokens 24.1 / 20.5, 301: 27.0 / 31.1, 512: 36.5 / 31.8, 1,023: 71.3 / 56.6; 3B 256: 32.0 / 27.3, 800 88.9 / 79.5; 8B
// 257: 89 / 107, 512: 123 / 109, 768: 201 / 139, 800: 209 / 206, 1,100: 257 / 222, 1,281: 318 / 289); the others from 1,024 tokens
// on, this kernel still where their pair tiles fill few SMs (1B, 1,280 tokens: output 15.6 / 26.4, down 38 / 84, 1,700 QKV 21.5 /
// 28.9; 8B 1,280 down 120 / 155).
SP_API int sp_tc_mid_or_pairs(int mode, int M, int N, int K, int multiple) {
    const bool gated = mode == MODE_SILU_MUL;
    if (M <= 128 || (!gated && M < 1024)) return 0;
    const int walkers = (sp_sm_count() > 0 ? sp_sm_count() : 148) / 2, row_tiles = (M + 255) / 256, num_kb = (K + BK - 1) / BK;
    auto rounds = [&](int bn) { return (row_tiles * ((N + bn - 1) / bn) + walkers - 1) / walkers; };
    const double start = rounds(128) > 1 || num_kb > 16 ? 10000.0 : 6000.0 + 250.0 * num_kb;
    int best = 0;
    double best_t = 0;
    for (const int bn : {256, 192, 128}) {
        if ((gated && bn != 256) || (multiple > 1 && bn % multiple)) continue;
        const double t = gated ? 5000.0 + rounds(bn) * 3500.0 + num_kb * (360.0 + 323.0 * (rounds(bn) - 1))
                               : start + (double)rounds(bn) * num_kb * (bn == 256 ? 360.0 : bn == 192 ? 335.0 : 310.0);
        if (!best || t < best_t) { best = bn; best_t = t; }
    }
    double mine = 0;
    if (M > 2048 || !plan_of(mode, M, N, K, &mine).nt) return best;
    return (gated ? 1.12 : 1.0) * mine < best_t ? 0 : best;
}

// Whether this kernel takes the product (0) or another has to (1, the reason as the last error).
SP_API int sp_tc_mid_supported(const void* A, const void* W, int M, int N, int K, int lda, int ldw, int mode, int pair) {
    if (M <= 0 || M > 2048) SP_FAIL("tc_mid: built for 1 to 2048 tokens, got %d", M);
    if (K <= 0 || (K % 8) || (lda % 8) || (ldw % 8)) SP_FAIL("tc_mid: K and the leading dimensions must be multiples of 8 (16-byte rows for TMA)");
    if (N <= 0 || (N % 8)) SP_FAIL("tc_mid: a multiple of 8 rows of W, got %d", N);
    if (((uintptr_t)A & 15) || ((uintptr_t)W & 15)) SP_FAIL("tc_mid: operands must start on a 16-byte boundary");
    if (mode == MODE_SILU_MUL && (pair != BW || N % (2 * BW))) SP_FAIL("tc_mid: gate and up rows come in blocks of %d, got %d", BW, pair);
    return 0;
}

// The product with the epilogues of sp_tc_stream_fused (tc_stream.cu): mode 0 C = A·Wᵀ (bfloat16 or float32), 1 C (float32)
// += A·Wᵀ, 2 C [M, N/2] = act(gate)·up · mult over blocks of 128 gate and 128 up rows, 4 rotate and store; ``ep`` may be null.
SP_API int sp_tc_mid(const void* A, const void* W, void* C, int c_dt, int M, int N, int K, int lda, int ldw, int ldc, int mode,
                     int pair, const void* epp, int act, float mult, float limit, float slope, int* status, cudaStream_t stream) {
    if (N <= 0) return 0;
    const SpGate ga{act, mult, limit, slope};
    if (mode != MODE_STORE && mode != MODE_ACCUMULATE && mode != MODE_SILU_MUL && mode != MODE_QKV_ROPE) SP_FAIL("tc_mid: unknown mode %d", mode);
    if (mode == MODE_SILU_MUL && !sp_gate_built(ga)) SP_FAIL("tc_mid: activation code %d is not built for gated rows", act);
    if (mode == MODE_ACCUMULATE && c_dt != SP_DT_F32) SP_FAIL("tc_mid: accumulation needs a float32 C");
    if (sp_tc_mid_supported(A, W, M, N, K, lda, ldw, mode, pair)) return 1;
    EpiArgs ep;
    memset(&ep, 0, sizeof(ep));
    if (epp) ep = *(const EpiArgs*)epp;
    if (ep.row_ssq && (ep.n_ssq <= 0 || ep.norm_width <= 0)) SP_FAIL("tc_mid: the row statistics need their count and the norm's width");
    if (ep.row_ssq && mode == MODE_ACCUMULATE) SP_FAIL("tc_mid: row statistics do not go with mode %d", mode);
    if (ep.xw && (mode != MODE_ACCUMULATE || !ep.next_w || !ep.ssq_out))
        SP_FAIL("tc_mid: preparing the next norm's input belongs to the accumulating epilogue and needs its weight and a place for the sums");
    if (ep.xw && (((uintptr_t)ep.xw & 7) || ((uintptr_t)ep.next_w & 7))) SP_FAIL("tc_mid: the next norm's weight and input must start on an 8-byte boundary");
    if (mode == MODE_QKV_ROPE) {
        if (ep.hd != 64 && ep.hd != 128) SP_FAIL("tc_mid: the rotate-and-store epilogue is built for head sizes 64 and 128, got %d", ep.hd);
        if (ep.nh <= 0 || ep.nkv <= 0 || N != (ep.nh + 2 * ep.nkv) * ep.hd) SP_FAIL("tc_mid: W has %d rows, %d q and %d kv heads of %d need %d", N, ep.nh, ep.nkv, ep.hd, (ep.nh + 2 * ep.nkv) * ep.hd);
        if (!ep.cs || !ep.tok_page || !ep.positions || !ep.q_out || !ep.kpool || !ep.vpool || ep.page_size <= 0)
            SP_FAIL("tc_mid: the rotate-and-store epilogue needs the angle table, the tokens' pages and positions, q and the cache");
        if (((uintptr_t)ep.cs & 15) || ((uintptr_t)ep.q_out & 7) || ((uintptr_t)ep.kpool & 7) || ((uintptr_t)ep.vpool & 7))
            SP_FAIL("tc_mid: the angle table must start on a 16-byte boundary, q and the cache on 8-byte boundaries");
    } else {
        if (((uintptr_t)C & 15) || (ldc % 4)) SP_FAIL("tc_mid: C must start on a 16-byte boundary and have rows of a multiple of 4 elements");
    }
    const Plan p = plan_of(mode, M, N, K);
    if (!p.nt) SP_FAIL("tc_mid: no division of %d tokens x %d x %d fits", M, N, K);
    const int parts = parts_of(mode), row_tiles = (N + BW * parts - 1) / (BW * parts);
    Args args{};
    args.ep = ep;
    args.rg = sp_range_host;
    args.ga = ga;
    args.C = C; args.status = status;
    args.c_dt = c_dt; args.M = M; args.N = N; args.K = K; args.ldc = ldc; args.mode = mode;
    args.nt = p.nt; args.pieces = p.pieces; args.stages = p.stages; args.tmem_cols = p.tmem_cols;
    CUtensorMap mw, ma;
    if (encode_map(&mw, W, N, K, ldw, BW)) return 1;
    if (encode_map(&ma, A, M, K, lda, p.nt)) return 1;
    if (parts == 2) return launch<true, false>(mw, ma, args, p, row_tiles, stream);
    return launch<false, false>(mw, ma, args, p, row_tiles, stream);
}

// Gated products of runs of rows of A [M, K], each with its expert's N rows (gate and up in blocks of 128) of the stacked W
// [w_rows, K]: C [M, N/2] = act(gate)·up, the clamped unit where ``slope`` is non-zero. ``tiles`` [n_tiles][3] on the device:
// (expert or -1, first row of A, rows: 1 to sp_tc_mid_run()); rows that no entry names are not written.
SP_API int sp_tc_mid_run() { return MAX_NT; }
SP_API int sp_tc_mid_grouped(const void* A, const void* W, void* C, int c_dt, int M, int N, int K, int lda, int ldw, int w_rows, int ldc,
                             const int* tiles, int n_tiles, float limit, float slope, int act, int* status, cudaStream_t stream) {
    if (M <= 0 || N <= 0 || n_tiles <= 0) return 0;
    const SpGate ga{slope != 0.0f ? (int)SP_ACT_CLAMPED : act, 1.0f, limit, slope};
    if (!sp_gate_built(ga)) SP_FAIL("tc_mid: activation code %d is not built for gated rows", ga.kind);
    if (sp_tc_mid_supported(A, W, 1, N, K, lda, ldw, MODE_SILU_MUL, BW)) return 1;
    if (((uintptr_t)C & 15) || (ldc % 4)) SP_FAIL("tc_mid: C must start on a 16-byte boundary and have rows of a multiple of 4 elements");
    if (n_tiles > 65535 || !tiles) SP_FAIL("tc_mid: a table of %d runs of rows", n_tiles);
    constexpr int parts = 2;
    const int row_tiles = N / (BW * parts);
    Plan p{n_tiles, MAX_NT, 1, 0, 0, 0};
    const int stage = parts * BW * BK * 2 + MAX_NT * BK * 2, num_kb = (K + BK - 1) / BK;
    p.stages = (SMEM_LIMIT - 1024) / stage;
    if (p.stages > num_kb) p.stages = num_kb;
    const int held = MAX_NT * BW * 4;
    p.smem = (p.stages * stage > held ? p.stages * stage : held) + 1024;
    p.tmem_cols = parts * MAX_NT;
    Args args{};
    args.rg = sp_range_host;
    args.ga = ga;
    args.C = C; args.status = status;
    args.c_dt = c_dt; args.M = M; args.N = N; args.K = K; args.ldc = ldc; args.mode = MODE_SILU_MUL;
    args.nt = p.nt; args.pieces = 1; args.stages = p.stages; args.tmem_cols = p.tmem_cols;
    args.tiles = tiles;
    CUtensorMap mw, ma;
    if (encode_map(&mw, W, w_rows, K, ldw, BW)) return 1;
    if (encode_map(&ma, A, M, K, lda, GROUP_BOX)) return 1;
    return launch<true, true>(mw, ma, args, p, row_tiles, stream);
}
