// Temperature / top-k / top-p sampling on the device, without sorting: a thread-block cluster per row of logits.
//
// Meaning, as in the reference (crates/spissa-runtime/src/ops.rs:377-430):
//   probs = softmax(logits / temperature); tokens ordered by falling probability,
//   equal ones by rising index (a stable sort); keep the first top_k (0 = all); of
//   those keep the shortest prefix whose mass reaches top_p; draw u·(kept mass) and
//   walk the kept list until the running mass reaches it. If nothing is hit, the most
//   probable token is returned (ops.rs:429).
//
// Every step of that walk asks the same question: which is the first token, in that order, at which a
// running total (a count for top-k, a mass for top-p and for the draw) reaches a target? The order is the
// rising order of a 64-bit key (inverted probability bits, then index), keys are unique, and the total up
// to a key is a plain sum over the tokens with smaller or equal keys. So the token can be found by descending
// the key four bits at a time: one pass over the row adds every token that is still in question into one
// of 16 sums by its next four key bits, the sums are added up in rising order until the target is
// reached, and the search goes on inside that one. A pass touches only tokens that share the bits chosen
// so far; once a single token is left it is looked up and the search ends (a peaked distribution is done
// after a few passes; equal probabilities are told apart by the index bits of the key).
//
// Finding the token by that descent alone took some twenty passes of three microseconds (8 rows of 128,256 logits: 80 us).
// Now one pass adds every token into one of 4,065 buckets, by the upper 14 bits of its probability (sign, exponent and five
// bits of the mantissa); a bucket's count and the sum of its tokens' lower 18 bits give its exact mass. The buckets' running
// totals stay in the cluster's shared memory for every question asked of the row, and each group of sixteen's in every CTA's:
// a question finds its bucket with one look at another CTA, the bucket's tokens go to all CTAs at once, each at a place that
// the counts have set aside, and behind that one barrier of the cluster every CTA finds the token among them for itself,
// by bins of the next ten bits. 8 rows 25 us (38 with the tokens gathered in one CTA and compared with one another by all,
// which took three trips between the CTAs and two barriers a question), 64 rows 101 (129), 64 of 32,000 37 (41). What is
// left are five barriers of the cluster, the softmax and the adding into buckets. Only where more than 1,024 tokens share
// the bucket (rows of nearly equal probabilities) the descent runs, from the three digits of the key that the bucket fixes
// (8 rows, top_k 50: logits N(0, 0.5) 23 us, by the descent from its first digit 55; all tokens equal 131 and 129:
// there a vote in front of the adding saves 12 us, which costs every other row 2).
//
// Sums are integers: a probability counts as floor(p · 2^44) and a token as 1 in the high bits of the same
// 64-bit word, so every total is exact and independent of the order of addition (the same draw always
// gives the same token), and finer than the 32-bit running sum of a serial walk. Each thread adds into
// words of its own in shared memory (no atomics); the CTAs of the cluster take slices of the row and add
// their 16 sums through distributed shared memory, so every CTA takes every decision alike.
#include "common.cuh"

SP_API const char* sp_sampling_last_error() { return sp_error_text; }
SP_DEFINE_RANGE_API(sampling)

namespace {

constexpr int SS_CLUSTER = 8;                      // CTAs per row; 256 threads each, 1024 when few rows leave SMs idle
constexpr int SS_SEGS = 16;                        // sums per pass: four key bits
constexpr int MASS_BITS = 45;                      // low bits: mass in units of 2^-44 (a row's total stays below 2^45)
constexpr unsigned long long MASS_MASK = (1ull << MASS_BITS) - 1;
constexpr unsigned long long ONE_TOKEN = 1ull << MASS_BITS;      // the count lives in the 19 bits above
constexpr float MASS_UNIT = 17592186044416.0f;     // 2^44
constexpr int SS_MAX_V = (1 << (64 - MASS_BITS)) - 1;

__device__ __forceinline__ unsigned ss_cluster_rank() {
    unsigned r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ void ss_cluster_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ unsigned ss_peer_addr(const void* local, unsigned rank) {
    unsigned ra;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(ra) : "r"((unsigned)__cvta_generic_to_shared(local)), "r"(rank));
    return ra;
}
__device__ __forceinline__ unsigned long long ss_ld_peer_u64(const void* local, unsigned rank) {
    unsigned long long v;
    asm volatile("ld.shared::cluster.u64 %0, [%1];" : "=l"(v) : "r"(ss_peer_addr(local, rank)) : "memory");
    return v;
}
__device__ __forceinline__ void ss_st_peer_f32(const void* local, unsigned rank, float v) {
    asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(ss_peer_addr(local, rank)), "f"(v) : "memory");
}

__device__ __forceinline__ unsigned long long ss_key(unsigned prob_bits, unsigned idx) {
    return ((unsigned long long)(~prob_bits) << 32) | idx;
}
// One token and its mass floor(p · 2^44), p in [0, 1], from the float's fields: (1.m) · 2^(e - 127 + 44 - 23).
__device__ __forceinline__ unsigned long long ss_weight(unsigned prob_bits) {
    const int e = (int)(prob_bits >> 23);                     // the sign bit is clear
    const unsigned long long m = (unsigned long long)((prob_bits & 0x7fffffu) | 0x800000u);
    const int up = e - 106;                                    // e - 127 + 21
    const unsigned long long q = e == 0 ? 0ull : (up >= 0 ? m << up : (up > -24 ? m >> -up : 0ull));
    return ONE_TOKEN + q;
}

struct Shared {
    unsigned long long* acc;                       // [16][threads]: every thread's own 16 sums (dynamic shared memory)
    unsigned long long seg[2][SS_SEGS];            // this CTA's sums of a pass (two buffers: peers read one while the next fills)
    unsigned long long total[SS_SEGS];             // the cluster's sums
    unsigned long long loc;                        // this CTA's find of a lookup (0: none)
    float stat[2][SS_CLUSTER];                     // the CTAs' maxima / sums of exponentials
    float red[32];
};

struct Row {
    const unsigned* bits;      // probability bits of this CTA's slice of the row: bits[i - i0], in shared memory when it fits
    int i0, i1;                // the slice
    int idx_digits;            // four-bit digits that hold an index
};

constexpr int SS_KNOWN = 3;                        // digits of the key that are known from the buckets

// The first key (rising) at which the running count (by_mass false) or mass reaches ``target``, where it begins with the
// SS_KNOWN digits of ``prefix`` and the tokens before those come to ``below``. ``upto``: the packed total up to and
// including it. Every thread of the cluster runs this alike.
template <int THREADS>
__device__ void ss_descend(Shared* sh, const Row& row, bool by_mass, unsigned long long target, unsigned long long prefix,
                           unsigned long long below, unsigned& parity, unsigned long long& key, unsigned long long& upto) {
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    unsigned long long* acc = sh->acc;
    const int n_digits = 8 + row.idx_digits;
    for (int d = SS_KNOWN; d < n_digits; ++d) {
        const int shift = d < 8 ? 60 - 4 * d : 4 * (n_digits - 1 - d);
        const unsigned long long above = ~0ull << (shift + 4);          // bits above this digit: a token must share them with the prefix
#pragma unroll
        for (int s = 0; s < SS_SEGS; ++s) acc[s * THREADS + tid] = 0ull;
        if (d < 8) {
            // a digit of the probability: 32-bit arithmetic on the key's upper half
            const unsigned pre_hi = (unsigned)(prefix >> 32), above_hi = (unsigned)(above >> 32);
            const int sh_hi = shift - 32;
            for (int i = row.i0 + tid; i < row.i1; i += THREADS) {
                const unsigned b = row.bits[i - row.i0];
                const unsigned kb = ~b;
                if (((kb ^ pre_hi) & above_hi) == 0u)
                    acc[((kb >> sh_hi) & 15u) * THREADS + tid] += ss_weight(b);
            }
        } else {
            for (int i = row.i0 + tid; i < row.i1; i += THREADS) {
                const unsigned b = row.bits[i - row.i0];
                const unsigned long long k = ss_key(b, (unsigned)i);
                if (((k ^ prefix) & above) == 0ull) acc[((k >> shift) & 15u) * THREADS + tid] += ss_weight(b);
            }
        }
        __syncthreads();
        // this CTA's 16 sums: the first 16 warps (or 8, two segments each) add up a segment's words
        constexpr int WARPS = THREADS / 32, PER_WARP = WARPS >= SS_SEGS ? 1 : SS_SEGS / WARPS;
        if (warp * PER_WARP < SS_SEGS) {
#pragma unroll
            for (int h = 0; h < PER_WARP; ++h) {
                const int s = PER_WARP * warp + h;
                unsigned long long v = 0ull;
#pragma unroll 8
                for (int k = 0; k < THREADS / 32; ++k) v += acc[s * THREADS + lane + 32 * k];
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
                if (lane == 0) sh->seg[parity][s] = v;
            }
        }
        ss_cluster_sync();                                     // every CTA's sums are written (and the acc reads are done)
        if (tid < SS_SEGS) {
            unsigned long long v = 0ull;
#pragma unroll
            for (unsigned r = 0; r < SS_CLUSTER; ++r) v += ss_ld_peer_u64(&sh->seg[parity][tid], r);
            sh->total[tid] = v;
        }
        parity ^= 1u;
        __syncthreads();
        int chosen = SS_SEGS - 1;
        unsigned long long cum = below;
        for (int s = 0; s < SS_SEGS; ++s) {
            const unsigned long long t = sh->total[s];
            if (t >= ONE_TOKEN) {                               // tokens in this segment
                const unsigned long long with = cum + t;
                if ((by_mass ? (with & MASS_MASK) : (with >> MASS_BITS)) >= target) { chosen = s; break; }
                cum = with;
            }
        }
        below = cum;
        prefix |= (unsigned long long)chosen << shift;
        const unsigned long long in_segment = sh->total[chosen];
        __syncthreads();                                       // sh->total is read by all before the next pass rewrites it
        if ((in_segment >> MASS_BITS) == 1ull || d == n_digits - 1) {
            // one token left: look it up (its remaining key bits are not known yet)
            const unsigned long long fixed = ~0ull << shift;
            if (tid == 0) sh->loc = 0ull;
            __syncthreads();
            for (int i = row.i0 + tid; i < row.i1; i += THREADS) {
                const unsigned long long k = ss_key(row.bits[i - row.i0], (unsigned)i);
                if (((k ^ prefix) & fixed) == 0ull) sh->loc = k + 1ull;       // at most one thread of the cluster
            }
            __syncthreads();
            ss_cluster_sync();
            unsigned long long found = 0ull;
#pragma unroll
            for (unsigned r = 0; r < SS_CLUSTER; ++r) found += ss_ld_peer_u64(&sh->loc, r);
            ss_cluster_sync();                                 // all have read before anyone's loc is reset
            key = found - 1ull;
            upto = below + in_segment;
            return;
        }
    }
}

// ---------------------------------------------------------------- the buckets
constexpr int BK_SHIFT = 18;                       // bits of a probability below its bucket
constexpr int BK_N = 4096;                         // probabilities are at most 1: bucket 4,064 is the last in use
constexpr int BK_PER = BK_N / SS_CLUSTER;          // positions (buckets by falling probability) whose totals a CTA keeps
constexpr int BK_LIST = 1024;                      // tokens of a bucket that are compared with one another
constexpr unsigned BK_CARRY = 1u << 20;            // in a bucket's count: its sum of lower bits has passed 2^32 (a slice has less than 2^20 tokens)

constexpr int BK_GROUP = 16;                       // positions (buckets by falling probability) whose total every CTA knows
constexpr int BK_GROUPS = BK_N / BK_GROUP;
constexpr int RF_BINS = 1024;                      // bins by which a list is searched
// In dynamic shared memory, in the place of the descent's words (which spoils them for the questions that follow).
struct Search {
    unsigned long long list[BK_LIST];              // a bucket's keys
    unsigned bin_count[RF_BINS], bin_low[RF_BINS];
};
struct Lists {
    unsigned count[BK_N];                          // this CTA's tokens of each bucket; later the place of the first of them in the bucket's list
    union { unsigned low[BK_N]; Search find; };    // their lower bits' contributions; later what a question needs
};
struct Buckets {
    unsigned long long scan[BK_PER];               // running totals (count and mass packed) of this CTA's positions
    unsigned long long groups[BK_GROUPS];          // running totals at the end of each group, from the first position of its CTA on
    unsigned long long warp_total[32];
    unsigned long long below, through;             // running totals before and through what was chosen
    unsigned long long key;
    int chosen, alone;
    int n_list[4], n_spoilt[4];                    // (a list's length has a word for each question: none has to be set back)
};

// What the lower 18 bits of a probability add to its mass, in the bucket's own unit (see bk_mass).
__device__ __forceinline__ unsigned bk_low(unsigned b) {
    const int e = (int)(b >> 23), down = 106 - e;                      // mass = mantissa >> down (or << -down)
    const unsigned l = b & ((1u << BK_SHIFT) - 1u);
    return e == 0 ? 0u : down <= 0 ? l : down <= BK_SHIFT ? l >> down : 0u;
}
// The mass of ``count`` tokens of a bucket whose bk_low add up to ``low``: the sum of ss_weight's masses, exactly. With
// mantissa = H · 2^18 + L, floor(mantissa / 2^d) is H · 2^(18 - d) + floor(L / 2^d) for d ≤ 18, and floor(H / 2^(d - 18)) beyond.
__device__ __forceinline__ unsigned long long bk_mass(int bucket, unsigned long long count, unsigned long long low) {
    const int e = bucket >> 5, down = 106 - e;
    const unsigned long long H = (unsigned long long)((bucket & 31) | 32);
    if (e == 0) return 0ull;
    if (down <= 0) return ((count * H << BK_SHIFT) + low) << -down;
    if (down <= BK_SHIFT) return (count * H << (BK_SHIFT - down)) + low;
    return down < 24 ? count * (H >> (down - BK_SHIFT)) : 0ull;
}
__device__ __forceinline__ unsigned long long bk_total(int bucket, unsigned long long count, unsigned long long low) {
    return (count << MASS_BITS) + bk_mass(bucket, count, low);
}
__device__ __forceinline__ bool bk_reached(unsigned long long total, bool by_mass, unsigned long long target) {
    return total >= ONE_TOKEN && (by_mass ? (total & MASS_MASK) : (total >> MASS_BITS)) >= target;
}

// Every CTA: its slice into buckets, then the running totals of its 512 positions of the row's buckets. What the questions
// need of them goes to every CTA at once: the groups' totals, and where in a bucket's list each CTA's own tokens begin.
template <int THREADS>
__device__ void bk_fill(Buckets* bk, Lists* li, const Row& row) {
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int n = row.i1 - row.i0;
    const bool carries = n >= 1 << (32 - BK_SHIFT);                    // a bucket's lower bits could pass 2^32
    for (int j = tid; j < n; j += THREADS) {
        const unsigned b = row.bits[j], low = bk_low(b);
        unsigned one = 1u;
        if (carries) {
            if (low && atomicAdd(&li->low[b >> BK_SHIFT], low) + low < low) one += BK_CARRY;
        } else if (low) {
            atomicAdd(&li->low[b >> BK_SHIFT], low);
        }
        atomicAdd(&li->count[b >> BK_SHIFT], one);
    }
    __syncthreads();
    ss_cluster_sync();
    constexpr int MINE = BK_PER / (THREADS < BK_PER ? THREADS : BK_PER);          // positions per thread
    const int rank = (int)ss_cluster_rank();
    unsigned long long part[MINE], run = 0ull;
#pragma unroll
    for (int i = 0; i < MINE; ++i) {
        part[i] = 0ull;
        const int pos = rank * BK_PER + tid * MINE + i, bucket = BK_N - 1 - pos;
        if (tid * MINE < BK_PER) {
            unsigned c[SS_CLUSTER], l[SS_CLUSTER];
#pragma unroll
            for (unsigned r = 0; r < SS_CLUSTER; ++r) {
                asm volatile("ld.shared::cluster.u32 %0, [%1];" : "=r"(c[r]) : "r"(ss_peer_addr(&li->count[bucket], r)) : "memory");
                asm volatile("ld.shared::cluster.u32 %0, [%1];" : "=r"(l[r]) : "r"(ss_peer_addr(&li->low[bucket], r)) : "memory");
            }
            unsigned count = 0u;
            unsigned long long low = 0ull;
#pragma unroll
            for (unsigned r = 0; r < SS_CLUSTER; ++r) {                // nobody else reads or writes this bucket's words here
                if (c[r]) asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(ss_peer_addr(&li->count[bucket], r)), "r"(count) : "memory");
                count += c[r] & (BK_CARRY - 1u);
                low += l[r] + ((unsigned long long)(c[r] / BK_CARRY) << 32);
            }
            part[i] = bk_total(bucket, count, low);
        }
        run += part[i];
    }
    // inclusive sums over the threads
    unsigned long long up = run;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const unsigned long long v = __shfl_up_sync(0xffffffffu, up, o);
        if (lane >= o) up += v;
    }
    if (lane == 31) bk->warp_total[warp] = up;
    __syncthreads();
    unsigned long long before = up - run;
    for (int w = 0; w < warp && w < BK_PER / MINE / 32; ++w) before += bk->warp_total[w];
#pragma unroll
    for (int i = 0; i < MINE; ++i) {
        before += part[i];
        const int p = tid * MINE + i;
        if (p < BK_PER) {
            bk->scan[p] = before;
            if ((p & (BK_GROUP - 1)) == BK_GROUP - 1) {
#pragma unroll
                for (unsigned r = 0; r < SS_CLUSTER; ++r)
                    asm volatile("st.shared::cluster.u64 [%0], %1;" ::"r"(ss_peer_addr(&bk->groups[(rank * BK_PER + p) / BK_GROUP], r)), "l"(before) : "memory");
            }
        }
    }
    __syncthreads();
    ss_cluster_sync();                                                 // the counts are not read any more
}

// The first key (rising) among the ``m`` keys of a list, all of ``bucket``, at which the running total from ``below`` on reaches
// the target, and the total up to and including it. A CTA searches for itself: the keys fall into bins by the next bits of the
// key, the bins' running totals tell which one holds the boundary, and its keys go on to the next bits until one is left (for
// most lists that is the first or the second pass; equal probabilities go on to the bits of their index). Arrives at the
// cluster's barrier as soon as the keys are in registers: the next list may then be written.
template <int THREADS>
__device__ void bk_refine(Buckets* bk, Search* se, int m, int bucket, bool by_mass, unsigned long long target,
                          unsigned long long below, unsigned long long& key, unsigned long long& upto) {
    constexpr int PER = BK_LIST / THREADS, BINS = RF_BINS / THREADS;   // keys and bins of a thread
    static_assert(PER >= 1 && BINS >= 1, "at most 1,024 threads");
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    unsigned long long mine[PER];
    bool in[PER];
#pragma unroll
    for (int i = 0; i < PER; ++i) {
        in[i] = tid + THREADS * i < m;
        mine[i] = in[i] ? se->list[tid + THREADS * i] : 0ull;
    }
    __syncwarp();
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    // digits of a key below its bucket: 10 and 8 bits of the probability, 10 and 9 of the index
#pragma unroll 1
    for (int d = 0; d < 4; ++d) {
        const int shift = d == 0 ? 40 : d == 1 ? 32 : d == 2 ? 9 : 0;
        const unsigned mask = d == 0 || d == 2 ? 1023u : d == 1 ? 255u : 511u;
#pragma unroll
        for (int i = 0; i < BINS; ++i) se->bin_count[tid * BINS + i] = se->bin_low[tid * BINS + i] = 0u;
        __syncthreads();
        unsigned bin[PER];
#pragma unroll
        for (int i = 0; i < PER; ++i) {
            bin[i] = (unsigned)(mine[i] >> shift) & mask;
            if (in[i]) {
                atomicAdd(&se->bin_count[bin[i]], 1u);
                const unsigned low = bk_low(~(unsigned)(mine[i] >> 32));
                if (low) atomicAdd(&se->bin_low[bin[i]], low);
            }
        }
        __syncthreads();
        // running counts and sums (1,024 keys of 18 bits: both fit 32 bits; scanned as one word)
        unsigned long long part[BINS], run = 0ull;
#pragma unroll
        for (int i = 0; i < BINS; ++i) {
            part[i] = ((unsigned long long)se->bin_count[tid * BINS + i] << 32) | se->bin_low[tid * BINS + i];
            run += part[i];
        }
        unsigned long long up = run;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const unsigned long long v = __shfl_up_sync(0xffffffffu, up, o);
            if (lane >= o) up += v;
        }
        if (lane == 31) bk->warp_total[warp] = up;
        __syncthreads();
        unsigned long long before = up - run, t = lane < THREADS / 32 && lane < warp ? bk->warp_total[lane] : 0ull;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
        before += t;
#pragma unroll
        for (int i = 0; i < BINS; ++i) {
            const unsigned long long after = before + part[i];
            if (part[i] >> 32) {
                const unsigned long long with = below + bk_total(bucket, after >> 32, after & 0xffffffffull);
                const unsigned long long without = below + bk_total(bucket, before >> 32, before & 0xffffffffull);
                if (bk_reached(with, by_mass, target) && !bk_reached(without, by_mass, target)) {
                    bk->chosen = tid * BINS + i;                       // one bin
                    bk->alone = part[i] >> 32 == 1ull;
                    bk->below = without;
                    bk->through = with;
                }
            }
            before = after;
        }
        __syncthreads();
        const unsigned chosen = (unsigned)bk->chosen;
        const bool last = bk->alone || d == 3;
        below = bk->below;
        upto = bk->through;
#pragma unroll
        for (int i = 0; i < PER; ++i) {
            in[i] = in[i] && bin[i] == chosen;
            if (last && in[i]) bk->key = mine[i];                      // keys are unique: one thread
        }
        if (last) break;
    }
    __syncthreads();
    key = bk->key;
}

// The token at which the running count or mass reaches ``target``, among all of the row: its key, and the packed total up to
// and including it. False when even the total does not (``upto``: the total). Every CTA alike. ``question``: 0, 1, ... within
// a row. ``spoilt``: a descent has overwritten where the CTAs' tokens begin in a list. ``arrived``: at the cluster's barrier, for
// which is waited before it is used again.
template <int THREADS>
__device__ bool bk_find(Shared* sh, Buckets* bk, Lists* li, const Row& row, int question, bool by_mass, unsigned long long target,
                        unsigned& parity, bool& spoilt, bool& arrived, unsigned long long& key, unsigned long long& upto) {
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    constexpr int PER_CTA = BK_GROUPS / SS_CLUSTER;                    // groups of a CTA: one for each lane of a warp
    static_assert(PER_CTA == 32 && THREADS >= BK_GROUPS, "a warp looks at the groups of one CTA");
    unsigned long long total = 0ull;
#pragma unroll
    for (int r = 0; r < SS_CLUSTER; ++r) total += bk->groups[r * PER_CTA + PER_CTA - 1];
    if (!bk_reached(total, by_mass, target)) { upto = total; return false; }
    if (warp < SS_CLUSTER) {
        unsigned long long base = 0ull;
        for (int r = 0; r < warp; ++r) base += bk->groups[r * PER_CTA + PER_CTA - 1];
        const unsigned long long with = base + bk->groups[tid];
        const unsigned long long without = base + (lane ? bk->groups[tid - 1] : 0ull);
        const unsigned here = __ballot_sync(0xffffffffu, bk_reached(with, by_mass, target) && !bk_reached(without, by_mass, target));
        if (here) {                                                    // one warp: the group's positions, from the CTA that has them
            const int group = warp * PER_CTA + __ffs(here) - 1;
            const unsigned long long before = __shfl_sync(0xffffffffu, without, __ffs(here) - 1);
            const int pos = group * BK_GROUP + lane;
            unsigned long long w = lane < BK_GROUP ? base + ss_ld_peer_u64(&bk->scan[pos % BK_PER], (unsigned)warp) : 0ull;
            unsigned long long wo = __shfl_up_sync(0xffffffffu, w, 1);
            if (lane == 0) wo = before;
            if (lane < BK_GROUP && bk_reached(w, by_mass, target) && !bk_reached(wo, by_mass, target)) {         // one lane
                bk->chosen = pos;
                bk->below = wo;
                bk->through = w;
            }
        }
    }
    __syncthreads();
    const int position = bk->chosen;
    const unsigned bucket = (unsigned)(BK_N - 1 - position);
    const unsigned long long below = bk->below;
    const unsigned long long n_in = (bk->through - below) >> MASS_BITS;
    if (arrived) asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
    arrived = false;
    if (n_in > BK_LIST) {
        // from the first of the four buckets that share the key's first SS_KNOWN digits
        const int first = position & ~3, owner = first / BK_PER, i = first % BK_PER;
        unsigned long long before = i ? ss_ld_peer_u64(&bk->scan[i - 1], (unsigned)owner) : 0ull;
        for (int r = 0; r < owner; ++r) before += bk->groups[r * PER_CTA + PER_CTA - 1];
        const unsigned long long prefix = (unsigned long long)((16383u - (unsigned)(BK_N - 1 - first)) >> 2) << 52;
        __syncthreads();                                               // what was chosen is read by all
        ss_descend<THREADS>(sh, row, by_mass, target, prefix, before, parity, key, upto);
        spoilt = true;
        return true;
    }
    // the bucket's tokens, to every CTA: a place of its own for each, in the order of the CTAs (within a CTA any order will do)
    const unsigned start = spoilt ? 0u : li->count[bucket];
    for (int i = row.i0 + tid; i < row.i1; i += THREADS) {
        const unsigned b = row.bits[i - row.i0];
        if (b >> BK_SHIFT == bucket) {
            unsigned at;
            if (spoilt) asm volatile("atom.shared::cluster.add.u32 %0, [%1], 1;" : "=r"(at) : "r"(ss_peer_addr(&bk->n_spoilt[question], 0u)) : "memory");
            else at = start + (unsigned)atomicAdd(&bk->n_list[question], 1);
            if (at < BK_LIST) {
#pragma unroll
                for (unsigned r = 0; r < SS_CLUSTER; ++r)
                    asm volatile("st.shared::cluster.u64 [%0], %1;" ::"r"(ss_peer_addr(&li->find.list[at], r)), "l"(ss_key(b, (unsigned)i)) : "memory");
            }
        }
    }
    __syncthreads();
    ss_cluster_sync();
    bk_refine<THREADS>(bk, &li->find, (int)n_in, (int)bucket, by_mass, target, below, key, upto);
    arrived = true;
    return true;
}

constexpr int INLINE_ROWS = 64;
struct Draws { float u[INLINE_ROWS]; };            // the rows' uniform numbers, with the launch itself: no copy to the device

template <int THREADS>
__host__ __device__ constexpr size_t words_bytes() {                   // the descent's words, or the lists
    constexpr size_t a = (size_t)SS_SEGS * THREADS * 8, b = (sizeof(Lists) + 15) / 16 * 16;
    return a > b ? a : b;
}

// ``cached`` tokens of a slice fit the dynamic shared memory: the passes then read the probabilities from there,
// else from the scratch row in global memory (``scratch`` may be null when every slice fits).
template <int THREADS>
__global__ void __launch_bounds__(THREADS)
sample_rows_kernel(const float* __restrict__ logits, int ld, int V, float temperature, int top_k, float top_p,
                   const float* __restrict__ u, const __grid_constant__ Draws draws, unsigned* __restrict__ scratch, int cached,
                   int* __restrict__ out) {
    extern __shared__ __align__(16) unsigned char dyn_smem[];
    __shared__ Shared sh_;
    Shared* sh = &sh_;
    sh->acc = (unsigned long long*)dyn_smem;                   // every thread writes the same value
    unsigned* slice_cache = (unsigned*)(dyn_smem + words_bytes<THREADS>());
    Lists* li = (Lists*)dyn_smem;
    __shared__ Buckets bk_;
    Buckets* bk = &bk_;
    const int tid = threadIdx.x;
    for (int i = tid; i < BK_N; i += THREADS) li->count[i] = li->low[i] = 0u;
    if (tid < 4) bk->n_list[tid] = bk->n_spoilt[tid] = 0;
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");          // this CTA's shared memory may be written to
    const unsigned rank = ss_cluster_rank();
    const int row_id = blockIdx.x / SS_CLUSTER;
    const float* x = logits + (size_t)row_id * ld;
    const int per = (V + SS_CLUSTER - 1) / SS_CLUSTER;
    Row row;
    row.i0 = min(V, (int)rank * per);
    row.i1 = min(V, row.i0 + per);
    unsigned* bits = per <= cached ? slice_cache : scratch + (size_t)row_id * V + row.i0;
    row.bits = bits;
    row.idx_digits = 1;
    while (row.idx_digits < 8 && (V - 1) >> (4 * row.idx_digits)) ++row.idx_digits;
    const int n = row.i1 - row.i0;

    // softmax of logits / temperature: exp(x - max) divided by the sum; every thread keeps to its own tokens, in registers
    // where it has few (all of its loads are then in flight together), so what it wrote to the slice it reads back itself
    constexpr int KEEP = 16;
    const bool few = n <= KEEP * THREADS;
    float held[KEEP];
    float mx = -INFINITY;
    if (few) {
#pragma unroll
        for (int i = 0; i < KEEP; ++i) {
            const int j = tid + THREADS * i;
            held[i] = j < n ? x[row.i0 + j] : 0.0f;
        }
#pragma unroll
        for (int i = 0; i < KEEP; ++i) {
            held[i] = held[i] / temperature;
            if (tid + THREADS * i < n) mx = fmaxf(mx, held[i]);
        }
    } else {
#pragma unroll 8
        for (int j = tid; j < n; j += THREADS) {
            const float v = x[row.i0 + j] / temperature;
            bits[j] = __float_as_uint(v);
            mx = fmaxf(mx, v);
        }
    }
    mx = sp_block_max(mx, sh->red);
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
    if (tid < SS_CLUSTER) ss_st_peer_f32(&sh->stat[0][rank], (unsigned)tid, mx);
    __syncwarp();
    ss_cluster_sync();
    mx = -INFINITY;
#pragma unroll
    for (unsigned r = 0; r < SS_CLUSTER; ++r) mx = fmaxf(mx, sh->stat[0][r]);
    float sum = 0.0f;
    if (few) {
#pragma unroll
        for (int i = 0; i < KEEP; ++i) {
            held[i] = expf(held[i] - mx);
            if (tid + THREADS * i < n) sum += held[i];
        }
    } else {
#pragma unroll 4
        for (int j = tid; j < n; j += THREADS) {
            const float e = expf(__uint_as_float(bits[j]) - mx);
            bits[j] = __float_as_uint(e);
            sum += e;
        }
    }
    sum = sp_block_sum(sum, sh->red);
    if (tid < SS_CLUSTER) ss_st_peer_f32(&sh->stat[1][rank], (unsigned)tid, sum);
    __syncwarp();
    ss_cluster_sync();
    sum = 0.0f;
#pragma unroll
    for (unsigned r = 0; r < SS_CLUSTER; ++r) sum += sh->stat[1][r];       // in rank order, alike in every CTA
    auto probability = [&](float e) {
        float p = e / sum;
        if (!(p >= 0.0f)) p = 0.0f;                           // NaN logits never win
        if (p > 1.0f) p = 1.0f;
        return __float_as_uint(p);
    };
    if (few) {
#pragma unroll
        for (int i = 0; i < KEEP; ++i)
            if (tid + THREADS * i < n) bits[tid + THREADS * i] = probability(held[i]);
    } else {
#pragma unroll 4
        for (int j = tid; j < n; j += THREADS) bits[j] = probability(__uint_as_float(bits[j]));
    }

    bk_fill<THREADS>(bk, li, row);
    int question = 0;
    unsigned parity = 0;
    bool spoilt = false, arrived = false;
    auto first_at = [&](bool by_mass, unsigned long long target, unsigned long long& key, unsigned long long& upto) -> bool {
        return bk_find<THREADS>(sh, bk, li, row, question++, by_mass, target, parity, spoilt, arrived, key, upto);
    };
    unsigned long long key = 0ull, upto = 0ull, limit_mass = 0ull;
    const bool limited = top_k > 0 && top_k < V && first_at(false, (unsigned long long)top_k, key, upto);       // the first top_k tokens
    if (limited) limit_mass = upto & MASS_MASK;
    // of those the shortest prefix whose mass reaches top_p; its mass
    const unsigned long long enough = __float2ull_rz(top_p * MASS_UNIT);
    unsigned long long kept_mass = limit_mass;                 // the first top_k weigh less
    if (!limited || limit_mass >= enough) {
        first_at(true, enough, key, upto);
        kept_mass = upto & MASS_MASK;
    }
    // the draw: u is a multiple of 2^-24, the target u · mass is taken exactly; it lies among the kept tokens
    const unsigned long long n_u = (unsigned long long)((u ? u[row_id] : draws.u[row_id]) * 16777216.0f);
    const unsigned long long target = (__umul64hi(kept_mass, n_u) << 40) | ((kept_mass * n_u) >> 24);
    if (!first_at(true, target, key, upto)) first_at(true, 0ull, key, upto);                    // the most probable token
    if (arrived) asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
    // (behind the last question's barrier of the cluster nobody reads or writes a peer's shared memory: all may leave)
    if (rank == 0 && tid == 0) out[row_id] = (int)(unsigned)(key & 0xffffffffu);
}

}  // namespace

constexpr int SS_CACHE_BYTES = 128 * 1024;         // of a slice's probabilities in shared memory

// 64-bit words of scratch: one 32-bit probability per token (unused when a slice fits the shared memory)
SP_API long long sp_sample_scratch_keys(int rows, int V) {
    return ((long long)rows * V + 1) / 2;
}

static int sample_rows_any(const float* logits, int ld, int rows, int V, float temperature, int top_k, float top_p, const float* u,
                           const Draws& draws, void* scratch, long long scratch_keys, int* out, cudaStream_t stream);

SP_API int sp_sample_rows(const float* logits, int ld, int rows, int V, float temperature, int top_k,
                          float top_p, const float* u, void* scratch, long long scratch_keys, int* out,
                          cudaStream_t stream) {
    if (!u && rows > 0) SP_FAIL("sample: the rows' uniform numbers are missing");
    return sample_rows_any(logits, ld, rows, V, temperature, top_k, top_p, u, Draws{}, scratch, scratch_keys, out, stream);
}

// The same with the uniform numbers in host memory, for up to 64 rows.
SP_API int sp_sample_rows_inline_max() { return INLINE_ROWS; }
SP_API int sp_sample_rows_inline(const float* logits, int ld, int rows, int V, float temperature, int top_k, float top_p, const float* u,
                                 void* scratch, long long scratch_keys, int* out, cudaStream_t stream) {
    if (rows > INLINE_ROWS) SP_FAIL("sample: %d rows of draws do not go with a launch (%d at most)", rows, INLINE_ROWS);
    Draws draws{};
    for (int r = 0; r < rows; ++r) draws.u[r] = u[r];
    return sample_rows_any(logits, ld, rows, V, temperature, top_k, top_p, nullptr, draws, scratch, scratch_keys, out, stream);
}

static int sample_rows_any(const float* logits, int ld, int rows, int V, float temperature, int top_k, float top_p, const float* u,
                           const Draws& draws, void* scratch, long long scratch_keys, int* out, cudaStream_t stream) {
    if (rows <= 0) return 0;
    if (V <= 0) SP_FAIL("sample: empty rows");
    if (!(temperature > 0.0f)) SP_FAIL("sample: temperature must be positive here (greedy rows use argmax)");
    if (!(top_p > 0.0f && top_p <= 1.0f)) SP_FAIL("sample: top_p must be in (0, 1], got %g", (double)top_p);
    if (top_k < 0) SP_FAIL("sample: top_k must not be negative");
    if (V > SS_MAX_V) SP_FAIL("sample: a vocabulary of %d is beyond this kernel's counters (%d at most)", V, SS_MAX_V);
    const int per = (V + SS_CLUSTER - 1) / SS_CLUSTER;
    const bool fits = (long long)per * 4 <= SS_CACHE_BYTES;
    if (!fits && scratch_keys < sp_sample_scratch_keys(rows, V))
        SP_FAIL("sample: scratch holds %lld words, %lld are needed", scratch_keys, sp_sample_scratch_keys(rows, V));
    const int cached = fits ? per : 0;
    const size_t cache_bytes = fits ? (((size_t)per * 4 + 15) / 16) * 16 : 0;
    static SpPerDevice configured;
    if (!configured.done()) {
        cudaError_t e = cudaFuncSetAttribute(sample_rows_kernel<256>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                             SS_CACHE_BYTES + (int)words_bytes<256>());
        if (e == cudaSuccess)
            e = cudaFuncSetAttribute(sample_rows_kernel<1024>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     SS_CACHE_BYTES / 2 + (int)words_bytes<1024>());
        if (e != cudaSuccess) SP_FAIL("sample: cannot reserve shared memory: %s", cudaGetErrorString(e));
        configured.mark();
    }
    // few rows: 1,024 threads per CTA (one CTA per SM, a quarter of the tokens per thread); many rows: 256, several CTAs per SM
    if (rows * SS_CLUSTER <= 128 && cache_bytes <= SS_CACHE_BYTES / 2)
        SP_CHECK_CALL("sample_rows", sp_launch_cluster(sample_rows_kernel<1024>, dim3(rows * SS_CLUSTER), dim3(1024),
                                                       cache_bytes + words_bytes<1024>(), stream, SS_CLUSTER, logits, ld, V,
                                                       temperature, top_k, top_p, u, draws, (unsigned*)scratch, cached, out));
    else
        SP_CHECK_CALL("sample_rows", sp_launch_cluster(sample_rows_kernel<256>, dim3(rows * SS_CLUSTER), dim3(256),
                                                       cache_bytes + words_bytes<256>(), stream, SS_CLUSTER, logits, ld, V,
                                                       temperature, top_k, top_p, u, draws, (unsigned*)scratch, cached, out));
    return 0;
}
