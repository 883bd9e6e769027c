// fsb_fullrow.cu - the full-vocabulary kernel of the B200 batched token sampler (sm_100a).
//
// Rows whose effective candidate count k exceeds kMaxK - above all `top_k == 0`, where the reference sorts the
// whole vocabulary (src/sampler.cpp:32-35 of paragontasx/ferro) - cannot keep their candidates in one CTA.  A
// cluster of four, five, six or eight CTAs works on one such row.  Every CTA keeps its slice of the row in shared memory
// (softcap and penalty applied once, src/model_gemma4.cpp:521 and src/sampler.cpp:11-18), so the row is read from
// HBM exactly once; everything after that reads shared memory:
//   1. the row's largest and smallest candidate key                                            (src/sampler.cpp:38)
//   2. if k < n: the k-th candidate, by a radix descent over the keys that counts                      (:27-31)
//   3. one pass over the weights e_i = exp((double)(x_i - max) / T) as 2^-62 fixed point: a histogram of them, exact,
//      over kBins bins of equal width in the logit.  Its cluster-wide cumulative sums end with the softmax denominator
//      (:40-41) and tell for any cumulative weight in which bin it is reached, and what the bins before it weigh.
//   4. with top-p (:44) or min-p (:43): the bins that can hold kept candidates are known now.  Their candidates, tens to
//      some hundreds as a rule, go to the first CTA, which orders them and does the rest of the row's work on the
//      ordered list: exact cumulative weights, both cuts and the draw (:45-49).  Without a cut, or when there are too
//      many, a cumulative weight is resolved on its own: the ordered candidates of its bin go there.
// If even one bin's candidates do not fit the first CTA's list (thousands of equal logits), a radix descent over the
// candidate keys resolves it: MSB-first over 8-bit digits, at every level each CTA histograms the candidates of its
// slice that match the prefix, all CTAs read all histograms through distributed shared memory and walk the digits - the
// same integer arithmetic everywhere, so no broadcast is needed - until a digit holds a single candidate.
// Sums of weights are integers, so they do not depend on the order in which threads add: the result is deterministic
// and differs from the reference's sequential fp64 sums by rounding only (~1e-13).
// What bounds it: the instructions of the passes over a slice, one CTA per SM, and latency of cluster-wide steps; not HBM.  Weighing
// a logit takes 19 fp64 operations, a conversion each way and some 40 others.  512 threads with 128 registers: with 1024 and 64 the
// passes spilled, and what all warps compute alike was issued eight times per scheduler instead of four.  What one warp can compute for
// all is left to one, and CTAs hand values to one another by counted stores (inbox_put): the cluster's barrier and its fences take 1 us.
// us by time stamps, 16 x 131072 in clusters of six, top-p 0.95: slice 2.3, extremes 0.6, weights, cumulative sums and the plan of what to look at
// 15.3, the rest 7 (29 where every crossing is resolved with a look at the slice of its own); 8 x 65536 in clusters of eight: 1.6, 0.6, 8.5, 5 (11).
#include <cuda_runtime.h>

#include <algorithm>

#include "fsb_device.cuh"

namespace fsb {
namespace {

constexpr int kFullThreads = 512;
constexpr int kFullWarps = kFullThreads / 32;
static_assert(kFullWarps <= 32, "the block reductions read one partial per lane");
constexpr int kMaxCluster = 8;                  // most CTAs per row
constexpr int kSliceCache = 32768;              // logits of a slice that are kept in shared memory
constexpr int kBins = 1024, kBinsEach = kBins / kFullThreads;   // a thread looks after two bins
constexpr int kShiftedFrom = 512;               // rows from this length on have slices that start on 16-byte boundaries
constexpr int kMostListed = 768;                // candidates that are worth a list
constexpr float kBinned = 19.4f;                // the bins cover this many temperatures below the maximum (weights down to 2^-28), the last one all the rest
constexpr int kSendCap = 512;                   // candidates a CTA can hand to the first one
constexpr int kShort = 256;                     // lists of up to this many candidates are ordered by counting
constexpr int kAhead = 4;                       // logits that a thread looks at together in a descent
constexpr int kStripes = 8;                     // copies of the level histogram (by warp): fewer warps hit one word at once
constexpr int kLimbs = 4;                       // a weight is added to a histogram as four 16-bit limbs (32-bit native atomics)

struct U128 {
    u64 hi, lo;
};
__device__ __forceinline__ U128 u128_add(U128 a, U128 b) {
    U128 r;
    r.lo = a.lo + b.lo;
    r.hi = a.hi + b.hi + (r.lo < a.lo ? 1ull : 0ull);
    return r;
}
__device__ __forceinline__ U128 u128_sub(U128 a, U128 b) {
    U128 r;
    r.lo = a.lo - b.lo;
    r.hi = a.hi - b.hi - (a.lo < b.lo ? 1ull : 0ull);
    return r;
}
__device__ __forceinline__ bool u128_ge(U128 a, U128 b) { return a.hi > b.hi || (a.hi == b.hi && a.lo >= b.lo); }
__device__ __forceinline__ double u128_to_double(U128 a) {
    return __dadd_rn(__dmul_rn(__ull2double_rn(a.hi), 18446744073709551616.0), __ull2double_rn(a.lo));
}
// smallest U128 that is >= d (d >= 0, finite, below 2^127)
__device__ __forceinline__ U128 double_to_u128_ceil(double d) {
    U128 r{0ull, 0ull};
    if (!(d > 0.0)) return r;
    const double hi_d = floor(d * (1.0 / 18446744073709551616.0));
    r.hi = __double2ull_rz(hi_d);
    const double rest = d - hi_d * 18446744073709551616.0;   // exact: both are multiples of ulp(d)
    r.lo = __double2ull_ru(rest);
    if (rest >= 18446744073709551616.0) { r.hi += 1ull; r.lo = 0ull; }
    return r;
}

// ---- the cluster ---------------------------------------------------------------------------------------------------
// The cluster's barrier: arrive releases this thread's shared-memory writes to the cluster, wait acquires the others'.
__device__ __forceinline__ void cluster_sync_all() {
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// Address of a shared-memory location of CTA `rank` of the cluster, and loads from there.
__device__ __forceinline__ unsigned map_to_rank(const void* p, unsigned rank) {
    unsigned a;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(smem_u32(p)), "r"(rank));
    return a;
}
__device__ __forceinline__ u64 ld_cluster_u64(unsigned addr) {
    u64 v;
    asm volatile("ld.shared::cluster.u64 %0, [%1];" : "=l"(v) : "r"(addr) : "memory");
    return v;
}
__device__ __forceinline__ unsigned ld_cluster_u32(unsigned addr) {
    unsigned v;
    asm volatile("ld.shared::cluster.u32 %0, [%1];" : "=r"(v) : "r"(addr) : "memory");
    return v;
}

// ---- shared memory of a CTA -------------------------------------------------------------------------------------------
// What is known about a row once its weights have been added up; one warp works it out.
struct RowPlan {
    U128 S, target_p;          // all weights; the cumulative weight that top-p wants
    double sum, min_thr, u, below;   // (below: where min-p flips, from the largest logit)
    float x_sure, x_never;     // min-p keeps logits above the first and none below the second
    int draw_lo, draw_hi, cut_lo, cut_hi;   // bins that the draw may fall into, and where the kept set may end (none: nothing is cut)
    int top_p, min_p;          // which cuts may end it there
    unsigned about;            // how many candidates those bins hold, about
};
struct FullShared {
    // A descent's level histogram (kStripes copies): [stripe][limb 0..3, then the candidate count][digit], four words of
    // padding between stripes; a limb sum stays below 2^32 while a stripe sees fewer than 65537 candidates, i.e. for
    // rows of up to 4 M logits.  In the first CTA also the lists of candidates that the CTAs hand over (list()).
    union {
        alignas(16) unsigned h[kStripes][(kLimbs + 1) * 256 + 4];
        struct {   // while the weights are added up:
            unsigned hist[kLimbs][kBins];      // this CTA's weights by bin, as sums of their 16-bit limbs
        };
    };
    u64 x_lo[2][256];          // this CTA's sum of them, which the other CTAs read; double buffered by level: a CTA may
    u64 x_hi[2][256];          // build the next level while others still read this one
    unsigned x_cnt[2][256];
    u64 x_small[2][4];         // small values exchanged across the cluster (extremes, sums), double buffered by use
    u64 x_all[2][kMaxCluster * 4];   // ... and every CTA's copy of all of them
    double table[64];          // 2^(j / 64)
    u64 part[2][kBins + 8];   // the CTAs' weights of the bins that this CTA adds up: the sums of their lower 32 bits and of the rest
    u64 cum[2][kBins];         // cluster-wide: weight of bins 0 .. b, the sums of the weights' lower 32 bits and of the rest
    unsigned cum_n[kBins];     // ... and about how many candidates they hold (see estimated_count)
    // suffix sums of the walk
    u64 w_lo[8], w_hi[8];
    unsigned w_cnt[8];
    int res_digit;
    unsigned res_cnt;          // candidates in the chosen digit
    unsigned res_above_cnt;    // candidates before it
    u64 res_above_lo, res_above_hi;
    u64 red[kFullWarps];
    u64 red_hi[kFullWarps];
    unsigned red_cnt[kFullWarps];
    RowPlan plan;
    // counted stores from the cluster's CTAs (inbox_put): extremes, parts of bins, their sums, and at the end numbers of candidates,
    // candidates and whether the first CTA takes them
    u64 in_slice, in_extremes, in_parts, in_sums, in_counts, in_list, in_verdict;
    u64 extremes[2][kMaxCluster], counts[kMaxCluster], verdict;
    int late;                  // a wait of this CTA has run out
    unsigned gone;             // ... of another CTA of the cluster: see step_aside
    int sent;                  // candidates this CTA has handed over
    unsigned got[2][kMaxCluster];   // ... every CTA of the cluster has, double buffered by use
    int first_p, first_u;      // places in the ordered list
    u64 kw_lo, kw_hi;          // weight of the kept set
    u64 cross[5];              // a resolved crossing: candidate, weight above (two words), count above, found
    __device__ __forceinline__ U128 weight_to(int b) const {   // of the bins up to b, b included (-1: none)
        return b < 0 ? U128{0ull, 0ull} : u128_add(U128{0ull, cum[0][b]}, U128{cum[1][b] >> 32, cum[1][b] << 32});
    }
    __device__ __forceinline__ u64* list() { return reinterpret_cast<u64*>(&h[0][0]); }
};
static_assert(sizeof(FullShared) + kSliceCache / 8 + 4 + 16 + (kSliceCache + 4) * sizeof(float) <= 227 * 1024, "a CTA's shared memory");
static_assert(sizeof(u64) * (kMaxCluster * kSendCap + kShort) <= sizeof(FullShared::h), "the lists, and room to order a short one, lie in the histogram's memory");

struct FullArgs {
    const float* logits;
    const RowDesc* rows;      // the rows of this kernel
    const int32_t* hist;
    const int32_t* drafts;    // ids staged with a resident verification call
    int32_t* pool;            // id pool of the resident histories (rows with kRowAppend store their token there)
    int32_t* tokens;
    int32_t* tokens_host;     // mirror of the tokens in mapped host memory, or null
    unsigned* status_host;    // takes a non-zero word whenever a status bit is set, or null
    int32_t* kept_ids;        // [rows][kMaxK]
    double* kept_pr;          // [rows][kMaxK]; also the staging of the kept set's first candidates while they are gathered
    int32_t* kept_n;
    unsigned* status;
    int32_t n_vocab;
    int32_t vocab_offset;
    int32_t write_back;
    int32_t record;           // the caller wants the kept sets (their memory is used as a staging area either way)
    float softcap;
    u64* trace;               // diagnostics: time stamps of the last row's phases, or null
};

// A weight in 2^-62 units: up * 2^31 + down.
struct Weight {
    unsigned up;
    int down;
    __device__ __forceinline__ u64 value() const { return ((u64)up << 31) + (u64)(long long)down; }
};

// What the passes of a row share.
struct RowCtx {
    const float* vals;        // the slice in shared memory (as the sampler sees it), or null: read and transform the row
    const float* row;         // the row in global memory
    const unsigned* bitmap;   // penalised columns of the slice (bit i = column lo + i), or null
    float pen, cap;
    int lo, main, n;          // first column of this CTA's slice, columns from there on, and all its columns
    int id_base;              // token id of column 0
    float mx;                 // the row's maximum
    double temp, inv_temp;    // T and 1 / T
    float cut;                // x - max below this weighs nothing
    bool odd;                 // an infinite maximum, or a temperature that makes `cut` overflow
    const double* table;      // 2^(j / 64)
    u64 floor_c;              // candidates are those at or above this composite (0: all)
    float bin_scale;          // bins per logit
    __device__ __forceinline__ float seen(float x, int i) const {   // what the sampler sees of logit i of the slice
        if (cap != 0.0f) x = __fmul_rn(cap, tanhf(__fdiv_rn(x, cap)));
        if (bitmap && ((bitmap[i >> 5] >> (i & 31)) & 1u)) x = x > 0.0f ? __fdiv_rn(x, pen) : __fmul_rn(x, pen);
        return x;
    }
    __device__ __forceinline__ float at(int i) const { return vals ? vals[i] : seen(row[lo + i], i); }
    // Logits i, i + kFullThreads, ... of the slice, kAhead of them; what lies past its end is NaN.  A descent's pass is bound by latency - of
    // reads from L2, where the row is not in shared memory, and of the weights' chains of fp64 operations - with 16 warps per SM to hide it:
    // four reads and four weights at a time.  us, one logit at a time / four reads, weights one by one / both / eight reads: 4 x 300000 358, 329,
    // 307, 323; 4 x 900000 1001, 908, 845, 892; 8 x 65536, k = 3000 52.1, 52.4, 46.6, 48.8.  With the next four on their way, too, 343.
    __device__ __forceinline__ void ahead(int i, float (&x)[kAhead]) const {
        const float nan = __int_as_float(0x7fc00000);
#pragma unroll
        for (int q = 0; q < kAhead; ++q) {
            const int at = i + q * kFullThreads;
            x[q] = at >= n ? nan : vals ? vals[at] : row[lo + at];
        }
        if (vals) return;
#pragma unroll
        for (int q = 0; q < kAhead; ++q)
            if (i + q * kFullThreads < n) x[q] = seen(x[q], i + q * kFullThreads);
    }
    // (the up to three columns before the row's first 16-byte boundary come last in the first slice)
    __device__ __forceinline__ u64 comp(float x, int i) const { return make_comp(x, (i < main ? lo + i : i - main) + id_base); }
    // (x - max) / T for a finite difference, correctly rounded: a quotient from the rounded reciprocal and one exact correction
    // step (Markstein 1990), three fused operations in place of a division.  Both operands are floats: a quotient of two 24-bit
    // significands is at least 2^-25 ulp away from the middle of two doubles, and the correction is off by some 2^-52 ulp.
    __device__ __forceinline__ double scaled(float diff) const {
        const double d = (double)diff, q = __dmul_rn(d, inv_temp);
        return __fma_rn(__fma_rn(-q, temp, d), inv_temp, q);
    }
    // src/sampler.cpp:40-41 (a masked logit is infinitely far below the maximum: no correction step)
    __device__ __forceinline__ double probability(float x, double sum) const { return __ddiv_rn(exp(__ddiv_rn((double)__fsub_rn(x, mx), temp)), sum); }
    // src/sampler.cpp:40, exp(y) as 2^-62 fixed point in two parts.  Table-driven (P. Tang, "Table-driven implementation of the
    // exponential function", ACM TOMS 15, 1989): y = (64 e + j) ln2 / 64 + r, exp(y) = 2^e 2^(j/64) (1 + p(r)) with |r| <=
    // ln2 / 128, where the Taylor polynomial of degree 5 is off by less than 2^-54.  Adding 1.5 * 2^(52 - b) rounds to a multiple
    // of 2^-b and leaves that multiple in the low word: b = 31 gives the first part, b = 62 what is left.  Seventeen fp64
    // operations and no branch (exp() and conversions took twice as long).
    // Logits 45 temperatures below the maximum and NaNs weigh nothing.
    __device__ __noinline__ Weight odd_weight(float x) const {   // (an infinite maximum alone has weight)
        const double e = x == mx ? 1.0 : x == x ? exp(__ddiv_rn((double)__fsub_rn(x, mx), temp)) : 0.0;
        const u64 w = __double2ull_rn(__dmul_rn(e, 4611686018427387904.0));
        return Weight{(unsigned)(w >> 31), (int)(w & 0x7FFFFFFFull)};
    }
    __device__ __forceinline__ Weight weight(float x) const { return odd ? odd_weight(x) : finite_weight(x); }
    __device__ __forceinline__ Weight finite_weight(float x) const {   // (of a row that is not odd)
        const double y = scaled(fmaxf(__fsub_rn(x, mx), cut));
        const double magic = 6755399441055744.0;   // 1.5 * 2^52
        const double t = __fma_rn(y, 92.33248261689366, magic);   // 64 / ln 2
        const int n = __double2loint(t);
        const double k = __dsub_rn(t, magic);
        // ln2 / 64 in two parts, the first with 32 significant bits: k times it is exact
        double r = __fma_rn(k, -0.010830424693267559632658958435, y);
        r = __fma_rn(k, -2.9815858269852933e-12, r);
        double q = __fma_rn(r, 1.0 / 120.0, 1.0 / 24.0);
        q = __fma_rn(r, q, 1.0 / 6.0);
        q = __fma_rn(r, q, 0.5);
        q = __fma_rn(__dmul_rn(r, r), q, r);
        const double s = table[n & 63];
        const double v = __fma_rn(s, q, s);
        const double w = __hiloint2double(__double2hiint(v) + ((n & ~63) << 14), __double2loint(v));   // times 2^(n >> 6)
        const double m1 = 3145728.0, m2 = 0.00146484375;   // 1.5 * 2^21, 1.5 * 2^-10
        const double t1 = __dadd_rn(w, m1);
        const double t2 = __dadd_rn(__dsub_rn(w, __dsub_rn(t1, m1)), m2);
        return Weight{(unsigned)__double2loint(t1), __double2loint(t2)};
    }
    __device__ __forceinline__ bool is_candidate(float x, int i) const { return x == x && (floor_c == 0ull || comp(x, i) >= floor_c); }
    // bin of a logit: never decreases as the logit falls
    __device__ __forceinline__ int bin(float x) const { return min(kBins - 1, __float2int_rd(__fmul_rn(__fsub_rn(mx, x), bin_scale))); }
};

__device__ __forceinline__ u64 block_max_u64(u64 v, FullShared* sh) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int o = 16; o; o >>= 1) v = max(v, __shfl_xor_sync(0xffffffffu, v, o));
    if (lane == 0) sh->red[warp] = v;
    __syncthreads();
    u64 r = lane < kFullWarps ? sh->red[lane] : 0ull;   // one partial per lane
#pragma unroll
    for (int o = 16; o; o >>= 1) r = max(r, __shfl_xor_sync(0xffffffffu, r, o));
    __syncthreads();
    return r;
}

// Exchanges up to four 64-bit values per CTA across the cluster: every CTA gets all C x 4 values.
// `use` alternates 0/1 between consecutive exchanges.  Contains one cluster barrier.
template <int C>
__device__ __forceinline__ void cluster_exchange(FullShared* sh, int use, const u64 (&mine)[4], u64 (&all)[C][4]) {
    if (threadIdx.x < 4) sh->x_small[use][threadIdx.x] = mine[threadIdx.x];
    cluster_sync_all();
    // one warp fetches the remote words; everybody else reads the local copy
    if (threadIdx.x < C * 4)
        sh->x_all[use][threadIdx.x] = ld_cluster_u64(map_to_rank(&sh->x_small[use][threadIdx.x & 3], threadIdx.x >> 2));
    __syncthreads();
#pragma unroll
    for (int r = 0; r < C; ++r)
#pragma unroll
        for (int j = 0; j < 4; ++j) all[r][j] = sh->x_all[use][r * 4 + j];
}

// Adds (digit, weight, one candidate) to the level histogram: native 32-bit shared-memory atomics on the count and on
// the weight's non-zero 16-bit limbs.  The lanes of a warp spread over the stripes, and the stripes start in
// different banks, so that lanes with the same digit seldom meet in one word.
__device__ __forceinline__ void hist_add(FullShared* sh, bool active, int digit, u64 weight, bool weighted, unsigned stripe_mask) {
    if (!active) return;
    unsigned* h = &sh->h[threadIdx.x & stripe_mask][digit];
    atomicAdd(h + kLimbs * 256, 1u);
    if (weighted) {
        const unsigned l0 = (unsigned)(weight & 0xFFFFull), l1 = (unsigned)((weight >> 16) & 0xFFFFull);
        const unsigned l2 = (unsigned)((weight >> 32) & 0xFFFFull), l3 = (unsigned)(weight >> 48);
        if (l0) atomicAdd(h, l0);
        if (l1) atomicAdd(h + 256, l1);
        if (l2) atomicAdd(h + 512, l2);
        if (l3) atomicAdd(h + 768, l3);
    }
}

// What a descent found: the candidate at which the accumulated weight (or count) reaches the target, the weight and
// the number of candidates strictly before it, and whether there was such a candidate at all.
struct Crossing {
    u64 c;
    U128 above;
    unsigned above_cnt;
    bool found;
};

// One level's histogram of this CTA (the stripes added up) goes to the exchange buffer `par`; after the cluster's
// barrier every CTA adds up all CTAs' histograms (thread d < 256 owns digit d) and walks the digits from the top:
// the crossing digit is the highest digit d that holds a candidate and whose suffix sum (the weight of all higher
// digits and its own, plus `above`) reaches the target.  Leaves digit, its candidate count and the weight and count
// before it in shared memory; digit -1 if the target is beyond all candidates.  All threads of all CTAs of the cluster must call.
template <int C>
__device__ __forceinline__ void level_reduce_and_walk(FullShared* sh, int par, U128 target, U128 above, unsigned above_cnt, bool by_count,
                                                      unsigned stripe_mask) {
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    u64 lo = 0ull, hi = 0ull;
    unsigned cnt = 0u;
    if (tid < 256) {
        u64 l0 = 0ull, l1 = 0ull, l2 = 0ull, l3 = 0ull;   // limb sums over the stripes: below 2^35 each
        unsigned c = 0u;
#pragma unroll
        for (int s = 0; s <= (int)stripe_mask; ++s) {
            l0 += sh->h[s][tid];
            l1 += sh->h[s][256 + tid];
            l2 += sh->h[s][512 + tid];
            l3 += sh->h[s][768 + tid];
            c += sh->h[s][kLimbs * 256 + tid];
        }
        U128 acc{0ull, l0};
        acc = u128_add(acc, U128{l1 >> 48, l1 << 16});
        acc = u128_add(acc, U128{l2 >> 32, l2 << 32});
        acc = u128_add(acc, U128{l3 >> 16, l3 << 48});
        sh->x_lo[par][tid] = acc.lo;
        sh->x_hi[par][tid] = acc.hi;
        sh->x_cnt[par][tid] = c;
    }
    cluster_sync_all();
    if (tid < 256) {
        u64 l[C], h[C];
        unsigned c[C];
#pragma unroll
        for (unsigned r = 0; r < (unsigned)C; ++r) {
            l[r] = ld_cluster_u64(map_to_rank(&sh->x_lo[par][tid], r));
            h[r] = ld_cluster_u64(map_to_rank(&sh->x_hi[par][tid], r));
            c[r] = ld_cluster_u32(map_to_rank(&sh->x_cnt[par][tid], r));
        }
#pragma unroll
        for (int r = 0; r < C; ++r) {
            lo += l[r];
            hi += h[r] + (lo < l[r] ? 1ull : 0ull);
            cnt += c[r];
        }
    }
    if (by_count) {   // the "weight" of a digit is its number of candidates
        lo = cnt;
        hi = 0ull;
    }
    // suffix sums over the digits: within a warp (digits warp * 32 .. + 31), then the warps above
    U128 suf{hi, lo};
    unsigned sufc = cnt;
    if (tid < 256) {
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const u64 l = __shfl_down_sync(0xffffffffu, suf.lo, o);
            const u64 h = __shfl_down_sync(0xffffffffu, suf.hi, o);
            const unsigned c = __shfl_down_sync(0xffffffffu, sufc, o);
            if (lane + o < 32) {
                suf = u128_add(suf, U128{h, l});
                sufc += c;
            }
        }
        if (lane == 0) {
            sh->w_lo[warp] = suf.lo;
            sh->w_hi[warp] = suf.hi;
            sh->w_cnt[warp] = sufc;
        }
    }
    if (tid == 0) sh->res_digit = -1;
    __syncthreads();
    U128 with{0ull, 0ull};
    unsigned with_c = 0u;
    if (tid < 256) {
        U128 higher = above;
        unsigned higher_c = above_cnt;
        for (int w = warp + 1; w < 8; ++w) {
            higher = u128_add(higher, U128{sh->w_hi[w], sh->w_lo[w]});
            higher_c += sh->w_cnt[w];
        }
        with = u128_add(suf, higher);        // everything from this digit up, and what came before the level
        with_c = sufc + higher_c;
        if (cnt != 0u && u128_ge(with, target)) atomicMax(&sh->res_digit, tid);   // the highest digit that reaches wins
    }
    __syncthreads();
    if (tid < 256 && tid == sh->res_digit) {
        const U128 before = u128_sub(with, U128{hi, lo});
        sh->res_above_lo = before.lo;
        sh->res_above_hi = before.hi;
        sh->res_above_cnt = with_c - cnt;
        sh->res_cnt = cnt;
    }
    __syncthreads();
}

// Radix descent over the candidates with composite in [floor_c, top_c] (the extremes of the candidate set): finds
// the candidate at which the accumulated weight - or, with by_count, the number of candidates - counted from the
// largest candidate down reaches `target`.  All threads of the cluster call.
template <int C>
__device__ __noinline__ Crossing cluster_descent(const RowCtx rc, FullShared* sh, u64 floor_c, u64 top_c, U128 target, bool by_count, int& use) {
    int par = use;
    const int tid = threadIdx.x;
    Crossing out{0ull, U128{0ull, 0ull}, 0u, false};
    u64 mask, pfx;
    int hb;
    if (top_c != floor_c) {
        const int hb0 = 63 - __clzll((long long)(top_c ^ floor_c));
        mask = (hb0 == 63) ? 0ull : (~0ull << (hb0 + 1));
        pfx = top_c & mask;
        hb = hb0;
    } else {
        mask = ~0ull;
        pfx = top_c;
        hb = -1;
    }
    U128 above{0ull, 0ull};
    unsigned above_cnt = 0u;
    bool first = true;
    while (hb >= 0) {
        const int w = hb + 1 < 8 ? hb + 1 : 8, lo = hb + 1 - w;
        const unsigned dmask = (1u << w) - 1u;
        // the first level sees every candidate, a few digits take most of them: eight stripes keep the lanes of a warp
        // apart.  Deeper levels see the few candidates that match the prefix: one stripe, an eighth of the clearing
        // and adding up.
        // (a 16-bit limb summed over one stripe stays below 2^32 for slices of up to 65536 logits)
        const unsigned stripe_mask = (first || rc.n > 65536) ? (unsigned)(kStripes - 1) : 0u;
        {
            for (int i = tid; i < (int)((stripe_mask + 1u) * sizeof(sh->h[0]) / sizeof(uint4)); i += kFullThreads)
                reinterpret_cast<uint4*>(&sh->h[0][0])[i] = make_uint4(0u, 0u, 0u, 0u);
            __syncthreads();
            for (int i0 = tid; i0 - (tid & 31) < rc.n; i0 += kAhead * kFullThreads) {   // (whole warps)
                float x[kAhead];
                rc.ahead(i0, x);
                int digit[kAhead];   // -1: takes no part
                bool some = false;
#pragma unroll
                for (int q = 0; q < kAhead; ++q) {
                    const u64 c = rc.comp(x[q], i0 + q * kFullThreads);
                    const bool in = x[q] == x[q] && c >= floor_c && (c & mask) == pfx;
                    digit[q] = in ? (int)((unsigned)(c >> lo) & dmask) : -1;
                    some = some || in;
                }
                if (!__any_sync(0xffffffffu, some)) continue;
                u64 w[kAhead];
                if (by_count) {
#pragma unroll
                    for (int q = 0; q < kAhead; ++q) w[q] = 0ull;
                } else if (rc.odd) {
#pragma unroll
                    for (int q = 0; q < kAhead; ++q) w[q] = rc.odd_weight(x[q]).value();
                } else {   // a weight is a chain of dependent fp64 operations: several at once
#pragma unroll
                    for (int q = 0; q < kAhead; ++q) w[q] = rc.finite_weight(x[q]).value();
                }
#pragma unroll
                for (int q = 0; q < kAhead; ++q) hist_add(sh, digit[q] >= 0, digit[q], w[q], !by_count, stripe_mask);
            }
            __syncthreads();
        }
        level_reduce_and_walk<C>(sh, par, target, above, above_cnt, by_count, stripe_mask);
        par ^= 1;
        first = false;
        const int d = sh->res_digit;
        const unsigned in_digit = sh->res_cnt;
        const U128 nabove{sh->res_above_hi, sh->res_above_lo};
        const unsigned nabove_cnt = sh->res_above_cnt;
        __syncthreads();   // the results may be overwritten
        if (d < 0) {   // the target lies beyond the candidates
            use = par;
            return out;
        }
        pfx |= (u64)(unsigned)d << lo;
        mask |= (u64)dmask << lo;
        above = nabove;
        above_cnt = nabove_cnt;
        hb = lo - 1;
        if (in_digit == 1u && hb >= 0) break;   // a single candidate matches the prefix: no need to resolve its other bits
    }
    if (hb >= 0) {
        // the single candidate that matches the prefix, wherever it lies: its owner finds it, the cluster takes the maximum
        u64 mine = 0ull;
        for (int i0 = tid; i0 < rc.n; i0 += kAhead * kFullThreads) {
            float x[kAhead];
            rc.ahead(i0, x);
#pragma unroll
            for (int q = 0; q < kAhead; ++q) {
                const u64 c = rc.comp(x[q], i0 + q * kFullThreads);
                if (x[q] == x[q] && c >= floor_c && (c & mask) == pfx) mine = c;
            }
        }
        // exactly one thread of the cluster holds it: that thread tells every CTA, one barrier makes it visible
        if (mine != 0ull) {
#pragma unroll
            for (unsigned r = 0; r < (unsigned)C; ++r) cluster_store_u64(map_to_rank(&sh->x_small[par][0], r), mine);
        }
        cluster_sync_all();
        pfx = sh->x_small[par][0];
        par ^= 1;
    }
    use = par;
    out.c = pfx;
    out.above = above;
    out.above_cnt = above_cnt;
    out.found = true;
    return out;
}

// ---- cumulative weights by bin ----------------------------------------------------------------------------------------
// About how many candidates a bin holds, from its weight (units of 2^-31): right to a few per cent unless the bins are wide.
// Clamped, so that sums do not overflow.
__device__ __forceinline__ unsigned estimated_count(const RowCtx& rc, int bin, u64 weight) {
    const float middle = ((float)bin + 0.5f) / (rc.bin_scale * (float)rc.temp);   // of the bin, below the maximum, in temperatures
    const float n = (float)weight * exp2f(fminf(middle * 1.442695f, 60.0f) - 31.0f);
    return n < 1e6f ? (unsigned)n + (weight ? 1u : 0u) : 1000000u;
}

// First bin whose cumulative weight reaches t (the last one if none does).  Whole warps call.
__device__ __forceinline__ int find_bin(const FullShared* sh, U128 t) {
    const int lane = threadIdx.x & 31;
    const unsigned group = __ballot_sync(0xffffffffu, u128_ge(sh->weight_to(32 * lane + 31), t));
    if (group == 0u) return kBins - 1;
    const int b = 32 * (__ffs(group) - 1);
    return b + __ffs(__ballot_sync(0xffffffffu, u128_ge(sh->weight_to(b + lane), t))) - 1;
}

// Sum of two words and a count over the CTA, left in x_small[use][0..2].  Contains one barrier; the sums are there after the
// next one.
__device__ __forceinline__ void block_sums(FullShared* sh, int use, u64 lo, u64 hi, unsigned cnt) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int o = 16; o; o >>= 1) {
        lo += __shfl_xor_sync(0xffffffffu, lo, o);
        hi += __shfl_xor_sync(0xffffffffu, hi, o);
    }
    cnt = __reduce_add_sync(0xffffffffu, cnt);
    if (lane == 0) {
        sh->red[warp] = lo;
        sh->red_hi[warp] = hi;
        sh->red_cnt[warp] = cnt;
    }
    __syncthreads();
    if (warp == 0) {
        lo = lane < kFullWarps ? sh->red[lane] : 0ull;
        hi = lane < kFullWarps ? sh->red_hi[lane] : 0ull;
        cnt = __reduce_add_sync(0xffffffffu, lane < kFullWarps ? sh->red_cnt[lane] : 0u);
#pragma unroll
        for (int o = 16; o; o >>= 1) {
            lo += __shfl_xor_sync(0xffffffffu, lo, o);
            hi += __shfl_xor_sync(0xffffffffu, hi, o);
        }
        if (lane == 0) {
            sh->x_small[use][0] = lo;
            sh->x_small[use][1] = hi;
            sh->x_small[use][2] = cnt;
        }
    }
}
// A sum of weights kept as the sums of their parts.
__device__ __forceinline__ U128 join_parts(u64 down, u64 up) { return u128_add(U128{(long long)down < 0 ? ~0ull : 0ull, down}, U128{up >> 33, up << 31}); }

// Four consecutive logits of the slice; what lies past its end is NaN.
__device__ __forceinline__ void load4(const RowCtx& rc, int i, float (&x)[4]) {
    if (rc.vals && i + 4 <= rc.n) {
        const float4 v = *reinterpret_cast<const float4*>(rc.vals + i);
        x[0] = v.x, x[1] = v.y, x[2] = v.z, x[3] = v.w;
        return;
    }
#pragma unroll
    for (int e = 0; e < 4; ++e) x[e] = i + e >= rc.n ? __int_as_float(0x7fc00000) : rc.vals ? rc.vals[i + e] : rc.row[rc.lo + i + e];
    if (rc.vals) return;
#pragma unroll
    for (int e = 0; e < 4; ++e)
        if (i + e < rc.n) x[e] = rc.seen(x[e], i + e);
}

// Hands this CTA's candidates of bins [b_lo, b_hi] to the first CTA of the cluster, and counts its candidates of the bins before
// them.  Returns whether everybody's candidates fitted.  After it the first CTA has the lists (CTA r's sh->got[par][r] candidates
// at list() + r * kSendCap), and every CTA's count is in its x_small[par].
template <int C>
__device__ __forceinline__ bool send_bins(const RowCtx& rc, FullShared* sh, unsigned rank, int b_lo, int b_hi, bool count, int par) {
    const int tid = threadIdx.x;
    if (tid == 0) sh->sent = 0;
    __syncthreads();
    const unsigned to = map_to_rank(sh->list() + rank * kSendCap, 0u);
    unsigned cnt = 0u;
    const int lane = tid & 31;
    bool full = false;   // (then nothing more is handed over: the lists are of no use)
    for (int i0 = 4 * (tid - lane); i0 < rc.n; i0 += 4 * kFullThreads) {
        float x[4];
        load4(rc, i0 + 4 * lane, x);
        bool give[4], some = false;
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const int b = rc.bin(x[e]);
            const bool in = b <= b_hi && rc.is_candidate(x[e], i0 + 4 * lane + e);
            give[e] = in && b >= b_lo;
            cnt += in && b < b_lo ? 1u : 0u;
            some = some || give[e];
        }
        if (__any_sync(0xffffffffu, some) && !full) {
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const unsigned hits = __ballot_sync(0xffffffffu, give[e]);
                if (hits == 0u) continue;
                int p = 0;
                if (lane == 0) p = atomicAdd(&sh->sent, __popc(hits));
                p = __shfl_sync(0xffffffffu, p, 0);
                full = full || p >= kSendCap;
                p += __popc(hits & ((1u << lane) - 1u));
                if (give[e] && p < kSendCap) cluster_store_u64(to + 8u * (unsigned)p, rc.comp(x[e], i0 + 4 * lane + e));
            }
        }
        if (full && !count) break;
    }
    if (count) block_sums(sh, par, 0ull, 0ull, cnt);
    else __syncthreads();
    if (tid < C) cluster_store_u32(map_to_rank(&sh->got[par][rank], (unsigned)tid), (unsigned)sh->sent);
    cluster_sync_all();
    bool fits = true;
#pragma unroll
    for (int r = 0; r < C; ++r) fits = fits && sh->got[par][r] <= (unsigned)kSendCap;
    return fits;
}

// The same for the candidates of bins [b0, b1] and [b2, b3] (b1 < b2, or the second range is empty), without a count; once per row.
// Nobody but the first CTA waits for the candidates: it counts what comes, and tells the others whether it has all of them.
// 1: it has, 0: it has not, -1: this CTA's wait has run out (the first one has told nobody anything then).
template <int C>
__device__ __forceinline__ int send_ranges(const RowCtx& rc, FullShared* sh, unsigned rank, int b0, int b1, int b2, int b3, int par) {
    const int tid = threadIdx.x;
    const unsigned to = map_to_rank(sh->list() + rank * kSendCap, 0u), bar = map_to_rank(&sh->in_list, 0u);
    // (a logit's bin is only worked out if the logit may lie in one of the ranges: the room on either side covers the rounding of the
    // bin, 2^-13 of its width, and of these limits)
    const float width = 1.0f / rc.bin_scale, room = 0.03f * width + 5e-7f * fabsf(rc.mx), inf = __int_as_float(0x7f800000);
    const bool two = b3 >= b2;
    const float hi1 = b0 > 0 ? rc.mx - (float)b0 * width + room : inf, lo1 = b1 < kBins - 1 ? rc.mx - (float)(b1 + 1) * width - room : -inf;
    const float hi2 = !two ? -inf : b2 > 0 ? rc.mx - (float)b2 * width + room : inf, lo2 = !two ? inf : b3 < kBins - 1 ? rc.mx - (float)(b3 + 1) * width - room : -inf;
    auto near = [&](float x) { return (x <= hi1 && x >= lo1) || (x <= hi2 && x >= lo2); };
    auto look = [&](float x, int i) {   // (few: a lane reserves for itself)
        const int b = rc.bin(x);
        if (((b >= b0 && b <= b1) || (b >= b2 && b <= b3)) && rc.is_candidate(x, i)) {
            const int p = atomicAdd(&sh->sent, 1);
            if (p < kSendCap) inbox_put(to + 8u * (unsigned)p, rc.comp(x, i), bar);
        }
    };
#pragma unroll 4
    for (int i = tid; i < rc.n >> 2; i += kFullThreads) {
        const float4 x = reinterpret_cast<const float4*>(rc.vals)[i];
        unsigned hits = (near(x.x) ? 1u : 0u) | (near(x.y) ? 2u : 0u) | (near(x.z) ? 4u : 0u) | (near(x.w) ? 8u : 0u);
        while (hits) {
            const int e = __ffs(hits) - 1;
            hits &= hits - 1u;
            look(e == 0 ? x.x : e == 1 ? x.y : e == 2 ? x.z : x.w, 4 * i + e);
        }
    }
    for (int i = (rc.n & ~3) + tid; i < rc.n; i += kFullThreads) look(rc.vals[i], i);
    __syncthreads();
    if (tid == 0) inbox_put(map_to_rank(&sh->counts[rank], 0u), (u64)(unsigned)sh->sent, map_to_rank(&sh->in_counts, 0u));
    if (rank != 0) return __syncthreads_or(!inbox_wait(&sh->in_verdict)) ? -1 : sh->verdict != 0ull ? 1 : 0;
    const bool counted = inbox_wait(&sh->in_counts);
    bool fits = true;
    unsigned words = 0u;
#pragma unroll
    for (int r = 0; r < C; ++r) {
        const unsigned n = (unsigned)sh->counts[r];
        fits = fits && n <= (unsigned)kSendCap;
        words += min(n, (unsigned)kSendCap);
        if (tid == r) sh->got[par][r] = n;
    }
    if (tid == 0 && counted) inbox_expect(&sh->in_list, 8u * words);
    if (!counted || !inbox_wait(&sh->in_list)) sh->late = 1;   // (also what is of no use: the lists' memory may be needed for a descent)
    __syncthreads();
    if (sh->late) return -1;
    if (tid > 0 && tid < C) inbox_put(map_to_rank(&sh->verdict, (unsigned)tid), fits ? 1ull : 0ull, map_to_rank(&sh->in_verdict, (unsigned)tid));
    return fits ? 1 : 0;
}

// What the first CTA does with the lists that send_bins left there takes T threads: 256 of them, one candidate each, if
// there are at most kShort (eight warps get through the barriers faster than sixteen), else all.
template <int T>
__device__ __forceinline__ void list_sync() { block_sync<T, T == kFullThreads ? 0 : 1>(); }

// Orders the lists: one list, largest first, at the returned address; `n` entries.
template <int C, int T>
__device__ __forceinline__ u64* order_lists(FullShared* sh, int use, int n) {
    const int tid = threadIdx.x, lane = tid & 31;
    u64* list = sh->list();
    u64* spare = list + kMaxCluster * kSendCap;
    constexpr int kPer = T == kFullThreads ? kMaxCluster * kSendCap / kFullThreads : 1;
    int off[C + 1];
    off[0] = 0;
#pragma unroll
    for (int r = 0; r < C; ++r) off[r + 1] = off[r] + (int)sh->got[use][r];
    u64 c[kPer];
#pragma unroll
    for (int q = 0; q < kPer; ++q) {
        const int e = q * T + tid;
        int from = 0;
#pragma unroll
        for (int r = 0; r < C; ++r) from = e >= off[r] ? r * kSendCap + e - off[r] : from;
        c[q] = e < n ? list[from] : 0ull;
    }
    list_sync<T>();
    if (T != kFullThreads) {   // ranks by counting: four lanes for an entry, two entries per read
        const int n8 = (n + 7) & ~7;
        if (tid < n8) list[tid] = c[0];
        list_sync<T>();
        const int part = tid & 3;
        for (int e0 = 0; e0 < n; e0 += T / 4) {
            const int e = e0 + (tid >> 2);
            if (e0 + ((tid & ~31) >> 2) >= n) break;   // (whole warps)
            const u64 mine = e < n ? list[e] : 0ull;
            int larger = 0;
#pragma unroll 4
            for (int j = 2 * part; j < n8; j += 8) {
                const ulonglong2 v = *reinterpret_cast<const ulonglong2*>(list + j);
                larger += (v.x > mine ? 1 : 0) + (v.y > mine ? 1 : 0);
            }
            larger += __shfl_xor_sync(0xffffffffu, larger, 1);
            larger += __shfl_xor_sync(0xffffffffu, larger, 2);
            if (part == 0 && e < n) spare[larger] = mine;
        }
        list_sync<T>();
        return spare;
    }
    if (n <= 2 * kFullThreads) {   // two runs of 32 per warp, ordered across the lanes; then the places of an entry in all runs
        const int runs = (n + 31) >> 5;
#pragma unroll
        for (int q = 0; q < 2; ++q) {
            if (q * kFullWarps + (tid >> 5) >= runs) continue;   // (whole warps)
#pragma unroll
            for (int k = 2; k <= 32; k <<= 1) {
#pragma unroll
                for (int j = k >> 1; j > 0; j >>= 1) {
                    const u64 o = __shfl_xor_sync(0xffffffffu, c[q], j);
                    c[q] = (((lane & k) == 0) == ((lane & j) == 0)) ? max(c[q], o) : min(c[q], o);
                }
            }
            list[q * kFullThreads + tid] = c[q];
        }
        __syncthreads();
        int rank[2] = {lane, lane};
#pragma unroll
        for (int p = 0; p < 2; ++p) {
            if (c[p] == 0ull) continue;
#pragma unroll 4
            for (int q = 0; q < runs; ++q) {
                const u64* run = list + 32 * q;
                int lo = 0;   // entries of the run above this one (0 .. 32)
#pragma unroll
                for (int st = 16; st > 0; st >>= 1)
                    if (run[lo + st - 1] > c[p]) lo += st;
                if (run[lo] > c[p]) lo += 1;
                rank[p] += q == p * kFullWarps + (tid >> 5) ? 0 : lo;
            }
        }
        __syncthreads();
#pragma unroll
        for (int p = 0; p < 2; ++p)
            if (c[p] != 0ull) list[rank[p]] = c[p];
        __syncthreads();
        return list;
    }
    int m = 4 * kFullThreads;
    while (m < n) m <<= 1;
#pragma unroll
    for (int q = 0; q < kPer; ++q)
        if (q * T + tid < m) list[q * T + tid] = c[q];
    for (int k = 2; k <= m; k <<= 1)   // bitonic, descending
        for (int j = k >> 1; j > 0; j >>= 1) {
            __syncthreads();
            for (int i = tid; i < m / 2; i += T) {
                const int lo = ((i & ~(j - 1)) << 1) | (i & (j - 1)), up = lo | j;
                const u64 x = list[lo], y = list[up];
                if ((x < y) == ((lo & k) == 0)) {
                    list[lo] = y;
                    list[up] = x;
                }
            }
        }
    __syncthreads();
    return list;
}

// Cumulative weights of the ordered list: every thread looks after up to four consecutive entries (`per` of them: fewer if
// the list is short).  Contains barriers.
template <int T>
struct ListScan {
    static constexpr int kPer = T == kFullThreads ? kMaxCluster * kSendCap / kFullThreads : 1;
    U128 before;     // weight before the thread's first entry
    u64 w[kPer];
    int per;
    // calls f(entry, weight before it, weight with it) for the thread's entries of the n
    template <class F>
    __device__ __forceinline__ void each(int n, F f) const {
        U128 cum = before;
#pragma unroll
        for (int q = 0; q < kPer; ++q) {
            const int e = (int)threadIdx.x * per + q;
            if (q < per && e < n) {
                const U128 with = u128_add(cum, U128{0ull, w[q]});
                f(e, cum, with);
                cum = with;
            }
        }
    }
};
template <int T>
__device__ __forceinline__ ListScan<T> scan_list(const RowCtx& rc, FullShared* sh, const u64* srt, int n, U128 above) {
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    ListScan<T> ls;
    ls.per = ListScan<T>::kPer == 1 ? 1 : (n + T - 1) / T;
    u64 lo = 0ull, hi = 0ull;
#pragma unroll
    for (int q = 0; q < ListScan<T>::kPer; ++q) {
        const int e = tid * ls.per + q;
        const Weight w = q < ls.per && e < n ? rc.weight(comp_value(srt[e])) : Weight{0u, 0};
        ls.w[q] = w.value();
        lo += (u64)(long long)w.down;
        hi += w.up;
    }
    u64 ilo = lo, ihi = hi;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const u64 l = __shfl_up_sync(0xffffffffu, ilo, o), h = __shfl_up_sync(0xffffffffu, ihi, o);
        if (lane >= o) {
            ilo += l;
            ihi += h;
        }
    }
    u64 wl = 0ull, wh = 0ull;
    if (n > 32) {
        list_sync<T>();
        if (lane == 31) {
            sh->red[warp] = ilo;
            sh->red_hi[warp] = ihi;
        }
        list_sync<T>();
        wl = lane < warp ? sh->red[lane] : 0ull;
        wh = lane < warp ? sh->red_hi[lane] : 0ull;
#pragma unroll
        for (int o = 16; o; o >>= 1) {
            wl += __shfl_xor_sync(0xffffffffu, wl, o);
            wh += __shfl_xor_sync(0xffffffffu, wh, o);
        }
    }
    ls.before = u128_add(above, join_parts(wl + ilo - lo, wh + ihi - hi));
    return ls;
}

// The first CTA's share of resolve(): the crossing among the candidates it was sent goes to every CTA of the cluster.
template <int C, int T>
__device__ __forceinline__ void cross_list(const RowCtx& rc, FullShared* sh, int use, int n, U128 target, U128 above, bool count) {
    u64 cnt = 0ull;
    if (count) {
#pragma unroll
        for (unsigned r = 0; r < (unsigned)C; ++r) cnt += ld_cluster_u64(map_to_rank(&sh->x_small[use][2], r));
    }
    const u64* srt = order_lists<C, T>(sh, use, n);
    const ListScan<T> ls = scan_list<T>(rc, sh, srt, n, above);
    ls.each(n, [&](int e, U128 before, U128 with) {
        if (u128_ge(with, target) && (!u128_ge(before, target) || e == 0)) {
#pragma unroll
            for (unsigned r = 0; r < (unsigned)C; ++r) {
                cluster_store_u64(map_to_rank(&sh->cross[0], r), srt[e]);
                cluster_store_u64(map_to_rank(&sh->cross[1], r), before.lo);
                cluster_store_u64(map_to_rank(&sh->cross[2], r), before.hi);
                cluster_store_u64(map_to_rank(&sh->cross[3], r), cnt + (u64)e);
                cluster_store_u64(map_to_rank(&sh->cross[4], r), 1ull);
            }
        }
    });
}
template <int C>
__device__ __forceinline__ int listed(const FullShared* sh, int use) {
    int n = 0;
#pragma unroll
    for (int r = 0; r < C; ++r) n += (int)sh->got[use][r];
    return n;
}

// The end of a row all of whose candidates that can be kept are in the first CTA's lists: min-p, top-p, draw, record.
struct RowCuts {
    U128 target_p;
    double u, sum, min_thr;
    bool top_p, min_p;
};
template <int C, int T>
__device__ __forceinline__ int finish_list(const RowCtx& rc, FullShared* sh, int use, int n, const RowCuts& cuts, const FullArgs& a, int out) {
    const int tid = threadIdx.x;
    if (tid == 0) {
        sh->first_p = 0x7fffffff;
        sh->first_u = 0x7fffffff;
    }
    const u64* srt = order_lists<C, T>(sh, use, n);
    const ListScan<T> ls = scan_list<T>(rc, sh, srt, n, U128{0ull, 0ull});
    ls.each(n, [&](int e, U128 before, U128 with) {
        if (cuts.top_p && u128_ge(with, cuts.target_p) && !u128_ge(before, cuts.target_p)) atomicMin(&sh->first_p, e + 1);
        if (cuts.min_p && rc.probability(comp_value(srt[e]), cuts.sum) < cuts.min_thr) atomicMin(&sh->first_p, max(e, 1));
    });
    list_sync<T>();
    const int keep = min(sh->first_p, n);
    ls.each(keep, [&](int e, U128, U128 with) {
        if (e == keep - 1) {
            sh->kw_lo = with.lo;
            sh->kw_hi = with.hi;
        }
    });
    list_sync<T>();
    const U128 target = double_to_u128_ceil(__dmul_rn(cuts.u, u128_to_double(U128{sh->kw_hi, sh->kw_lo})));
    ls.each(keep, [&](int e, U128, U128 with) {
        if (u128_ge(with, target)) atomicMin(&sh->first_u, e);
        if (a.record && e < kMaxK) {
            a.kept_ids[(size_t)out * kMaxK + e] = comp_id(srt[e]);
            a.kept_pr[(size_t)out * kMaxK + e] = rc.probability(comp_value(srt[e]), cuts.sum);
        }
    });
    list_sync<T>();
    if (a.record && tid == 0) a.kept_n[out] = keep;
    return comp_id(srt[min(sh->first_u, keep - 1)]);   // (a target beyond the list, by rounding, takes the last)
}

// The end of a row whose first CTA has the candidates of the bins that the draw may fall into and of those where the kept set may
// end: the cut, the weight of the kept set, the draw.
template <int C, int T>
__device__ __forceinline__ int finish_bins(const RowCtx& rc, FullShared* sh, int use, int n) {
    const RowPlan& ends = sh->plan;
    const int tid = threadIdx.x;
    const bool cut = ends.cut_hi >= ends.cut_lo;
    const U128 above = cut ? sh->weight_to(ends.cut_lo - 1) : ends.S;   // the kept set if it ends before the cut's bins
    if (tid == 0) {
        sh->first_p = 0x7fffffff;
        sh->first_u = 0x7fffffff;
        sh->kw_lo = above.lo;
        sh->kw_hi = above.hi;
    }
    const u64* srt = order_lists<C, T>(sh, use, n);
    const ListScan<T> ls = scan_list<T>(rc, sh, srt, n, sh->weight_to(ends.draw_lo - 1));
    // what lies between the two ranges is not in the list
    const U128 gap = cut ? u128_sub(sh->weight_to(max(ends.cut_lo - 1, ends.draw_hi)), sh->weight_to(ends.draw_hi)) : U128{0ull, 0ull};
    list_sync<T>();
    if (cut) {
        ls.each(n, [&](int e, U128 before, U128 with) {
            const float x = comp_value(srt[e]);
            const int b = rc.bin(x);
            if (b < ends.cut_lo) return;
            if (b > ends.draw_hi) {
                before = u128_add(before, gap);
                with = u128_add(with, gap);
            }
            if (ends.top_p && u128_ge(with, ends.target_p) && !u128_ge(before, ends.target_p)) atomicMin(&sh->first_p, e + 1);
            if (ends.min_p && rc.probability(x, ends.sum) < ends.min_thr) atomicMin(&sh->first_p, e);
        });
        list_sync<T>();
    }
    const int keep = min(sh->first_p, n);
    if (cut) {
        ls.each(keep, [&](int e, U128, U128 with) {
            const int b = rc.bin(comp_value(srt[e]));
            if (e != keep - 1 || b < ends.cut_lo) return;
            if (b > ends.draw_hi) with = u128_add(with, gap);
            sh->kw_lo = with.lo;
            sh->kw_hi = with.hi;
        });
        list_sync<T>();
    }
    const U128 kept{sh->kw_hi, sh->kw_lo};
    U128 target = double_to_u128_ceil(__dmul_rn(ends.u, u128_to_double(kept)));
    if (!u128_ge(kept, target)) target = kept;   // (beyond it by rounding: the last one)
    ls.each(keep, [&](int e, U128, U128 with) {
        if (rc.bin(comp_value(srt[e])) > ends.draw_hi) with = u128_add(with, gap);
        if (u128_ge(with, target)) atomicMin(&sh->first_u, e);
    });
    list_sync<T>();
    return comp_id(srt[max(0, min(sh->first_u, keep - 1))]);
}

// The candidate at which the cumulative weight reaches `target`; every CTA gets it.  Bins if they are of use, else a descent.
// `count`: the number of candidates before it is wanted.
template <int C>
__device__ __noinline__ Crossing resolve(const RowCtx rc, FullShared* sh, unsigned rank, bool binned, bool count, u64 floor_c, u64 top_c, U128 target, int& par) {
    const int tid = threadIdx.x;
    if (binned) {
        const int bin = find_bin(sh, target);
        if (tid == 0) sh->cross[4] = 0ull;
        const bool fits = send_bins<C>(rc, sh, rank, bin, bin, count, par);
        if (fits) {
            if (rank == 0) {
                const int n = listed<C>(sh, par);
                const U128 above = sh->weight_to(bin - 1);
                if (n > kShort) cross_list<C, kFullThreads>(rc, sh, par, n, target, above, count);
                else if (tid < kShort) cross_list<C, kShort>(rc, sh, par, n, target, above, count);
            }
            par ^= 1;
            cluster_sync_all();
            return Crossing{sh->cross[0], U128{sh->cross[2], sh->cross[1]}, (unsigned)sh->cross[3], sh->cross[4] != 0ull};
        }
        par ^= 1;
    }
    return cluster_descent<C>(rc, sh, floor_c, top_c, target, false, par);
}

// What a CTA does whose wait has run out, and those of its row that learn of it: the row is reported and gets token 0, nothing that
// was waited for is used.  `tell`: the others learn of it at their next look at `gone` - all of them are still there, since none leaves the
// kernel without a word from this CTA that it has not given, or its arrival at a barrier.  Then the CTA keeps to the cluster's barriers until
// the others have left or do the same (the barrier does not count threads that have exited; kMostBarriers is more than a row has between
// its last wait for a word and its look at `gone`: nine of a descent, two for the sums, one before the look): its memory is there for whoever
// reads it or stores to it.
constexpr int kMostBarriers = 32;
struct RowOutputs {   // (by value: the address of a kernel's argument would put a copy of all of them in local memory)
    unsigned *status, *status_host;
    int32_t *tokens, *tokens_host, *append_at, *kept_n;
    int out;
};
template <int C>
__device__ __noinline__ void step_aside(FullShared* sh, unsigned rank, bool tell, bool copying, const RowOutputs o) {
    const int tid = threadIdx.x;
    if (tid == 0) report_status(o.status, o.status_host, kStatusLate);
    if (tell && tid < C) cluster_store_u32(map_to_rank(&sh->gone, (unsigned)tid), 1u);
    for (int i = 0; i < kMostBarriers; ++i) {
        __syncwarp();
        cluster_sync_all();
    }
    if (copying) inbox_wait(&sh->in_slice);   // (a copy that is still on its way)
    if (rank == 0 && tid == 0) {
        if (o.kept_n) o.kept_n[o.out] = 0;
        if (o.append_at) *o.append_at = 0;
        put_token(o.tokens, o.tokens_host, o.out, 0);
    }
}

template <int C>
__global__ void __launch_bounds__(kFullThreads, 1) full_row_kernel(const FullArgs a, int cache_slice) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    FullShared* sh = reinterpret_cast<FullShared*>(smem_raw);
    const int tid = threadIdx.x;
    const unsigned rank = cluster_rank();
    const RowDesc d = a.rows[blockIdx.x / C];
    const int V = a.n_vocab;
    // the slices: equal runs of columns, a multiple of four each
    // (from the row's first 16-byte boundary on, so that they can be copied in one piece; the columns before it belong to the first CTA)
    const float* row = a.logits + d.logits_off;
    const bool shifted = cache_slice && V >= kShiftedFrom;
    const int head = shifted ? (int)((0u - ((unsigned)reinterpret_cast<uintptr_t>(row) >> 2)) & 3u) : 0;
    const int per = (((V - head + C - 1) / C) + 3) & ~3;
    const int lo = min(V, head + (int)rank * per), main = min(V, lo + per) - lo, n = main + (rank == 0 ? head : 0);
    unsigned* bitmap = reinterpret_cast<unsigned*>(smem_raw + sizeof(FullShared));
    float* vals = reinterpret_cast<float*>(smem_raw + sizeof(FullShared) + (size_t)((per + 3 + 31) / 32) * sizeof(unsigned));
    vals = reinterpret_cast<float*>(((uintptr_t)vals + 15) & ~(uintptr_t)15);
    const int id_base = a.vocab_offset;
    int par = 0;
#define FTR(n)                                                                                   \
    do {                                                                                         \
        if (a.trace && blockIdx.x == gridDim.x - C && tid == 0) a.trace[(n)] = global_timer_ns(); \
    } while (0)
    FTR(0);
    constexpr int kMine = (kBins + C - 1) / C;   // bins that a CTA adds up (six CTAs: 171, and C * kMine is two more than there are threads)
    static_assert(C * kMine <= kBins + 8, "the parts' memory");
    if (tid == 0) {
        for (u64* bar : {&sh->in_slice, &sh->in_extremes, &sh->in_parts, &sh->in_sums, &sh->in_counts, &sh->in_list, &sh->in_verdict}) inbox_init(bar);
        inbox_inits_fence();
        inbox_expect(&sh->in_extremes, 16u * C);
        inbox_expect(&sh->in_parts, 16u * C * (unsigned)max(0, min(kMine, kBins - (int)rank * kMine)));
        inbox_expect(&sh->in_sums, 16u * kBins);
        inbox_expect(&sh->in_counts, 8u * C);
        inbox_expect(&sh->in_verdict, 8u);
        sh->sent = 0;
        sh->late = 0;
        sh->gone = 0u;
    }
    if (tid == 32) {   // (while the first loads are on their way)
        double w = __dmul_rn(__ull2double_rn(d.rng_word), 5.42101086242752217003726400434970855712890625e-20);   // 2^-64
        if (w >= 1.0) w = __longlong_as_double(0x3FEFFFFFFFFFFFFFll);
        sh->plan.u = w;
        sh->plan.below = d.min_p > 0.0f ? (double)d.temperature * log((double)d.min_p) : 0.0;
    }
    cluster_arrive_relaxed();   // (waited for before the first access to another CTA's shared memory)
    if (tid < 64) sh->table[tid] = exp2((double)tid / 64.0);

    // ---- 0. the slice as the sampler sees it: softcap, penalty, optional write-back
    const int n4 = (reinterpret_cast<uintptr_t>(row + lo) & 15u) == 0 ? main >> 2 : 0;
    const bool has_pen = (d.flags & kRowPenalty) != 0;
    const int32_t* const window = a.hist + d.hist_begin;
    const int n_drafts = has_pen ? d.flags >> kRowDraftShift : 0, window_len = has_pen ? d.hist_len + n_drafts : 0, words = (n + 31) >> 5;
    auto window_id = [&](int i) { return i < d.hist_len ? window[i] : a.drafts[d.draft_off + i - d.hist_len]; };
    RowCtx rc{nullptr, row, has_pen ? bitmap : nullptr, d.penalty, a.softcap, lo, main, n, id_base, 0.0f, (double)d.temperature, 0.0, -45.0f * d.temperature, false, sh->table, 0ull, 0.0f};
    const float ninf = -__int_as_float(0x7f800000);
    float mx = ninf, mn = -ninf;
    unsigned valid = 0u;
    auto take = [&](float x, int i, bool hit) {   // logit i of the slice as loaded: transform, note the extremes, write back
        if (a.softcap != 0.0f) x = __fmul_rn(a.softcap, tanhf(__fdiv_rn(x, a.softcap)));
        if (hit) x = x > 0.0f ? __fdiv_rn(x, d.penalty) : __fmul_rn(x, d.penalty);
        mx = fmaxf(mx, x);   // (NaNs take no part)
        mn = fminf(mn, x);
        valid += x == x ? 1u : 0u;
        if (a.write_back && (a.softcap != 0.0f || hit)) const_cast<float*>(row)[lo + i] = x;
        return x;
    };
    const bool copied = cache_slice && n4 > 0;
    auto aside = [&](bool tell) {
        step_aside<C>(sh, rank, tell, copied,
                      RowOutputs{a.status, a.status_host, a.tokens, a.tokens_host, d.flags & kRowAppend ? a.pool + d.hist_begin + d.hist_len : nullptr, a.record ? a.kept_n : nullptr, d.out_index});
    };
    if (copied) {
        // The usual way, a slice on a 16-byte boundary: one bulk copy, and the penalty where the window says so.  (Loads and stores by all threads, with a
        // look at the window's bits for every logit: 5.7 us for 21848 logits, this way 2.3.)
        if (tid == 0) {
            inbox_expect(&sh->in_slice, 16u * (unsigned)n4);
            bulk_copy(vals, row + lo, 16u * (unsigned)n4, &sh->in_slice);
        }
        int id = tid < window_len ? window_id(tid) : 0;
        if (has_pen)
            for (int i = tid; i < words; i += kFullThreads) bitmap[i] = 0u;
        auto column = [&](int i) { return i < main ? lo + i : i - main; };
        for (int i = 4 * n4 + tid; i < n; i += kFullThreads) vals[i] = __ldcs(row + column(i));
        __syncthreads();   // (the barriers are initialised)
        if (!inbox_wait(&sh->in_slice)) sh->late = 1;
        __syncthreads();
        if (sh->late) {
            cluster_wait_acquire();
            aside(true);
            return;
        }
        if (a.softcap != 0.0f) {
            for (int i = tid; i < n; i += kFullThreads) {
                const float x = __fmul_rn(a.softcap, tanhf(__fdiv_rn(vals[i], a.softcap)));
                vals[i] = x;
                if (a.write_back) const_cast<float*>(row)[column(i)] = x;
            }
            __syncthreads();
        }
        if (has_pen) {
            for (int i = tid; i < window_len; i += kFullThreads) {
                if (i != tid) id = window_id(i);
                const int col = id - id_base;
                if (col < 0 || col >= V) continue;   // (and no overflow)
                const int c = col >= lo && col < lo + main ? col - lo : rank == 0 && col < head ? main + col : -1;
                if (c < 0) continue;
                const unsigned bit = 1u << (c & 31);
                if (atomicOr(&bitmap[c >> 5], bit) & bit) continue;   // an id counts once however often it occurs
                const float x = vals[c], y = x > 0.0f ? __fdiv_rn(x, d.penalty) : __fmul_rn(x, d.penalty);
                vals[c] = y;
                if (a.write_back) const_cast<float*>(row)[col] = y;
            }
            __syncthreads();
        }
        auto seen = [&](float x) {   // (NaNs take no part)
            mx = fmaxf(mx, x);
            mn = fminf(mn, x);
            valid += x == x ? 1u : 0u;
        };
#pragma unroll 4
        for (int i = tid; i < n4; i += kFullThreads) {
            const float4 x = reinterpret_cast<const float4*>(vals)[i];
            seen(x.x);
            seen(x.y);
            seen(x.z);
            seen(x.w);
        }
        for (int i = 4 * n4 + tid; i < n; i += kFullThreads) seen(vals[i]);
    } else {
        // anything else by loads, and the window's columns in a bitmap
        if (has_pen) {
            for (int i = tid; i < words; i += kFullThreads) bitmap[i] = 0u;
            __syncthreads();
            for (int i = tid; i < window_len; i += kFullThreads) {
                const int c = window_id(i) - id_base - lo;
                if (c >= 0 && c < n) atomicOr(&bitmap[c >> 5], 1u << (c & 31));
            }
            __syncthreads();
        }
        for (int i0 = 0; i0 < n; i0 += 8 * kFullThreads) {   // what is left, or a row that does not lie on 16-byte boundaries
            float y[8];
#pragma unroll
            for (int u = 0; u < 8; ++u) {
                const int i = i0 + u * kFullThreads + tid;
                y[u] = i < n ? __ldcs(row + lo + i) : 0.0f;
            }
#pragma unroll
            for (int u = 0; u < 8; ++u) {
                const int i = i0 + u * kFullThreads + tid;
                if (i < n) {
                    const float x = take(y[u], i, has_pen && ((bitmap[i >> 5] >> (i & 31)) & 1u));
                    if (cache_slice) vals[i] = x;
                }
            }
        }
    }
    if (cache_slice) {
        rc.vals = vals;
    } else if (a.write_back) {   // the row in memory now holds the transformed values: read it as final
        __syncthreads();
        rc.bitmap = nullptr;
        rc.cap = 0.0f;
    }
    FTR(1);
    // ---- 1. the row's extremes and its number of logits
    {
        const int lane = tid & 31, warp = tid >> 5;
        unsigned kx = __reduce_max_sync(0xffffffffu, float_key(mx)), kn = __reduce_min_sync(0xffffffffu, float_key(mn));
        unsigned cnt = __reduce_add_sync(0xffffffffu, valid);
        if (lane == 0) {
            sh->red[warp] = ((u64)kx << 32) | kn;
            sh->red_cnt[warp] = cnt;
        }
        __syncthreads();
        cluster_wait_acquire();
        if (warp == 0) {
            const u64 both = lane < kFullWarps ? sh->red[lane] : 0xFFFFFFFFull;
            kx = __reduce_max_sync(0xffffffffu, (unsigned)(both >> 32));
            kn = __reduce_min_sync(0xffffffffu, (unsigned)both);
            cnt = __reduce_add_sync(0xffffffffu, lane < kFullWarps ? sh->red_cnt[lane] : 0u);
            if (lane < C) {   // one lane per CTA of the cluster tells it
                const unsigned bar = map_to_rank(&sh->in_extremes, (unsigned)lane);
                inbox_put(map_to_rank(&sh->extremes[0][rank], (unsigned)lane), ((u64)kx << 32) | kn, bar);
                inbox_put(map_to_rank(&sh->extremes[1][rank], (unsigned)lane), (u64)cnt, bar);
            }
        }
        if (!inbox_wait(&sh->in_extremes)) sh->late = 1;
        __syncthreads();
        if (sh->late) {
            aside(true);
            return;
        }
        kx = 0u;
        kn = ~0u;
        valid = 0u;
#pragma unroll
        for (int r = 0; r < C; ++r) {
            kx = max(kx, (unsigned)(sh->extremes[0][r] >> 32));
            kn = min(kn, (unsigned)sh->extremes[0][r]);
            valid += (unsigned)sh->extremes[1][r];
        }
        mx = key_float(kx);
        mn = key_float(kn);
    }
    // bounds of the candidates' composites, for the descents
    const u64 cmax = ((u64)float_key(mx) << 32) | 0xFFFFFFFFull, cmin = (u64)float_key(mn) << 32;
    const int out = d.out_index;
    auto finish = [&](int token) {   // one thread: the row's token to wherever it is wanted
        if (d.flags & kRowAppend) a.pool[d.hist_begin + d.hist_len] = token;
        put_token(a.tokens, a.tokens_host, out, token);
    };
    if (valid == 0u) {   // nothing but NaNs
        if (rank == 0 && tid == 0) {
            report_status(a.status, a.status_host, kStatusEmptyRow);
            a.kept_n[out] = 0;
            finish(0);
        }
        __syncwarp();
        cluster_sync_all();   // (a CTA that steps aside may still tell this one)
        return;
    }
    rc.mx = mx;
    rc.inv_temp = __ddiv_rn(1.0, rc.temp);
    rc.odd = !(mx < -ninf && mx > ninf) || d.temperature > 1e36f;
    FTR(2);

    // ---- 2. the k-th candidate (k < n only)
    u64 c_k = cmin;
    if (d.k < V) {
        const Crossing ck = cluster_descent<C>(rc, sh, 0ull, cmax, U128{0ull, (u64)d.k}, true, par);
        if (ck.found) c_k = rc.floor_c = max(cmin, ck.c);
    }
    FTR(3);
    // ---- 3. the weights' exact sum, the number of candidates, and the histogram
    // (a row whose largest logit is infinite, or that is too long for shared memory, is left to the descents)
    const float inf = -ninf;
    const bool binned = rc.vals != nullptr && !rc.odd;
    // What lies further down than kBinned temperatures - most of a row, often - is one bin, added up in registers: the other bins are
    // narrow, and a crossing's list short.  A cumulative weight that is reached there (all of it weighs less than 2^-28 of the largest per
    // logit, 1 part in 1000 of a row of 262144 at the most) is resolved by a descent.
    rc.bin_scale = (float)(kBins - 1) / fminf(kBinned * d.temperature, mx - mn);
    if (!(rc.bin_scale < inf)) rc.bin_scale = 0.0f;
    U128 S;
    const unsigned n_cand = rc.floor_c != 0ull ? (unsigned)d.k : valid;
    if (binned) {
#pragma unroll
        for (int l = 0; l < kLimbs * kBinsEach; ++l) (&sh->hist[0][0])[l * kFullThreads + tid] = 0u;
        u64 rest_lo = 0ull, rest_hi = 0ull;   // of the last bin
        __syncthreads();
        auto add = [&](float x, u64 w) {
            const int b = rc.bin(x);
            const unsigned lo = (unsigned)w, hi = (unsigned)(w >> 32);
            if (b < kBins - 1) {
                unsigned* h = &sh->hist[0][b];
                atomicAdd(h, lo & 0xFFFFu);
                atomicAdd(h + kBins, lo >> 16);
                atomicAdd(h + 2 * kBins, hi & 0xFFFFu);
                if (hi >> 16) atomicAdd(h + 3 * kBins, hi >> 16);
            } else {
                rest_lo += lo;
                rest_hi += hi;
            }
        };
        for (int i = tid; i < n >> 2; i += kFullThreads) {
            const float4 v = reinterpret_cast<const float4*>(rc.vals)[i];
            float x[4] = {v.x, v.y, v.z, v.w};
            if (rc.floor_c != 0ull) {
#pragma unroll
                for (int e = 0; e < 4; ++e) x[e] = rc.is_candidate(x[e], 4 * i + e) ? x[e] : ninf;
            }
            u64 w[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) w[e] = rc.weight(x[e]).value();
#pragma unroll
            for (int e = 0; e < 4; ++e) add(x[e], w[e]);
        }
        for (int i = (n & ~3) + tid; i < n; i += kFullThreads)
            if (rc.is_candidate(rc.vals[i], i)) add(rc.vals[i], rc.weight(rc.vals[i]).value());
        const int lane = tid & 31, warp = tid >> 5;
        {   // the last bin
#pragma unroll
            for (int o = 16; o; o >>= 1) {
                rest_lo += __shfl_xor_sync(0xffffffffu, rest_lo, o);
                rest_hi += __shfl_xor_sync(0xffffffffu, rest_hi, o);
            }
            if (lane == 0) {
                sh->red[warp] = rest_lo;
                sh->red_hi[warp] = rest_hi;
            }
        }
        __syncthreads();
        // Every CTA adds up kMine of the bins, from what the others send it, and sends the sums to all: a thread looks after one bin of
        // its CTA, then after a bin and the CTA that its sum goes to.
        {
            u64 r0 = 0ull, r1 = 0ull;
            if (warp == kFullWarps - 1) {
                r0 = lane < kFullWarps ? sh->red[lane] : 0ull;
                r1 = lane < kFullWarps ? sh->red_hi[lane] : 0ull;
#pragma unroll
                for (int o = 16; o; o >>= 1) {
                    r0 += __shfl_xor_sync(0xffffffffu, r0, o);
                    r1 += __shfl_xor_sync(0xffffffffu, r1, o);
                }
            }
#pragma unroll
            for (int q = 0; q < kBinsEach; ++q) {
                const int bin = q * kFullThreads + tid;
                u64 p0 = (u64)sh->hist[0][bin] + ((u64)sh->hist[1][bin] << 16), p1 = (u64)sh->hist[2][bin] + ((u64)sh->hist[3][bin] << 16);
                if (bin == kBins - 1) {
                    p0 += r0;
                    p1 += r1;
                }
                const unsigned owner = (unsigned)(bin / kMine), at = rank * kMine + (unsigned)(bin % kMine), bar = map_to_rank(&sh->in_parts, owner);
                inbox_put(map_to_rank(&sh->part[0][at], owner), p0, bar);
                inbox_put(map_to_rank(&sh->part[1][at], owner), p1, bar);
            }
        }
        const bool parts = inbox_wait(&sh->in_parts);
        if (!parts) sh->late = 1;
        for (int t = tid; parts && t < C * kMine; t += kFullThreads) {
            const int dst = t / kMine, bin = (int)rank * kMine + t % kMine;
            if (bin >= kBins) continue;
            u64 c0 = 0ull, c1 = 0ull;
#pragma unroll
            for (int r = 0; r < C; ++r) {
                c0 += sh->part[0][r * kMine + t % kMine];
                c1 += sh->part[1][r * kMine + t % kMine];
            }
            const unsigned bar = map_to_rank(&sh->in_sums, (unsigned)dst);
            inbox_put(map_to_rank(&sh->cum[0][bin], (unsigned)dst), c0, bar);
            inbox_put(map_to_rank(&sh->cum[1][bin], (unsigned)dst), c1, bar);
        }
        if (!inbox_wait(&sh->in_sums)) sh->late = 1;
        // inclusive sums over the bins, largest logits first
        u64 own0[kBinsEach], own1[kBinsEach], c0 = 0ull, c1 = 0ull;
        unsigned own_est[kBinsEach], est = 0u;
#pragma unroll
        for (int q = 0; q < kBinsEach; ++q) {   // (consecutive ones)
            const int bin = kBinsEach * tid + q;
            const u64 w0 = sh->cum[0][bin], w1 = sh->cum[1][bin];
            own0[q] = c0 += w0;
            own1[q] = c1 += w1;
            own_est[q] = est += estimated_count(rc, bin, (w1 << 1) + (w0 >> 31));
        }
        const u64 mine0 = c0, mine1 = c1;
        const unsigned mine_est = est;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const u64 t0 = __shfl_up_sync(0xffffffffu, c0, o), t1 = __shfl_up_sync(0xffffffffu, c1, o);
            const unsigned e = __shfl_up_sync(0xffffffffu, est, o);
            if (lane >= o) {
                c0 += t0;
                c1 += t1;
                est += e;
            }
        }
        if (lane == 31) {   // (red was last read before this CTA's parts went out)
            sh->red[warp] = c0;
            sh->red_hi[warp] = c1;
            sh->red_cnt[warp] = est;
        }
        __syncthreads();
        if (sh->late) {
            aside(true);
            return;
        }
        u64 t0 = lane < warp ? sh->red[lane] : 0ull, t1 = lane < warp ? sh->red_hi[lane] : 0ull;
        est += __reduce_add_sync(0xffffffffu, lane < warp ? sh->red_cnt[lane] : 0u);
#pragma unroll
        for (int o = 16; o; o >>= 1) {
            t0 += __shfl_xor_sync(0xffffffffu, t0, o);
            t1 += __shfl_xor_sync(0xffffffffu, t1, o);
        }
#pragma unroll
        for (int q = 0; q < kBinsEach; ++q) {
            const int bin = kBinsEach * tid + q;
            sh->cum[0][bin] = c0 - mine0 + t0 + own0[q];
            sh->cum[1][bin] = c1 - mine1 + t1 + own1[q];
            sh->cum_n[bin] = est - mine_est + own_est[q];
        }
        __syncthreads();
        S = sh->weight_to(kBins - 1);
    } else {
        u64 wl = 0ull, wh = 0ull;   // sums of the weights' lower and upper parts
        for (int i = 4 * tid; i < n; i += 4 * kFullThreads) {
            float x[4];
            load4(rc, i, x);
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const Weight w = rc.weight(rc.floor_c == 0ull || rc.is_candidate(x[e], i + e) ? x[e] : ninf);
                wl += (u64)(long long)w.down;
                wh += w.up;
            }
        }
        block_sums(sh, par, wl, wh, 0u);
        cluster_sync_all();
        if (tid < C * 4) sh->x_all[par][tid] = ld_cluster_u64(map_to_rank(&sh->x_small[par][tid & 3], (unsigned)tid >> 2));
        __syncthreads();
        wl = wh = 0ull;
#pragma unroll
        for (int r = 0; r < C; ++r) {
            wl += sh->x_all[par][4 * r];
            wh += sh->x_all[par][4 * r + 1];
        }
        S = join_parts(wl, wh);
        par ^= 1;
        cluster_sync_all();   // (the next use of x_small)
    }
    // what follows from it, by one warp: sixteen of them would issue the same instructions four times per scheduler
    if (tid < 32) {
        RowPlan& pl = sh->plan;   // (all lanes store the same)
        const double total = __dmul_rn(u128_to_double(S), 2.168404344971008868014905601739883422851562500e-19);   // * 2^-62
        // (top-p: the first candidate at which the cumulative probability reaches it, included)
        const U128 reach = double_to_u128_ceil(__dmul_rn(__dmul_rn((double)d.top_p, total), 4611686018427387904.0));
        pl.S = S;
        pl.sum = total;
        pl.target_p = reach;
        bool by_top_p = d.top_p < 1.0f && u128_ge(S, reach), by_min_p = d.min_p > 0.0f;
        int cut_lo = 0, cut_hi = -1;
        if (by_top_p && binned) cut_lo = cut_hi = find_bin(sh, reach);
        if (by_min_p) {
            pl.min_thr = __dmul_rn(__ddiv_rn(1.0, total), (double)d.min_p);
            // (the test is monotone in the logit and flips near mx + T * ln(min_p): only logits within a band around that value need the
            // exact arithmetic, those above it are kept, those below it are not)
            const double x_flip = (double)mx + pl.below, band = 1e-3 * (fabs(x_flip) + rc.temp + 1.0);
            const float x_sure = (float)(x_flip + band), x_never = (float)(x_flip - band);
            pl.x_sure = x_sure;
            pl.x_never = x_never;
            const int sure = max(0, rc.bin(x_sure)), never = max(0, rc.bin(x_never));
            if (by_top_p && cut_hi < sure) {
                by_min_p = false;   // (top-p ends the kept set earlier)
            } else if (by_top_p && never < cut_lo) {
                by_top_p = false;
                cut_lo = sure;
                cut_hi = never;
            } else {
                cut_lo = by_top_p ? min(cut_lo, sure) : sure;
                cut_hi = by_top_p ? max(cut_hi, never) : never;
            }
        }
        if (binned) {
            // the kept set weighs between `least` and `most`: the draw's place follows, up to a bin or two
            const bool cut = cut_hi >= cut_lo;
            const double w = pl.u;
            auto drawn = [&](U128 kept) {
                const U128 t = double_to_u128_ceil(__dmul_rn(w, u128_to_double(kept)));
                return find_bin(sh, u128_ge(kept, t) ? t : kept);
            };
            const int draw_hi = drawn(cut ? sh->weight_to(cut_hi) : S), draw_lo = cut ? drawn(sh->weight_to(cut_lo - 1)) : draw_hi;
            auto held = [&](int lo, int hi) { return sh->cum_n[hi] - (lo > 0 ? sh->cum_n[lo - 1] : 0u); };
            pl.about = held(draw_lo, draw_hi) + (cut ? held(cut_lo, cut_hi) : 0u);
            pl.draw_lo = draw_lo;
            pl.draw_hi = draw_hi;
        }
        pl.cut_lo = cut_lo;
        pl.cut_hi = cut_hi;
        pl.top_p = by_top_p ? 1 : 0;
        pl.min_p = by_min_p ? 1 : 0;
    }
    __syncthreads();
    const RowPlan& plan = sh->plan;
    const double sum = plan.sum, min_thr = plan.min_thr, u = plan.u;
    const U128 target_p = plan.target_p;
    FTR(4);

    // ---- 4. the usual way: the candidates of the bins where the kept set may end, and of those that the draw may fall into, go to the
    // first CTA, which finishes the row
    int sent = 0;
    if (binned && !a.record) {
        if (plan.about <= (unsigned)kMostListed) sent = send_ranges<C>(rc, sh, rank, plan.draw_lo, plan.draw_hi, max(plan.cut_lo, plan.draw_hi + 1), plan.cut_hi, par);
        if (sent > 0) {
            FTR(5);
            if (rank != 0) return;   // nobody reads this CTA's memory any more
            const int m = listed<C>(sh, par);
            int token;
            if (m > kShort) {
                token = finish_bins<C, kFullThreads>(rc, sh, par, m);
            } else {
                if (tid >= kShort) return;
                token = finish_bins<C, kShort>(rc, sh, par, m);
            }
            if (tid == 0) finish(token);
            FTR(6);
            return;
        }
        par ^= 1;
        if (sent < 0 && rank == 0) {
            aside(true);
            return;
        }
    }
    __syncwarp();
    cluster_sync_all();   // whoever goes on from here needs all CTAs of the row
    if (sh->gone) {
        aside(false);
        return;
    }
    if (sent < 0) {   // the first CTA's verdict came late: it is here by now, from a CTA that has passed the barrier with it or has left
        if (__syncthreads_or(!inbox_wait(&sh->in_verdict))) {
            aside(false);
            return;
        }
        if (sh->verdict) return;   // (the row is finished)
    }

    // ---- 4a. the usual way with a cut: everything that can be kept goes to the first CTA, which finishes the row
    if (binned && (d.top_p < 1.0f || d.min_p > 0.0f)) {
        int b_hi = kBins - 1;
        if (d.top_p < 1.0f) b_hi = find_bin(sh, target_p);
        if (d.min_p > 0.0f) b_hi = min(b_hi, rc.bin(plan.x_never));
        // (a list of more than a thousand is ordered too slowly: 22 us for 2000, two crossings take 15)
        if (sh->cum_n[b_hi] <= (unsigned)kMostListed && send_bins<C>(rc, sh, rank, 0, b_hi, false, par)) {
            FTR(5);
            if (rank != 0) return;   // nobody reads this CTA's memory any more
            const RowCuts cuts{target_p, u, sum, min_thr, d.top_p < 1.0f, d.min_p > 0.0f};
            const int m = listed<C>(sh, par);
            int token;
            if (m > kShort) {
                token = finish_list<C, kFullThreads>(rc, sh, par, m, cuts, a, out);
            } else {
                if (tid >= kShort) return;
                token = finish_list<C, kShort>(rc, sh, par, m, cuts, a, out);
            }
            if (tid == 0) finish(token);
            FTR(6);
            return;
        }
        par ^= 1;
    }

    // ---- 4b. the cuts one by one: min-p
    u64 c_keep = c_k;
    if (d.min_p > 0.0f) {
        u64 lowest = ~0ull;
        for (int i = tid; i < n; i += kFullThreads) {
            const float x = rc.at(i);
            if (!rc.is_candidate(x, i) || x < plan.x_never) continue;
            if (x > plan.x_sure || !(rc.probability(x, sum) < min_thr)) lowest = min(lowest, rc.comp(x, i));
        }
        lowest = ~block_max_u64(~lowest, sh);
        u64 v[4] = {~lowest, 0ull, 0ull, 0ull}, all[C][4];
        cluster_exchange<C>(sh, par, v, all);
        par ^= 1;
        for (int r = 0; r < C; ++r) lowest = min(lowest, ~all[r][0]);
        if (lowest == ~0ull) lowest = cmax & 0xFFFFFFFF00000000ull;   // keep at least the best
        c_keep = max(c_keep, lowest);
    }
    // ---- top-p
    bool keep_from_top_p = false;
    Crossing cp{0ull, U128{0ull, 0ull}, 0u, false};
    if (d.top_p < 1.0f) {
        cp = resolve<C>(rc, sh, rank, binned, a.record != 0, c_k, cmax, target_p, par);
        if (cp.found && cp.c >= c_keep) {
            c_keep = cp.c;
            keep_from_top_p = true;
        }
    }
    FTR(6);
    // ---- 4c. total weight and size of the kept set: known from the crossing when top-p made the cut, the whole
    // candidate set when nothing cut, otherwise one pass
    U128 KW = S;
    unsigned n_keep = n_cand;
    if (keep_from_top_p) {
        KW = u128_add(cp.above, U128{0ull, rc.weight(comp_value(cp.c)).value()});
        n_keep = cp.above_cnt + 1u;
    } else if (c_keep != c_k) {
        u64 wl = 0ull, wh = 0ull;
        unsigned pc = 0u;
        for (int i = tid; i < n; i += kFullThreads) {
            const float x = rc.at(i);
            if (x == x && rc.comp(x, i) >= c_keep) {
                const Weight w = rc.weight(x);
                wl += (u64)(long long)w.down;
                wh += w.up;
                ++pc;
            }
        }
        block_sums(sh, par, wl, wh, pc);
        cluster_sync_all();
        wl = wh = 0ull;
        n_keep = 0u;
        for (unsigned r = 0; r < (unsigned)C; ++r) {
            wl += ld_cluster_u64(map_to_rank(&sh->x_small[par][0], r));
            wh += ld_cluster_u64(map_to_rank(&sh->x_small[par][1], r));
            n_keep += (unsigned)ld_cluster_u64(map_to_rank(&sh->x_small[par][2], r));
        }
        KW = join_parts(wl, wh);
        par ^= 1;
    }
    FTR(7);
    // ---- 4d. the draw: first kept candidate whose cumulative weight reaches u * (kept weight)
    {
        U128 target = double_to_u128_ceil(__dmul_rn(u, u128_to_double(KW)));
        if (!u128_ge(KW, target)) target = KW;   // (beyond it by rounding: the last one)
        const Crossing ct = resolve<C>(rc, sh, rank, binned, false, c_k, cmax, target, par);
        const u64 c_tok = ct.found && ct.c >= c_keep ? ct.c : c_keep;
        if (rank == 0 && tid == 0) finish(comp_id(c_tok));
    }
    FTR(8);

    // ---- 5. the kept set's record: its size, and its first kMaxK candidates in order with their probabilities
    if (a.record) {
        const int want = (int)min(n_keep, (unsigned)kMaxK);
        u64 c_first = c_keep;   // the last of the first `want` kept candidates
        if ((unsigned)want < n_keep) {
            const Crossing cf = cluster_descent<C>(rc, sh, c_k, cmax, U128{0ull, (u64)want}, true, par);
            if (cf.found) c_first = max(c_keep, cf.c);
        }
        // every CTA appends its candidates >= c_first to the row's staging area (the probabilities' memory, as keys);
        // the kept-set size doubles as the fill counter until the first CTA has ordered them
        u64* stage = reinterpret_cast<u64*>(a.kept_pr + (size_t)out * kMaxK);
        if (rank == 0 && tid == 0) a.kept_n[out] = 0;
        __threadfence();
        cluster_sync_all();
        for (int i = tid; i < n; i += kFullThreads) {
            const float x = rc.at(i);
            if (x == x) {
                const u64 c = rc.comp(x, i);
                if (c >= c_first) {
                    const int p = atomicAdd(&a.kept_n[out], 1);
                    if (p < kMaxK) stage[p] = c;
                }
            }
        }
        __threadfence();
        cluster_sync_all();
        if (rank == 0) {
            u64* srt = reinterpret_cast<u64*>(vals);   // the first CTA's slice is no longer needed
            u64 c = 0ull;
            if (tid < want) c = __ldcg(stage + tid);
            __syncthreads();
            if (tid < want) srt[tid] = c;
            __syncthreads();
            if (tid < want) {
                int rank_in = 0;
                for (int j = 0; j < want; ++j) rank_in += srt[j] > c ? 1 : 0;
                a.kept_ids[(size_t)out * kMaxK + rank_in] = comp_id(c);
                a.kept_pr[(size_t)out * kMaxK + rank_in] = rc.probability(comp_value(c), sum);
            }
            if (tid == 0) a.kept_n[out] = (int)n_keep;
        }
    }
    cluster_sync_all();   // no CTA leaves while another may still read its shared memory
}

}  // namespace

namespace {
int slice_of(int n_vocab, int cluster) { return (((n_vocab + cluster - 1) / cluster) + 3) & ~3; }
size_t full_row_smem_bytes(int n_vocab, int cluster) {
    const int per = slice_of(n_vocab, cluster);
    const size_t bitmap = sizeof(unsigned) * (size_t)((per + 3 + 31) / 32);   // (three columns may come before the first slice)
    // (the kept set's record is ordered in the slice's memory: kMaxK 64-bit words)
    const size_t slice = per <= kSliceCache ? sizeof(float) * (size_t)std::max(per + 4, 2 * kMaxK) : sizeof(u64) * (size_t)kMaxK;
    return sizeof(FullShared) + bitmap + 16 + slice;
}
template <int C>
void fill_config(cudaLaunchConfig_t& cfg, cudaLaunchAttribute* attr, int n_rows, int n_vocab) {
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = C;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.gridDim = dim3((unsigned)(n_rows * C));
    cfg.blockDim = dim3(kFullThreads);
    cfg.dynamicSmemBytes = full_row_smem_bytes(n_vocab, C);
    cfg.attrs = attr;
    cfg.numAttrs = 1;
}
template <int C>
int launch_full(const FullArgs& a, int n_rows, cudaStream_t stream) {
    cudaLaunchAttribute attr[1];
    cudaLaunchConfig_t cfg{};
    fill_config<C>(cfg, attr, n_rows, a.n_vocab);
    cfg.stream = stream;
    return (int)cudaLaunchKernelEx(&cfg, full_row_kernel<C>, a, slice_of(a.n_vocab, C) <= kSliceCache ? 1 : 0);
}
// How many clusters of C CTAs run at once.  A cluster lies in one GPC, so this is less than SMs / C: 15 of eight on B200's
// 148 SMs (of seven, too), 22 of six, 26 of five, 33 of four.
int g_at_once[4] = {0, 0, 0, 0};   // of four, five, six, eight
template <int C>
int prepare_full(int& at_once) {
    // the largest request of any row length, whatever the engine's: the attribute is the kernel's, and engines of several sizes
    // may be alive.  Rows that still fit the slice cache need the most.
    const size_t most = full_row_smem_bytes(C * kSliceCache, C);
    cudaError_t e = cudaFuncSetAttribute(full_row_kernel<C>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)most);
    if (e != cudaSuccess || at_once > 0) return (int)e;
    cudaLaunchAttribute attr[1];
    cudaLaunchConfig_t cfg{};
    fill_config<C>(cfg, attr, 64, C * kSliceCache);
    return (int)cudaOccupancyMaxActiveClusters(&at_once, full_row_kernel<C>, &cfg);
}
}  // namespace

int prepare_full_row_kernel() {
    for (int e : {prepare_full<8>(g_at_once[3]), prepare_full<6>(g_at_once[2]), prepare_full<5>(g_at_once[1]), prepare_full<4>(g_at_once[0])})
        if (e != 0) return e;
    return 0;
}

int launch_full_row_kernel(const float* logits, const RowDesc* rows, int n_rows, const int32_t* hist, const int32_t* drafts, int32_t* pool, int32_t* tokens, int32_t* tokens_host,
                           int32_t* kept_ids, double* kept_pr, int32_t* kept_n, int record, uint32_t* status, uint32_t* status_host, int n_vocab,
                           int vocab_offset, int write_back, float softcap, uint64_t* trace, void* stream) {
    if (n_vocab > (1 << 22)) return (int)cudaErrorInvalidValue;   // the histogram's limb sums are sized for 4 M logits
    FullArgs a{};
    a.logits = logits;
    a.rows = rows;
    a.hist = hist;
    a.drafts = drafts;
    a.pool = pool;
    a.tokens = tokens;
    a.tokens_host = tokens_host;
    a.status_host = status_host;
    a.kept_ids = kept_ids;
    a.kept_pr = kept_pr;
    a.kept_n = kept_n;
    a.status = status;
    a.n_vocab = n_vocab;
    a.vocab_offset = vocab_offset;
    a.write_back = write_back;
    a.record = record;
    a.softcap = softcap;
    a.trace = reinterpret_cast<u64*>(trace);
    // The more CTAs per row the shorter the passes, but a second wave of clusters costs as much as the first.  Measured on B200 with top-p
    // 0.95 (us, four / five / six / eight CTAs): 8 x 16384 14.7 each, 8 x 65536 23.7 / 22.9 / 21.2 / 18.8, 16 x 131072 42 / 34.2 / 32.1 / 43.1,
    // 23 x 131072 42 / 33.1 / 49.3 / 44.4, 32 x 65536 24.9 / 40.0 / 37.4 / 45.4.  The rule's terms: steps, and passes over a slice.
    int best = 8;
    double cost = 1e30;
    for (int i = 3; i >= 0; --i) {
        const int c = i == 3 ? 8 : 4 + i, per = slice_of(n_vocab, c), at_once = std::max(1, g_at_once[i]);
        if (c < 8 && per > kSliceCache) continue;
        const double t = ((n_rows + at_once - 1) / at_once) * (11.0 + 0.92 * per / 1024.0);
        if (t < cost) {
            cost = t;
            best = c;
        }
    }
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    switch (best) {
        case 8: return launch_full<8>(a, n_rows, st);
        case 6: return launch_full<6>(a, n_rows, st);
        case 5: return launch_full<5>(a, n_rows, st);
        default: return launch_full<4>(a, n_rows, st);
    }
}

}  // namespace fsb
