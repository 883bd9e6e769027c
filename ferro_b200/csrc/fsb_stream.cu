// fsb_stream.cu - the streaming candidate kernel of the B200 batched token sampler (sm_100a).
//
// One launch samples every row of a batch whose effective k is at most kMaxK (greedy rows are k = 1):
//   repetition penalty (src/sampler.cpp:11-18) -> greedy argmax (:19-23) or top-k candidates (:25-35)
//   -> fp64 softmax (:37-41) -> min-p (:43) -> top-p (:44) -> seeded draw (:45-49).
// (reference paths are relative to the paragontasx/ferro project root)
#include <cuda_runtime.h>

#include "../../include/ferro_sampler_b200.h"
#include <algorithm>
#include <cfloat>
#include <type_traits>
#include <cstring>

#include "fsb_device.cuh"

namespace fsb {
namespace {

// How it works.
// A row is cut into 1 to 8 equal segments, one CTA each; the CTAs of a row are a thread-block cluster.  A CTA reads its
// segment once, in chunks of four 16-byte cells per thread.  Every thread copies its own cells to shared memory
// asynchronously (cp.async), two chunks ahead, and reads back only what it copied itself: no barrier between copy and
// look, 32 KB per CTA in flight, four CTAs per SM.
// The look works on raw logits and leaves the penalised ones out.  A thread keeps two running maxima (of different cells);
// from all threads' maxima the CTA derives a bound that at least k logits of the segment reach (cta_bound), at chunks 0, 1,
// 3, 7, 15, ...  A cell whose maximum reaches the bound is listed in shared memory, data and all: about 100 in each of these
// intervals for k = 64.  Every warp has a list of its own and keeps its length in a register: votes, but no atomics and
// nothing to wait for.  Should a list overflow, the segment is gone through once more with the final bound.  A segment that
// fits the ring (8192 or 32768 logits) is not listed: it is looked at again when its bound is known.
// At the end the listed cells are taken apart: the logits that reach the final bound are candidates, and with them the
// penalised logits of the window that do so once penalised, each id once.  The softcap is applied here too, to candidates
// only: it is monotone up to the rounding of tanhf, and a margin under the bound covers that.
// For k <= 64 the final bound is the row's (publish_most, key_bound), so a row has about 1.4 k candidates however many CTAs work
// on it, and the few in each go straight to the first CTA, which orders them and finishes the row.  For k > 64 a CTA keeps to
// its segment's bound, and the first one picks the k best of what they send.
// What bounds it: the stream (HBM) for large batches, for small ones a chain of about ten dependent steps.  A step's
// latency is its instruction count: a warp alone issues a dependent instruction every four to five cycles, and 32 warps that
// all do the same take eight times their share of a scheduler, so steps after the stream are left to one warp or eight, and
// what several CTAs need of one another goes by counted stores (inbox_put) instead of the cluster's barrier and its fences.
// us per launch with launches chained (form 2): 1 x 65536, k = 40 7.9, 32 x 131072, k = 40 11.2, 72 x 131072, k = 50 16.9, 64 x 262144, k = 64
// 20.6, 512 x 32768, k = 40 24.5; with a bound per segment and the cluster's barrier 2.3, 3.2, 4.1, 2.7 and 1.0 more.
// The exact path (exact_select) makes no assumption: a radix selection over the transformed segment that reads it again
// (from L2) per digit.  It runs when hundreds of equal logits reach the final bound.
// Waits for another CTA end after a second or so at the latest.  A CTA whose wait has run out reports the row (kStatusLate) and uses nothing of
// what it waited for: without the row's keys it goes on with a bound that no finite logit (under the softcap: hardly one) reaches, and the
// first one without all candidates finishes a row of none.  It stays until the others have left or gave up, too: what is still on its way to it
// finds its memory there.

constexpr int kCells = 4;                               // cells of a thread per chunk
constexpr int kStages = 2;
constexpr int kPenCap = 1024;                           // penalised columns of a segment that are looked up ahead
constexpr int kPickCap = 1024;                          // candidates of a segment
constexpr int kMergeList = 2048;                        // candidates of all segments, an equal share of it each
constexpr int kCellSlots = 4096, kCellIds = 2048;       // penalised cells: slots of their table, and the longest window that may use it
constexpr int kSelectSmemMax = 224 * 1024;
static_assert(kMergeList >= 2 * kMaxK, "the epilogue's scratch lives in the merge list's memory");
static_assert((kPickCap + 32 + kMaxK) * 8 + 256 * 4 <= kStages * kCells * 256 * 16 - kCellSlots * 4, "candidates, the rare paths' counters and the table lie in a small CTA's ring");

// Columns of the longest segment.
int segment_columns(int n_vocab, int nseg) { return 4 * ((n_vocab / 4 + nseg - 1) / nseg) + 8; }
// A segment's penalised columns: logits and numbers of the first kPenCap, and a bitmap.
size_t window_bytes(int seg_cols) { return seg_cols > 0 ? kPenCap * (sizeof(float) + sizeof(int)) + (size_t)((seg_cols + 32 + 127) / 128) * 16 : 0; }

// The same where a bit per cell will do (see CellSegment): a group of 32 words per chunk of small CTAs.
size_t cell_bits_bytes(int seg_cols) { return seg_cols > 0 ? (size_t)(seg_cols / 4 + 1024) / 1024 * 128 : 0; }

struct Segment {
    const float* row;          // the row's logits
    unsigned* bitmap;          // penalised columns (bit 0 = column bit0), valid when has_pen
    const int32_t* hist;       // the penalty window: these ids ...
    const int32_t* drafts;     // ... then these
    int hist_len, window_len;  // ids in the first part, in both
    int lo, hi;                // columns
    int bit0;
    int id_base;               // token id of column 0
    bool has_pen;
    float pen, cap;
};

__device__ __forceinline__ int window_id(const Segment& s, int i) { return i < s.hist_len ? s.hist[i] : s.drafts[i - s.hist_len]; }
__device__ __forceinline__ float penalise(float x, float pen) { return x > 0.0f ? __fdiv_rn(x, pen) : __fmul_rn(x, pen); }   // src/sampler.cpp:17
__device__ __forceinline__ bool penalised(const Segment& s, int c) { return s.has_pen && ((s.bitmap[(c - s.bit0) >> 5] >> ((c - s.bit0) & 31)) & 1u); }

// A whole row whose penalised logits are kept by cells, on small CTAs: a bit per cell - a quarter of the memory, and one
// 16-byte read per warp and chunk - marks the cells that hold some.  Marked cells take no part in the bounds, but are listed as
// others are if the largest of them, penalised or not, can reach the bound; at the end a hash table in the ring's memory says
// which columns of the listed ones the window holds.  (Set aside as a whole and fetched again at the end, 800 random reads for a
// window of 1024, they took 16 us of the 106 of a launch of 512 x 262144, all rows at the same time.)
constexpr int kMarked = 1 << 30;   // in a listed cell's number
struct CellSegment : Segment {
    int* table;                // kCellSlots, or half of them, x (cell << 4 | penalised columns of it), -1: free
    const unsigned* edges;     // penalised ones of the logits outside the cells
    int head, n_cells;
    int slots;
};
__device__ __forceinline__ int cell_word(int cell) { return (cell >> 10) * 32 + ((cell >> 5) & 7) * 4 + ((cell >> 8) & 3); }
__device__ __forceinline__ unsigned cell_slot(int cell, int slots) { return __umulhi((unsigned)cell * 2654435761u, (unsigned)slots); }
__device__ __forceinline__ int edge_index(const CellSegment& s, int c) { return c < s.head ? c : 4 + c - s.head - 4 * s.n_cells; }
__device__ __forceinline__ bool outside_cells(const CellSegment& s, int c) { return c < s.head || c >= s.head + 4 * s.n_cells; }
// The penalised columns of a marked cell.
__device__ __forceinline__ int penalised_of(const CellSegment& s, int cell) {
    for (unsigned h = cell_slot(cell, s.slots);; h = (h + 1u) & (unsigned)(s.slots - 1)) {   // (at least half of the slots are free)
        const int v = s.table[h];
        if (v < 0) return 0;
        if ((v >> 4) == cell) return v & 15;
    }
}
__device__ __forceinline__ bool penalised(const CellSegment& s, int c) {
    if (!s.has_pen) return false;
    if (outside_cells(s, c)) return (*s.edges >> edge_index(s, c)) & 1u;
    const int cell = (c - s.head) >> 2, e = (c - s.head) & 3;
    return ((s.bitmap[cell_word(cell)] >> (cell & 31)) & 1u) && ((penalised_of(s, cell) >> e) & 1);
}

struct StreamCtl : SharedCtl {
    CellSegment seg;           // what the steps after the stream need to know: registers are scarce while it runs
    RowDesc desc;
    u64 keyed, counted, sent;  // barriers: the row's keys have come; in its first CTA, the numbers of candidates, the candidates
    u64 count[8];              // from segment r: its number of candidates, whether they are in the second part of its share, and how many words it has sent
    unsigned bound;
    int late;                  // a wait has run out
    int pad[2];
};
static_assert(sizeof(StreamCtl) % 16 == 0, "what follows the control block is read 16 bytes at a time");

// Sizes that go with T, the threads of a CTA.
template <int T>
struct Geometry {
    static constexpr int kWarps = T / 32;
    static constexpr int kChunkCells = kCells * T;
    static constexpr size_t kRingBytes = (size_t)kStages * kChunkCells * sizeof(float4);
    // cells a warp can list; with k > 64; where penalised cells are listed with the others (a window of a thousand ids may hold the
    // hundred largest logits: with 64 a few rows in 512 went through their segment twice)
    static constexpr int kWarpCells = 64, kWarpCellsLong = T == 256 ? 128 : 64, kWarpCellsMarked = 88;
    static_assert((kPickCap + 32 + kMaxK + kMergeList + 32) * sizeof(u64) <= kRingBytes, "everything after the stream lives in the ring's memory");
    // keys that the warps of a row hand over (publish_most): 8 per warp, at most 256
    __host__ __device__ static constexpr int key_words(int nseg) { return T == 256 && nseg == 1 ? 64 : 256; }
    // dynamic shared memory: ring, listed cells (data, numbers), penalised logits (data, columns), control block, keys,
    // receive buffer, bitmap of the penalised columns of the segment (its first word: the up to three columns before the cells)
    static size_t smem_bytes(int nseg, int kmax, int seg_cols, bool marked = false) {
        const size_t cells = (size_t)kWarps * (kmax > 64 ? kWarpCellsLong : marked ? kWarpCellsMarked : kWarpCells) * (sizeof(float4) + sizeof(int));
        return kRingBytes + cells + sizeof(StreamCtl) + key_words(nseg) * sizeof(unsigned) + (nseg > 1 ? kMergeList : 0) * sizeof(u64) + window_bytes(seg_cols);
    }
};

// Logit of column c as the sampler sees it.
template <class S>
__device__ __forceinline__ float transform(float x, int c, const S& s) {
    if (s.cap != 0.0f) x = softcap_call(x, s.cap);
    if (penalised(s, c)) x = penalise(x, s.pen);
    return x;
}

// A bound that at least k logits of the segment reach, from the threads' maxima (each a logit of its own; two per
// thread, of different cells).  Minus infinity - and what is no number - never reaches a bound.  All threads get the same
// value; contains one barrier; buffers alternate, so that the next call may write while a slow warp still reads.
//  The r-th largest maximum of every warp, r = ceil(k / warps), minimum over the warps: 1.3 k to 2 k logits reach it.  r warp
//  reductions take the largest out one after the other; keys give up their low bits to be distinct, which lowers the bound
//  by less than 2^-17 of its value.  k <= 64 does with one maximum per thread.  (Ranks by counting over shared memory took
//  2.6 us per call with 32 warps, this 0.4; the k-th largest of all threads' maxima lets fewer through but costs more.)
template <int T, int BAR>
__device__ __forceinline__ float cta_bound(float run_a, float run_b, int k, int buf, SharedCtl* ctl) {
    constexpr int kWarps = T / 32;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    unsigned ka = (float_key(run_a) & ~63u) | (unsigned)(2 * lane), kb = (float_key(run_b) & ~63u) | (unsigned)(2 * lane + 1), top;
    if (k <= 64) {
        ka = max(ka, kb);
        top = __reduce_max_sync(0xffffffffu, ka);
        for (int r = (k - 1) / kWarps; r > 0; --r) {
            if (ka == top) ka = 0u;
            top = __reduce_max_sync(0xffffffffu, ka);
        }
    } else {
        top = __reduce_max_sync(0xffffffffu, max(ka, kb));
        for (int r = (k - 1) / kWarps; r > 0; --r) {
            if (ka == top) ka = 0u;
            if (kb == top) kb = 0u;
            top = __reduce_max_sync(0xffffffffu, max(ka, kb));
        }
    }
    if (lane == 0) ctl->top[buf][warp] = top & ~63u;
    block_sync<T, BAR>();
    const unsigned m = __reduce_min_sync(0xffffffffu, ctl->top[buf][lane & (kWarps - 1)]);
    return fmaxf(key_float(m), -FLT_MAX);   // (also for the patterns just below minus infinity's key, which are no numbers)
}

// For k <= 64 the final bound is the row's, however many CTAs it has: every warp hands its `most` largest lane maxima - each lane's
// is a logit of its own; keys, their low bits cut off - to all CTAs of the row, and each finds a value that at least k of all those
// keys reach, and not many more: about 1.1 k to 1.7 k logits do.
// How many that is in a row of `cells` cells and nseg CTAs of n_warps warps: 1.6 k of them in all, but no more than 8 a warp.
__host__ __device__ __forceinline__ int keys_per_warp(int cells, int nseg, int n_warps, int k) {
    const int groups = ((cells + nseg - 1) / nseg + 31) >> 5, sources = nseg * (groups < n_warps ? groups : n_warps);   // (warps that have any cells)
    int most = 1;
    while (most < 8 && 5 * most * sources < 8 * k) most *= 2;
    return most;
}
template <int T>
__device__ __forceinline__ void publish_most(float run, int most, int seg, int nseg, unsigned* keys, u64* inbox) {
    constexpr int kWarps = T / 32;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    unsigned key = (float_key(run) & ~31u) | (unsigned)lane;
    unsigned* own = keys + (seg * kWarps + warp) * most;
    unsigned at = 0u, bar = 0u;
    if (nseg > 1 && lane < nseg) {
        at = cluster_map_shared(smem_u32(own), (unsigned)lane);
        bar = cluster_map_shared(smem_u32(inbox), (unsigned)lane);
    }
    for (int r = 0; r < most; ++r) {
        const unsigned top = __reduce_max_sync(0xffffffffu, key);
        if (key == top) key = 0u;
        if (nseg == 1) {
            if (lane == 0) own[r] = top & ~31u;
        } else if (lane < nseg) {
            inbox_put(at + 4u * (unsigned)r, top & ~31u, bar);
        }
    }
}
// One warp; `n` (8 .. 256) keys.  Bisection by votes, over the integers between the smallest and the largest key, until between k and
// 9/8 k keys are at or above the middle (four or five steps of 50 cycles as a rule; counting all ranks took 1200).
__device__ __forceinline__ unsigned key_bound(int n, int k, const unsigned* keys) {
    const int lane = threadIdx.x & 31;
    unsigned q[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) q[i] = 32 * i + lane < n ? keys[32 * i + lane] : 0u;
    auto reach = [&](unsigned t) {
        int c = 0;
#pragma unroll
        for (int i = 0; i < 4; ++i) c += __popc(__ballot_sync(0xffffffffu, q[i] >= t));
        if (n > 128) {
#pragma unroll
            for (int i = 4; i < 8; ++i) c += __popc(__ballot_sync(0xffffffffu, q[i] >= t));
        }
        return c;
    };
    unsigned top = 0u;
#pragma unroll
    for (int i = 0; i < 8; ++i) top = max(top, q[i]);
    unsigned lo = 0x00800000u, hi = __reduce_max_sync(0xffffffffu, top) + 1u;   // lo: the key of -FLT_MAX
    if (hi <= lo || reach(lo) < k) return 0u;
    unsigned low = hi;
#pragma unroll
    for (int i = 0; i < 8; ++i) low = min(low, q[i] >= lo ? q[i] : hi);
    lo = __reduce_min_sync(0xffffffffu, low);
    while (hi - lo > 1u) {
        const unsigned mid = lo + ((hi - lo) >> 1);
        const int c = reach(mid);
        if (c >= k) {
            lo = mid;
            if (8 * c <= 9 * k) break;
        } else {
            hi = mid;
        }
    }
    return lo;
}

// Keeps those of a warp's n <= 128 listed cells that reach `admit`, in order, and those whose number has a bit of `always`;
// returns how many they are.
__device__ __noinline__ int prune_cells(float4* cells, int* nums, int n, float admit, int always) {
    const int lane = threadIdx.x & 31;
    int w = 0;
    for (int p0 = 0; p0 < n; p0 += 32) {
        float4 x = make_float4(0.f, 0.f, 0.f, 0.f);
        int num = 0;
        bool keep = false;
        if (p0 + lane < n) {
            x = cells[p0 + lane];
            num = nums[p0 + lane];
            keep = fmaxf(fmaxf(x.x, x.y), fmaxf(x.z, x.w)) >= admit || (num & always) != 0;
        }
        const unsigned m = __ballot_sync(0xffffffffu, keep);
        if (keep) {   // (never ahead of what is still to be read)
            const int q = w + __popc(m & ((1u << lane) - 1u));
            cells[q] = x;
            nums[q] = num;
        }
        w += __popc(m);
        __syncwarp();
    }
    return w;
}

// Exact selection of the min(k, candidates) largest composites of the transformed segment into list (unordered);
// returns their number.  `bins`: 256 words.  MSB-first over 8-bit digits of the composites: count the digits of the composites that match
// the prefix, walk the counts from the top, go on in the digit in which the k-th lies; stops early when a digit is
// taken whole.  Every digit reads the segment again.  All threads call, after a barrier.
template <int T, class S>
__device__ __noinline__ int exact_select(const S s, int k, u64* list, unsigned* bins, SharedCtl* ctl) {
    const int tid = threadIdx.x, lane = tid & 31;
    u64 prefix = 0ull, mask = 0ull;
    int need = k;
    const int rounds = (s.hi - s.lo + T - 1) / T;
    for (int shift = 56; shift >= 0; shift -= 8) {
        if (tid < 256) bins[tid] = 0u;
        __syncthreads();
        for (int i = 0; i < rounds; ++i) {
            const int c = s.lo + i * T + tid;
            unsigned digit = 256u;
            if (c < s.hi) {
                const float x = transform(__ldcg(s.row + c), c, s);
                const u64 m = make_comp(x, c + s.id_base);
                if (x == x && (m & mask) == prefix) digit = (unsigned)(m >> shift) & 255u;
            }
            const unsigned peers = __match_any_sync(0xffffffffu, digit);   // equal logits would meet in one counter
            if (digit < 256u && lane == __ffs(peers) - 1) atomicAdd(&bins[digit], (unsigned)__popc(peers));
        }
        __syncthreads();
        if (tid < 32) {   // lane l owns digits 255 - 8 l .. 248 - 8 l
            int mine = 0;
#pragma unroll
            for (int d = 0; d < 8; ++d) mine += (int)bins[255 - 8 * lane - d];
            int inc = mine;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int t = __shfl_up_sync(0xffffffffu, inc, o);
                if (lane >= o) inc += t;
            }
            const int total = __shfl_sync(0xffffffffu, inc, 31);
            int above = inc - mine;
            if (total < need) {   // first digit only: fewer than k candidates, all are taken
                if (lane == 0) ctl->sel_in_bin = -1;
            } else if (above < need && inc >= need) {
                for (int d = 0; d < 8; ++d) {
                    const int in = (int)bins[255 - 8 * lane - d];
                    if (above + in >= need) {
                        ctl->sel_prefix = prefix | ((u64)(255 - 8 * lane - d) << shift);
                        ctl->sel_need = need - above;
                        ctl->sel_in_bin = in;
                        break;
                    }
                    above += in;
                }
            }
        }
        __syncthreads();
        const int in_bin = ctl->sel_in_bin;
        if (in_bin < 0) {
            prefix = 0ull;
            break;
        }
        prefix = ctl->sel_prefix;
        need = ctl->sel_need;
        mask |= 255ull << shift;
        if (in_bin == need) break;
    }
    __syncthreads();
    if (tid == 0) ctl->kept_n = 0;
    __syncthreads();
    for (int i = 0; i < rounds; ++i) {
        const int c = s.lo + i * T + tid;
        if (c >= s.hi) continue;
        const float x = transform(__ldcg(s.row + c), c, s);
        const u64 m = make_comp(x, c + s.id_base);
        if (x == x && m >= prefix) list[atomicAdd(&ctl->kept_n, 1)] = m;   // at most k
    }
    __syncthreads();
    return ctl->kept_n;
}

// A segment with fewer than k logits above minus infinity (masked vocabularies): its first columns that hold minus
// infinity are candidates too.  Appends up to k - n of them to the list; returns the new length.  All threads call.
template <int T, class S>
__device__ __noinline__ int append_masked(const S s, int n, int k, u64* list, unsigned* counts) {
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    __syncthreads();
    for (int c0 = s.lo; c0 < s.hi && n < k; c0 += T) {
        const int c = c0 + tid;
        const bool hit = c < s.hi && transform(__ldcg(s.row + c), c, s) == -__int_as_float(0x7f800000);
        const unsigned m = __ballot_sync(0xffffffffu, hit);
        if (lane == 0) counts[warp] = (unsigned)__popc(m);
        __syncthreads();
        int before = n, total = 0;
        for (int w = 0; w < T / 32; ++w) {
            if (w < warp) before += (int)counts[w];
            total += (int)counts[w];
        }
        before += __popc(m & ((1u << lane) - 1u));
        if (hit && before < k) list[before] = make_comp(-__int_as_float(0x7f800000), c + s.id_base);
        n = min(k, n + total);
        __syncthreads();
    }
    return n;
}

// Write-back: the transformed logits go to the caller's row.  Nothing reads the raw row after this.
template <int T>
__device__ __noinline__ void write_back(const Segment s) {
    float* row = const_cast<float*>(s.row);
    __syncthreads();
    if (s.cap != 0.0f) {
        for (int c = s.lo + threadIdx.x; c < s.hi; c += T) row[c] = transform(__ldcg(row + c), c, s);
        return;
    }
    for (int i = threadIdx.x; i < s.window_len; i += T) {
        const int c = window_id(s, i) - s.id_base;
        if (c < s.lo || c >= s.hi) continue;
        const unsigned bit = 1u << ((c - s.bit0) & 31);   // an id counts once however often it occurs in the window
        if (atomicAnd(&s.bitmap[(c - s.bit0) >> 5], ~bit) & bit) row[c] = penalise(__ldcg(row + c), s.pen);
    }
}

__device__ __forceinline__ unsigned lanes_below() {
    unsigned m;
    asm("mov.u32 %0, %%lanemask_lt;" : "=r"(m));
    return m;
}
__device__ __forceinline__ float cell_max(const float4& x) { return fmaxf(max3(x.x, x.y, x.z), x.w); }

// Where a segment lies in its row: the row's whole 16-byte cells are cut into nseg runs.  Up to three logits before the
// first cell belong to the first segment, up to three after the last cell to the last one: rows may start anywhere.
struct RowSpan {
    const float4* cells;   // cell 0
    int head;              // columns before it
    int n_cells, c_lo, c_hi;
    // column of the segment's e-th logit outside the whole cells (e < 8), or -1
    __device__ __forceinline__ int edge_column(int e, int n_vocab, int seg, int nseg) const {
        if (e < 4) return seg == 0 && e < head ? e : -1;
        return seg == nseg - 1 && e - 4 < n_vocab - head - 4 * n_cells ? head + 4 * n_cells + e - 4 : -1;
    }
};
__device__ __forceinline__ RowSpan row_span(const float* row_ptr, int V, int seg, int nseg) {
    RowSpan w;
    w.head = min(V, (int)((0u - ((unsigned)reinterpret_cast<uintptr_t>(row_ptr) >> 2)) & 3u));
    w.n_cells = (V - w.head) >> 2;
    const int lseg = 31 - __clz(nseg), per = (w.n_cells + nseg - 1) >> lseg;   // nseg is a power of two
    w.c_lo = min(seg * per, w.n_cells);
    w.c_hi = min(w.c_lo + per, w.n_cells);
    w.cells = reinterpret_cast<const float4*>(row_ptr + w.head);
    return w;
}
__device__ __forceinline__ Segment make_segment(const StreamArgs& a, const RowSpan& w, const float* row_ptr, int seg, int nseg, unsigned* bitmap) {
    Segment s;
    s.row = row_ptr;
    s.bitmap = bitmap;
    s.hist = s.drafts = nullptr;
    s.hist_len = s.window_len = 0;
    s.lo = seg == 0 ? 0 : w.head + 4 * w.c_lo;
    s.hi = seg == nseg - 1 ? a.n_vocab : w.head + 4 * w.c_hi;
    s.bit0 = w.head + 4 * w.c_lo - 32;
    s.id_base = a.vocab_offset;
    s.has_pen = false;
    s.pen = 1.0f;
    s.cap = a.softcap;
    return s;
}

__device__ __forceinline__ void set_window(Segment& s, const int32_t* hist, const int32_t* drafts, const RowDesc& d) {
    s.hist = hist + d.hist_begin;
    s.hist_len = d.hist_len;
    s.drafts = drafts + d.draft_off;
    s.window_len = d.hist_len + (d.flags >> kRowDraftShift);
}

// The first ids of the window, up to 1024, which a CTA asks for before its copies fill the memory pipes.
template <int T>
struct FirstIds {
    static constexpr int kPer = 1024 / T;
    int id[kPer];
    __device__ __forceinline__ void load(const Segment& s) {
#pragma unroll
        for (int q = 0; q < kPer; ++q) id[q] = (int)threadIdx.x + q * T < s.window_len ? window_id(s, threadIdx.x + q * T) : 0;
    }
    // calls f(in the window, id) for every id of the window, whole warps at a time
    template <class F>
    __device__ __forceinline__ void each(const Segment& s, F f) const {
        const int tid = threadIdx.x, i0 = tid & ~31;
#pragma unroll
        for (int q = 0; q < kPer; ++q)
            if (i0 + q * T < s.window_len) f(tid + q * T < s.window_len, id[q]);
        for (int i = tid + 1024; (i & ~31) < s.window_len; i += T) f(i < s.window_len, i < s.window_len ? window_id(s, i) : 0);
    }
};
__device__ __forceinline__ void clear_bits(unsigned* bitmap, int quads, int threads) {
    for (int i = threadIdx.x; i < quads; i += threads) reinterpret_cast<uint4*>(bitmap)[i] = make_uint4(0u, 0u, 0u, 0u);
}

// The window's columns of the segment: sets their bits (cleared before), and lists each once - an id counts once however often it
// occurs - with its logit, which is fetched now (the copies belong to the next group that the thread commits) and needed at the end.
// All threads call, after a barrier; another has to follow.
template <int T>
__device__ __forceinline__ void collect_penalised(const Segment& s, const FirstIds<T>& ids, SharedCtl* ctl, float* pen_raw, int* pen_col) {
    const int lane = threadIdx.x & 31;
    ids.each(s, [&](bool in, int id) {
        const int c = id - s.id_base;
        bool first = false;
        if (in && c >= s.lo && c < s.hi) {
            const unsigned bit = 1u << ((c - s.bit0) & 31);
            first = (atomicOr(&s.bitmap[(c - s.bit0) >> 5], bit) & bit) == 0u;
        }
        const unsigned hits = __ballot_sync(0xffffffffu, first);
        if (hits) {
            int p = 0;
            if (lane == 0) p = atomicAdd(&ctl->pen_n, __popc(hits));
            p = __shfl_sync(0xffffffffu, p, 0) + __popc(hits & lanes_below());
            if (first && p < kPenCap) {
                pen_col[p] = c;
                cp_async4(smem_u32(pen_raw + p), s.row + c);
            }
        }
    });
}
// Calls f(valid, raw logit, column) for every penalised column; whole warps call it together.
template <int T, class F>
__device__ __forceinline__ void for_each_penalised(const Segment& s, int n_pen, const float* pen_raw, const int* pen_col, F f) {
    const int tid = threadIdx.x, lane = tid & 31;
    if (n_pen <= kPenCap) {
        for (int i0 = tid & ~31; i0 < n_pen; i0 += T) {
            const bool in = i0 + lane < n_pen;
            f(in, in ? pen_raw[i0 + lane] : 0.0f, in ? pen_col[i0 + lane] : 0);
        }
    } else {   // a long window: whatever the bitmap holds
        const int words = (s.hi - s.bit0 + 31) >> 5;
        for (int w0 = tid & ~31; w0 < words; w0 += T) {
            unsigned bits = w0 + lane < words ? s.bitmap[w0 + lane] : 0u;
            while (__any_sync(0xffffffffu, bits != 0u)) {
                const int col = s.bit0 + 32 * (w0 + lane) + __ffs(bits) - 1;
                f(bits != 0u, bits ? __ldcg(s.row + col) : 0.0f, col);
                bits &= bits - 1u;
            }
        }
    }
}
// Penalised logits of a thread's cells of a chunk (`j`: its first cell, counted from the segment's first; `left`: cells of
// the segment from this chunk on) become minus infinity: they are looked at on their own.
template <int T>
__device__ __forceinline__ void mask_penalised(float4 (&x)[kCells], const unsigned* bitmap, int j, int left) {
    const float ninf = -__int_as_float(0x7f800000);
    const unsigned* w = bitmap + (j >> 3) + 1;
    const int sh = 4 * (j & 7);
    unsigned bits[kCells];
#pragma unroll
    for (int u = 0; u < kCells; ++u) bits[u] = (int)threadIdx.x + u * T < left ? w[u * (T / 8)] >> sh : 0u;
    if ((bits[0] | bits[1] | bits[2] | bits[3]) & 15u) {
#pragma unroll
        for (int u = 0; u < kCells; ++u) {
            if (bits[u] & 1u) x[u].x = ninf;
            if (bits[u] & 2u) x[u].y = ninf;
            if (bits[u] & 4u) x[u].z = ninf;
            if (bits[u] & 8u) x[u].w = ninf;
        }
    }
}
// The window's cells: sets their bits (cleared before, as `edges` is) before the stream, and fills the table after it.  All threads
// call; a barrier has to follow.
template <int T>
__device__ __forceinline__ void collect_cells(const CellSegment& s, const FirstIds<T>& ids, unsigned* edges) {
    ids.each(s, [&](bool in, int id) {
        const int c = id - s.id_base;
        if (!in || c < s.lo || c >= s.hi) return;
        const int cell = (c - s.head) >> 2;
        if (outside_cells(s, c)) atomicOr(edges, 1u << edge_index(s, c));
        else atomicOr(&s.bitmap[cell_word(cell)], 1u << (cell & 31));
    });
}
template <int T>
__device__ __forceinline__ void fill_table(const CellSegment& s) {
    for (int i = threadIdx.x; i < s.slots / 4; i += T) reinterpret_cast<int4*>(s.table)[i] = make_int4(-1, -1, -1, -1);
    __syncthreads();
    for (int i = threadIdx.x; i < s.window_len; i += T) {
        const int c = window_id(s, i) - s.id_base;
        if (c < s.lo || c >= s.hi || outside_cells(s, c)) continue;
        const int cell = (c - s.head) >> 2, bit = 1 << ((c - s.head) & 3);
        for (unsigned h = cell_slot(cell, s.slots);; h = (h + 1u) & (unsigned)(s.slots - 1)) {   // (no more cells than ids: at most half of the slots)
            const int v = atomicCAS(&s.table[h], -1, cell << 4 | bit);
            if (v == -1) break;
            if ((v >> 4) == cell) {
                atomicOr(&s.table[h], bit);
                break;
            }
        }
    }
}
// Largest of the lanes' composites.
__device__ __forceinline__ u64 warp_max_u64(u64 v) {
    const unsigned hi = __reduce_max_sync(0xffffffffu, (unsigned)(v >> 32));
    const unsigned lo = __reduce_max_sync(0xffffffffu, (unsigned)(v >> 32) == hi ? (unsigned)v : 0u);
    return ((u64)hi << 32) | lo;
}
// The row's candidates in order: softmax, cuts, draw, and whatever the caller wants of them.
__device__ __forceinline__ void finish_row(const StreamArgs& a, const RowDesc& d, const u64* out, int kk, double* work, SharedCtl* ctl) {
    const RowTail rt{d.rng_word, d.temperature, d.top_p, d.min_p, d.flags, d.out_index, d.hist_begin + d.hist_len};
    const TailOut tout{a.tokens, a.tokens_host, a.status_host, a.pool, a.kept_ids, a.kept_pr, a.kept_n, reinterpret_cast<u64*>(a.shard_out), a.shard_n, a.shard_stride, a.status};
    row_epilogue(out, kk, rt, work, ctl, tout);
}

// For callers whose logits live in host memory: the penalised values at the window's ids, in window order, go straight to
// pinned host memory, where the host waits for every one and stores it into its row (src/sampler.cpp:17); it computes nothing.
template <int T>
__device__ __noinline__ void send_patched(const Segment s, float* out) {
    for (int i = threadIdx.x; i < s.window_len; i += T) {
        const int c = window_id(s, i) - s.id_base;
        if (c >= s.lo && c < s.hi) *reinterpret_cast<volatile float*>(out + i) = transform(__ldcg(s.row + c), c, s);
    }
}

__device__ __forceinline__ void trace_mark(const StreamArgs& a, int slot) {
    if (a.trace && threadIdx.x == 0 && blockIdx.x < 4096u) {
        a.trace[(size_t)blockIdx.x * 8 + slot] = slot == 0 ? global_timer_ns() : (u64)clock64();
        if (slot == 0) a.trace[(size_t)blockIdx.x * 8 + 7] = (u64)clock64();
    }
}

// Room in a list for every value of the warp that reaches `bound`: one shared-memory atomic per warp (lanes of a warp
// that add to one word are served one after the other, 8 cycles each).  hit[i]: the lanes whose i-th value does; entries go
// in order of i, then of lanes.  All lanes call.
template <int N>
__device__ __forceinline__ int warp_reserve(const float (&v)[N], float bound, unsigned (&hit)[N], int* counter) {
    int total = 0;
#pragma unroll
    for (int i = 0; i < N; ++i) {
        hit[i] = __ballot_sync(0xffffffffu, v[i] >= bound);
        total += __popc(hit[i]);
    }
    int p = 0;
    if ((threadIdx.x & 31) == 0 && total) p = atomicAdd(counter, total);
    return __shfl_sync(0xffffffffu, p, 0);
}

// A launch's arguments: with NDESC > 0 the row descriptors come with them - no CTA waits for a read of global memory before
// it knows its row - and with few rows the staged window ids, too, if they are few: such a batch needs no copy to the device.
// (4 KB of arguments cost 0.6 us, reading 256 ids from them 0.2; 1000 ids would take 1.3, more than a copy.)
constexpr int kFewRows = 8, kArgRows = 64, kArgIds = 256;
template <int NDESC>
struct SelectArgs {
    StreamArgs a;
    RowDesc rows[NDESC > 0 ? NDESC : 1];
    int32_t ids[NDESC == kFewRows ? kArgIds : 1];
    __device__ __forceinline__ const int32_t* hist() const { return NDESC == kFewRows && !a.hist ? ids : a.hist; }
    __device__ __forceinline__ const int32_t* drafts() const { return NDESC == kFewRows && !a.drafts ? ids : a.drafts; }
};

template <int T, int NDESC, bool LONG, bool CELLS>
__global__ void __launch_bounds__(T, T == 256 && NDESC > 0 ? 2 : 1024 / T) stream_select_kernel(const __grid_constant__ SelectArgs<NDESC> args) {
    using G = Geometry<T>;
    constexpr int kChunkCells = G::kChunkCells, kWarps = G::kWarps;
    const StreamArgs& a = args.a;
    extern __shared__ __align__(128) unsigned char smem_raw[];
    float4* ring = reinterpret_cast<float4*>(smem_raw);
    u64* picked = reinterpret_cast<u64*>(smem_raw);   // after the stream: candidates, the row's candidates in order, merge list
    u64* out = picked + kPickCap + 32;
    u64* list = out + kMaxK;
    float4* listed = reinterpret_cast<float4*>(smem_raw + G::kRingBytes);
    const int tid = threadIdx.x, lane = tid & 31;
    constexpr int cell_cap = LONG ? G::kWarpCellsLong : CELLS ? G::kWarpCellsMarked : G::kWarpCells;
    int* listed_num = reinterpret_cast<int*>(listed + kWarps * cell_cap);
    float* pen_raw = reinterpret_cast<float*>(listed_num + kWarps * cell_cap);
    int* pen_col = reinterpret_cast<int*>(pen_raw + (a.penalised && !CELLS ? kPenCap : 0));
    StreamCtl* ctl = reinterpret_cast<StreamCtl*>(pen_col + (a.penalised && !CELLS ? kPenCap : 0));
    unsigned* keys = reinterpret_cast<unsigned*>(ctl + 1);   // the largest logits that the row's warps have seen
    u64* recv = reinterpret_cast<u64*>(keys + G::key_words(a.nseg));
    u64* lists = reinterpret_cast<u64*>(listed);
    listed += (tid >> 5) * cell_cap;   // the warp's own
    listed_num += (tid >> 5) * cell_cap;
    pdl_launch_dependents();
    trace_mark(a, 0);
    // Mode 1 waits only before its first write (unless it stores into the logits); otherwise only the launch's latency -
    // placing the CTAs on the SMs - overlaps the end of the launch before it.
    if (a.write_back || a.overlap != 1) pdl_wait_prior();

    const int nseg = a.nseg, row = (int)cluster_id(), seg = (int)cluster_rank();
    const RowDesc& dp = NDESC > 0 ? args.rows[row] : a.rows[row];
    const float* row_ptr = a.logits + (a.row_ld >= 0 ? (int64_t)row * a.row_ld : dp.logits_off);

    const int V = a.n_vocab;
    const RowSpan span = row_span(row_ptr, V, seg, nseg);
    const int head = span.head, n_cells = span.n_cells, c_lo = span.c_lo, c_hi = span.c_hi;
    const float4* cells = span.cells;
    const float qnan = __int_as_float(0x7fc00000), ninf = -__int_as_float(0x7f800000);
    const unsigned slot0 = smem_u32(ring + tid);
    // chunk c of this thread: cells j, j + T, ... go to stage c % kStages
    auto fetch = [&](int c) {
        const int j = c_lo + c * kChunkCells + tid;
        const unsigned dst = slot0 + (unsigned)((c % kStages) * kChunkCells) * (unsigned)sizeof(float4);
#pragma unroll
        for (int u = 0; u < kCells; ++u)
            if (j + u * T < c_hi) cp_async16(dst + (unsigned)(u * T * sizeof(float4)), cells + j + u * T);
        cp_async_commit();
    };
    using Seg = std::conditional_t<CELLS, CellSegment, Segment>;
    unsigned* const bitmap = reinterpret_cast<unsigned*>(recv + (nseg > 1 ? kMergeList : 0));
    const bool has_pen = (dp.flags & kRowPenalty) != 0;
    const int k = dp.k;
    const int most = LONG ? 0 : keys_per_warp(n_cells, nseg, kWarps, k);
    if (tid < 8) {   // the logits outside the whole cells
        const int c = span.edge_column(tid, V, seg, nseg);
        if (c >= 0) cp_async4(smem_u32(&ctl->edge[tid]), row_ptr + c);
        else ctl->edge[tid] = qnan;
    }
    if (tid >= 32 && tid < 40) reinterpret_cast<u64*>(&ctl->desc)[tid - 32] = reinterpret_cast<const u64*>(&dp)[tid - 32];
    if (tid == 0) {
        ctl->lost = 0;
        ctl->kept_n = 0;
        ctl->pen_n = 0;
        ctl->late = 0;
        if (nseg > 1 && !LONG) {
            inbox_init(&ctl->keyed);
            inbox_init(&ctl->counted);
            inbox_init(&ctl->sent);
            inbox_inits_fence();
            inbox_expect(&ctl->keyed, (unsigned)(4 * most * kWarps * nseg));
            inbox_expect(&ctl->counted, (unsigned)(8 * nseg));
        }
    }
    if (nseg > 1) cluster_arrive_relaxed();   // (waited for before the first store to another CTA's shared memory)
    {
        Seg s;
        static_cast<Segment&>(s) = make_segment(a, span, row_ptr, seg, nseg, bitmap);
        s.has_pen = has_pen;
        s.pen = dp.penalty;
        if (has_pen) set_window(s, args.hist(), args.drafts(), dp);
        if constexpr (CELLS) {
            s.table = reinterpret_cast<int*>(smem_raw + G::kRingBytes) - kCellSlots;   // (the list's memory, but for what the rare paths keep there)
            s.slots = s.window_len <= kCellIds / 2 ? kCellSlots / 2 : kCellSlots;
            s.edges = reinterpret_cast<const unsigned*>(&ctl->pen_n);
            s.head = head;
            s.n_cells = n_cells;
        }
        if (tid == 0) static_cast<Seg&>(ctl->seg) = s;
        // Of the stream's copies those of the first chunk go out before the window's bits are set, the others after: a copy takes the
        // load/store unit 16 cycles per warp, and what works on shared memory queues behind them.
        if (has_pen) {
            FirstIds<T> ids;
            ids.load(s);
            clear_bits(bitmap, CELLS ? 8 * ((n_cells + 1023) >> 10) : (s.hi - s.bit0 + 127) >> 7, T);
            fetch(0);
            __syncthreads();
            if constexpr (CELLS) collect_cells<T>(s, ids, reinterpret_cast<unsigned*>(&ctl->pen_n));
            else collect_penalised<T>(s, ids, ctl, pen_raw, pen_col);
            for (int c = 1; c < kStages; ++c) fetch(c);
        } else {
            for (int c = 0; c < kStages; ++c) fetch(c);
        }
    }
    __syncthreads();
    const Seg& s = ctl->seg;
    trace_mark(a, 1);

    // ---- the stream
    const float cap = a.softcap;
    // A segment that fits the ring is only looked at when its final bound is known: nothing is listed.
    const bool held = !LONG && !CELLS && c_hi - c_lo <= kStages * kChunkCells;
    float run_a = ninf, run_b = ninf, thr = -FLT_MAX, admit = -FLT_MAX, seen = ninf;
    int refreshes = 0;
    int wn = 0;           // cells in the warp's list
    bool fresh = false;   // the bound takes in everything seen so far
    bool lost = false;    // a list was too short
    bool again = false;   // the second time through: the bound is final
    const bool raised = CELLS && has_pen && s.pen < 1.0f;
again_from_the_start:
    for (int c = 0, j0 = c_lo + tid;; ++c, j0 += kChunkCells) {
        const int left = c_hi - (j0 - tid);   // cells of the segment from this chunk on
        cp_async_wait<kStages - 1>();
        const float4* st = ring + (c % kStages) * kChunkCells + tid;
        float4 x[kCells];
#pragma unroll
        for (int u = 0; u < kCells; ++u) x[u] = st[u * T];
        if (!CELLS && has_pen) mask_penalised<T>(x, bitmap, j0 - c_lo, left);
        float m[kCells];
#pragma unroll
        for (int u = 0; u < kCells; ++u) m[u] = cell_max(x[u]);
        if (left < kChunkCells) {
#pragma unroll
            for (int u = 0; u < kCells; ++u)
                if (tid + u * T >= left) m[u] = ninf;
        }
        unsigned marked = 0u;
        if (CELLS && has_pen) {
            const uint4 bits = reinterpret_cast<const uint4*>(bitmap)[8 * c + (tid >> 5)];
            marked = ((bits.x >> lane) & 1u) | ((bits.y >> lane) & 1u) << 1 | ((bits.z >> lane) & 1u) << 2 | ((bits.w >> lane) & 1u) << 3;
            float r[kCells];
#pragma unroll
            for (int u = 0; u < kCells; ++u) r[u] = (marked >> u) & 1u ? ninf : m[u];
            run_a = max3(run_a, max3(r[0], r[1], r[2]), r[3]);
            if (raised) {   // a penalty below 1 makes logits larger
#pragma unroll
                for (int u = 0; u < kCells; ++u)
                    if ((marked >> u) & 1u) m[u] = cap != 0.0f ? -ninf : penalise(m[u], s.pen);
            }
        } else if (LONG) {
            run_a = max3(run_a, m[0], m[1]);
            run_b = max3(run_b, m[2], m[3]);
        } else {
            run_a = max3(run_a, max3(m[0], m[1], m[2]), m[3]);
        }
        fetch(c + kStages);   // into the stage just read
        if (held) {
            if (left <= kChunkCells) break;
            continue;
        }
        fresh = !again && ((c & (c + 1)) == 0 || thr <= -FLT_MAX || (k > 64 && c < 4));
        if (fresh) {
            thr = cta_bound<T, 0>(run_a, run_b, k, refreshes++ & 1, ctl);
            admit = thr;
            if (cap != 0.0f) softcap_admit(thr, cap, admit, seen);
            if (wn > cell_cap / 4) wn = prune_cells(listed, listed_num, wn, admit, CELLS && raised ? kMarked : 0);
        }
        if (__any_sync(0xffffffffu, fmaxf(max3(m[0], m[1], m[2]), m[3]) >= admit)) {   // the warp's own list: no atomics
#pragma unroll
            for (int u = 0; u < kCells; ++u) {
                const unsigned hits = __ballot_sync(0xffffffffu, m[u] >= admit);
                const int q = wn + __popc(hits & lanes_below());
                if (m[u] >= admit && q < cell_cap) {
                    listed[q] = x[u];
                    listed_num[q] = (j0 + u * T) | (CELLS && ((marked >> u) & 1u) ? kMarked : 0);
                }
                wn += __popc(hits);
            }
            if (wn > cell_cap) {
                lost = true;
                wn = cell_cap;
            }
        }
        if (left <= kChunkCells) break;
    }
    cp_async_wait<0>();   // (also the penalised logits and those outside the cells: a group has been committed after them)
    if (lost && lane == 0) ctl->lost = 1;
    trace_mark(a, 4);

    // ---- candidates: logits that reach the final bound
    if constexpr (LONG) {
        if (fresh || again) {
            __syncthreads();
        } else {
            thr = cta_bound<T, 0>(run_a, run_b, k, refreshes++ & 1, ctl);
            admit = thr;
        }
        if (cap != 0.0f && !again) softcap_bounds(thr, cap, admit, seen);   // (softcap_admit leaves `seen` to the final bound)
    } else if (again) {
        __syncthreads();
    } else {
        if (nseg > 1) cluster_wait_acquire();   // every CTA of the row runs: its shared memory may be written
        publish_most<T>(run_a, most, seg, nseg, keys, &ctl->keyed);
        if (nseg == 1) __syncthreads();
        if (tid < 32) {
            if (nseg > 1 && !inbox_wait(&ctl->keyed)) {
                ctl->late = 1;
                report_status(a.status, a.status_host, kStatusLate);
            }
            __syncwarp();
            const unsigned least = key_bound(most * kWarps * nseg, k, keys);
            if (lane == 0) ctl->bound = least;
        }
        __syncthreads();
        thr = ctl->late ? -ninf : fmaxf(key_float(ctl->bound), -FLT_MAX);
        admit = thr;
        if (cap != 0.0f) softcap_bounds(thr, cap, admit, seen);
    }
    const bool bounded = thr > -FLT_MAX;
    if (cap == 0.0f) seen = thr;      // (minus infinity is not among the listed ones)
    lost = ctl->lost != 0;
    if (lost && bounded && !again) {   // the early bounds let too much through: the final one will not, unless many logits are equal
        __syncthreads();
        if (tid == 0) ctl->lost = 0;
        for (int c = 0; c < kStages; ++c) fetch(c);
        wn = 0;
        lost = false;
        again = true;
        __syncthreads();
        goto again_from_the_start;
    }
    // Candidates go to a list of this CTA; those of a row of several CTAs straight to the first one's (k <= 64).  A CTA's share of it
    // ends with room for a list that it makes again (64).
    const bool direct = !LONG && nseg > 1;
    const int lseg = 31 - __clz(nseg), share = direct ? min(kPickCap, (kMergeList >> lseg) - 64) : kPickCap;
    unsigned first_recv = 0u, sent_bar = 0u;
    if (direct) {
        first_recv = cluster_map_shared(smem_u32(recv + (kMergeList >> lseg) * seg), 0u);
        sent_bar = cluster_map_shared(smem_u32(&ctl->sent), 0u);
    } else if (held) {
        picked = lists;   // (the ring is still being read)
    }
    auto put = [&](int p, u64 m) {
        if (p >= share) return;
        if (direct) inbox_put(first_recv + 8u * (unsigned)p, m, sent_bar);
        else picked[p] = m;
    };
    auto pick = [&](bool hit, float y, int col) {   // all lanes of the warp
        const unsigned hits = __ballot_sync(0xffffffffu, hit);
        if (hits == 0u) return;
        int p = 0;
        if (lane == 0) p = atomicAdd(&ctl->kept_n, __popc(hits));
        p = __shfl_sync(0xffffffffu, p, 0) + __popc(hits & lanes_below());
        if (hit) put(p, make_comp(y, col + s.id_base));
    };
    auto pick_cell = [&](const float4& v, int col, int pen) {   // a cell per lane, `pen`: penalised ones of its columns
        float xs[4] = {v.x, v.y, v.z, v.w};
        if (s.cap != 0.0f) {
#pragma unroll
            for (int e = 0; e < 4; ++e) xs[e] = xs[e] >= admit || (CELLS && ((pen >> e) & 1)) ? softcap_call(xs[e], s.cap) : ninf;
        }
        if (CELLS && pen) {
#pragma unroll
            for (int e = 0; e < 4; ++e)
                if ((pen >> e) & 1) xs[e] = penalise(xs[e], s.pen);
        }
        const float least = fmaxf(seen, -FLT_MAX);
        if constexpr (LONG) {
            unsigned hit[4];
            int q = warp_reserve<4>(xs, least, hit, &ctl->kept_n);
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                if (xs[e] >= least) put(q + __popc(hit[e] & lanes_below()), make_comp(xs[e], col + e + s.id_base));
                q += __popc(hit[e]);
            }
        } else {   // few: a lane reserves for itself
            const int hits = (xs[0] >= least ? 1 : 0) + (xs[1] >= least ? 1 : 0) + (xs[2] >= least ? 1 : 0) + (xs[3] >= least ? 1 : 0);
            if (hits) {
                int q = atomicAdd(&ctl->kept_n, hits);
#pragma unroll
                for (int e = 0; e < 4; ++e)
                    if (xs[e] >= least) put(q++, make_comp(xs[e], col + e + s.id_base));
            }
        }
    };
    if constexpr (CELLS) {
        if (s.has_pen) {
            fill_table<T>(s);
            __syncthreads();
        }
    }
    if (!lost) {
        if (held) {
            auto cell = [&](int i) {   // the thread's i-th cell of the ring, which holds the segment in order
                const int j = i * T + tid;
                float4 v = make_float4(ninf, ninf, ninf, ninf);
                if (j < c_hi - c_lo) {
                    v = ring[j];
                    if (s.has_pen) {
                        const unsigned bits = s.bitmap[(j >> 3) + 1] >> (4 * (j & 7));
                        if (bits & 1u) v.x = ninf;
                        if (bits & 2u) v.y = ninf;
                        if (bits & 4u) v.z = ninf;
                        if (bits & 8u) v.w = ninf;
                    }
                }
                return v;
            };
            unsigned mine = 0u;
            if (run_a >= admit) {
#pragma unroll
                for (int i = 0; i < kStages * kCells; ++i) mine |= (cell_max(cell(i)) >= admit ? 1u : 0u) << i;
            }
            while (mine) {   // (lanes on their own)
                const int i = __ffs(mine) - 1;
                mine &= mine - 1u;
                pick_cell(cell(i), head + 4 * (c_lo + i * T + tid), 0);
            }
        } else {
            for (int p0 = 0; p0 < wn; p0 += 32) {
                float4 v = make_float4(ninf, ninf, ninf, ninf);
                int col = 0, pen = 0;
                bool reach = false;
                if (p0 + lane < wn) {
                    v = listed[p0 + lane];
                    const int num = listed_num[p0 + lane], cell = num & ~kMarked;
                    col = head + 4 * cell;
                    reach = cell_max(v) >= admit;
                    if constexpr (CELLS) {
                        if (num != cell && (reach || raised)) {
                            pen = penalised_of(s, cell);
                            reach = true;
                        }
                    }
                }
                if (LONG || reach) pick_cell(v, col, pen);
            }
        }
        if (tid < 32 && V != 4 * n_cells) {
            float x = lane < 8 ? ctl->edge[lane] : qnan;
            const bool pen = CELLS && s.has_pen && lane < 8 && ((ctl->pen_n >> lane) & 1);
            if (!CELLS && s.has_pen && x == x && penalised(s, lane < 4 ? lane : head + 4 * n_cells + lane - 4)) x = qnan;   // (looked at on its own)
            float y = s.cap != 0.0f ? softcap_call(x, s.cap) : x;
            if (pen) y = penalise(y, s.pen);
            pick((pen ? y > ninf : x >= admit) && y >= seen, y, lane < 4 ? lane : head + 4 * n_cells + lane - 4);
        }
        if (!CELLS && s.has_pen)
            for_each_penalised<T>(s, ctl->pen_n, pen_raw, pen_col, [&](bool in, float x, int col) {
                const float y = penalise(s.cap != 0.0f ? softcap_call(x, s.cap) : x, s.pen);
                pick(in && y >= seen && y > ninf, y, col);
            });
    }
    __syncthreads();
    int n = ctl->kept_n;
    lost = lost || n > share;
    // (the softcap makes a finite logit of minus infinity, equal to or above others: without a raw bound such columns count, too)
    const bool exact = lost || (LONG && n < k && bounded) || (cap != 0.0f && admit <= -FLT_MAX);
    u64 report = 0ull;   // (to the first CTA)
    if (exact || (n < k && !(direct && bounded))) {
        const int kept = min(n, share);
        if (exact) n = exact_select<T>(s, k, picked, reinterpret_cast<unsigned*>(list), ctl);
        else n = append_masked<T>(s, n, k, picked, reinterpret_cast<unsigned*>(list));
        if (direct) {   // (these work on a list of the CTA's own)
            __syncthreads();
            const int from = exact ? 0 : kept;
            for (int i = from + tid; i < n; i += T) inbox_put(first_recv + 8u * (unsigned)((exact ? share : 0) + i), picked[i], sent_bar);
            report = (u64)(unsigned)(kept + n - from) << 32 | (exact ? 1ull << 16 : 0ull) | (u64)(unsigned)n;
        }
    } else {
        report = (u64)(unsigned)n << 32 | (u64)(unsigned)n;
    }
    if (!CELLS && a.write_back) write_back<T>(s);
    if (!CELLS && a.patched && s.has_pen) send_patched<T>(s, a.patched + dp.gather_off);
    trace_mark(a, 2);
    if (a.trace && tid == 0 && blockIdx.x < 4096u) a.trace[(size_t)blockIdx.x * 8 + 3] = (u64)n;
    if (a.overlap == 1) pdl_wait_prior();   // from here on this launch writes what the previous launch in the stream may still be using

    // ---- the row: the k best of all its segments' candidates, in order
    if (direct) {
        if (tid == 0) inbox_put(cluster_map_shared(smem_u32(&ctl->count[seg]), 0u), report, cluster_map_shared(smem_u32(&ctl->counted), 0u));
        if (seg != 0) {
            trace_mark(a, 6);
            if (ctl->late) outlast_cluster();
            return;
        }
    }
    if (tid >= kPost) return;   // eight warps finish the row (no barrier of the whole CTA or by all threads of the cluster from here on)
    u64* all = picked;
    if (direct) {
        constexpr u64 kUnknown = 1ull << 48;   // (more words than there can be, and no candidate)
        const bool counted = inbox_wait(&ctl->counted);
        const u64 said = !counted ? kUnknown : lane < nseg ? ctl->count[lane] : 0ull;
        const int n_q = (int)(said & 0xFFFFu);
        n = __reduce_add_sync(0xffffffffu, n_q);
        const int words = __reduce_add_sync(0xffffffffu, (int)(said >> 32));
        if (tid == 0 && words < (int)(kUnknown >> 32)) inbox_expect(&ctl->sent, 8u * (unsigned)words);
        const int from = tid >> 5;   // one list: warp w copies segment w's part
        const int before = __reduce_add_sync(0xffffffffu, lane < from ? n_q : 0), mine = __shfl_sync(0xffffffffu, n_q, from);
        const u64* src = recv + (kMergeList >> lseg) * from + ((__shfl_sync(0xffffffffu, (unsigned)said, from) >> 16) & 1u ? share : 0);
        const bool here = inbox_wait(&ctl->sent) && counted;
        if (!here) ctl->late = 1;
        for (int i = lane; here && i < mine; i += 32) list[before + i] = src[i];
        all = list;
        block_sync<kPost, 1>();
        if (ctl->late) {
            n = 0;
            if (tid == 0) report_status(a.status, a.status_host, kStatusLate);
            outlast_cluster();
        }
    } else if (LONG && nseg > 1) {
        cluster_wait_acquire();   // every CTA of the row runs: the first one's shared memory may be written
        const int send_cap = min(kPickCap, kMergeList >> lseg);
        const unsigned dst = cluster_map_shared(smem_u32(recv + seg * send_cap), 0u);
        if (n > send_cap) {       // (many equal logits, or k > 64 and eight segments)
            rank_emit(picked, n, k, list, ctl, [&](int rank, u64 m) { cluster_store_u64(dst + 8u * (unsigned)rank, m); });
            n = min(n, k);
        } else {
            for (int i = tid; i < n; i += kPost) cluster_store_u64(dst + 8u * (unsigned)i, picked[i]);
        }
        if (tid == 0) cluster_store_u32(cluster_map_shared(smem_u32(&ctl->recv_n[seg]), 0u), (unsigned)n);
        __syncwarp();
        cluster_arrive_release();
        if (seg != 0) {
            trace_mark(a, 6);
            return;
        }
        if (tid == 0) ctl->out_cnt = 0;
        cluster_wait_acquire();
        // a bound that k of them reach, then those that reach it (thread t looks after every (256 / nseg)-th candidate of one segment)
        const int q = tid & (nseg - 1), n_q = ctl->recv_n[q];
        const u64* from = recv + q * send_cap;
        run_a = run_b = ninf;
        for (int i = tid >> lseg; i < n_q; i += kPost >> lseg) {
            const float y = comp_value(from[i]);
            if (i & (kPost >> lseg)) run_b = fmaxf(run_b, y);
            else run_a = fmaxf(run_a, y);
        }
        const float floor_y = cta_bound<kPost, 1>(run_a, run_b, k, refreshes & 1, ctl);
        const float least = floor_y > -FLT_MAX ? floor_y : ninf;
        const int most = __reduce_max_sync(0xffffffffu, n_q);   // (every warp has threads of every segment)
        for (int i = tid >> lseg; (i - (tid >> lseg)) < most; i += kPost >> lseg) {
            const u64 m = i < n_q ? from[i] : 0ull;
            const bool hit = m != 0ull && comp_value(m) >= least;
            const unsigned hits = __ballot_sync(0xffffffffu, hit);
            if (hits == 0u) continue;
            int p = 0;
            if ((tid & 31) == 0) p = atomicAdd(&ctl->out_cnt, __popc(hits));
            p = __shfl_sync(0xffffffffu, p, 0) + __popc(hits & lanes_below());
            if (hit) list[p] = m;
        }
        block_sync<kPost, 1>();
        n = ctl->out_cnt;
        all = list;
    }
    rank_emit(all, n, k, all == list ? picked : list, ctl, [&](int rank, u64 m) { out[rank] = m; });
    block_sync<kPost, 1>();
    trace_mark(a, 5);
    finish_row(a, ctl->desc, out, min(n, k), reinterpret_cast<double*>(list), ctl);
    trace_mark(a, 6);
}

// Launches whose rows are all greedy (a verification step at temperature 0, the static entry point): the same stream, but
// a thread keeps the best cell it has seen in registers ("strictly larger" keeps the first of equals, because a thread
// meets its cells in ascending order), the CTA takes the largest composite, and one warp finishes the row.  No bound, no
// lists, no barrier before the end.  (Not with a softcap, which makes different logits equal, nor with write-back or patched values for the host.)
// PEN: some row has a penalty window.  Where none has, the kernel does not know windows: their code between the first copies and the
// stream, passed by, and the looks at whether there is one cost a launch that is waited for 700 cycles of 7550 (136 x 65536, by the SM's
// counter); us per launch in a train, one kernel for both and two: 8.12, 8.03; with windows of 128 ids 9.28, 9.10.
template <int T>
size_t argmax_smem_bytes(int seg_cols) {
    return Geometry<T>::kRingBytes + sizeof(SharedCtl) + window_bytes(seg_cols);
}

template <int T, int NDESC, bool PEN>
__global__ void __launch_bounds__(T, 1024 / T) argmax_kernel(const __grid_constant__ SelectArgs<NDESC> args) {
    constexpr int kChunkCells = Geometry<T>::kChunkCells;
    const StreamArgs& a = args.a;
    extern __shared__ __align__(128) unsigned char smem_raw[];
    float4* ring = reinterpret_cast<float4*>(smem_raw);
    u64* best_of = reinterpret_cast<u64*>(smem_raw);   // after the stream: the warps' best, then the first masked columns
    SharedCtl* ctl = reinterpret_cast<SharedCtl*>(smem_raw + Geometry<T>::kRingBytes);
    constexpr int pen_cap = PEN ? kPenCap : 0;
    float* pen_raw = reinterpret_cast<float*>(ctl + 1);
    int* pen_col = reinterpret_cast<int*>(pen_raw + pen_cap);
    const int tid = threadIdx.x, lane = tid & 31;
    pdl_launch_dependents();
    trace_mark(a, 0);
    if (a.overlap != 1) pdl_wait_prior();

    const int nseg = a.nseg, lseg = 31 - __clz(nseg);
    const int row = (int)(blockIdx.x >> lseg), seg = (int)(blockIdx.x & (unsigned)(nseg - 1));
    const RowDesc& dp = NDESC > 0 ? args.rows[row] : a.rows[row];
    const float* row_ptr = a.logits + (a.row_ld >= 0 ? (int64_t)row * a.row_ld : dp.logits_off);
    const RowSpan w = row_span(row_ptr, a.n_vocab, seg, nseg);
    const float ninf = -__int_as_float(0x7f800000), qnan = __int_as_float(0x7fc00000);
    const unsigned slot0 = smem_u32(ring + tid);
    auto fetch = [&](int c) {
        const int j = w.c_lo + c * kChunkCells + tid;
        const unsigned dst = slot0 + (unsigned)((c % kStages) * kChunkCells) * (unsigned)sizeof(float4);
#pragma unroll
        for (int u = 0; u < kCells; ++u)
            if (j + u * T < w.c_hi) cp_async16(dst + (unsigned)(u * T * sizeof(float4)), w.cells + j + u * T);
        cp_async_commit();
    };
    if constexpr (!PEN)
        for (int c = 0; c < kStages; ++c) fetch(c);
    float edge = qnan;
    int edge_col = -1;
    if (tid < 8) {
        edge_col = w.edge_column(tid, a.n_vocab, seg, nseg);
        if (edge_col >= 0) edge = __ldcg(row_ptr + edge_col);
    }
    if (nseg > 1) cluster_arrive_relaxed();
    Segment s = make_segment(a, w, row_ptr, seg, nseg, reinterpret_cast<unsigned*>(pen_col + pen_cap));
    if constexpr (PEN) {   // (without windows nobody waits for the descriptor before the end)
        s.has_pen = (dp.flags & kRowPenalty) != 0;
        s.pen = dp.penalty;
    }
    if (PEN && s.has_pen) {
        set_window(s, args.hist(), args.drafts(), dp);
        FirstIds<T> ids;
        ids.load(s);
        if (tid == 0) ctl->pen_n = 0;
        clear_bits(s.bitmap, (s.hi - s.bit0 + 127) >> 7, T);
        fetch(0);
        __syncthreads();
        collect_penalised<T>(s, ids, ctl, pen_raw, pen_col);
        for (int c = 1; c < kStages; ++c) fetch(c);
        __syncthreads();
        if (edge_col >= 0 && penalised(s, edge_col)) edge = qnan;
    } else if constexpr (PEN) {
        for (int c = 0; c < kStages; ++c) fetch(c);
    }
    trace_mark(a, 1);

    float best = ninf, floor_x = ninf;
    float4 best_cell = make_float4(0.f, 0.f, 0.f, 0.f);
    int best_num = -1;
    for (int c = 0, j0 = w.c_lo + tid;; ++c, j0 += kChunkCells) {
        const int left = w.c_hi - (j0 - tid);
        cp_async_wait<kStages - 1>();
        const float4* st = ring + (c % kStages) * kChunkCells + tid;
        float4 x[kCells];
#pragma unroll
        for (int u = 0; u < kCells; ++u) x[u] = st[u * T];
        float m[kCells];
#pragma unroll
        for (int u = 0; u < kCells; ++u) m[u] = tid + u * T < left ? cell_max(x[u]) : ninf;
        // (`floor_x` is the warp's best so far: what does not exceed it cannot win, and a warp rarely sees more than ten such chunks)
        if (__any_sync(0xffffffffu, fmaxf(max3(m[0], m[1], m[2]), m[3]) > floor_x)) {
            if (PEN && s.has_pen) {
                mask_penalised<T>(x, s.bitmap, j0 - w.c_lo, left);
#pragma unroll
                for (int u = 0; u < kCells; ++u)
                    if (tid + u * T < left) m[u] = cell_max(x[u]);
            }
#pragma unroll
            for (int u = 0; u < kCells; ++u) {
                if (m[u] > best) {
                    best = m[u];
                    best_cell = x[u];
                    best_num = j0 + u * T;
                }
            }
            floor_x = key_float(__reduce_max_sync(0xffffffffu, float_key(best)));
        }
        fetch(c + kStages);
        if (left <= kChunkCells) break;
    }
    cp_async_wait<0>();
    if (PEN && s.has_pen) __syncthreads();   // the penalised logits were fetched by other threads
    trace_mark(a, 4);

    u64 top = 0ull;
    if (best_num >= 0) {
        const int e = best_cell.x == best ? 0 : best_cell.y == best ? 1 : best_cell.z == best ? 2 : 3;
        top = make_comp(best, w.head + 4 * best_num + e + s.id_base);
    }
    if (edge > ninf) top = max(top, make_comp(edge, edge_col + s.id_base));
    if (PEN && s.has_pen)
        for_each_penalised<T>(s, ctl->pen_n, pen_raw, pen_col, [&](bool in, float x, int col) {
            const float y = penalise(x, s.pen);
            if (in && y > ninf) top = max(top, make_comp(y, col + s.id_base));
        });
    top = warp_max_u64(top);
    __syncthreads();   // the ring's memory is free
    if (lane == 0) best_of[tid >> 5] = top;
    if (__syncthreads_or(top != 0ull) == 0) {   // nothing above minus infinity: the first column that holds it, if any
        u64* found = best_of + 32;
        const int n = append_masked<T>(s, 0, 1, found, reinterpret_cast<unsigned*>(found + 8));
        __syncthreads();
        if (tid == 0 && n > 0) best_of[0] = found[0];
        __syncthreads();
    }
    trace_mark(a, 2);
    if (tid >= 32) return;
    top = warp_max_u64(lane < T / 32 ? best_of[lane] : 0ull);
    if (a.overlap == 1) pdl_wait_prior();
    if (nseg > 1) {
        cluster_wait_acquire();   // every CTA of the row runs: the first one's shared memory may be written
        if (lane == 0) cluster_store_u64(cluster_map_shared(smem_u32(&ctl->red[seg]), 0u), top);
        __syncwarp();
        cluster_arrive_release();
        if (seg != 0) return;
        cluster_wait_acquire();
        top = warp_max_u64(lane < nseg ? ctl->red[lane] : 0ull);
    }
    trace_mark(a, 5);
    if (lane == 0) best_of[0] = top;
    __syncwarp();
    finish_row(a, dp, best_of, top != 0ull ? 1 : 0, reinterpret_cast<double*>(best_of + 8), ctl);
    trace_mark(a, 6);
}

template <int T, int NDESC>
int launch_select(cudaLaunchConfig_t& cfg, const StreamArgs& a, const RowDesc* rows, const int32_t* ids, int n_ids) {
    const int seg_cols = a.penalised ? segment_columns(a.n_vocab, a.nseg) : 0;
    cfg.blockDim = dim3(T);
    cfg.dynamicSmemBytes = Geometry<T>::smem_bytes(a.nseg, a.kmax, seg_cols);
    if (cfg.dynamicSmemBytes > (size_t)kSelectSmemMax) return (int)cudaErrorInvalidValue;
    if (a.kmax <= 64) {   // the keys that the warps of a row hand over have to fit (they do in every layout that plan_select gives)
        // (a row has at least so many whole cells, and more cells or a smaller k mean no more keys)
        const int cells = (a.n_vocab > 3 ? a.n_vocab - 3 : 0) / 4;
        if (keys_per_warp(cells, a.nseg, T / 32, a.kmax) * (T / 32) * a.nseg > Geometry<T>::key_words(a.nseg)) return (int)cudaErrorInvalidValue;
    }
    SelectArgs<NDESC> args;
    args.a = a;
    if (NDESC > 0) std::memcpy(args.rows, rows, sizeof(RowDesc) * (size_t)a.n_rows);
    if (NDESC == kFewRows && n_ids > 0) std::memcpy(args.ids, ids, sizeof(int32_t) * (size_t)n_ids);
    if (a.all_greedy && a.softcap == 0.0f && !a.write_back && !a.patched) {
        cfg.dynamicSmemBytes = argmax_smem_bytes<T>(seg_cols);
        return (int)(a.penalised ? cudaLaunchKernelEx(&cfg, argmax_kernel<T, NDESC, true>, args) : cudaLaunchKernelEx(&cfg, argmax_kernel<T, NDESC, false>, args));
    }
    if constexpr (T == 256 && NDESC == 0) {
        // Whole rows on small CTAs, four per SM, that do not fit the ring: a bit per column costs every thread four words per chunk, and
        // above 65536 columns the bitmap leaves room for three CTAs or two.  us per launch (chained), bit per column -> per cell, windows
        // of 512 ids: 512 x 16384 22.6 -> 17.6, 200 x 49152 31.0 -> 27.5, 512 x 49152 35.0 -> 31.2, 160 x 16384 22.3 -> 19.3; of 128 ids 512 x
        // 32768 24.4 -> 21.0, of 1024 36.2 -> 26.6.  Windows of more than kCellIds ids would fill more than half of the table.
        if (a.penalised && a.nseg == 1 && a.kmax <= 64 && a.n_vocab >= 4 * kStages * Geometry<T>::kChunkCells + 8 && a.window_max <= kCellIds && !a.write_back && !a.patched) {
            cfg.dynamicSmemBytes = Geometry<T>::smem_bytes(1, a.kmax, 0, true) + cell_bits_bytes(seg_cols);
            return (int)cudaLaunchKernelEx(&cfg, stream_select_kernel<T, NDESC, false, true>, args);
        }
    }
    return (int)(a.kmax > 64 ? cudaLaunchKernelEx(&cfg, stream_select_kernel<T, NDESC, true, false>, args) : cudaLaunchKernelEx(&cfg, stream_select_kernel<T, NDESC, false, false>, args));
}
template <int T>
int launch_select(cudaLaunchConfig_t& cfg, const StreamArgs& a, const RowDesc* rows, const int32_t* ids, int n_ids) {
    if (rows && a.n_rows <= kFewRows) return launch_select<T, kFewRows>(cfg, a, rows, ids, n_ids);
    if (rows && a.n_rows <= kArgRows) return launch_select<T, kArgRows>(cfg, a, rows, nullptr, 0);
    return launch_select<T, 0>(cfg, a, nullptr, nullptr, 0);
}
template <int T, int NDESC>
int prepare_select() {
    cudaError_t e = cudaFuncSetAttribute(argmax_kernel<T, NDESC, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, kSelectSmemMax);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(argmax_kernel<T, NDESC, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, kSelectSmemMax);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(stream_select_kernel<T, NDESC, false, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, kSelectSmemMax);
    if constexpr (T == 256 && NDESC == 0)
        if (e == cudaSuccess) e = cudaFuncSetAttribute(stream_select_kernel<T, NDESC, false, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, kSelectSmemMax);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(stream_select_kernel<T, NDESC, true, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, kSelectSmemMax);
    return (int)e;
}

}  // namespace

// Per-device set-up (the current device): opt in to the large dynamic shared memory.
int prepare_device_kernels() {
    for (int e : {prepare_select<256, 0>(), prepare_select<256, kFewRows>(), prepare_select<256, kArgRows>(), prepare_select<1024, 0>(),
                  prepare_select<1024, kFewRows>(), prepare_select<1024, kArgRows>()})
        if (e != 0) return e;
    return 0;
}

bool rows_fit_launch(int n_rows, int64_t n_ids) { return n_ids == 0 ? n_rows <= kArgRows : n_rows <= kFewRows && n_ids <= kArgIds; }

int launch_stream_kernel(StreamArgs a, const RowDesc* host_rows, const int32_t* host_ids, int n_ids, bool ids_are_windows, void* stream) {
    if (n_ids > 0) {   // the staged ids go with the launch: the windows themselves, or the drafts behind windows in the id pool
        a.drafts = nullptr;
        if (ids_are_windows) a.hist = nullptr;
    }
    // Plain stream order, too, is launched with programmatic serialization where that pays: every CTA waits for the launch before to be
    // complete (pdl_wait_prior), and only placing the CTAs overlaps its end.  us per launch in a train, without -> with: 1 x 65536 10.4 ->
    // 7.8, 32 x 131072 14.0 -> 11.1, 64 x 262144 22.8 -> 20.5, 148 x 131072 23.9 -> 21.2, 512 x 32768 22.8 -> 20.6.  Not where a few small CTAs
    // per SM are the whole launch: placed while others still run, they pile up on some SMs (200 x 131072 31.4 -> 41.0, 300 x 65536 26.3 -> 29.3);
    // clusters do not (37 x 65536, k = 16, 296 CTAs 15.4 -> 13.3).
    const int ctas = a.n_rows * a.nseg;
    const bool chained = a.overlap == 0 && !a.unchained && (a.wide || ctas <= (a.nseg > 1 ? 2 : 1) * a.sms || ctas >= 3 * a.sms);
    cudaLaunchAttribute attr[2];
    int n = 0;
    if (a.overlap || chained) {
        attr[n].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[n].val.programmaticStreamSerializationAllowed = 1;
        ++n;
    }
    if (a.nseg > 1) {
        attr[n].id = cudaLaunchAttributeClusterDimension;
        attr[n].val.clusterDim.x = (unsigned)a.nseg;
        attr[n].val.clusterDim.y = 1;
        attr[n].val.clusterDim.z = 1;
        ++n;
    }
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3((unsigned)(a.n_rows * a.nseg));
    cfg.stream = static_cast<cudaStream_t>(stream);
    cfg.attrs = attr;
    cfg.numAttrs = n;
    return a.wide ? launch_select<1024>(cfg, a, host_rows, host_ids, n_ids) : launch_select<256>(cfg, a, host_rows, host_ids, n_ids);
}

// How a launch is laid out: small CTAs (256 threads) or large ones (1024), and the segments of a row.  Measured on B200,
// us per launch with windows of 512 ids; s1 = small, one segment (c: penalised logits by cells), w2 = large, two.
// Few rows: small CTAs, the row cut as finely as two per SM allow and segments of 2048 logits (4096, and a CTA per SM at the most, for
// more than eight rows): 1 x 65536, k = 40: s2 11.8, s4 9.5, s8 7.9, w4 8.9; 8 x 16384: s2 9.2, s8 8.0; 30 x 16384: s2 8.7, s4 8.2, s8 8.5.
// Long rows, as many as there are clusters of eight large CTAs that run at once (15): those, from 100000 logits on (1 x 262144: s8
// 12.9, w8 10.7; 14 x 131072: s8 11.6, w4 11.1, w8 10.4; 6 x 90000: s8 9.5, w8 9.9; 16 x 131072: w4 10.4, w8 15.5).
// Medium batches: large CTAs, one per SM, in clusters of four or two while those run at once (clusters of four on 132 SMs only: 37 x
// 262144 w4 24.7, w2 19.6; 64 x 131072: s4 16.1, w1 19.5, w2 16.2; 148 x 131072: s1 28.8, s2 23.3, w1 21.3); four small ones below 65536
// logits up to 64 rows (44 x 40000: s4 9.9, w2 10.8; 64 x 49152: 11.5, 12.8; 70 x 40000: 11.8 both; 50 x 65536: 12.3, 11.9).
// Many rows: a small CTA per row, several per SM, so that the steps of one run beside the stream of the others (plain order: 200 x
// 131072, k = 40: s1 31.5, s2 41.5, w1 38.2; 160 x 65536: s1 24.9, s2 24.8, w1 28.6; 296 x 262144: s1 57.3, s2 63.8, w1 63.0; 512 x 32768: s1
// 20.8, w1 40.4).
// k > 64: a small CTA has longer lists and more bounds to find: large ones, in two segments while a pair per row runs at once (32 x
// 65536, k = 200: w1 22.3, w2 17.9, s4 23.0), and above that where logits times k are many (512 x 65536, k = 100: s1 51.4, w1 67.4; k = 200 66.5,
// 80.9; k = 256 87.3, 86.2; 300 x 100000, k = 200 59.1, 68.8; 512 x 131072, k = 100 73.8, 86.1; k = 256 134, 109; 300 x 262144, k = 100 102, 92).
// All greedy: little after the stream.  Up to three CTAs per SM two segments pay (200 x 262144: s1 37.4, s2 35.2); windows of more than
// 65536 columns leave room for three or two CTAs per SM, and one large one streams better than a second wave (512 x 262144: s1 104, w1 88).
SelectPlan plan_select(int n_rows, int n_vocab, int sms, int kmax, bool all_greedy, bool penalised) {
    SelectPlan pl;
    auto fits = [&](int nseg, int most, int columns = 8192) { return n_rows * nseg <= most && n_vocab / nseg >= columns; };
    if (kmax > 64) {
        pl.wide = n_rows <= sms || (int64_t)n_vocab * kmax >= (kmax > 224 ? 10000000 : 24000000);
        if (fits(2, sms) && n_vocab >= 32768) pl.nseg = 2;
    } else if (n_rows > sms) {
        if (all_greedy && n_vocab >= 65536 && n_rows <= sms + sms / 2) pl.nseg = 2;
        pl.wide = penalised && all_greedy && n_vocab > 65536 && n_rows > 3 * sms;
    } else {
        pl.wide = n_rows > sms / 4 || (kmax > 32 && n_rows > 8 && n_vocab >= 65536);
        if (pl.wide) pl.nseg = fits(4, sms - sms / 10) ? 4 : fits(2, sms) ? 2 : 1;
        if (n_vocab >= 100000 && fits(8, sms - sms / 5)) {
            pl.wide = true;
            pl.nseg = 8;
        }
        if (pl.wide && !all_greedy && n_vocab < 65536 && n_rows > sms / 4 && fits(4, 2 * sms - sms / 4)) {
            pl.wide = false;
            pl.nseg = 4;
        }
    }
    // (the bitmap of a very long segment - above 380000 columns - does not fit beside a large CTA's ring, but always beside a small one's)
    if (pl.wide && penalised && Geometry<1024>::smem_bytes(pl.nseg, kmax, segment_columns(n_vocab, pl.nseg)) > (size_t)kSelectSmemMax) pl = SelectPlan{};
    if (!pl.wide && n_rows <= sms)
        while (pl.nseg < 8 && (fits(2 * pl.nseg, 2 * sms) || fits(2 * pl.nseg, n_rows <= 8 ? 2 * sms : sms, n_rows <= 8 ? 2048 : 4096))) pl.nseg *= 2;
    return pl;
}

}  // namespace fsb

// ---------------------------------------------------------------------------------------------- fsb_argmax_rows_static
// Greedy tokens of device-resident rows with no allocation at all: the streaming kernel above, with its row descriptors
// and status word in one array that is part of this library's image.
namespace fsb {
namespace {

constexpr int kStaticMaxRows = FSB_STATIC_MAX_ROWS;
constexpr size_t kStaticStatusOff = sizeof(RowDesc) * kStaticMaxRows;   // behind RowDesc[kStaticMaxRows]
static __device__ __align__(256) unsigned char g_static_scratch[kStaticStatusOff + 256];

constexpr int kStaticMaxDevices = 64;
struct StaticDevice {
    void* base = nullptr;   // device address of g_static_scratch on this device
    int sms = 0;            // its multiprocessors
};
StaticDevice g_static_dev[kStaticMaxDevices];

// Row descriptors of plain greedy rows (no penalty window): row r starts at r * ld, its token goes to tokens[r].
// The kernel also clears the status word a previous call may have left set (a call that was not waited for and whose
// kernel reported an error): stream order puts this before the streaming kernel.
__global__ void static_greedy_rows_kernel(RowDesc* rows, int n_rows, int64_t ld, uint32_t* status) {
    const int r = threadIdx.x;
    if (r == 0) *status = 0u;
    if (r >= n_rows) return;
    RowDesc d{};
    d.logits_off = (int64_t)r * ld;
    d.k = 1;
    d.k_global = 1;
    d.temperature = 0.0f;
    d.top_p = 1.0f;
    d.penalty = 1.0f;
    d.flags = kRowGreedy;
    d.out_index = r;
    rows[r] = d;
}

}  // namespace
}  // namespace fsb

extern "C" int fsb_argmax_rows_static(int device, const float* logits_dev, int64_t ld, int n_rows, int n_vocab, int32_t* tokens_dev,
                                      void* cuda_stream, unsigned flags) {
    using namespace fsb;
    if (!logits_dev || !tokens_dev || n_rows < 0 || n_vocab <= 0 || ld < n_vocab || (flags & ~FSB_STATIC_WAIT)) return FSB_ERR_INVALID;
    if (n_rows > kStaticMaxRows) return FSB_ERR_CAPACITY;   // the static array holds FSB_STATIC_MAX_ROWS descriptors, no more
    if (device < 0 || device >= kStaticMaxDevices) return FSB_ERR_NO_DEVICE;
    if (n_rows == 0) return FSB_OK;
    int prev = -1;
    if (cudaGetDevice(&prev) != cudaSuccess) return FSB_ERR_NO_DEVICE;
    if (cudaSetDevice(device) != cudaSuccess) return FSB_ERR_NO_DEVICE;
    int rc = FSB_OK;
    StaticDevice& sd = g_static_dev[device];
    if (!sd.base) {   // first call on this device (it is current): where the array lives, how many SMs there are
        void* p = nullptr;
        int sms = 0;
        if (cudaGetSymbolAddress(&p, g_static_scratch) != cudaSuccess || !p) rc = FSB_ERR_CUDA;
        if (rc == FSB_OK && prepare_device_kernels() != 0) rc = FSB_ERR_CUDA;
        if (rc == FSB_OK && cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device) != cudaSuccess) rc = FSB_ERR_CUDA;
        if (rc == FSB_OK) {
            sd.sms = sms > 0 ? sms : 1;
            sd.base = p;
        }
    }
    if (rc == FSB_OK) {
        unsigned char* base = static_cast<unsigned char*>(sd.base);
        cudaStream_t st = static_cast<cudaStream_t>(cuda_stream);
        RowDesc* rows = reinterpret_cast<RowDesc*>(base);
        uint32_t* status = reinterpret_cast<uint32_t*>(base + kStaticStatusOff);
        static_greedy_rows_kernel<<<1, kStaticMaxRows, 0, st>>>(rows, n_rows, ld, status);
        if (cudaGetLastError() != cudaSuccess) rc = FSB_ERR_CUDA;
        StreamArgs a{};
        a.logits = logits_dev;
        a.rows = rows;
        a.tokens = tokens_dev;
        a.status = status;
        a.row_ld = ld;
        a.n_rows = n_rows;
        a.n_vocab = n_vocab;
        a.kmax = 1;
        a.all_greedy = 1;
        a.sms = sd.sms;
        a.unchained = 1;   // (the stream may be capturing, for all that is known here)
        const SelectPlan pl = plan_select(n_rows, n_vocab, sd.sms, 1, true, false);
        a.nseg = pl.nseg;
        a.wide = pl.wide ? 1 : 0;
        if (rc == FSB_OK && launch_stream_kernel(a, nullptr, nullptr, 0, false, st) != 0) rc = FSB_ERR_CUDA;
        if (rc == FSB_OK && (flags & FSB_STATIC_WAIT)) {
            uint32_t word = 0;
            if (cudaMemcpyAsync(&word, status, sizeof word, cudaMemcpyDeviceToHost, st) != cudaSuccess || cudaStreamSynchronize(st) != cudaSuccess) rc = FSB_ERR_CUDA;
            else if (word != 0u) rc = FSB_ERR_DEVICE;
        }
    }
    if (prev >= 0 && prev != device) cudaSetDevice(prev);
    return rc;
}
