// fsb_device.cuh - device-side building blocks of the sampling kernels (sm_100a).
//
//  * order-preserving 64-bit candidate keys ("composites"): (logit descending, token id ascending) becomes plain
//    unsigned descending order, with -0.0f and +0.0f mapped to the same key - the order of the reference's
//    comparator `a.first > b.first || (a.first == b.first && a.second < b.second)` (src/sampler.cpp:31,34);
//  * thread-block cluster and programmatic-launch primitives;
//  * a CTA-wide ordering of the k largest composites of a list;
//  * the per-row epilogue: softmax in fp64 with the reference's sequential sums, min-p, top-p and the draw
//    (src/sampler.cpp:37-49).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include <cfloat>
#include <type_traits>

#include "fsb_internal.h"

namespace fsb {

using u64 = unsigned long long;

// ---------------------------------------------------------------------------------------------- composites
__device__ __forceinline__ u64 make_comp(float x, int id) {
    unsigned u = __float_as_uint(x);
    if (u == 0x80000000u) u = 0u;                                     // -0.0f ties with +0.0f
    const unsigned key = (u & 0x80000000u) ? ~u : (u | 0x80000000u);  // monotone: larger float -> larger key
    return ((u64)key << 32) | (u64)(0xFFFFFFFFu - (unsigned)id);      // lower id -> larger composite
}
__device__ __forceinline__ float comp_value(u64 c) {
    const unsigned key = (unsigned)(c >> 32);
    return __uint_as_float((key & 0x80000000u) ? (key & 0x7FFFFFFFu) : ~key);
}
__device__ __forceinline__ int comp_id(u64 c) { return (int)(0xFFFFFFFFu - (unsigned)(c & 0xFFFFFFFFull)); }

// Order-preserving 32-bit key of a float (the upper half of a composite) and its inverse.
__device__ __forceinline__ unsigned float_key(float x) {
    unsigned u = __float_as_uint(x);
    if (u == 0x80000000u) u = 0u;
    return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
__device__ __forceinline__ float key_float(unsigned key) { return __uint_as_float((key & 0x80000000u) ? (key & 0x7FFFFFFFu) : ~key); }

// max of three floats in one instruction (sm_100)
__device__ __forceinline__ float max3(float a, float b, float c) {
    float d;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
    return d;
}

// ---------------------------------------------------------------------------------------------- softcap
static __device__ __noinline__ float softcap_call(float x, float cap) { return __fmul_rn(cap, tanhf(__fdiv_rn(x, cap))); }   // src/model_gemma4.cpp:521
// The softcap y(x) = cap * tanhf(x / cap) is monotone up to rounding: the division, tanhf (2 ulp) and the product are
// together off by less than cap * 2^-22.  For a raw bound `thr`: `seen` is a value that every logit x >= thr reaches
// after the softcap, `admit` a raw value below which no logit reaches `seen` - the raw bound moved down until the
// softcap's value is a margin of cap * 2^-20 below `seen` (lane j tries 2^j times a small step).
__device__ __forceinline__ void softcap_bounds(float thr, float cap, float& admit, float& seen) {
    if (thr <= -FLT_MAX) {
        admit = -FLT_MAX;
        seen = -__int_as_float(0x7f800000);
        return;
    }
    const float t0 = fminf(thr, 1e38f), margin = cap * 9.5367431640625e-7f;
    seen = softcap_call(t0, cap) - margin;
    const float t = t0 - ldexpf((fabsf(t0) + cap) * 9.5367431640625e-7f, threadIdx.x & 31);
    const unsigned ok = __ballot_sync(0xffffffffu, softcap_call(t, cap) <= seen - margin);
    admit = ok ? __shfl_sync(0xffffffffu, t, __ffs(ok) - 1) : -FLT_MAX;
    admit = fmaxf(admit, -FLT_MAX);
}

// `admit` alone, for a bound that will be refined: up to four caps from zero the softcap's slope is at least 1 - tanh(4)^2 = 0.0013, so what
// lies 0.005 caps further down is 6.7e-6 caps below after it - more than the margin of 2^-20 caps and three roundings of 2^-22 - and
// so below whatever a higher bound makes `seen`.  (All warps work out softcap_bounds alike, 1000 cycles of 32 warps' issue slots at every
// refresh: 1.6 us of a launch of 64 x 262144.)
__device__ __forceinline__ void softcap_admit(float thr, float cap, float& admit, float& seen) {
    if (fabsf(thr) <= 4.0f * cap) admit = fmaxf(thr - 0.005f * cap, -FLT_MAX);
    else softcap_bounds(thr, cap, admit, seen);
}

// Asynchronous 16-byte copies global -> shared memory; a thread waits for its own, by groups.
__device__ __forceinline__ void cp_async16(unsigned dst, const void* src) { asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory"); }
__device__ __forceinline__ void cp_async4(unsigned dst, const void* src) { asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(dst), "l"(src) : "memory"); }
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

__device__ __forceinline__ unsigned smem_u32(const void* p) { return (unsigned)__cvta_generic_to_shared(p); }

// ---------------------------------------------------------------------------------------------- launch order
// Programmatic dependent launch: let the next launch in the stream begin as resources free up, and wait for the
// previous launch to be complete (and its memory visible) before touching anything it wrote.
__device__ __forceinline__ void pdl_launch_dependents() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void pdl_wait_prior() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// Thread-block clusters (the CTAs that share a row): the address of a shared-memory location in another CTA of the
// cluster, stores to it, and the cluster's barrier (arrive releases this thread's stores to the cluster, wait acquires
// the others').
__device__ __forceinline__ unsigned cluster_rank() {
    unsigned r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ unsigned cluster_id() {
    unsigned r;
    asm volatile("mov.u32 %0, %%clusterid.x;" : "=r"(r));
    return r;
}
__device__ __forceinline__ unsigned cluster_map_shared(unsigned local_addr, unsigned rank) {
    unsigned a;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(local_addr), "r"(rank));
    return a;
}
__device__ __forceinline__ void cluster_store_u64(unsigned addr, u64 v) { asm volatile("st.shared::cluster.u64 [%0], %1;" ::"r"(addr), "l"(v) : "memory"); }
__device__ __forceinline__ void cluster_store_u32(unsigned addr, unsigned v) { asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(addr), "r"(v) : "memory"); }
// An arrival that releases nothing ("this CTA has started"): it does not wait for the thread's copies in flight.
__device__ __forceinline__ void cluster_arrive_relaxed() { asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_arrive_release() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait_acquire() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }
// Ends when all other CTAs of the cluster have left or are here, too (the barrier does not count threads that have exited).  Whole warps.
__device__ __forceinline__ void outlast_cluster() {
    __syncwarp();
    cluster_arrive_release();
    cluster_wait_acquire();
}

// Stores to another CTA's shared memory that a barrier there counts, by bytes: the receiver waits for what it expects, and nobody
// for a fence (a release of the cluster's barrier takes 1200 cycles).  One thread of the receiver initialises the barrier, and
// expects the bytes, before or after they come; inbox_inits_fence before that CTA arrives at the cluster's barrier.
__device__ __forceinline__ void inbox_init(u64* bar) { asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(bar)) : "memory"); }
__device__ __forceinline__ void inbox_inits_fence() { asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory"); }
__device__ __forceinline__ void inbox_expect(u64* bar, unsigned bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ void inbox_put(unsigned addr, unsigned v, unsigned bar) {
    asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.b32 [%0], %1, [%2];" ::"r"(addr), "r"(v), "r"(bar) : "memory");
}
__device__ __forceinline__ void inbox_put(unsigned addr, u64 v, unsigned bar) {
    asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.b64 [%0], %1, [%2];" ::"r"(addr), "l"(v), "r"(bar) : "memory");
}
// A bulk copy global -> own shared memory (16-byte aligned, a multiple of 16 bytes), counted by such a barrier, too.
__device__ __forceinline__ void bulk_copy(void* dst, const void* src, unsigned bytes, u64* bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(smem_u32(dst)), "l"(src), "r"(bytes), "r"(smem_u32(bar)) : "memory");
}
// Waits until everything expected has come; gives up (false) after a million looks, for each of which the hardware may suspend the
// thread for a microsecond.  Threads of a CTA may differ in what they get.  (A test has waits run out.)
#ifndef FSB_INBOX_LOOKS
#define FSB_INBOX_LOOKS (1 << 20)
#endif
__device__ __forceinline__ bool inbox_wait(u64* bar) {
    for (int i = FSB_INBOX_LOOKS; i > 0; --i) {
        unsigned done;
        asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], 0, 1000;\n\tselp.u32 %0, 1, 0, p;\n\t}"
                     : "=r"(done) : "r"(smem_u32(bar)) : "memory");
        if (done) return true;
    }
    return false;
}

__device__ __forceinline__ u64 global_timer_ns() {
    u64 t;
    asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
    return t;
}

// ---------------------------------------------------------------------------------------------- shared control block
// A barrier of the CTA's first T threads.  BAR 0: the whole CTA; BAR 1: those that are still at work when the others have
// left (the steps after the stream are short chains: more than eight warps would only issue the same instructions more
// often).
template <int T, int BAR>
__device__ __forceinline__ void block_sync() { asm volatile("bar.sync %0, %1;" ::"n"(BAR), "n"(T) : "memory"); }

constexpr int kPost = 256;   // threads that finish a row
static_assert(kPost == kMaxK && kMaxK % 16 == 0, "the epilogue has a thread per candidate and reads them 16 at a time");

struct SharedCtl {
    alignas(16) unsigned top[2][32];          // per-warp bounds (keys), double buffered
    float edge[8];                            // the row's logits outside its whole 16-byte cells (NaN: none)
    u64 red[2 * kPost / 32];                  // cross-warp reduction scratch
    int sum[3];                               // rotating counters of the selection steps
    int lost;                                 // a warp's list of cells was too short
    int kept_n;                               // candidates picked from the lists
    int pen_n;                                // penalised columns of the segment
    int out_cnt;
    int recv_n[8];                            // clusters: candidates that segment r of the row has sent
    u64 sel_prefix;
    int sel_need, sel_in_bin;
};

// ---------------------------------------------------------------------------------------------- top-k selection
// Smallest and largest of the composites the threads hold (each thread passes the extremes of its own; threads
// with nothing pass ~0 and 0).  All of the first kPost threads must call.
__device__ __forceinline__ void cta_minmax(u64& mn, u64& mx, SharedCtl* ctl) {
    constexpr int T = kPost;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int o = 16; o; o >>= 1) {
        mn = min(mn, __shfl_xor_sync(0xffffffffu, mn, o));
        mx = max(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    }
    if (lane == 0) {
        ctl->red[warp] = mn;
        ctl->red[T / 32 + warp] = mx;
    }
    block_sync<kPost, 1>();
    mn = ctl->red[0];
    mx = ctl->red[T / 32];
#pragma unroll
    for (int w = 1; w < T / 32; ++w) {
        mn = min(mn, ctl->red[w]);
        mx = max(mx, ctl->red[T / 32 + w]);
    }
    block_sync<kPost, 1>();   // the scratch may be written again
}

// Bound L of the k largest among n > k distinct composites held by the first kPost threads: exactly k composites
// are >= L.  count_ge(t) = how many of this thread's composites are >= t.  MSB-first bisection from the highest bit
// in which the composites differ: every step is one warp reduction, one shared-memory add per warp and one
// barrier, and the search stops as soon as a trial bound is passed by exactly k composites.
template <class Count>
__device__ __forceinline__ u64 bisect_bound(int k, u64 mn, u64 mx, SharedCtl* ctl, Count count_ge) {
    if (mx == mn) return mn;
    const int tid = threadIdx.x;
    const int hb = 63 - __clzll((long long)(mx ^ mn));
    u64 pfx = (hb == 63) ? 0ull : (mx & (~0ull << (hb + 1)));
    if (tid == 0) ctl->sum[0] = 0;
    block_sync<kPost, 1>();
    int step = 0;
#pragma unroll 1
    for (int b = hb; b >= 0; --b, ++step) {
        const u64 trial = pfx | (1ull << b);
        const int wsum = __reduce_add_sync(0xffffffffu, count_ge(trial));
        if ((tid & 31) == 0 && wsum) atomicAdd(&ctl->sum[step % 3], wsum);
        if (tid == 0) ctl->sum[(step + 1) % 3] = 0;   // last read two barriers ago
        block_sync<kPost, 1>();
        const int total = ctl->sum[step % 3];
        if (total >= k) pfx = trial;
        if (total == k) break;
    }
    return pfx;
}

// Keeps the k largest of list[0..n) (distinct composites in shared memory) in list[0..k), unordered, and returns
// min(n, k).  `tmp` is scratch for k composites outside the list.  The first kPost threads call.
static __device__ __noinline__ int select_list_topk(u64* list, int n, int k, u64* tmp, SharedCtl* ctl) {
    constexpr int T = kPost;
    if (n <= k) return n;
    const int tid = threadIdx.x;
    u64 mn = ~0ull, mx = 0ull;
#pragma unroll 1
    for (int i = tid; i < n; i += T) {
        const u64 c = list[i];
        mn = min(mn, c);
        mx = max(mx, c);
    }
    cta_minmax(mn, mx, ctl);
    const u64 L = bisect_bound(k, mn, mx, ctl, [&](u64 t) {
        int c = 0;
#pragma unroll 1
        for (int i = tid; i < n; i += T) c += list[i] >= t ? 1 : 0;
        return c;
    });
    if (tid == 0) ctl->out_cnt = 0;
    block_sync<kPost, 1>();
#pragma unroll 1
    for (int i = tid; i < n; i += T) {
        const u64 c = list[i];
        if (c >= L) {
            const int p = atomicAdd(&ctl->out_cnt, 1);
            if (p < k) tmp[p] = c;
        }
    }
    block_sync<kPost, 1>();
#pragma unroll 1
    for (int i = tid; i < k; i += T) list[i] = tmp[i];
    block_sync<kPost, 1>();
    return k;
}

// Ranks the composites buf[0..n) (distinct but for zeros, which rank last; shared memory, 16-byte aligned, room for
// 64 more entries) and calls emit(rank, composite) once for each that ranks below k.
//  n <= 128: by counting.  Four lanes count for an entry, or for two of them, each a quarter of the list, two entries per 16-byte
//    broadcast read and no dependency between the reads (the quarters are interleaved: no bank conflicts); no atomics, one barrier.
//    The list is padded to 64 or 128 entries, so that all reads are under way at once (64: 670 cycles, 900 without).
//  n <= kRankCap: in runs of 32 that the warps sort across their lanes; an entry's rank is its place in its run plus the
//    larger entries of the other runs, by binary searches that do not depend on one another.
//  longer lists are first cut down to k by bisection (`tmp`: scratch for k composites).
// The first kPost threads call, after a barrier that made buf visible.
constexpr int kRankCap = 1024;
template <class Emit>
__device__ __forceinline__ void rank_emit(u64* buf, int n, int k, u64* tmp, SharedCtl* ctl, Emit emit) {
    constexpr int T = kPost;
    const int tid = threadIdx.x;
    if (n > kRankCap) n = select_list_topk(buf, n, k, tmp, ctl);
    if (n <= 128) {
        const int padded = n <= 64 ? 64 : 128;
        if (tid < padded - n) buf[n + tid] = 0ull;   // padding: 0 is below every composite
        block_sync<kPost, 1>();
        const int e = tid >> 2, part = tid & 3;
        auto rank = [&](auto full) {   // of entry e, and of entry e + 64 of a list of more than 64
            constexpr int kEntries = decltype(full)::value;
            const u64 c0 = buf[e], c1 = kEntries > 64 ? buf[e + 64] : 0ull;
            int l0 = 0, l1 = 0;
#pragma unroll
            for (int j = 0; j < kEntries; j += 8) {
                const ulonglong2 v = *reinterpret_cast<const ulonglong2*>(buf + 2 * part + j);
                l0 += (v.x > c0 ? 1 : 0) + (v.y > c0 ? 1 : 0);
                if (kEntries > 64) l1 += (v.x > c1 ? 1 : 0) + (v.y > c1 ? 1 : 0);
            }
            l0 += l1 << 16;
            l0 += __shfl_xor_sync(0xffffffffu, l0, 1);
            l0 += __shfl_xor_sync(0xffffffffu, l0, 2);
            l1 = l0 >> 16;
            l0 &= 0xFFFF;
            if (part == 0 && c0 != 0ull && l0 < k) emit(l0, c0);
            if (kEntries > 64 && part == 1 && c1 != 0ull && l1 < k) emit(l1, c1);
        };
        if (n <= 64) rank(std::integral_constant<int, 64>{});
        else rank(std::integral_constant<int, 128>{});
        return;
    }
    const int lane = tid & 31, runs = (n + 31) >> 5;
    for (int q = tid >> 5; q < runs; q += T / 32) {
        u64 c = 32 * q + lane < n ? buf[32 * q + lane] : 0ull;
#pragma unroll
        for (int kk = 2; kk <= 32; kk <<= 1) {   // bitonic, descending
#pragma unroll
            for (int j = kk >> 1; j > 0; j >>= 1) {
                const u64 o = __shfl_xor_sync(0xffffffffu, c, j);
                const bool down = (lane & kk) == 0, low = (lane & j) == 0;
                c = (down == low) ? max(c, o) : min(c, o);
            }
        }
        buf[32 * q + lane] = c;
    }
    block_sync<kPost, 1>();
    for (int e = tid; e < 32 * runs; e += T) {
        const u64 c = buf[e];
        if (lane >= k) continue;
        int r = lane;
#pragma unroll 4
        for (int q = 0; q < runs; ++q) {
            const u64* run = buf + 32 * q;
            int lo = 0;   // entries of the run above c (0 .. 32)
#pragma unroll
            for (int s = 16; s > 0; s >>= 1)
                if (run[lo + s - 1] > c) lo += s;
            if (run[lo] > c) lo += 1;
            r += q == e >> 5 ? 0 : lo;
        }
        if (c != 0ull && r < k) emit(r, c);
    }
}

// ---------------------------------------------------------------------------------------------- row epilogue
// What the epilogue needs to know about a row.
struct RowTail {
    u64 rng_word;
    float temperature, top_p, min_p;
    int flags;
    int out_index;
    long long append_at;    // resident histories: where the token goes in the id pool (used with kRowAppend)
};

struct TailOut {
    int32_t* tokens;
    int32_t* tokens_host;   // mirror of the tokens in mapped host memory, or null
    unsigned* status_host;  // takes a non-zero word whenever a status bit is set, or null
    int32_t* pool;          // id pool of the resident histories
    int32_t* kept_ids;
    double* kept_pr;
    int32_t* kept_n;
    u64* shard_out;
    int32_t* shard_n;       // null: the count goes to the header word of the row's list
    int shard_stride;
    unsigned* status;
};

// A status bit for the host: the device word collects the bits, the host mirror (if any) just becomes non-zero - before
// the token that the host may be waiting for.
__device__ __forceinline__ void report_status(unsigned* status, unsigned* status_host, unsigned bit) {
    atomicOr(status, bit);
    if (status_host) {
        *reinterpret_cast<volatile unsigned*>(status_host) = bit;
        __threadfence_system();
    }
}
// A row's token: to the device array and, if the caller reads its own memory, to the host mirror, from where the host may
// take it as soon as it lands.
__device__ __forceinline__ void put_token(int32_t* tokens, int32_t* tokens_host, int index, int token) {
    tokens[index] = token;
    if (tokens_host) *reinterpret_cast<volatile int32_t*>(tokens_host + index) = token;
}

// The cuts and the draw with the reference's own arithmetic, by one warp: probabilities p[i] = x[i] / s, their sequential sums
// c[i] = p[0] + ... + p[i] (src/sampler.cpp:42-49).  Leaves p in `e` and c in `x`; returns keep | pick << 16.
static __device__ __noinline__ int exact_cuts(double* x, double* e, int kk, double s, double min_p, double top_p, double u) {
    const int lane = threadIdx.x & 31;
    int keep = 0;
    for (int b = 0; b < kk; b += 32) {   // min-p keeps those not below p[0] * min_p (they do not increase, p[0] is 1 / s)
        const bool in = b + lane < kk;
        const double p = in ? __ddiv_rn(x[b + lane], s) : 0.0;
        if (in) e[b + lane] = p;
        const bool cut = min_p > 0.0 && p < __dmul_rn(__ddiv_rn(1.0, s), min_p);
        keep += __popc(__ballot_sync(0xffffffffu, in && !cut));
    }
    __syncwarp();
    // top-p keeps the shortest prefix whose sum reaches top_p, the crossing candidate included
    double c = 0.0;
    int i = 0;
    while (i < keep) {
        double v[16];
        const int n = min(16, keep - i);
#pragma unroll
        for (int q = 0; q < 16; ++q) v[q] = q < n ? e[i + q] : 0.0;
#pragma unroll
        for (int q = 0; q < 16; ++q) {
            c = __dadd_rn(c, v[q]);
            if (lane == q) x[i + q] = c;
        }
        i += n;
        if (c >= top_p) break;
    }
    __syncwarp();
    for (int b = 0; b < i; b += 32) {
        const unsigned m = __ballot_sync(0xffffffffu, b + lane < i && x[b + lane] >= top_p);
        if (m) {
            keep = min(keep, b + __ffs(m));
            break;
        }
    }
    const double r = __dadd_rn(__dmul_rn(u, x[keep - 1]), 0.0);   // r = u * tot + 0.0
    int pick = keep - 1;
    for (int b = 0; b < keep; b += 32) {
        const unsigned m = __ballot_sync(0xffffffffu, b + lane < keep && r <= x[b + lane]);
        if (m) {
            pick = b + __ffs(m) - 1;
            break;
        }
    }
    return keep | pick << 16;
}

// srt[0..kk) holds the row's candidates in order (largest first).  Either hands them out (vocabulary-sharded mode)
// or finishes the row: softmax over the candidates in fp64, sequential sums in candidate order, min-p, top-p,
// draw.  `work` is scratch for 2 * kMaxK doubles, 16-byte aligned, that does not overlap srt.  The first kPost threads call it
// with the same arguments; it is the last thing they do (no barrier at the end).
// Exponentials are one thread's work each.  Their sum follows the reference's order of additions exactly: a warp runs the
// chain of dependent adds, 9 cycles each, all lanes alike over broadcast reads, and keeps the partial sums S[i].  The
// reference then adds up the probabilities x[i] / S in the same way; both its cuts and its draw compare such a sum with a
// number, and that sum differs from S[i] / S by less than (2 * 256 + 5) * 2^-53 of it, the rounding of three chains of at most
// 256 terms.  A comparison that S[i] decides by more than 1e-12 - seventeen times that - comes out the same, so the second
// chain and the divisions run only where one is closer (equal logits with a cut between them), or where the probabilities are
// recorded: they would take 1.1 us of a launch of 24 x 100003, k = 50, 1.2 of 64 x 262144, k = 64, and 4.2 of 512 x 65536, k = 200.
__device__ __forceinline__ void row_epilogue(const u64* srt, int kk, const RowTail r, double* work, SharedCtl* ctl, const TailOut o) {
    const int tid = threadIdx.x, lane = tid & 31;
    double* e = work;
    double* P = work + kMaxK;
    if (o.shard_out) {
        u64* list = o.shard_out + (size_t)r.out_index * o.shard_stride;
        if (kk <= 0 && tid == 0) report_status(o.status, o.status_host, kStatusEmptyRow);
        if (o.shard_n) {
            if (tid < kk) list[tid] = srt[tid];
            if (tid == 0) o.shard_n[r.out_index] = kk;
        } else {
            if (tid < kk) list[1 + tid] = srt[tid];
            if (tid == 0) list[0] = (u64)kk;
        }
        return;
    }
    int token = 0, keep = 0;
    if (kk > 0 && !(r.flags & kRowGreedy)) {
        // x[i] = exp((double)(x_i - x_0) / T)   (fp32 subtraction, fp64 division, src/sampler.cpp:40)
        double x = 0.0;
        if (tid < kk) {
            const float diff = __fsub_rn(comp_value(srt[tid]), comp_value(srt[0]));
            x = exp(__ddiv_rn(diff == 0.0f ? 1.0 : (double)diff, (double)r.temperature));
            if (diff == 0.0f) x = 1.0;   // (a zero takes the division's slow path, and the largest candidate's is one)
        }
        P[tid] = x;   // (kMaxK == kPost: zeros behind the last candidate)
        block_sync<kPost, 1>();
        if (tid >= 32) return;
        // one engine output -> U[0,1) as libstdc++ does it
        double u = __dmul_rn(__ull2double_rn(r.rng_word), 5.42101086242752217003726400434970855712890625e-20);   // 2^-64
        if (u >= 1.0) u = __longlong_as_double(0x3FEFFFFFFFFFFFFFll);
        double s = 0.0;
        for (int i = 0; i < kk; i += 16) {
            double2 v[8];
#pragma unroll
            for (int q = 0; q < 8; ++q) v[q] = *reinterpret_cast<const double2*>(P + i + 2 * q);
#pragma unroll
            for (int q = 0; q < 8; ++q) {
                v[q].x = s = __dadd_rn(s, v[q].x);
                v[q].y = s = __dadd_rn(s, v[q].y);
            }
            if (lane == 0) {
#pragma unroll
                for (int q = 0; q < 8; ++q) *reinterpret_cast<double2*>(e + i + 2 * q) = v[q];
            }
        }
        __syncwarp();
        int pick = 0;
        const double close = 1e-12 * s;
        bool sure = s < 1e300 && !o.kept_n;   // (an infinite logit makes the sum no number)
        keep = kk;
        if (sure && r.min_p > 0.0f) {
            const double min_p = (double)r.min_p, low = min_p - 1e-12 * min_p, high = min_p + 1e-12 * min_p;
            keep = 0;
            int most = 0;
            for (int b = 0; b < kk; b += 32) {
                const double v = b + lane < kk ? P[b + lane] : 0.0;
                keep += __popc(__ballot_sync(0xffffffffu, v >= high));
                most += __popc(__ballot_sync(0xffffffffu, v >= low));
            }
            sure = keep == most;
        }
        // first of the n kept candidates whose sum reaches t (n if there is none); notes when one is too close to tell
        auto first_to_reach = [&](double t, int n) {
            const double low = t - close, high = t + close;
            for (int b = 0; b < n; b += 32) {
                const double v = b + lane < n ? e[b + lane] : 0.0;
                const unsigned m = __ballot_sync(0xffffffffu, b + lane < n && v >= low), h = __ballot_sync(0xffffffffu, b + lane < n && v >= high);
                if (m) {
                    sure = sure && __ffs(m) == __ffs(h);
                    return b + __ffs(m) - 1;
                }
            }
            return n;
        };
        if (sure) {
            if (r.top_p < 1.0f) keep = min(keep, first_to_reach((double)r.top_p * s, keep) + 1);
            pick = min(first_to_reach(u * e[keep - 1], keep), keep - 1);
        }
        if (!sure) {
            const int both = exact_cuts(P, e, kk, s, (double)r.min_p, r.top_p < 1.0f ? (double)r.top_p : 2.0, u);
            keep = both & 0xFFFF;
            pick = both >> 16;
        }
        token = comp_id(srt[pick]);
    } else {
        if (tid >= 32) return;
        if (kk > 0) token = comp_id(srt[0]);   // greedy: first index of the maximum (src/sampler.cpp:19-23)
    }
    if (o.kept_n) {
        for (int i = lane; i < keep; i += 32) {
            o.kept_ids[(size_t)r.out_index * kMaxK + i] = comp_id(srt[i]);
            o.kept_pr[(size_t)r.out_index * kMaxK + i] = e[i];
        }
        if (lane == 0) o.kept_n[r.out_index] = keep;
    }
    if (lane == 0) {
        if (kk <= 0) report_status(o.status, o.status_host, kStatusEmptyRow);   // nothing but NaNs in the row
        if (r.flags & kRowAppend) o.pool[r.append_at] = token;
        put_token(o.tokens, o.tokens_host, r.out_index, token);
    }
}

}  // namespace fsb
