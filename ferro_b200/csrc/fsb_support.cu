// fsb_support.cu - the small kernels around the two sampling kernels of the B200 batched token sampler (sm_100a):
// the merge of per-shard candidate lists (vocabulary sharding), the device side of resident histories and resident
// verification windows (src/server.cpp:598-636 of paragontasx/ferro is the host loop they replace), and the gather
// that lets a host caller see the penalised values without any host arithmetic.
#include <cuda_runtime.h>

#include <cstring>

#include "fsb_device.cuh"

namespace fsb {
namespace {

constexpr int kThreads = kPost;   // of the list merge
constexpr size_t kSmemMerge = (size_t)(kMergeCap + 32 + kMaxK) * sizeof(u64) + sizeof(SharedCtl);   // gathered lists, ordered candidates, control

// Merge of per-shard candidate lists: one CTA per row gathers the row's n_lists ordered lists (already in this
// device's memory, list g of row r at lists + (g * n_rows + r) * list_stride) and finishes the row exactly as the
// streaming kernel does after its own selection - the k best of the whole row are among the shards' k best, and
// the order (value descending, id ascending) does not depend on the split.  With list_n the lists are bare and
// list_n[g * n_rows + r] gives their lengths; without it a list starts with a header word that holds its length.
__global__ void __launch_bounds__(kThreads, 1) merge_lists_kernel(const u64* lists, const int32_t* list_n, int n_lists, int list_stride, int n_rows,
                                                                 const RowDesc* rows, int32_t* tokens, int32_t* kept_ids, double* kept_pr,
                                                                 int32_t* kept_n, unsigned* status) {
    extern __shared__ __align__(128) unsigned char smem_raw[];
    u64* buf = reinterpret_cast<u64*>(smem_raw);
    u64* out = buf + kMergeCap + 32;
    SharedCtl* ctl = reinterpret_cast<SharedCtl*>(out + kMaxK);
    const int row = blockIdx.x, tid = threadIdx.x;
    if (row >= n_rows) return;
    const RowDesc d = rows[row];
    const int hdr = list_n ? 0 : 1;
    int total = 0;   // the same in every thread
    auto list_at = [&](int g) { return lists + ((size_t)g * n_rows + row) * (size_t)list_stride; };
    auto length = [&](int g) {
        const long long stated = list_n ? (long long)list_n[(size_t)g * n_rows + row] : (long long)list_at(g)[0];
        return (int)max(0ll, min(stated, (long long)min(kMaxK, list_stride - hdr)));
    };
    // Thirty-two lists at a time: every warp reads all their lengths at once, and copies some of the lists, two words per lane on their
    // way together.  (List after list, the next length read when the one before was known: 8.6 us for eight lists of 41, this way 6.6.)
    const int lane = tid & 31;
    for (int g0 = 0; g0 < n_lists; g0 += 32) {
        const int mine = g0 + lane < n_lists ? length(g0 + lane) : 0;
        for (int g = g0; g < min(g0 + 32, n_lists); ++g) {
            const int n = __shfl_sync(0xffffffffu, mine, g - g0);
            if (total + n > kMergeCap) {
                if (tid == 0) atomicOr(status, kStatusMergeOverflow);
                continue;
            }
            if ((g & (kThreads / 32 - 1)) == tid >> 5) {
                const u64* src = list_at(g) + hdr;
                for (int i = lane; i < n; i += 64) {
                    const u64 c0 = src[i], c1 = i + 32 < n ? src[i + 32] : 0ull;
                    buf[total + i] = c0;
                    if (i + 32 < n) buf[total + i + 32] = c1;
                }
            }
            total += n;
        }
    }
    block_sync<kPost, 1>();
    const TailOut tout{tokens, nullptr, nullptr, nullptr, kept_ids, kept_pr, kept_n, nullptr, nullptr, 0, status};
    const RowTail rt{d.rng_word, d.temperature, d.top_p, d.min_p, d.flags & ~kRowAppend, d.out_index, 0};
    rank_emit(buf, total, d.k_global, out, ctl, [&](int rank, u64 c) { out[rank] = c; });
    block_sync<kPost, 1>();
    row_epilogue(out, min(total, d.k_global), rt, reinterpret_cast<double*>(buf), ctl, tout);
}

// Write-back for callers whose logits live in host memory: after a launch with write-back on the device copy, the
// values at the rows' window ids (the only entries the penalty touches) are gathered, one float per window id in
// window order, so that the host can store them into the caller's rows without redoing any arithmetic.
__global__ void gather_patched_kernel(const float* logits, const RowDesc* rows, int n_rows, const int32_t* hist, int n_vocab, int vocab_offset,
                                      float* out) {
    const int row = blockIdx.x;
    if (row >= n_rows) return;
    const RowDesc d = rows[row];
    for (int i = threadIdx.x; i < d.hist_len; i += blockDim.x) {
        const int c = hist[d.hist_begin + i] - vocab_offset;
        out[d.gather_off + i] = (c >= 0 && c < n_vocab) ? logits[d.logits_off + c] : 0.0f;
    }
}

// Resident verification windows, after the launch: per stream the accept loop of src/server.cpp:630-636 over the sampled
// tokens (accept while the token equals the next draft, at most `lim` rows), and the accepted tokens are stored behind
// the history.  Table entry of a stream: first row, rows m, limit, unused, end of the history in the pool (two words), then
// the m - 1 drafts.
__global__ void accept_windows_kernel(const int32_t* table, int n_streams, const int32_t* tokens, int32_t* pool) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n_streams) return;
    const int32_t* t = table + (size_t)i * kWindowTableInts;
    const int r0 = t[0], m = t[1], lim = t[2];
    const int64_t end = ((int64_t)t[5] << 32) | (uint32_t)t[4];
    int acc = 0;
    for (int r = 0; r < lim; ++r) {
        acc = r + 1;
        if (r + 1 < m && tokens[r0 + r] == t[6 + r]) continue;
        break;
    }
    for (int r = 0; r < acc; ++r) pool[end + r] = tokens[r0 + r];
}

// Prompt-lookup drafting over resident histories (lookup_draft, src/server.cpp:552-564): the tokens that followed
// the most recent earlier occurrence of the history's last n tokens, n = 4, 3, ... min_n - at most kmax of them, cut
// at the end-of-sequence id; an occurrence whose continuation is empty is passed over.  One CTA per stream, one pass: at every
// position a thread finds how many ids up to there are those the history ends with (up to four; the five ids it needs are on their
// way at once), and the last position of every length is noted; the longest one wins, and a warp copies the draft.  (A pass per length,
// an id read when the one before had matched: 5.5 us for eight histories of 1024 ids, this way 4.8.)
// out[i * stride] = number of drafts of stream i, then the drafts; `out` is the caller's pinned memory, where the host
// waits for the number and for every draft (a system-wide fence between the two would cost 7 us).
struct LookupArgs {
    LookupDesc d[kLookupArgs];
};
__global__ void lookup_drafts_kernel(const int32_t* pool, const __grid_constant__ LookupArgs args, const LookupDesc* desc, int n_streams, int32_t* out, int stride) {
    __shared__ int last[5];   // of the positions whose longest match is n ids, the last (-1: none)
    const int i = blockIdx.x;
    if (i >= n_streams) return;
    const LookupDesc d = desc ? desc[i] : args.d[i];
    const int32_t* h = pool + d.begin;
    const int L = d.len;
    if (threadIdx.x < 5) last[threadIdx.x] = -1;
    __syncthreads();
    if (d.kmax > 0 && L > 1) {
        int32_t end[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) end[j] = h[max(L - 1 - j, 0)];
#pragma unroll 4
        for (int q = L - 2 - (int)threadIdx.x; q >= 0; q -= (int)blockDim.x) {   // the match ends at q
            const int32_t next = h[q + 1];
            int32_t id[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) id[j] = h[max(q - j, 0)];
            int n = 0;
#pragma unroll
            for (int j = 3; j >= 0; --j) n = q >= j && id[j] == end[j] ? n + 1 : 0;
            if (n >= max(d.min_n, 1) && next != d.eos) atomicMax(&last[n], q);   // (an occurrence followed by the end-of-sequence id drafts nothing)
        }
    }
    __syncthreads();
    int found_n = 0, best = -1;
    for (int n = 4, q = -1; n >= max(d.min_n, 1); --n) {   // a match of n ids is one of n - 1, too
        q = max(q, last[n]);
        if (q >= 0) {
            found_n = n;
            best = q - n + 1;
            break;
        }
    }
    if (threadIdx.x >= 32) return;
    const int lane = threadIdx.x, most = found_n > 0 ? min(min(d.kmax, stride - 1), L - best - found_n) : 0;
    volatile int32_t* to = out + (size_t)i * stride;
    int cnt = 0;
    for (int k0 = 0; k0 < most; k0 += 32) {
        const int id = k0 + lane < most ? h[best + found_n + k0 + lane] : d.eos;
        const unsigned stop = __ballot_sync(0xffffffffu, k0 + lane >= most || id == d.eos);
        const int n = stop ? __ffs(stop) - 1 : 32;
        if (lane < n) to[1 + k0 + lane] = id;
        cnt = k0 + n;
        if (n < 32) break;
    }
    if (lane == 0) to[0] = cnt;
}

}  // namespace

int launch_lookup_drafts(const int32_t* pool, const LookupDesc* host_desc, const LookupDesc* desc, int n_streams, int32_t* out, int stride, void* stream) {
    LookupArgs args;
    const bool sent = n_streams <= kLookupArgs;
    if (sent) std::memcpy(args.d, host_desc, sizeof(LookupDesc) * (size_t)n_streams);
    lookup_drafts_kernel<<<n_streams, 256, 0, static_cast<cudaStream_t>(stream)>>>(pool, args, sent ? nullptr : desc, n_streams, out, stride);
    return (int)cudaGetLastError();
}

int prepare_support_kernels() {
    return (int)cudaFuncSetAttribute(merge_lists_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemMerge);
}

int launch_merge_lists(const void* lists, const int32_t* list_n, int n_lists, int list_stride, int n_rows, const RowDesc* rows, int32_t* tokens,
                       int32_t* kept_ids, double* kept_pr, int32_t* kept_n, uint32_t* status, void* stream) {
    merge_lists_kernel<<<n_rows, kThreads, kSmemMerge, static_cast<cudaStream_t>(stream)>>>(static_cast<const u64*>(lists), list_n, n_lists, list_stride,
                                                                                           n_rows, rows, tokens, kept_ids, kept_pr, kept_n, status);
    return (int)cudaGetLastError();
}

int launch_gather_patched(const float* logits, const RowDesc* rows, int n_rows, const int32_t* hist, int n_vocab, int vocab_offset, float* out,
                          void* stream) {
    gather_patched_kernel<<<n_rows, 128, 0, static_cast<cudaStream_t>(stream)>>>(logits, rows, n_rows, hist, n_vocab, vocab_offset, out);
    return (int)cudaGetLastError();
}

int launch_accept_windows(const int32_t* table, int n_streams, const int32_t* tokens, int32_t* pool, void* stream) {
    accept_windows_kernel<<<(n_streams + 63) / 64, 64, 0, static_cast<cudaStream_t>(stream)>>>(table, n_streams, tokens, pool);
    return (int)cudaGetLastError();
}

}  // namespace fsb
