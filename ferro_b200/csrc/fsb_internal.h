// fsb_internal.h - structures shared by the host shim (fsb_shim.cpp) and the CUDA kernels.
#pragma once
#include <stddef.h>
#include <stdint.h>

namespace fsb {

// ---- compile-time geometry -----------------------------------------------------------------------------------
constexpr int kMaxK = 256;                    // largest k of the candidate path (== FSB_MAX_CANDIDATE_K)
constexpr int kMergeCap = 2400;               // candidates of one row that the list merge can gather

// status word bits written by kernels (0 = fine)
enum : uint32_t {
    kStatusMergeOverflow = 4u,   // the candidate lists of a row hold more than the merge has room for
    kStatusEmptyRow = 8u,        // a row produced no candidate (all logits NaN)
    kStatusLate = 16u            // what another CTA of the row had to send did not come
};

// row flags
enum : int32_t {
    kRowGreedy = 1,       // temperature <= 0 or top_k == 1: argmax, no draw
    kRowPenalty = 2,      // the row has a non-empty penalty window and penalty != 1
    kRowAppend = 4        // resident histories: the row's token is appended at hist_begin + hist_len of the id pool
};
// Resident verification windows: the drafts before a row are the last ids of its window.  They are not in the id pool:
// bits 8 and up of the flags hold their number, draft_off the first one's place among the ids staged with the call.
constexpr int kRowDraftShift = 8;

constexpr int kWindowTableInts = 72;          // int32 words per stream of a resident verification call: 6 + up to 66 drafts

// One row of a batch, as the kernels see it (64 bytes).
struct RowDesc {
    uint64_t rng_word;     // raw 64-bit engine output of this row's draw (unused for greedy rows)
    int64_t logits_off;    // element offset of the row from the logits base pointer
    int64_t hist_begin;    // first id of the penalty window in the device history array
    int32_t hist_len;      // ids in the window (0: no penalty)
    int32_t k;             // effective candidate count: 1 for greedy, else (0 < top_k < n) ? top_k : n
    float temperature;
    float top_p;
    float min_p;
    float penalty;
    int32_t flags;
    int32_t out_index;     // position of the row's token in the output array
    int32_t k_global;      // vocabulary sharding: candidate count of the whole row (k is the shard's); otherwise == k
    union {
        int32_t gather_off;   // where the row's window values go when patched entries are gathered for a host caller
        int32_t draft_off;    // resident verification windows: see kRowDraftShift
    };
};
static_assert(sizeof(RowDesc) == 64, "RowDesc layout");

// Arguments of the streaming candidate kernel.
struct StreamArgs {
    const float* logits;       // base of the [rows][ld] matrix
    const RowDesc* rows;       // n_rows descriptors (only rows of the candidate path)
    const int32_t* hist;       // packed penalty-window ids (or the id pool)
    const int32_t* drafts;     // ids staged with a resident verification call
    float* patched;            // optional: the transformed logits at the window ids, indexed by RowDesc::gather_off + place in the window
    int32_t* pool;             // id pool of the resident histories (rows with kRowAppend store their token there)
    int32_t* tokens;           // output tokens, indexed by RowDesc::out_index
    uint32_t* status;          // one word, OR of kStatus* bits
    // optional mirror in mapped host memory (device addresses of pinned host words; null = off): tokens are stored
    // there as well, and a non-zero word is stored to status_host whenever a status bit is set, so that a synchronous
    // caller needs no copy back - it waits for the stream and reads its own memory
    int32_t* tokens_host;
    uint32_t* status_host;
    // optional kept-set record, indexed by out_index (null = off)
    int32_t* kept_ids;         // [rows][kMaxK]
    double* kept_pr;           // [rows][kMaxK]
    int32_t* kept_n;           // [rows]
    // optional per-row sorted candidates for the vocabulary-sharded mode (null = run the epilogue here)
    uint64_t* shard_out;       // [rows][shard_stride] composites, descending
    int32_t* shard_n;          // [rows] their number; null: a list starts with a header word that holds it
    int32_t shard_stride;      // 64-bit words per row of shard_out
    uint64_t* trace;           // optional [grid][8] timestamps (diagnostics), null = off
    int64_t row_ld;            // >= 0: row r starts at r * row_ld (no descriptor read before the first load)
    int32_t n_rows;
    int32_t n_vocab;
    int32_t nseg;              // CTAs per row (1..8), a thread-block cluster when more than one
    int32_t wide;              // large CTAs (see SelectPlan)
    int32_t kmax;              // largest k of the rows
    int32_t all_greedy;        // every row is greedy
    int32_t window_max;        // ids of the longest penalty window
    int32_t penalised;         // some row has a penalty window
    int32_t write_back;        // store penalised values into the caller's rows
    int32_t vocab_offset;      // token id of column 0
    float softcap;             // 0 = off
    int32_t overlap;           // see fsb_set_launch_overlap
    int32_t sms;               // multiprocessors of the device
    int32_t unchained;         // no launch attribute unless `overlap` asks for it
};

// How a launch of n_rows rows is laid out on a device of `sms` multiprocessors: CTAs per row, and whether they are large
// ones (1024 threads, one per SM) or small ones (256 threads, several per SM).
struct SelectPlan {
    int nseg = 1;
    bool wide = false;
};
SelectPlan plan_select(int n_rows, int n_vocab, int sms, int kmax, bool all_greedy, bool penalised);

// All return a cudaError_t as int (0 = success).
int prepare_device_kernels();
// Whether a batch's descriptors and staged ids can be arguments of the launch.
bool rows_fit_launch(int n_rows, int64_t n_ids);
// host_rows: the descriptors in host memory (sent with the launch when they are few), or null.  host_ids: n_ids staged ids
// that go with the launch instead of a.hist (ids_are_windows) or a.drafts.
int launch_stream_kernel(StreamArgs a, const RowDesc* host_rows, const int32_t* host_ids, int n_ids, bool ids_are_windows, void* stream);

// One stream of a prompt-lookup drafting call: where its history lies in the id pool and what to look for.
struct LookupDesc {
    int64_t begin;         // first id of the history in the id pool
    int32_t len;           // ids in the history
    int32_t kmax;          // most drafts wanted
    int32_t min_n;         // shortest suffix that may be matched (>= 1)
    int32_t eos;           // end-of-sequence id: a draft stops before it
};
static_assert(sizeof(LookupDesc) == 24, "LookupDesc layout");
constexpr int kDraftStride = 68;              // int32 words per stream of a drafting call: the count, then up to 67 drafts

constexpr int kLookupArgs = 64;               // drafting calls of up to this many streams send the descriptors with the launch

// Defined in fsb_support.cu.
int prepare_support_kernels();
int launch_lookup_drafts(const int32_t* pool, const LookupDesc* host_desc, const LookupDesc* desc, int n_streams, int32_t* out, int stride, void* stream);
int launch_merge_lists(const void* lists, const int32_t* list_n, int n_lists, int list_stride, int n_rows, const RowDesc* rows, int32_t* tokens,
                       int32_t* kept_ids, double* kept_pr, int32_t* kept_n, uint32_t* status, void* stream);
int launch_accept_windows(const int32_t* table, int n_streams, const int32_t* tokens, int32_t* pool, void* stream);
int launch_gather_patched(const float* logits, const RowDesc* rows, int n_rows, const int32_t* hist, int n_vocab, int vocab_offset,
                          float* out, void* stream);

// Defined in fsb_fullrow.cu.
int prepare_full_row_kernel();
int launch_full_row_kernel(const float* logits, const RowDesc* rows, int n_rows, const int32_t* hist, const int32_t* drafts, int32_t* pool, int32_t* tokens, int32_t* tokens_host,
                           int32_t* kept_ids, double* kept_pr, int32_t* kept_n, int record, uint32_t* status, uint32_t* status_host, int n_vocab,
                           int vocab_offset, int write_back, float softcap, uint64_t* trace, void* stream);

}  // namespace fsb

// fsb_sample_batch and fsb_verify_windows with one history array per row / stream instead of a packed one; for the
// Python binding (fsb_python.cpp), whose callers hold one array per slot.
struct fsb_handle;
extern "C" {
__attribute__((visibility("default"))) int fsb_sample_batch_lists(fsb_handle* h, int n_rows, const int* stream_ids, const float* logits, int64_t ld,
                                                                  int n_vocab, const int32_t* const* hist_lists, const int64_t* hist_lens,
                                                                  int32_t* tokens_out, unsigned flags);
__attribute__((visibility("default"))) int fsb_verify_windows_lists(fsb_handle* h, int n_streams, const int* stream_ids, const int* row_off,
                                                                    const int32_t* rows_flat, const float* logits, int64_t ld, int n_vocab,
                                                                    const int32_t* const* hist_lists, const int64_t* hist_lens, const int* max_accept,
                                                                    int32_t* tokens_out, int* acc_out, int* confirmed_out, unsigned flags);
}
