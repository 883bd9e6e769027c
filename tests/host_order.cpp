// host_order.cpp - the host shim (fsb_shim.cpp) over a device that does nothing until it has to: what is queued on a stream
// runs when somebody waits for it, in order, and a copy reads its source only then.  The kernels are stand-ins: a row's token
// is the lower 31 bits of the engine output that its launch saw.  Prints "ok", or what went wrong.
#include <cuda_runtime.h>

#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <deque>
#include <functional>
#include <string>
#include <vector>

#include "../ferro_b200/csrc/fsb_internal.h"
#include "../include/ferro_sampler_b200.h"

#include <random>

namespace {
using Op = std::function<void()>;
std::deque<std::pair<Op, const void*>> queue_;   // operations, and the event that one records
std::vector<Op> graph_;
bool capturing_ = false;
std::vector<int> overlaps_;                      // mode of every streaming launch

void enqueue(Op op, const void* event = nullptr) {
    if (capturing_) graph_.push_back(op);
    else queue_.emplace_back(std::move(op), event);
}
void run_until(const void* event) {              // null: everything
    if (event) {
        bool there = false;
        for (auto& q : queue_) there = there || q.second == event;
        if (!there) return;
    }
    while (!queue_.empty()) {
        auto q = queue_.front();
        queue_.pop_front();
        q.first();
        if (event && q.second == event) return;
    }
}
}  // namespace

extern "C" {
cudaError_t cudaGetDeviceCount(int* n) { *n = 1; return cudaSuccess; }
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaGetDeviceProperties(cudaDeviceProp* p, int) {
    std::memset(p, 0, sizeof *p);
    p->major = 10;
    p->multiProcessorCount = 148;
    return cudaSuccess;
}
cudaError_t cudaGetLastError() { return cudaSuccess; }
const char* cudaGetErrorString(cudaError_t) { return "fake device"; }
cudaError_t cudaMalloc(void** p, size_t n) { *p = std::calloc(1, n); return cudaSuccess; }
cudaError_t cudaFree(void* p) { std::free(p); return cudaSuccess; }
cudaError_t cudaMallocHost(void** p, size_t n) { *p = std::calloc(1, n); return cudaSuccess; }
cudaError_t cudaFreeHost(void* p) { std::free(p); return cudaSuccess; }
cudaError_t cudaHostGetDevicePointer(void** d, void* h, unsigned) { *d = h; return cudaSuccess; }
cudaError_t cudaMemset(void* p, int v, size_t n) { std::memset(p, v, n); return cudaSuccess; }
cudaError_t cudaMemsetAsync(void* p, int v, size_t n, cudaStream_t) { enqueue([=] { std::memset(p, v, n); }); return cudaSuccess; }
cudaError_t cudaMemcpy(void* d, const void* s, size_t n, cudaMemcpyKind) { run_until(nullptr); std::memcpy(d, s, n); return cudaSuccess; }
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind, cudaStream_t) { enqueue([=] { std::memcpy(d, s, n); }); return cudaSuccess; }
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) { *s = reinterpret_cast<cudaStream_t>(16); return cudaSuccess; }
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { run_until(nullptr); return cudaSuccess; }
cudaError_t cudaStreamQuery(cudaStream_t) { run_until(nullptr); return cudaSuccess; }
cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, unsigned) { return cudaSuccess; }
cudaError_t cudaStreamIsCapturing(cudaStream_t, cudaStreamCaptureStatus* s) {
    *s = capturing_ ? cudaStreamCaptureStatusActive : cudaStreamCaptureStatusNone;
    return cudaSuccess;
}
cudaError_t cudaThreadExchangeStreamCaptureMode(cudaStreamCaptureMode*) { return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { *e = static_cast<cudaEvent_t>(std::malloc(1)); return cudaSuccess; }
cudaError_t cudaEventDestroy(cudaEvent_t e) { std::free(e); return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t) { enqueue([] {}, e); return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t e) { run_until(e); return cudaSuccess; }
}

namespace fsb {
int prepare_device_kernels() { return 0; }
int prepare_support_kernels() { return 0; }
int prepare_full_row_kernel() { return 0; }
SelectPlan plan_select(int, int, int, int, bool, bool) { return {}; }
bool rows_fit_launch(int n_rows, int64_t n_ids) { return n_ids == 0 ? n_rows <= 64 : n_rows <= 8 && n_ids <= 256; }
int launch_stream_kernel(StreamArgs a, const RowDesc* host_rows, const int32_t*, int, bool, void*) {
    overlaps_.push_back(a.overlap);
    std::vector<RowDesc> sent;
    if (host_rows && a.n_rows <= 64) sent.assign(host_rows, host_rows + a.n_rows);   // arguments are taken when the launch is queued
    enqueue([=] {
        for (int i = 0; i < a.n_rows; ++i) {
            const RowDesc& d = sent.empty() ? a.rows[i] : sent[(size_t)i];
            const int32_t token = (int32_t)(d.rng_word & 0x7fffffffull);
            a.tokens[d.out_index] = token;
            if (a.tokens_host) a.tokens_host[d.out_index] = token;
            if (d.flags & kRowAppend) a.pool[d.hist_begin + d.hist_len] = token;
        }
    });
    return 0;
}
int launch_full_row_kernel(const float*, const RowDesc*, int, const int32_t*, const int32_t*, int32_t*, int32_t*, int32_t*, int32_t*, double*, int32_t*, int,
                           uint32_t*, uint32_t*, int, int, int, float, uint64_t*, void*) { return 1; }
// the "drafts" are the history's last kmax ids
int launch_lookup_drafts(const int32_t* pool, const LookupDesc* host_desc, const LookupDesc*, int n_streams, int32_t* out, int stride, void*) {
    for (int i = 0; i < n_streams; ++i) {
        const LookupDesc d = host_desc[i];
        enqueue([=] {
            for (int k = 0; k < d.kmax; ++k) out[(size_t)i * stride + 1 + k] = pool[d.begin + d.len - d.kmax + k];
            out[(size_t)i * stride] = d.kmax;
        });
    }
    return 0;
}
int launch_merge_lists(const void*, const int32_t*, int, int, int n_rows, const RowDesc* rows, int32_t* tokens, int32_t*, double*, int32_t*, uint32_t*, void*) {
    enqueue([=] {
        for (int i = 0; i < n_rows; ++i) tokens[rows[i].out_index] = (int32_t)(rows[i].rng_word & 0x7fffffffull);
    });
    return 0;
}
int launch_accept_windows(const int32_t*, int, const int32_t*, int32_t*, void*) { return 0; }
int launch_gather_patched(const float*, const RowDesc*, int, const int32_t*, int, int, float*, void*) { return 0; }
}  // namespace fsb

namespace {
int bad(const char* what, int at, long long got, long long want) {
    std::printf("%s: %d: %lld, not %lld\n", what, at, got, want);
    return 1;
}
struct Setup {
    fsb_handle* h = nullptr;
    std::vector<int> sid;
    std::vector<std::mt19937_64> rng;
    explicit Setup(int rows, float penalty = 1.0f) {
        if (fsb_create(0, rows, 1000, rows * 1024, &h) != FSB_OK) std::abort();
        for (int i = 0; i < rows; ++i) {
            ferro_sampler_params p;
            fsb_params_default(&p);
            p.repetition_penalty = penalty;
            p.seed = (uint64_t)(100 + i);
            int s = 0;
            if (fsb_stream_open(h, &p, &s) != FSB_OK) std::abort();
            sid.push_back(s);
            rng.emplace_back(p.seed);
        }
    }
    fsb_batch* prepare() {
        std::vector<int64_t> off(sid.size() + 1, 0);
        fsb_batch* b = nullptr;
        if (fsb_batch_prepare(h, (int)sid.size(), sid.data(), 1000, 1000, nullptr, off.data(), 0, &b) != FSB_OK) std::abort();
        return b;
    }
    std::vector<int32_t> next() {   // what the rows draw next
        std::vector<int32_t> t;
        for (auto& r : rng) t.push_back((int32_t)(r() & 0x7fffffffull));
        return t;
    }
};
float logits_[1000];

// Steps that are queued without waiting: every launch draws what the redraw before it drew.
// (`waited`: the first two of them are waited for, as by a caller that changes its ways.)
int queued_steps(int rows, bool merge, bool waited = false) {
    Setup s(rows);
    fsb_batch* b = s.prepare();
    std::vector<uint64_t> lists((size_t)rows * 52);
    std::vector<std::vector<int32_t>> seen(6, std::vector<int32_t>((size_t)rows)), want;
    for (int step = 0; step < 6; ++step) {
        if (step > 0 && fsb_batch_redraw(s.h, b) != FSB_OK) return bad("redraw", step, 1, 0);
        want.push_back(s.next());
        const int rc = merge ? fsb_batch_merge_launch_packed(s.h, b, lists.data(), 52, 1, 0, rows) : fsb_batch_launch(s.h, b, logits_);
        if (rc != FSB_OK) return bad("launch", step, rc, 0);
        int32_t* to = seen[(size_t)step].data();
        const int32_t* from = fsb_batch_tokens_device(b);
        enqueue([=] { std::memcpy(to, from, sizeof(int32_t) * (size_t)rows); });
        if (waited && step < 2 && fsb_batch_check(s.h, b) != FSB_OK) return bad("check", step, 1, 0);
    }
    run_until(nullptr);
    for (int step = 0; step < 6; ++step)
        for (int i = 0; i < rows; ++i)
            if (seen[(size_t)step][(size_t)i] != want[(size_t)step][(size_t)i])
                return bad("token of a queued step", step * 1000 + i, seen[(size_t)step][(size_t)i], want[(size_t)step][(size_t)i]);
    return 0;
}

// A captured launch that is replayed after a redraw draws the new outputs.
int replayed_launch(int rows) {
    Setup s(rows);
    fsb_batch* b = s.prepare();
    s.next();
    capturing_ = true;
    const int rc = fsb_batch_launch(s.h, b, logits_);
    capturing_ = false;
    if (rc != FSB_OK) return bad("captured launch", 0, rc, 0);
    for (int step = 0; step < 3; ++step) {
        if (fsb_batch_redraw(s.h, b) != FSB_OK) return bad("redraw", step, 1, 0);
        const auto want = s.next();
        for (auto& op : graph_) enqueue(op);
        std::vector<int32_t> got((size_t)rows);
        if (fsb_batch_tokens(s.h, b, got.data()) != FSB_OK) return bad("tokens", step, 1, 0);
        for (int i = 0; i < rows; ++i)
            if (got[(size_t)i] != want[(size_t)i]) return bad("token of a replay", step * 1000 + i, got[(size_t)i], want[(size_t)i]);
    }
    return 0;
}

// Overlap mode 1: launches whose windows lie in the id pool, where the launch before appends its tokens, wait for it.
int overlapped_windows() {
    for (float penalty : {1.0f, 1.3f}) {
        Setup s(4, penalty);
        fsb_set_launch_overlap(s.h, 1);
        const int32_t ids[3] = {1, 2, 3};
        for (int sid : s.sid) fsb_stream_history_set(s.h, sid, ids, 3);
        std::vector<int32_t> tok(4);
        overlaps_.clear();
        for (int step = 0; step < 2; ++step)
            if (fsb_sample_batch_resident(s.h, 4, s.sid.data(), logits_, 1000, 1000, tok.data(), FSB_APPEND_SAMPLED) != FSB_OK) return bad("step", step, 1, 0);
        fsb_batch* b = s.prepare();
        fsb_batch_launch(s.h, b, logits_);
        const int want[3] = {penalty == 1.0f ? 1 : 2, penalty == 1.0f ? 1 : 2, 1};
        for (int i = 0; i < 3; ++i)
            if (overlaps_[(size_t)i] != want[i]) return bad("mode of launch", i, overlaps_[(size_t)i], want[i]);
    }
    return 0;
}

// An engine that leaves a stream, the default stream among them, leaves nothing behind that the next one would have to wait for.
int switched_streams() {
    Setup s(1);
    const int32_t ids[3] = {1, 2, 3};
    int n = 0;
    for (uintptr_t to : {0, 32, 0}) {
        if (fsb_set_cuda_stream(s.h, reinterpret_cast<void*>(to)) != FSB_OK) return bad("stream", n, 1, 0);
        if (!queue_.empty()) return bad("operations left on a stream", n, (long long)queue_.size(), 0);
        fsb_stream_history_set(s.h, s.sid[0], ids, 3);
        ++n;
    }
    fsb_destroy(s.h);
    return queue_.empty() ? 0 : bad("operations left on a stream", n, (long long)queue_.size(), 0);
}

// Every 32-bit value is a token id of a history, and of the drafts that are taken from it.
int any_draft() {
    Setup s(1);
    const int32_t ids[4] = {INT32_MIN, 7, INT32_MIN, INT32_MAX};
    fsb_stream_history_set(s.h, s.sid[0], ids, 4);
    int32_t drafts[4] = {0, 0, 0, 0};
    int n = 0;
    const int most = 4, least = 2;
    const int rc = fsb_lookup_drafts_resident(s.h, 1, s.sid.data(), &most, &least, 99, drafts, 4, &n);
    if (rc != FSB_OK || n != 4) return bad("drafts", 0, rc, 0);
    for (int i = 0; i < 4; ++i)
        if (drafts[i] != ids[i]) return bad("draft", i, drafts[i], ids[i]);
    return 0;
}
}  // namespace

int main(int argc, char** argv) {
    const std::string what = argc > 1 ? argv[1] : "";
    const int rows = argc > 2 ? std::atoi(argv[2]) : 8;
    const int rc = what == "queued" ? queued_steps(rows, false) : what == "merged" ? queued_steps(rows, true) : what == "waited" ? queued_steps(rows, false, true)
                   : what == "replayed" ? replayed_launch(rows)
                   : what == "overlap" ? overlapped_windows() : what == "switched" ? switched_streams() : what == "drafts" ? any_draft() : 2;
    if (rc == 0) std::puts("ok");
    return rc;
}
