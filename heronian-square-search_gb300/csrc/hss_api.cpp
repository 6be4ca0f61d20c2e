// hss_api.cpp - C ABI over the sm_103a search kernels (include/hss.h).
//
// Replaces the reference's in-process boundary: Search::prepare builds the
// factor cache (gpu_search_v42.cu:354-391), Search::run uploads it and loops
// launch / synchronise / harvest over batches of at most 512 roots
// (gpu_search_v42.cu:393-495).  Here the cache and its sorted layout are built
// once per handle on the device and stay resident; each search call is one
// launch sequence on a private stream (batched: rows and items planned on the
// host, one persistent launch, the shared-prime kernels for what it leaves;
// plain: one launch per <= 512 roots), timed with CUDA events, and its counters
// and hits are copied back once.
#include <cuda_runtime.h>
#include <stdio.h>
#include <string.h>
#include <time.h>

#include <algorithm>
#include <array>
#include <condition_variable>
#include <deque>
#include <map>
#include <mutex>
#include <string>
#include <thread>
#include <vector>

#include "hss_api_status.h"
#include "hss_ctx.h"
#include "hss_kernels.h"
#include "hss_prep.h"

using namespace hss;

namespace {

constexpr uint32_t kDefaultHitCap = 4096;      // gpu_search_v42.cu:177-178
constexpr uint32_t kPlainBatch = 512;          // gpu_search_v42.cu:457
constexpr uint32_t kDefaultItemTarget = 1u << 23;
constexpr uint32_t kTileCap = 16384;           // largest m-range of one item
constexpr uint32_t kTileMin = 32;
constexpr uint32_t kBucketShift = 10;          // item ordering granularity in m
constexpr uint64_t kArcLeast = 1000;            // handles from this limit on have the arc layout
constexpr uint64_t kArcLimit = 10000;          // and long calls use it from this one on (see run_batched)
constexpr size_t kArcRows = 64;
constexpr uint64_t kMergedCap = 96ull << 20;   // shared-prime queue entries
constexpr uint32_t kDescChunk = 1u << 24;       // shared-prime pairs set up per chunk (192 bytes each: 3 GB)
// Where every search goes by arcs only the rest list's pairs come by the
// shared-prime kernels: the queues start small (0.1 GB; opening, one search and closing at LIMIT
// 10^7 took 23.3 ms so, 25.1 ms with the full ones of 2.4 GB) and are enlarged
// to the full ones when a call first needs more (a plain scan may need more still).
// Where there is no room the call goes on with what there is, in smaller launches.
constexpr uint64_t kArcMergedCap = 48ull << 20;
constexpr uint32_t kArcDescChunk = 1u << 23;
constexpr uint64_t kArcMergedStart = 2ull << 20;
constexpr uint32_t kArcDescStart = 1u << 19;


}  // namespace

namespace {

int fail(hss_t* h, int status, const std::string& msg) {
    if (h) h->err = msg;
    return status;
}

// (a refused call's error also stays with the thread until it is read, and the
// check behind the next kernel launch would report it: it is taken out here)
#define HSS_CUDA(h, call)                                                                          \
    do {                                                                                           \
        cudaError_t e_ = (call);                                                                   \
        if (e_ != cudaSuccess) {                                                                   \
            cudaGetLastError();                                                                    \
            return fail(h, HSS_ERR_CUDA, std::string(#call) + ": " + cudaGetErrorString(e_));      \
        }                                                                                          \
    } while (0)

uint64_t now_ns() {
    timespec ts;
    clock_gettime(CLOCK_MONOTONIC, &ts);
    return (uint64_t)ts.tv_sec * 1000000000ull + (uint64_t)ts.tv_nsec;
}

template <class T>
int device_alloc(hss_t* h, T** out, size_t count) {
    void* p = nullptr;
    if (count == 0) count = 1;
    cudaError_t e = cudaMalloc(&p, count * sizeof(T));
    if (e != cudaSuccess) {
        cudaGetLastError();
        return fail(h, HSS_ERR_MEMORY, std::string("cudaMalloc: ") + cudaGetErrorString(e));
    }
    h->allocations.push_back(p);
    *out = static_cast<T*>(p);
    return HSS_OK;
}

void device_free(hss_t* h, void* p) {
    if (!p) return;
    auto it = std::find(h->allocations.begin(), h->allocations.end(), p);
    if (it != h->allocations.end()) h->allocations.erase(it);
    cudaFree(p);
}

// Replaces an array of *cap elements (of `per` T each) by one of n.  Where it
// cannot be had the old one stays: memory for both being short, the old one is
// given up first and allocated again if that was not enough.  Only where that
// fails too is the array gone, and its capacity 0: no capacity ever claims
// more than its array holds.
template <class T, class Cap>
int device_grow(hss_t* h, T** p, Cap* cap, size_t n, size_t per = 1) {
    T* larger = nullptr;
    int s = device_alloc(h, &larger, n * per);
    if (s && *cap) {
        const size_t old = *cap;
        device_free(h, *p);
        *p = nullptr;
        *cap = 0;
        if ((s = device_alloc(h, &larger, n * per)) && device_alloc(h, p, old * per) == HSS_OK) *cap = (Cap)old;
    }
    if (s) return s;
    device_free(h, *p);
    *p = larger;
    *cap = (Cap)n;
    return HSS_OK;
}

// The same for pinned host memory, whose contents are not kept.
template <class T>
int host_grow(hss_t* h, T** p, size_t* cap, size_t n) {
    if (*p) cudaFreeHost(*p);
    *p = nullptr;
    *cap = 0;
    HSS_CUDA(h, cudaMallocHost(p, n * sizeof(T)));
    *cap = n;
    return HSS_OK;
}

template <class T>
int upload(hss_t* h, T** out, const T* src, size_t count) {
    int s = device_alloc(h, out, count);
    if (s) return s;
    HSS_CUDA(h, cudaMemcpy(*out, src, count * sizeof(T), cudaMemcpyHostToDevice));
    return HSS_OK;
}

uint32_t free_count(const hss_t* h, uint64_t x) { return h->seg_off[x + 1] - h->seg_off[x] - 1; }

// Upper bound on the pairs of row l that share a split prime with m in
// [l, N]: inclusion-exclusion over the distinct split primes of l.
uint64_t merged_bound(const hss_t* h, uint64_t l) {
    NumberFactors f = factor_number(h->spf.data(), l);
    if (f.count == 0) return 0;
    uint64_t n = h->limit, total = 0;
    for (uint32_t mask = 1; mask < (1u << f.count); ++mask) {
        uint64_t prod = 1;
        int bits = 0;
        bool over = false;
        for (uint32_t i = 0; i < f.count; ++i)
            if (mask & (1u << i)) {
                prod *= f.primes[i];
                ++bits;
                if (prod > n) over = true;
            }
        if (over) continue;
        uint64_t cnt = n / prod - (l - 1) / prod;
        if (bits & 1) total += cnt;
        else total -= cnt;
    }
    return total;
}

int ensure_rows(hss_t* h, size_t rows) {
    const size_t cap = std::max(rows, (size_t)1024);
    if (rows > h->rows_cap)
        if (int s = device_grow(h, &h->d_rows, &h->rows_cap, cap)) return s;
    if (rows > h->h_rows_cap)
        if (int s = host_grow(h, &h->h_rows, &h->h_rows_cap, cap)) return s;
    return HSS_OK;
}

// Grows the shared-prime queue (entries of 16 bytes) to hold `n` pairs.
// A handle with the arc layout starts with smaller queues: its chunk of
// descriptors grows here too, where there is room (the pairs of a queue are set
// up in as many chunks as it takes).
int ensure_merged(hss_t* h, uint64_t n) {
    const uint32_t chunk = n > kArcMergedCap ? kDescChunk : kArcDescChunk;
    if (n > h->desc_chunk && h->desc_chunk < chunk) {
        HSS_CUDA(h, cudaStreamSynchronize(h->stream));
        const int s = device_grow(h, &h->d_desc, &h->desc_chunk, chunk, kBigEntryWords);
        if (s && !h->desc_chunk) return s;
    }
    if (n <= h->merged_cap) return HSS_OK;
    if (n >= UINT32_MAX) return fail(h, HSS_ERR_OVERFLOW, "shared-prime queue beyond 32-bit indexing");
    HSS_CUDA(h, cudaStreamSynchronize(h->stream));
    uint64_t cap = n <= kArcMergedCap ? kArcMergedCap : n + n / 8;
    if (cap >= UINT32_MAX) cap = UINT32_MAX - 1;
    int s = device_grow(h, &h->d_merged, &h->merged_cap, (size_t)cap);
    if (s && cap > n) s = device_grow(h, &h->d_merged, &h->merged_cap, (size_t)n);
    return s;
}

// A launch group whose exact work outgrew the exact queue, or whose big
// shared-prime pairs outgrew the big-pair queue, is incomplete: the queue
// that overflowed is enlarged 4x (exact: up to 2^28 items; big pairs: up to
// 2^24 descriptors of 192 bytes) and the caller runs the whole call again.
int grow_overflowed(hss_t* h) {
    if (!h->exact_overflow && !h->big_overflow) return HSS_ERR_OVERFLOW;
    HSS_CUDA(h, cudaStreamSynchronize(h->stream));
    if (h->exact_overflow) {
        h->exact_overflow = false;
        const uint64_t cap = (uint64_t)h->exact_cap * 4;
        if (cap > (1ull << 28)) return HSS_ERR_OVERFLOW;
        if (int s = device_grow(h, &h->d_exact, &h->exact_cap, (size_t)cap)) return s;
    }
    if (h->big_overflow) {
        h->big_overflow = false;
        const uint64_t cap = (uint64_t)h->big_cap * 4;
        if (cap > (1ull << 24)) return HSS_ERR_OVERFLOW;
        if (int s = device_grow(h, &h->d_big, &h->big_cap, (size_t)cap, kBigEntryWords)) return s;
    }
    return HSS_OK;
}

// Runs `call` again after enlarging the queue that overflowed (4x per rerun;
// h->call_reruns counts the reruns).
template <class Call>
int with_exact_retry(hss_t* h, Call call) {
    for (uint32_t attempt = 0;; ++attempt) {
        h->exact_overflow = h->big_overflow = false;
        h->call_reruns = attempt;
        const int s = call();
        if (s == HSS_ERR_OVERFLOW && (h->exact_overflow || h->big_overflow) && grow_overflowed(h) == HSS_OK)
            continue;
        return s;
    }
}

// Room for a launch group's rows, rest list and items (`bytes` in all) and
// its rows' values; growing waits for the stream.
int ensure_group(hss_t* h, size_t bytes, size_t values) {
    if (bytes > h->group_cap) {
        HSS_CUDA(h, cudaStreamSynchronize(h->stream));
        device_free(h, h->d_group);
        h->d_group = nullptr;
        h->group_cap = 0;
        const size_t cap = std::max(bytes + bytes / 4, (size_t)1 << 18);
        if (int s = device_alloc(h, &h->d_group, cap)) return s;
        for (unsigned char*& p : h->h_group) {
            if (p) cudaFreeHost(p);
            p = nullptr;
            HSS_CUDA(h, cudaMallocHost(&p, cap));
        }
        h->group_cap = cap;
    }
    if (values > h->values_cap) {
        HSS_CUDA(h, cudaStreamSynchronize(h->stream));
        device_free(h, h->d_values);
        device_free(h, h->d_value_hot);
        h->d_values = nullptr;
        h->d_value_hot = nullptr;
        h->values_cap = 0;
        const size_t cap = std::max(values + values / 4, (size_t)1 << 14);
        if (int s = device_alloc(h, &h->d_values, cap)) return s;
        if (int s = device_alloc(h, &h->d_value_hot, cap)) return s;
        h->values_cap = cap;
    }
    return HSS_OK;
}

int ensure_items(hss_t* h, size_t n) {
    const size_t cap = std::max(n + n / 4, (size_t)1 << 16);
    if (n > h->items_cap)
        if (int s = device_grow(h, &h->d_items, &h->items_cap, cap)) return s;
    if (n > h->h_items_cap)
        if (int s = host_grow(h, &h->h_items, &h->h_items_cap, cap)) return s;
    return HSS_OK;
}

// The shared-prime, big-pair, descriptor and exact-work queues at their first
// size, those that are not there (at open, or after a growth that lost one).
int ensure_queues(hss_t* h) {
    const uint64_t merged = !h->plan ? kMergedCap : h->limit < kArcLimit ? kArcMergedCap : kArcMergedStart;
    const uint32_t chunk = !h->plan ? kDescChunk : h->limit < kArcLimit ? kArcDescChunk : kArcDescStart;
    const uint32_t exact = h->opts.exact_capacity ? std::min<uint32_t>(h->opts.exact_capacity, 1u << 28) : 1u << 24;
    int s = HSS_OK;
    if (!h->merged_cap && (s = device_grow(h, &h->d_merged, &h->merged_cap, merged))) return s;
    if (!h->big_cap && (s = device_grow(h, &h->d_big, &h->big_cap, 1u << 20, kBigEntryWords))) return s;
    if (!h->desc_chunk && (s = device_grow(h, &h->d_desc, &h->desc_chunk, chunk, kBigEntryWords))) return s;
    if (!h->exact_cap && (s = device_grow(h, &h->d_exact, &h->exact_cap, exact))) return s;
    return HSS_OK;
}

// The buffers of one launch sequence (hits, control words, the shared-prime,
// big-pair, descriptor and exact-work queues, row counters), its stream and
// call events.  A handle has one set; serving gives each of its lanes another
// set over the same cache.
int alloc_launch_buffers(hss_t* h) {
    h->hit_cap = h->opts.hit_capacity ? h->opts.hit_capacity : kDefaultHitCap;
    int s = HSS_OK;
    if ((!h->d_hits && (s = device_alloc(h, &h->d_hits, h->hit_cap))) ||
        (!h->d_ctrl && (s = device_alloc(h, &h->d_ctrl, 8))) || (s = ensure_queues(h)) || (s = ensure_rows(h, 1024)))
        return s;
    if ((!h->stream && cudaStreamCreateWithFlags(&h->stream, cudaStreamNonBlocking) != cudaSuccess) ||
        cudaEventCreate(&h->ev0) != cudaSuccess || cudaEventCreate(&h->ev1) != cudaSuccess)
        return fail(h, HSS_ERR_CUDA, "stream or event creation failed");
    return HSS_OK;
}

LaunchBuffers buffers(const hss_t* h, size_t row_offset) {
    LaunchBuffers b;
    b.rows = h->d_rows + row_offset;
    b.hits = h->d_hits;
    b.hit_count = h->d_ctrl + 0;
    b.hit_cap = h->hit_cap;
    b.merged_queue = h->d_merged;
    b.merged_count = h->d_ctrl + 1;
    b.merged_cap = h->merged_cap;
    b.next_item = h->d_ctrl + 2;
    b.error_flags = h->d_ctrl + 3;
    b.tables = h->d_tables;
    b.row_info = h->d_row_info + row_offset;
    b.exact_queue = h->d_exact;
    b.exact_count = h->d_ctrl + 5;
    b.exact_cap = h->exact_cap;
    b.big_queue = h->d_big;
    b.big_count = h->d_ctrl + 4;
    b.big_next = h->d_ctrl + 6;
    b.big_cap = h->big_cap;
    b.pair_desc = h->d_desc;
    b.desc_chunk = h->desc_chunk;
    b.desc_next = h->d_ctrl + 7;
    return b;
}

int take_events(hss_t* h, std::array<cudaEvent_t, 3>* out) {
    for (int i = 0; i < 3; ++i) {
        if (h->events_used == h->event_pool.size()) {
            cudaEvent_t e;
            HSS_CUDA(h, cudaEventCreate(&e));
            h->event_pool.push_back(e);
        }
        (*out)[i] = h->event_pool[h->events_used++];
    }
    return HSS_OK;
}

// A row of a launch: root l and its index in the call's row counters.
struct RowRef {
    uint64_t l;
    uint32_t index;
};

// Work items of the given rows: each row's m-range [l, N] cut into ranges of
// about item_target alpha*beta evaluations (at most kTileCap roots), then
// ordered by m so that concurrently running items read the same m-side
// records from L2; the last wave is cut finer.  Returns the number of items
// and sets *alpha_cap to the largest row segment.
size_t build_items(hss_t* h, const RowRef* rows, size_t nrows, uint32_t* alpha_cap, uint32_t min_tile) {
    const uint64_t n = h->limit;
    const uint32_t target = h->opts.item_target ? h->opts.item_target : kDefaultItemTarget;
    std::vector<uint32_t> tile(nrows);
    size_t total = 0;
    uint32_t acap = 1;
    for (size_t r = 0; r < nrows; ++r) {
        uint64_t l = rows[r].l;
        uint32_t na = free_count(h, l) + 1;
        acap = std::max(acap, na);
        double per_m = (double)(h->seg_off[n + 1] - h->seg_off[l]) / (double)(n - l + 1);
        double t = (double)target / ((double)na * std::max(per_m, 1.0));
        uint32_t tm = t >= kTileCap ? kTileCap : (uint32_t)t;
        tm = std::max(min_tile, tm & ~(kTileMin - 1));
        tile[r] = tm;
        total += (n - l + 1 + tm - 1) / tm;
    }
    // the last wave of items (four per SM: two per CTA of the default shape)
    // is cut in four, so that the CTAs run out of work closer together
    const size_t tail = std::min(total, (size_t)h->sm_count * 4);
    if (ensure_items(h, total + 3 * tail)) return (size_t)-1;
    // counting sort by m-bucket of the item start
    const size_t nb = (n >> kBucketShift) + 2;
    std::vector<uint32_t> count(nb + 1, 0);
    for (size_t r = 0; r < nrows; ++r)
        for (uint64_t m = rows[r].l; m <= n; m += tile[r]) ++count[(m >> kBucketShift) + 1];
    for (size_t b = 1; b <= nb; ++b) count[b] += count[b - 1];
    for (size_t r = 0; r < nrows; ++r) {
        uint64_t l = rows[r].l;
        for (uint64_t m = l; m <= n; m += tile[r]) {
            uint64_t m1 = std::min<uint64_t>(m + tile[r], n + 1);
            h->h_items[count[m >> kBucketShift]++] =
                WorkItem{(uint32_t)l, (uint32_t)m, (uint32_t)m1, rows[r].index};
        }
    }
    std::vector<WorkItem> last(h->h_items + total - tail, h->h_items + total);
    size_t pos = total - tail;
    for (const WorkItem& it : last) {
        const uint32_t q = (it.m1 - it.m0 + 3) / 4;
        for (uint32_t s = it.m0; s < it.m1; s += q)
            h->h_items[pos++] = WorkItem{it.l, s, std::min(s + q, it.m1), it.row};
    }
    *alpha_cap = acap;
    return pos;
}

// Room for the constants of a call's rows; the stream is idle afterwards.
int ensure_row_info(hss_t* h, size_t rows) {
    HSS_CUDA(h, cudaStreamSynchronize(h->stream));
    const size_t cap = std::max(rows, (size_t)1024);
    if (rows > h->row_info_cap)
        if (int s = device_grow(h, &h->d_row_info, &h->row_info_cap, cap)) return s;
    if (rows > h->h_row_info_cap)
        if (int s = host_grow(h, &h->h_row_info, &h->h_row_info_cap, cap)) return s;
    return HSS_OK;
}

// Constants of the call's rows first .. first + count - 1 (row i of the call,
// root l_of(i), at index i).
template <class LOf>
int upload_row_info(hss_t* h, size_t first, size_t count, LOf l_of) {
    for (size_t i = first; i < first + count; ++i)
        fill_row_info(h->spf.data(), h->seg_off.data(), h->limit, l_of(i), &h->h_row_info[i]);
    HSS_CUDA(h, cudaMemcpyAsync(h->d_row_info + first, h->h_row_info + first, count * sizeof(RowInfo),
                                cudaMemcpyHostToDevice, h->stream));
    h->h2d_bytes += count * sizeof(RowInfo);
    return HSS_OK;
}

[[maybe_unused]] int check_errors(hss_t* h) {
    unsigned int ctrl[4];
    HSS_CUDA(h, cudaMemcpy(ctrl, h->d_ctrl, sizeof ctrl, cudaMemcpyDeviceToHost));
    if (ctrl[3] & 1u) return fail(h, HSS_ERR_OVERFLOW, "shared-prime queue over capacity");
    if (ctrl[3] & 2u) return fail(h, HSS_ERR_OVERFLOW, "shared-prime pair exceeds the list capacity");
    return HSS_OK;
}

// Captures the stream work of `enqueue` in a CUDA graph and launches it.  The
// handle keeps one executable graph and updates it in place from each new
// capture (item count, grid and buffer sizes change between calls); when the
// update is refused, the graph is instantiated again.
template <class Enqueue>
int run_captured(hss_t* h, Enqueue enqueue) {
    HSS_CUDA(h, cudaStreamBeginCapture(h->stream, cudaStreamCaptureModeThreadLocal));
    const int s = enqueue();
    cudaGraph_t g = nullptr;
    const cudaError_t ce = cudaStreamEndCapture(h->stream, &g);
    if (s || ce != cudaSuccess) {
        if (g) cudaGraphDestroy(g);
        if (s) return s;
        return fail(h, HSS_ERR_CUDA, std::string("cudaStreamEndCapture: ") + cudaGetErrorString(ce));
    }
    bool updated = false;
    if (h->graph_exec) {
        cudaGraphExecUpdateResultInfo info;
        if (cudaGraphExecUpdate(h->graph_exec, g, &info) == cudaSuccess) {
            updated = true;
        } else {
            cudaGetLastError();
            cudaGraphExecDestroy(h->graph_exec);
            h->graph_exec = nullptr;
        }
    }
    cudaError_t e = cudaSuccess;
    if (!updated) e = cudaGraphInstantiate(&h->graph_exec, g, 0);
    cudaGraphDestroy(g);
    if (e != cudaSuccess) return fail(h, HSS_ERR_CUDA, std::string("cudaGraphInstantiate: ") + cudaGetErrorString(e));
    HSS_CUDA(h, cudaGraphLaunch(h->graph_exec, h->stream));
    ++h->graph_launches;
    ++h->call_graphs;
    return HSS_OK;
}

int search_locked(hss_t* h, uint64_t first, uint64_t last, int mode, hss_counts* out, uint64_t* row_candidates,
                  hss_hit* hits, uint32_t hit_cap, uint32_t* nhits);
int search_many_locked(hss_t* h, const uint64_t* firsts, const uint64_t* lasts, uint32_t count, size_t rows,
                       hss_counts* per_interval, hss_counts* total, hss_hit* hits, uint32_t hit_cap,
                       uint32_t* nhits);

// Launches the batched sequence for a set of rows whose shared-prime pairs
// fit the queue: reset cursor/queue, items H2D, persistent kernel, shared-prime
// kernel.  Counters accumulate into d_rows[index].  pair_bound (at least those
// pairs) sets how many shared-prime chunks are launched.
int run_batched_rows(hss_t* h, const RowRef* rows, size_t nrows, uint64_t pair_bound) {
    // the pinned item buffer may still be read by the previous group's copy
    HSS_CUDA(h, cudaStreamSynchronize(h->stream));
    uint32_t acap = 1;
    const int threads = h->opts.block_threads ? (int)h->opts.block_threads : 256;
    // every warp of a CTA claims 128 roots at a time: items span at least that
    size_t n_items = build_items(h, rows, nrows, &acap, (uint32_t)threads / 32 * 128);
    if (n_items == (size_t)-1) return HSS_ERR_MEMORY;
    if (n_items == 0) return HSS_OK;
    BatchedConfig cfg;
    cfg.threads = h->opts.block_threads ? (int)h->opts.block_threads : 256;
    cfg.min_blocks = h->opts.ctas_per_sm ? (int)h->opts.ctas_per_sm : (cfg.threads == 128 ? 4 : cfg.threads == 512 ? 1 : 2);
    cfg.alpha_cap = acap;
    size_t smem = batched_smem_bytes(cfg.threads, acap);
    int per_sm = batched_max_ctas_per_sm(cfg.threads, cfg.min_blocks, smem);
    cfg.ctas = h->sm_count * per_sm;
    LaunchBuffers b = buffers(h, 0);
    std::array<cudaEvent_t, 3> ev;
    if (int e = take_events(h, &ev)) return e;
    // the group's stream work: items H2D, queue resets, the three kernels.
    // Inside a capture the timing events become event-record nodes
    // (cudaEventRecordExternal), so they still time the graph's kernels.
    const unsigned int rec = h->opts.use_graph ? cudaEventRecordExternal : cudaEventRecordDefault;
    uint32_t merged_launches = 0;
    auto enqueue = [&]() -> int {
        HSS_CUDA(h, cudaMemcpyAsync(h->d_items, h->h_items, n_items * sizeof(WorkItem), cudaMemcpyHostToDevice,
                                    h->stream));
        HSS_CUDA(h, cudaMemsetAsync(h->d_ctrl + 1, 0, 2 * sizeof(unsigned int), h->stream));
        HSS_CUDA(h, cudaMemsetAsync(h->d_ctrl + 4, 0, 3 * sizeof(unsigned int), h->stream));
        HSS_CUDA(h, cudaEventRecordWithFlags(ev[0], h->stream, rec));
        HSS_CUDA(h, launch_batched(h->dev, h->d_items, (uint32_t)n_items, cfg, b, h->stream));
        HSS_CUDA(h, cudaEventRecordWithFlags(ev[1], h->stream, rec));
        HSS_CUDA(h, launch_merged(h->dev, pair_bound, b, h->sm_count * 4, h->stream, &merged_launches));
        HSS_CUDA(h, launch_exact(h->dev, b, h->sm_count * 4, h->stream));
        HSS_CUDA(h, cudaEventRecordWithFlags(ev[2], h->stream, rec));
        return HSS_OK;
    };
    if (h->opts.use_graph) {
        if (int e = run_captured(h, enqueue)) return e;
    } else if (int e = enqueue()) {
        return e;
    }
    h->h2d_bytes += n_items * sizeof(WorkItem);
    h->marks.push_back(ev);
    h->launches += 2 + merged_launches;  // batched, shared-prime kernels, exact
    return HSS_OK;
}

// Splits rows into groups whose shared-prime bound fits the queue.
int run_products(hss_t* h, const std::vector<RowRef>& rows) {
    if (int s = ensure_row_info(h, rows.size())) return s;
    if (int s = upload_row_info(h, 0, rows.size(), [&](size_t i) { return rows[i].l; })) return s;
    size_t start = 0;
    while (start < rows.size()) {
        uint64_t bound = 0;
        size_t end = start;
        while (end < rows.size()) {
            uint64_t b = merged_bound(h, rows[end].l);
            if (end > start && bound + b > h->merged_cap) break;
            bound += b;
            ++end;
        }
        if (bound > h->merged_cap) return fail(h, HSS_ERR_OVERFLOW, "row exceeds the shared-prime queue");
        int s = run_batched_rows(h, rows.data() + start, end - start, bound);
        if (s) return s;
        start = end;
    }
    return HSS_OK;
}

// Launches the batched sequence for the rows collected in h->planner: reset
// cursors and queues, rows and items H2D, the rows' values, the persistent
// kernel, the shared-prime kernels over the rest list (when it holds any) and
// the exact kernel.  Counters accumulate into d_rows[index].
int run_planned(hss_t* h) {
    // (an executable graph is updated in place only when it does not run)
    if (h->opts.use_graph) HSS_CUDA(h, cudaStreamSynchronize(h->stream));
    ArcPlanner& p = h->planner;
    ArcConfig cfg;
    cfg.threads = h->opts.block_threads == 512 ? 512 : 768;
    cfg.ctas = h->sm_count * arc_max_ctas_per_sm(cfg.threads);
    if (p.entries > kArcValuesMost) return fail(h, HSS_ERR_OVERFLOW, "a launch group's values beyond 25-bit numbering");
    if (!p.finish(*h->plan, (uint32_t)cfg.ctas, arc_item_target(h->opts)))
        return fail(h, HSS_ERR_MEMORY, "no memory for a launch group's rows and items");
    if (p.rows.empty()) return HSS_OK;
    const size_t rows_b = p.rows.size() * sizeof(ArcRow), rest_b = p.rest.size() * sizeof(ArcRest),
                 items_b = p.items.size() * sizeof(ArcItem);
    auto align = [](size_t x) { return (x + 255) & ~(size_t)255; };
    const size_t rest_at = align(rows_b), items_at = rest_at + align(rest_b), bytes = items_at + items_b;
    if (int s = ensure_group(h, bytes, p.entries)) return s;
    // the pinned buffer of two groups ago: its copy is done
    const uint32_t turn = h->group_turn++ & 1u;
    unsigned char* host = h->h_group[turn];
    if (!h->group_copied[turn]) HSS_CUDA(h, cudaEventCreateWithFlags(&h->group_copied[turn], cudaEventDisableTiming));
    if (!h->opts.use_graph) HSS_CUDA(h, cudaEventSynchronize(h->group_copied[turn]));
    memcpy(host, p.rows.data(), rows_b);
    if (rest_b) memcpy(host + rest_at, p.rest.data(), rest_b);
    if (items_b) memcpy(host + items_at, p.items.data(), items_b);
    ArcBuffers b{buffers(h, 0), reinterpret_cast<const ArcRow*>(h->d_group), h->d_values, h->d_value_hot, h->d_arc_tabs};
    const ArcRest* rest = reinterpret_cast<const ArcRest*>(h->d_group + rest_at);
    const ArcItem* items = reinterpret_cast<const ArcItem*>(h->d_group + items_at);
    std::array<cudaEvent_t, 3> ev;
    if (int e = take_events(h, &ev)) return e;
    // Inside a capture the timing events become event-record nodes
    // (cudaEventRecordExternal), so they still time the graph's kernels.
    const unsigned int rec = h->opts.use_graph ? cudaEventRecordExternal : cudaEventRecordDefault;
    uint32_t launched = 0;
    auto enqueue = [&]() -> int {
        HSS_CUDA(h, cudaMemcpyAsync(h->d_group, host, bytes, cudaMemcpyHostToDevice, h->stream));
        if (!h->opts.use_graph) HSS_CUDA(h, cudaEventRecord(h->group_copied[turn], h->stream));
        HSS_CUDA(h, cudaMemsetAsync(h->d_ctrl + 1, 0, 2 * sizeof(unsigned int), h->stream));
        HSS_CUDA(h, cudaMemsetAsync(h->d_ctrl + 4, 0, 3 * sizeof(unsigned int), h->stream));
        HSS_CUDA(h, cudaEventRecordWithFlags(ev[0], h->stream, rec));
        HSS_CUDA(h, launch_arc_values(h->dev, (uint32_t)p.rows.size(), b, h->stream));
        HSS_CUDA(h, launch_arc(h->dev, items, (uint32_t)p.items.size(), cfg, b, h->stream));
        HSS_CUDA(h, cudaEventRecordWithFlags(ev[1], h->stream, rec));
        launched = 3;  // values, persistent, exact
        if (!p.rest.empty()) {
            uint32_t merged = 0;
            HSS_CUDA(h, launch_arc_rest(h->dev, rest, (uint32_t)p.rest.size(), b, h->sm_count * 8, h->stream));
            HSS_CUDA(h, launch_merged(h->dev, p.rest_pairs, b, h->sm_count * 4, h->stream, &merged));
            launched += 1 + merged;
        }
        HSS_CUDA(h, launch_arc_exact(h->dev, b, h->sm_count * 4, h->stream));
        HSS_CUDA(h, cudaEventRecordWithFlags(ev[2], h->stream, rec));
        return HSS_OK;
    };
    if (h->opts.use_graph) {
        if (int e = run_captured(h, enqueue)) return e;
    } else if (int e = enqueue()) {
        return e;
    }
    h->h2d_bytes += bytes;
    h->marks.push_back(ev);
    h->launches += launched;
    return HSS_OK;
}

// Splits the call's rows into launch groups whose values and rest pairs fit the
// buffers.  Of a long call the first eighth is a group by itself, so that the
// device works while the host plans the rest.
constexpr uint64_t kGroupValues = 8ull << 20;  // and one root more: 13.3 M at most, for 15,413,645 at LIMIT 3 10^7
static_assert(kGroupValues + (13ull << 20) <= kArcValuesMost, "a group's values can be numbered");
constexpr size_t kGroupRows = 1u << 20;
constexpr size_t kLongCall = 2048;

// Long calls below kArcLimit go by products: class lists are too short there
// for runs to pay (roots 80..4979 at LIMIT 5000: 3.3 ms by products, 4.1 ms by
// arcs; 100..7000 at 8000: 7.4 and 8.3; 4000..4100 at 5000: 0.39 and 0.46; but
// 3000..5000 at 11,000: 4.5 and 3.8).  Calls of at most kArcRows roots spend their
// time on launches and waits, of which the arc path has fewer (four roots at
// 8000: 0.36 ms by products, 0.13 by arcs; one at 2000 or 5000: 0.29 and 0.25, 0.39 and
// 0.18).
bool goes_by_arcs(const hss_t* h, size_t rows) { return h->plan && (h->limit >= kArcLimit || rows <= kArcRows); }

int run_batched(hss_t* h, const std::vector<RowRef>& rows) {
    if (!goes_by_arcs(h, rows.size())) return run_products(h, rows);
    h->planner.clear();
    size_t start = 0;
    bool grown = false;
    if (int s = ensure_row_info(h, rows.size())) return s;
    while (start < rows.size()) {
        const size_t piece = start == 0 && rows.size() >= kLongCall && !h->opts.use_graph ? rows.size() / 8 : rows.size() - start;
        if (int s = upload_row_info(h, start, piece, [&](size_t i) { return rows[i].l; })) return s;
        for (size_t i = start; i < start + piece; ++i) {
            h->planner.add(h->h_row_info[i], rows[i].index, h->limit, h->dev.max_exponent, 1, h->limit,
                           min_roots(h->limit, rows.size()));
            if (h->planner.rest_pairs >= h->merged_cap / 2 && h->merged_cap < kArcMergedCap && !grown) {
                // (once a call: without room for it the groups are smaller)
                grown = true;
                const int s = ensure_merged(h, kArcMergedCap);
                if (s && (s != HSS_ERR_MEMORY || !h->merged_cap || !h->desc_chunk)) return s;
            }
            const bool full = h->planner.entries >= kGroupValues || h->planner.rows.size() >= kGroupRows ||
                              h->planner.rest_pairs >= h->merged_cap / 2;
            if (!full && i + 1 < start + piece) continue;
            if (h->planner.rest_pairs > h->merged_cap)
                if (int s = ensure_merged(h, h->planner.rest_pairs)) return s;
            if (int s = run_planned(h)) return s;
            h->planner.clear();
        }
        start += piece;
    }
    return HSS_OK;
}

int run_plain(hss_t* h, uint64_t first, uint64_t last) {
    uint32_t nrows = 0;
    for (uint64_t b = first; b <= last; b += nrows) {
        nrows = (uint32_t)std::min<uint64_t>(kPlainBatch, last - b + 1);
        uint64_t bound = 0;
        uint32_t acap = 1;
        for (uint64_t l = b; l < b + nrows; ++l) {
            bound += merged_bound(h, l);
            acap = std::max(acap, free_count(h, l) + 1);
        }
        if (int s = ensure_merged(h, bound)) {
            // without room for the batch's pairs: as many of its rows as fit, at least one
            if (s != HSS_ERR_MEMORY || !h->merged_cap || !h->desc_chunk) return s;
            while (nrows > 1 && bound > h->merged_cap) bound -= merged_bound(h, b + --nrows);
            if (bound > h->merged_cap && (s = ensure_merged(h, bound))) return s;
        }
        HSS_CUDA(h, cudaMemsetAsync(h->d_ctrl + 1, 0, sizeof(unsigned int), h->stream));
        HSS_CUDA(h, cudaMemsetAsync(h->d_ctrl + 4, 0, 3 * sizeof(unsigned int), h->stream));
        LaunchBuffers buf = buffers(h, b - first);
        std::array<cudaEvent_t, 3> ev;
        if (int e = take_events(h, &ev)) return e;
        HSS_CUDA(h, cudaEventRecord(ev[0], h->stream));
        HSS_CUDA(h, launch_plain(h->dev, b, nrows, acap, buf, h->stream));
        HSS_CUDA(h, cudaEventRecord(ev[1], h->stream));
        uint32_t merged_launches = 0;
        HSS_CUDA(h, launch_merged(h->dev, bound, buf, h->sm_count * 4, h->stream, &merged_launches));
        HSS_CUDA(h, launch_exact(h->dev, buf, h->sm_count * 4, h->stream));
        HSS_CUDA(h, cudaEventRecord(ev[2], h->stream));
        h->marks.push_back(ev);
        h->launches += 2 + merged_launches;  // plain, shared-prime kernels, exact
    }
    return HSS_OK;
}

int begin_call(hss_t* h, size_t rows) {
    int s = ensure_rows(h, rows);
    if (!s) s = ensure_queues(h);
    if (s) return s;
    HSS_CUDA(h, cudaMemsetAsync(h->d_rows, 0, rows * sizeof(RowCounts), h->stream));
    HSS_CUDA(h, cudaMemsetAsync(h->d_ctrl, 0, 8 * sizeof(unsigned int), h->stream));
    HSS_CUDA(h, cudaEventRecord(h->ev0, h->stream));
    h->events_used = 0;
    h->marks.clear();
    h->launches = 0;
    h->call_graphs = 0;
    h->h2d_bytes = h->d2h_bytes = 0;
    return HSS_OK;
}

// Copies row counters and hits back; hits sorted by (l, m, n) and deduplicated.
int end_call(hss_t* h, size_t rows, double* ms, std::vector<DevHit>* hits, uint32_t* found,
             double* main_ms = nullptr, double* merged_ms = nullptr) {
    HSS_CUDA(h, cudaEventRecord(h->ev1, h->stream));
    HSS_CUDA(h, cudaMemcpyAsync(h->h_rows, h->d_rows, rows * sizeof(RowCounts), cudaMemcpyDeviceToHost,
                                h->stream));
    unsigned int ctrl[4];
    HSS_CUDA(h, cudaMemcpyAsync(ctrl, h->d_ctrl, sizeof ctrl, cudaMemcpyDeviceToHost, h->stream));
    HSS_CUDA(h, cudaStreamSynchronize(h->stream));
    float f = 0;
    HSS_CUDA(h, cudaEventElapsedTime(&f, h->ev0, h->ev1));
    *ms = f;
    double t_main = 0, t_merged = 0;
    for (auto& ev : h->marks) {
        float a = 0, b = 0;
        HSS_CUDA(h, cudaEventElapsedTime(&a, ev[0], ev[1]));
        HSS_CUDA(h, cudaEventElapsedTime(&b, ev[1], ev[2]));
        t_main += a;
        t_merged += b;
    }
    if (main_ms) *main_ms = t_main;
    if (merged_ms) *merged_ms = t_merged;
    h->d2h_bytes += rows * sizeof(RowCounts) + sizeof ctrl;
    if (ctrl[3] & 1u) return fail(h, HSS_ERR_OVERFLOW, "shared-prime queue over capacity");
    if (ctrl[3] & 2u) return fail(h, HSS_ERR_OVERFLOW, "shared-prime pair exceeds the list capacity");
    if (ctrl[3] & 12u) {
        h->exact_overflow = (ctrl[3] & 4u) != 0;
        h->big_overflow = (ctrl[3] & 8u) != 0;
        return fail(h, HSS_ERR_OVERFLOW, "exact work or big-pair queue over capacity");
    }
    if (ctrl[3] & ~15u) return fail(h, HSS_ERR_OVERFLOW, "a device index check failed (an event index out of range)");
    uint32_t nh = std::min(ctrl[0], h->hit_cap);
    hits->resize(nh);
    if (nh) HSS_CUDA(h, cudaMemcpy(hits->data(), h->d_hits, nh * sizeof(DevHit), cudaMemcpyDeviceToHost));
    h->d2h_bytes += nh * sizeof(DevHit);
    std::sort(hits->begin(), hits->end(), [](const DevHit& a, const DevHit& b) {
        if (a.l != b.l) return a.l < b.l;
        if (a.m != b.m) return a.m < b.m;
        return a.n < b.n;
    });
    hits->erase(std::unique(hits->begin(), hits->end(),
                            [](const DevHit& a, const DevHit& b) { return a.l == b.l && a.m == b.m && a.n == b.n; }),
                hits->end());
    *found = ctrl[0] > h->hit_cap ? ctrl[0] : (uint32_t)hits->size();
    return HSS_OK;
}

void add_row(hss_counts* c, const RowCounts& r) {
    c->processed += r.processed;
    c->products += r.products;
    c->candidates += r.candidates;
    c->r16 += r.r16;
    c->exact += r.exact;
    c->merged += r.merged;
    c->merged_products += r.mproducts;
    c->merged_candidates += r.mcandidates;
    c->merged_r16 += r.mr16;
}

void copy_hits(const std::vector<DevHit>& in, hss_hit* out, uint32_t cap) {
    for (size_t i = 0; i < in.size() && i < cap; ++i) {
        out[i].l = in[i].l;
        out[i].m = in[i].m;
        out[i].n = in[i].n;
        out[i].area4_lo = in[i].area4_lo;
        out[i].area4_hi = in[i].area4_hi;
        out[i].heron_ok = in[i].heron_ok;
        out[i].reserved = 0;
    }
}

// The arc layout of the handle's cache (h->dev, h->records), enqueued on the stream.
// It takes as much memory again as the cache: where the device has no room for it,
// the handle goes without and searches by products.
int open_arc_layout(hss_t* h) {
    if (h->limit < kArcLeast) return HSS_OK;
    auto plan = std::make_shared<ArcPlan>();
    ArcBuild b;
    std::string err;
    int s = plan_arc_blocks(h->dev.seg_off, h->limit, h->stream, plan.get(), &err);
    if (!s) s = build_arc_layout(h->dev, h->records, *plan, h->stream, &b, &err);
    if (s == HSS_ERR_MEMORY) return HSS_OK;
    if (s) return fail(h, s, err);
    h->allocations.insert(h->allocations.end(), b.owned.begin(), b.owned.end());
    h->dev.blocks = b.blocks;
    for (uint32_t f = 0; f < kFields; ++f) h->dev.arc_w[f] = b.w[f];
    h->dev.arc_ang = b.ang;
    h->dev.arc_part = b.part;
    h->dev.arc_src = b.src;
    h->dev.arc_m = b.m;
    h->dev.arc_xy = b.xy;
    h->dev.arc_index = b.index;
    h->dev.arc_mask = b.mask;
    h->dev.pos = b.pos;
    h->plan = std::move(plan);
    return HSS_OK;
}

// The handle's launch buffers; where the layout leaves no room for them, in its place.
int open_launch_buffers(hss_t* h) {
    const int s = alloc_launch_buffers(h);
    if (s != HSS_ERR_MEMORY || !h->plan) return s;
    HSS_CUDA(h, cudaStreamSynchronize(h->stream));
    device_free(h, const_cast<ArcBlock*>(h->dev.blocks));  // the first array of the layout's one allocation
    h->plan.reset();
    // (the product path's queues are larger)
    auto drop = [&](auto** p, uint32_t* cap) {
        device_free(h, *p);
        *p = nullptr;
        *cap = 0;
    };
    drop(&h->d_merged, &h->merged_cap);
    drop(&h->d_big, &h->big_cap);
    drop(&h->d_desc, &h->desc_chunk);
    drop(&h->d_exact, &h->exact_cap);
    return alloc_launch_buffers(h);
}

}  // namespace

// ------------------------------------------------------------------ exports

extern "C" {

const char* hss_version(void) { return "hss-gb300 1.0 (sm_103a)"; }

const char* hss_strerror(int status) {
    switch (status) {
        case HSS_OK: return "ok";
        case HSS_ERR_ARGUMENT: return "invalid argument";
        case HSS_ERR_CUDA: return "CUDA error";
        case HSS_ERR_MEMORY: return "out of memory";
        case HSS_ERR_LIMIT: return "limit not supported";
        case HSS_ERR_STATE: return "checkpoint does not match requested range";
        case HSS_ERR_OVERFLOW: return "internal capacity exceeded";
        case HSS_ERR_NOT_FOUND: return "unknown request";
        case HSS_ERR_BUSY: return "request still running";
        case HSS_ERR_NO_DEVICE: return "no sm_103 CUDA device";
        default: return "unknown status";
    }
}

const char* hss_last_error(const hss_t* h) { return h ? h->err.c_str() : "null handle"; }

int hss_cache_check(uint64_t limit, int device, uint64_t* mismatches, double* host_seconds,
                    double* device_seconds) {
    if (!mismatches || limit < 1 || limit > HSS_MAX_LIMIT) return HSS_ERR_ARGUMENT;
    int ndev = 0;
    if (cudaGetDeviceCount(&ndev) != cudaSuccess || device < 0 || device >= ndev || cudaSetDevice(device) != cudaSuccess)
        return HSS_ERR_NO_DEVICE;
    cudaDeviceProp prop;
    if (cudaGetDeviceProperties(&prop, device) != cudaSuccess) return HSS_ERR_NO_DEVICE;
    HostCache hc;
    std::string err;
    unsigned hw = std::thread::hardware_concurrency();
    int s = build_host_cache(limit, (int)(hw ? hw : 1), &hc, &err);
    if (s) return s;
    cudaStream_t st = nullptr;
    if (cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking) != cudaSuccess) return HSS_ERR_CUDA;
    DeviceBuild db;
    s = build_device_cache(limit, prop.multiProcessorCount, st, &db, &err);
    cudaStreamDestroy(st);
    if (s) return s;
    uint64_t bad = 0;
    auto compare = [&](const void* dev, const void* host, size_t count, size_t elem) -> int {
        std::vector<unsigned char> copy(count * elem);
        if (count && cudaMemcpy(copy.data(), dev, count * elem, cudaMemcpyDeviceToHost) != cudaSuccess)
            return HSS_ERR_CUDA;
        const unsigned char* h = static_cast<const unsigned char*>(host);
        for (size_t i = 0; i < count; ++i)
            if (memcmp(copy.data() + i * elem, h + i * elem, elem) != 0) ++bad;
        return HSS_OK;
    };
    bad += (db.records != hc.records) + (db.pp_count != hc.pp_hot.size()) +
           (db.reference_flattened != hc.reference_flattened) + (db.reference_cached != hc.reference_cached) +
           (db.max_exponent != hc.max_exponent);
    if (!bad) {
        if ((s = compare(db.spf, hc.spf.data(), hc.spf.size(), sizeof(uint32_t))) ||
            (s = compare(db.seg_off, hc.seg_off.data(), hc.seg_off.size(), sizeof(uint32_t))) ||
            (s = compare(db.hot, hc.hot.get(), hc.records, sizeof(HotRec))) ||
            (s = compare(db.exact, hc.exact.get(), hc.records, sizeof(ExactRec))) ||
            (s = compare(db.owner, hc.owner.get(), hc.records, sizeof(uint32_t))) ||
            (s = compare(db.pp_base, hc.pp_base.data(), hc.pp_base.size(), sizeof(uint32_t))) ||
            (s = compare(db.pp_hot, hc.pp_hot.data(), hc.pp_hot.size(), sizeof(HotRec))) ||
            (s = compare(db.pp_exact, hc.pp_exact.data(), hc.pp_exact.size(), sizeof(__int128)))) {
            for (void* p : db.owned) cudaFree(p);
            return s;
        }
        bad += (db.spf_host != hc.spf) + (db.seg_off_host != hc.seg_off);
    }
    for (void* p : db.owned) cudaFree(p);
    *mismatches = bad;
    if (host_seconds) *host_seconds = hc.seconds;
    if (device_seconds) *device_seconds = db.seconds;
    return HSS_OK;
}

int hss_open(uint64_t limit, int device, const hss_opts* opts, hss_t** out) {
    if (!out) return HSS_ERR_ARGUMENT;
    *out = nullptr;
    if (limit < 1 || limit > HSS_MAX_LIMIT) return HSS_ERR_LIMIT;
    hss_t* h = new hss_t();
    if (opts) h->opts = *opts;
    h->device = device;
    h->limit = limit;
    int ndev = 0;
    if (cudaGetDeviceCount(&ndev) != cudaSuccess || device < 0 || device >= ndev) {
        delete h;
        return HSS_ERR_NO_DEVICE;
    }
    cudaDeviceProp prop;
    if (cudaSetDevice(device) != cudaSuccess || cudaGetDeviceProperties(&prop, device) != cudaSuccess ||
        prop.major != 10 || prop.minor != 3) {
        delete h;
        return HSS_ERR_NO_DEVICE;
    }
    h->sm_count = prop.multiProcessorCount;
    int s = HSS_OK;
    if (cudaStreamCreateWithFlags(&h->stream, cudaStreamNonBlocking) != cudaSuccess) {
        delete h;
        return HSS_ERR_CUDA;
    }
    if (!h->opts.host_build) {
        // the cache built by kernels on the device (same arrays and values as the host build)
        DeviceBuild db;
        std::string err;
        auto take = [&] {
            h->records = db.records;
            h->dev.limit = limit;
            h->dev.spf = db.spf;
            h->dev.seg_off = db.seg_off;
            h->dev.hot = db.hot;
            h->dev.exact = db.exact;
            h->dev.owner = db.owner;
            h->dev.pp_base = db.pp_base;
            h->dev.pp_hot = db.pp_hot;
            h->dev.pp_exact = db.pp_exact;
            h->dev.max_exponent = db.max_exponent;
            return open_arc_layout(h);
        };
        s = build_device_cache(limit, h->sm_count, h->stream, &db, &err, take);
        if (s) {
            hss_close(h);
            return s;
        }
        h->allocations.insert(h->allocations.end(), db.owned.begin(), db.owned.end());
        if (db.longest > kItemRecords) {
            hss_close(h);
            return HSS_ERR_LIMIT;
        }
        h->ref_flattened = db.reference_flattened;
        h->ref_cached = db.reference_cached;
        h->prep_seconds = db.seconds;
        h->seg_off = std::move(db.seg_off_host);
        h->spf = std::move(db.spf_host);
    } else {
        HostCache hc;
        std::string err;
        unsigned hw = std::thread::hardware_concurrency();
        int threads = h->opts.prep_threads ? (int)h->opts.prep_threads : (int)(hw ? hw : 1);
        s = build_host_cache(limit, threads, &hc, &err);
        if (s) {
            hss_close(h);
            return s;
        }
        uint32_t longest = 0;
        for (uint64_t x = 1; x <= limit; ++x) longest = std::max(longest, hc.seg_off[x + 1] - hc.seg_off[x]);
        if (longest > kItemRecords) {
            hss_close(h);
            return HSS_ERR_LIMIT;
        }
        h->records = hc.records;
        h->ref_flattened = hc.reference_flattened;
        h->ref_cached = hc.reference_cached;
        h->prep_seconds = hc.seconds;
        uint32_t *spf, *seg, *owner, *ppb;
        HotRec *hot, *pph;
        ExactRec* ex;
        __int128* ppx;
        if ((s = upload(h, &spf, hc.spf.data(), hc.spf.size())) ||
            (s = upload(h, &seg, hc.seg_off.data(), hc.seg_off.size())) ||
            (s = upload(h, &hot, hc.hot.get(), hc.records)) || (s = upload(h, &ex, hc.exact.get(), hc.records)) ||
            (s = upload(h, &owner, hc.owner.get(), hc.records)) ||
            (s = upload(h, &ppb, hc.pp_base.data(), hc.pp_base.size())) ||
            (s = upload(h, &pph, hc.pp_hot.data(), hc.pp_hot.size())) ||
            (s = upload(h, &ppx, hc.pp_exact.data(), hc.pp_exact.size()))) {
            hss_close(h);
            return s;
        }
        h->dev.limit = limit;
        h->dev.spf = spf;
        h->dev.seg_off = seg;
        h->dev.hot = hot;
        h->dev.exact = ex;
        h->dev.owner = owner;
        h->dev.pp_base = ppb;
        h->dev.pp_hot = pph;
        h->dev.pp_exact = ppx;
        h->dev.max_exponent = hc.max_exponent;
        h->seg_off = std::move(hc.seg_off);
        h->spf = std::move(hc.spf);
        if (cudaDeviceSynchronize() != cudaSuccess || (s = open_arc_layout(h)) ||
            cudaStreamSynchronize(h->stream) != cudaSuccess) {
            hss_close(h);
            return s ? s : HSS_ERR_CUDA;
        }
    }
    std::vector<uint8_t> tables(kTableTotalBytes);
    build_residue_tables(tables.data());
    std::vector<uint8_t> arc_tabs(kArcTabBytes);
    build_arc_tables(arc_tabs.data());
    if ((s = upload(h, &h->d_tables, tables.data(), kTableTotalBytes)) ||
        (s = upload(h, &h->d_arc_tabs, arc_tabs.data(), kArcTabBytes)) || (s = open_launch_buffers(h))) {
        hss_close(h);
        return s;
    }
    *out = h;
    return HSS_OK;
}

int hss_serve_stop(hss_t* h);

void hss_close(hss_t* h) {
    if (!h) return;
    hss_serve_stop(h);
    cudaSetDevice(h->device);
    if (h->stream) cudaStreamSynchronize(h->stream);
    for (void* p : h->allocations) cudaFree(p);
    if (h->h_items) cudaFreeHost(h->h_items);
    for (unsigned char* p : h->h_group)
        if (p) cudaFreeHost(p);
    for (cudaEvent_t e : h->group_copied)
        if (e) cudaEventDestroy(e);
    if (h->h_rows) cudaFreeHost(h->h_rows);
    if (h->h_row_info) cudaFreeHost(h->h_row_info);
    if (h->h_ctrl) cudaFreeHost(h->h_ctrl);
    if (h->h_slots) cudaFreeHost(h->h_slots);
    if (h->ev0) cudaEventDestroy(h->ev0);
    if (h->ev1) cudaEventDestroy(h->ev1);
    for (cudaEvent_t e : h->event_pool) cudaEventDestroy(e);
    if (h->graph_exec) cudaGraphExecDestroy(h->graph_exec);
    if (h->stream) cudaStreamDestroy(h->stream);
    delete h;
}

int hss_int32_peak(int device, double* ops_per_second, double* ms) {
    int ndev = 0;
    if (cudaGetDeviceCount(&ndev) != cudaSuccess || device < 0 || device >= ndev) return HSS_ERR_NO_DEVICE;
    cudaDeviceProp prop;
    if (cudaGetDeviceProperties(&prop, device) != cudaSuccess) return HSS_ERR_CUDA;
    double v = int32_peak_ops(device, prop.multiProcessorCount, ms);
    if (ops_per_second) *ops_per_second = v;
    return v > 0 ? HSS_OK : HSS_ERR_CUDA;
}

int hss_info(const hss_t* h, uint64_t* limit, uint64_t* records, uint64_t* flattened, uint64_t* cached,
             double* prep_seconds) {
    if (!h) return HSS_ERR_ARGUMENT;
    if (limit) *limit = h->limit;
    if (records) *records = h->records;
    if (flattened) *flattened = h->ref_flattened;
    if (cached) *cached = h->ref_cached;
    if (prep_seconds) *prep_seconds = h->prep_seconds;
    return HSS_OK;
}

int hss_cache_inspect(uint64_t limit, uint64_t x, uint64_t* records, uint64_t* flattened, uint64_t* cached,
                      int64_t* re, int64_t* im, uint32_t cap, uint32_t* count) {
    if (limit < 1 || limit > HSS_MAX_LIMIT || x > limit) return HSS_ERR_ARGUMENT;
    HostCache hc;
    std::string err;
    unsigned hw = std::thread::hardware_concurrency();
    int s = build_host_cache(limit, (int)(hw ? hw : 1), &hc, &err);
    if (s) return s;
    if (records) *records = hc.records;
    if (flattened) *flattened = hc.reference_flattened;
    if (cached) *cached = hc.reference_cached;
    if (x) {
        uint32_t a = hc.seg_off[x], b = hc.seg_off[x + 1];
        if (count) *count = b - a;
        for (uint32_t i = a; i < b && i - a < cap; ++i) {
            if (re) re[i - a] = hc.exact[i].re;
            if (im) im[i - a] = hc.exact[i].im;
        }
    }
    return HSS_OK;
}

int hss_search(hss_t* h, uint64_t first, uint64_t last, int mode, hss_counts* out, uint64_t* row_candidates,
               hss_hit* hits, uint32_t hit_cap, uint32_t* nhits) {
    if (!h || !out) return HSS_ERR_ARGUMENT;
    if (first < 1 || first > last || last > h->limit)
        return fail(h, HSS_ERR_ARGUMENT, "need 1 <= first <= last <= limit");
    if (mode != HSS_MODE_PLAIN && mode != HSS_MODE_BATCHED) return fail(h, HSS_ERR_ARGUMENT, "unknown mode");
    std::lock_guard<std::mutex> lock(h->gpu_mu);
    HSS_CUDA(h, cudaSetDevice(h->device));
    return with_exact_retry(h, [&] { return search_locked(h, first, last, mode, out, row_candidates, hits, hit_cap,
                                                          nhits); });
}

}  // extern "C"

namespace {

int search_locked(hss_t* h, uint64_t first, uint64_t last, int mode, hss_counts* out, uint64_t* row_candidates,
                  hss_hit* hits, uint32_t hit_cap, uint32_t* nhits) {
    const size_t rows = (size_t)(last - first + 1);
    int s = begin_call(h, rows);
    if (s) return s;
    if (mode == HSS_MODE_PLAIN) {
        if ((s = ensure_row_info(h, rows)) || (s = upload_row_info(h, 0, rows, [&](size_t i) { return first + i; }))) return s;
        s = run_plain(h, first, last);
    } else {
        std::vector<RowRef> refs(rows);
        for (size_t r = 0; r < rows; ++r) refs[r] = RowRef{first + r, (uint32_t)r};
        s = run_batched(h, refs);
    }
    if (s) return s;
    std::vector<DevHit> found;
    uint32_t nfound = 0;
    double ms = 0, main_ms = 0, merged_ms = 0;
    if ((s = end_call(h, rows, &ms, &found, &nfound, &main_ms, &merged_ms))) return s;
    memset(out, 0, sizeof *out);
    out->main_ms = main_ms;
    out->merged_ms = merged_ms;
    out->launches = h->launches;
    out->graph_launches = h->call_graphs;
    out->reruns = h->call_reruns;
    out->h2d_bytes = h->h2d_bytes;
    out->d2h_bytes = h->d2h_bytes;
    for (size_t r = 0; r < rows; ++r) {
        add_row(out, h->h_rows[r]);
        out->pairs += h->limit - (first + r) + 1;
        if (row_candidates) row_candidates[r] = h->h_rows[r].candidates;
    }
    out->hits = nfound;
    out->kernel_ms = ms;
    if (hits) copy_hits(found, hits, hit_cap);
    if (nhits) *nhits = nfound;
    return HSS_OK;
}

}  // namespace

extern "C" {

int hss_autotune(hss_t* h, uint64_t first, uint64_t last, hss_opts* best, hss_tune_trial* trials,
                 uint32_t max_trials, uint32_t* ntrials) {
    if (!h) return HSS_ERR_ARGUMENT;
    struct Setting {
        uint32_t threads, ctas, target;
    };
    static const uint32_t kProducts[][2] = {{128, 4}, {128, 6}, {256, 2}, {256, 3}, {512, 1}};
    static const uint32_t kArcs[][2] = {{256, 2}, {512, 1}};  // 24 warps per CTA, and 16
    static const uint32_t kTargets[] = {0, 1u << 21, 1u << 22, 1u << 23, 1u << 24, 1u << 25};
    const hss_opts saved = h->opts;
    const bool arcs = first <= last && goes_by_arcs(h, last - first + 1);
    // the handle's own setting first, then every variant with every weight; the
    // product path's own weight is one of the list, the arc path's is 0
    Setting list[1 + 5 * 6];
    uint32_t n = 0;
    auto add = [&](const Setting& x) {
        for (uint32_t i = 0; i < n; ++i)
            if (list[i].threads == x.threads && list[i].ctas == x.ctas && list[i].target == x.target) return;
        list[n++] = x;
    };
    {
        const uint32_t threads = arcs ? (saved.block_threads == 512 ? 512u : 256u) : saved.block_threads ? saved.block_threads : 256u;
        const uint32_t ctas = !arcs && saved.ctas_per_sm ? saved.ctas_per_sm : threads == 128 ? 4u : threads == 512 ? 1u : 2u;
        add(Setting{threads, ctas, saved.item_target || arcs ? saved.item_target : kDefaultItemTarget});
    }
    for (uint32_t v = 0; v < (arcs ? 2u : 5u); ++v) {
        const uint32_t* variant = arcs ? kArcs[v] : kProducts[v];
        for (uint32_t target : kTargets)
            if (target || arcs) add(Setting{variant[0], variant[1], target});
    }
    hss_opts chosen = saved;
    float best_ms = 0;
    for (uint32_t i = 0; i < n; ++i) {
        h->opts.block_threads = list[i].threads;
        h->opts.ctas_per_sm = list[i].ctas;
        h->opts.item_target = list[i].target;
        hss_counts c;
        int s = hss_search(h, first, last, HSS_MODE_BATCHED, &c, nullptr, nullptr, 0, nullptr);  // warm
        if (!s) s = hss_search(h, first, last, HSS_MODE_BATCHED, &c, nullptr, nullptr, 0, nullptr);
        if (s) {
            h->opts = saved;
            return s;
        }
        float ms = (float)c.kernel_ms;
        if (trials && i < max_trials) trials[i] = hss_tune_trial{list[i].threads, list[i].ctas, list[i].target, ms};
        // By arcs a weight holds for calls of every size from then on, where the
        // planner's follows the call: it has to be worth 3 % (runs of one setting
        // differ by 2 %; at LIMIT 10^7 64 roots take 16.4 ms by the planner's and 16.4
        // to 17.8 ms with fixed ones, 512 roots 106.1 to 108.5 ms and 106.1 to 122.3).
        if (arcs && list[i].target) ms *= 1.03f;
        if (best_ms == 0 || ms < best_ms) {
            best_ms = ms;
            chosen = h->opts;
        }
    }
    h->opts = chosen;
    if (best) *best = chosen;
    if (ntrials) *ntrials = n;
    return HSS_OK;
}

int hss_search_many(hss_t* h, const uint64_t* firsts, const uint64_t* lasts, uint32_t count,
                    hss_counts* per_interval, hss_counts* total, hss_hit* hits, uint32_t hit_cap,
                    uint32_t* nhits) {
    if (!h || !firsts || !lasts || count == 0) return HSS_ERR_ARGUMENT;
    size_t rows = 0;
    for (uint32_t i = 0; i < count; ++i) {
        if (firsts[i] < 1 || firsts[i] > lasts[i] || lasts[i] > h->limit)
            return fail(h, HSS_ERR_ARGUMENT, "need 1 <= first <= last <= limit for every interval");
        rows += lasts[i] - firsts[i] + 1;
    }
    if (rows > UINT32_MAX) return fail(h, HSS_ERR_ARGUMENT, "too many rows");
    std::lock_guard<std::mutex> lock(h->gpu_mu);
    HSS_CUDA(h, cudaSetDevice(h->device));
    return with_exact_retry(h, [&] {
        return search_many_locked(h, firsts, lasts, count, rows, per_interval, total, hits, hit_cap, nhits);
    });
}

}  // extern "C"

namespace {

int search_many_locked(hss_t* h, const uint64_t* firsts, const uint64_t* lasts, uint32_t count, size_t rows,
                       hss_counts* per_interval, hss_counts* total, hss_hit* hits, uint32_t hit_cap,
                       uint32_t* nhits) {
    int s = begin_call(h, rows);
    if (s) return s;
    std::vector<RowRef> refs;
    refs.reserve(rows);
    for (uint32_t i = 0; i < count; ++i)
        for (uint64_t l = firsts[i]; l <= lasts[i]; ++l) refs.push_back(RowRef{l, (uint32_t)refs.size()});
    if ((s = run_batched(h, refs))) return s;
    std::vector<DevHit> found;
    uint32_t nfound = 0;
    double ms = 0, main_ms = 0, merged_ms = 0;
    if ((s = end_call(h, rows, &ms, &found, &nfound, &main_ms, &merged_ms))) return s;
    hss_counts sum{};
    sum.main_ms = main_ms;
    sum.merged_ms = merged_ms;
    sum.launches = h->launches;
    sum.graph_launches = h->call_graphs;
    sum.reruns = h->call_reruns;
    sum.h2d_bytes = h->h2d_bytes;
    sum.d2h_bytes = h->d2h_bytes;
    size_t r = 0;
    for (uint32_t i = 0; i < count; ++i) {
        hss_counts c{};
        for (uint64_t l = firsts[i]; l <= lasts[i]; ++l, ++r) {
            add_row(&c, h->h_rows[r]);
            c.pairs += h->limit - l + 1;
        }
        for (const DevHit& hit : found)
            if (hit.l >= firsts[i] && hit.l <= lasts[i]) ++c.hits;
        if (per_interval) per_interval[i] = c;
        sum.pairs += c.pairs;
        sum.processed += c.processed;
        sum.products += c.products;
        sum.candidates += c.candidates;
        sum.r16 += c.r16;
        sum.exact += c.exact;
        sum.merged += c.merged;
        sum.merged_products += c.merged_products;
        sum.merged_candidates += c.merged_candidates;
        sum.merged_r16 += c.merged_r16;
    }
    sum.hits = nfound;
    sum.kernel_ms = ms;
    if (total) *total = sum;
    if (hits) copy_hits(found, hits, hit_cap);
    if (nhits) *nhits = nfound;
    return HSS_OK;
}

}  // namespace

// ------------------------------------------------------------------ serving
//
// Continuous admission.  Requests queue at hss_submit; a background loop
// admits them while request slots and device state space are free, and runs
// waves - a bounded slice of every admitted request - on two lanes (launch
// buffers and a stream each, over the handle's cache), so one wave runs on
// the device while the host harvests the previous one and forms the next.
// Each admitted request owns a range of row records in a device arena sized
// from free HBM at serve start: every wave ends with a kernel that writes its
// row counters there, marked done, so a request's progress and counts stay
// on the device until it completes and are read back once.  Admission waits
// when the arena has no room for a request's rows.

namespace hss {

struct Request {
    uint64_t id = 0, first = 0, last = 0;
    uint64_t next_row = 0;  // next root to schedule
    uint64_t rows_done = 0;
    uint64_t inflight = 0;  // rows in waves not yet settled
    uint32_t slot = 0;      // first record of its rows in the device state arena
    uint64_t submitted_ns = 0, admitted_ns = 0, finished_ns = 0;
    double ms_weighted = 0; // wave device time x its logical pairs in the wave
    hss_counts counts{};
    std::vector<DevHit> hits;
    int status = HSS_ERR_BUSY;
    bool admitted = false;
};

// A wave on a lane: its rows (index i of the wave) and their requests.
struct Wave {
    std::vector<RowRef> rows;
    std::vector<Request*> owner;
    bool live = false;
};

}  // namespace hss

namespace {

// A lane: a second set of launch buffers and a stream over h's cache (the
// cache arrays and residue tables are shared, not owned).
hss_t* make_lane(hss_t* h, int* status) {
    hss_t* lane = new hss_t();
    lane->device = h->device;
    lane->limit = h->limit;
    lane->opts = h->opts;
    lane->opts.use_graph = 0;
    lane->sm_count = h->sm_count;
    lane->seg_off = h->seg_off;
    lane->spf = h->spf;
    lane->dev = h->dev;
    lane->d_tables = h->d_tables;
    lane->d_arc_tabs = h->d_arc_tabs;
    lane->plan = h->plan;
    int s = alloc_launch_buffers(lane);
    if (!s && cudaMallocHost(&lane->h_ctrl, 8 * sizeof(unsigned int)) != cudaSuccess) {
        cudaGetLastError();
        s = HSS_ERR_MEMORY;
    }
    if (s) {
        hss_close(lane);
        *status = s;
        return nullptr;
    }
    *status = HSS_OK;
    return lane;
}

int ensure_slots(hss_t* lane, size_t n) {
    const size_t cap = std::max(n, (size_t)1024);
    if (n > lane->slots_cap)
        if (int s = device_grow(lane, &lane->d_slots, &lane->slots_cap, cap)) return s;
    if (n > lane->h_slots_cap)
        if (int s = host_grow(lane, &lane->h_slots, &lane->h_slots_cap, cap)) return s;
    return HSS_OK;
}

// Enqueues a wave on its (idle) lane: row constants, the batched launch
// groups, the scatter of its row counters into the requests' device state,
// and the read-back of the control words.  Returns without waiting for the
// device.
int launch_wave(hss_t* h, hss_t* lane, const Wave& w) {
    const size_t n = w.rows.size();
    int s = begin_call(lane, n);
    if (s) return s;
    if ((s = ensure_slots(lane, n))) return s;
    for (size_t i = 0; i < n; ++i) lane->h_slots[i] = w.owner[i]->slot + (uint32_t)(w.rows[i].l - w.owner[i]->first);
    HSS_CUDA(lane, cudaMemcpyAsync(lane->d_slots, lane->h_slots, n * sizeof(uint32_t), cudaMemcpyHostToDevice,
                                   lane->stream));
    if ((s = run_batched(lane, w.rows))) return s;
    HSS_CUDA(lane, launch_scatter_rows(lane->d_rows, lane->d_slots, (uint32_t)n, h->d_state, lane->stream));
    HSS_CUDA(lane, cudaEventRecord(lane->ev1, lane->stream));
    HSS_CUDA(lane, cudaMemcpyAsync(lane->h_ctrl, lane->d_ctrl, 8 * sizeof(unsigned int), cudaMemcpyDeviceToHost,
                                   lane->stream));
    return HSS_OK;
}

// Waits for a lane's wave and collects its hits and device time; a wave whose
// exact-work or big-pair queue overflowed runs again (grown queue) before it
// counts.
int finish_wave(hss_t* h, hss_t* lane, const Wave& w, std::vector<DevHit>* hits, double* ms) {
    for (uint32_t attempt = 0;; ++attempt) {
        HSS_CUDA(lane, cudaStreamSynchronize(lane->stream));
        const unsigned int* ctrl = lane->h_ctrl;
        if ((ctrl[3] & 12u) && !(ctrl[3] & 3u)) {
            lane->exact_overflow = (ctrl[3] & 4u) != 0;
            lane->big_overflow = (ctrl[3] & 8u) != 0;
            if (grow_overflowed(lane) != HSS_OK)
                return fail(lane, HSS_ERR_OVERFLOW, "exact work or big-pair queue over capacity");
            if (int s = launch_wave(h, lane, w)) return s;
            continue;
        }
        if (ctrl[3] & 1u) return fail(lane, HSS_ERR_OVERFLOW, "shared-prime queue over capacity");
        if (ctrl[3] & 2u) return fail(lane, HSS_ERR_OVERFLOW, "shared-prime pair exceeds the list capacity");
        if (ctrl[3]) return fail(lane, HSS_ERR_OVERFLOW, "a device index check failed");
        const uint32_t nh = std::min(ctrl[0], lane->hit_cap);
        hits->resize(nh);
        if (nh) HSS_CUDA(lane, cudaMemcpy(hits->data(), lane->d_hits, nh * sizeof(DevHit), cudaMemcpyDeviceToHost));
        float f = 0;
        HSS_CUDA(lane, cudaEventElapsedTime(&f, lane->ev0, lane->ev1));
        *ms = f;
        return HSS_OK;
    }
}

// Sums a completed request's row records from the device state arena into
// its counters; every row must be marked done.
int read_request_state(hss_t* h, Request* r) {
    const size_t rows = (size_t)(r->last - r->first + 1);
    std::vector<RowCounts> state(rows);
    HSS_CUDA(h, cudaMemcpy(state.data(), h->d_state + r->slot, rows * sizeof(RowCounts), cudaMemcpyDeviceToHost));
    for (size_t i = 0; i < rows; ++i) {
        if (state[i].pad != 1) return fail(h, HSS_ERR_STATE, "a request row was not recorded on the device");
        add_row(&r->counts, state[i]);
        r->counts.pairs += h->limit - (r->first + i) + 1;
    }
    r->counts.d2h_bytes += rows * sizeof(RowCounts);
    return HSS_OK;
}

// Attributes a finished wave to its requests (under serve_mu) and completes
// those whose rows are all done: counters from the device state, slot range
// released.
void settle_wave(hss_t* h, Wave& w, int status, const std::vector<DevHit>& hits, double ms,
                 std::vector<Request*>& active) {
    std::lock_guard<std::mutex> lock(h->serve_mu);
    for (size_t i = 0; i < w.rows.size(); ++i) {
        Request* r = w.owner[i];
        --r->inflight;
        if (status) {
            r->status = status;
            r->next_row = r->last + 1;  // schedule nothing more
            continue;
        }
        r->ms_weighted += ms * (double)(h->limit - w.rows[i].l + 1);
        ++r->rows_done;
    }
    for (const DevHit& hit : hits)
        if (hit.row < w.owner.size()) w.owner[hit.row]->hits.push_back(hit);
    const uint64_t t = now_ns();
    for (size_t i = 0; i < active.size();) {
        Request* r = active[i];
        const uint64_t rows = r->last - r->first + 1;
        const bool failed = r->status != HSS_ERR_BUSY;
        // a request leaves when all its rows are done, or when it failed and
        // no wave in flight still writes its state records
        if (failed ? r->inflight > 0 : r->rows_done < rows) {
            ++i;
            continue;
        }
        if (!failed) {
            const int s = read_request_state(h, r);
            r->status = s ? s : HSS_OK;
            r->counts.kernel_ms = r->ms_weighted / (double)std::max<uint64_t>(r->counts.pairs, 1);
            r->counts.hits = r->hits.size();
        }
        r->finished_ns = t;
        h->arena.release(r->slot, (uint32_t)rows);
        active[i] = active.back();
        active.pop_back();
    }
    w.rows.clear();
    w.owner.clear();
    w.live = false;
    h->serve_cv.notify_all();
}

void serve_loop(hss_t* h) {
    cudaSetDevice(h->device);
    std::vector<Request*> active;
    Wave waves[2];
    int next_lane = 0;
    for (;;) {
        Wave w;
        {
            std::unique_lock<std::mutex> lock(h->serve_mu);
            auto schedulable = [&] {
                for (Request* r : active)
                    if (r->next_row <= r->last) return true;
                return false;
            };
            h->serve_cv.wait(lock, [&] {
                return h->serve_stop || !h->pending.empty() || schedulable() || waves[0].live || waves[1].live;
            });
            if (h->serve_stop) break;
            // admission: a request slot and room for its rows in the device state arena
            while (!h->pending.empty() && active.size() < h->max_active) {
                Request* r = h->requests[h->pending.front()];
                uint32_t slot = 0;
                if (!h->arena.alloc((uint32_t)(r->last - r->first + 1), &slot)) break;
                h->pending.pop_front();
                r->slot = slot;
                r->admitted = true;
                r->admitted_ns = now_ns();
                r->next_row = r->first;
                active.push_back(r);
            }
            // The wave: the oldest admitted request with rows left takes the
            // pair budget, every younger one a single row.  Large requests
            // then finish in arrival order, as one at a time would, while
            // every newcomer advances in every wave, so short requests end
            // within a few waves instead of waiting behind the large ones.
            std::vector<Request*> order;
            for (Request* r : active)
                if (r->next_row <= r->last) order.push_back(r);
            std::sort(order.begin(), order.end(), [](const Request* x, const Request* y) { return x->id < y->id; });
            const uint64_t budget = (uint64_t)h->wave_items << 20;
            for (size_t i = 0; i < order.size(); ++i) {
                Request* r = order[i];
                const uint64_t share = i == 0 ? budget : 0;
                uint64_t taken = 0;
                while (r->next_row <= r->last && (taken == 0 || taken + (h->limit - r->next_row + 1) <= share)) {
                    taken += h->limit - r->next_row + 1;
                    w.rows.push_back(RowRef{r->next_row, (uint32_t)w.rows.size()});
                    w.owner.push_back(r);
                    ++r->next_row;
                    ++r->inflight;
                }
            }
        }
        const bool launched = !w.rows.empty();
        if (launched) {
            hss_t* lane = h->lanes[next_lane];
            waves[next_lane] = std::move(w);
            waves[next_lane].live = true;
            const int s = launch_wave(h, lane, waves[next_lane]);
            if (s) {
                cudaStreamSynchronize(lane->stream);
                settle_wave(h, waves[next_lane], s, {}, 0, active);
            }
            next_lane ^= 1;
        }
        // Lanes alternate, so waves[next_lane] is the older wave.  After a
        // launch it is harvested (the new wave keeps the device busy
        // meanwhile); with nothing new to launch, the oldest live wave is.
        int i = next_lane;
        if (!waves[i].live && !launched) i ^= 1;
        if (waves[i].live) {
            std::vector<DevHit> hits;
            double ms = 0;
            const int s = finish_wave(h, h->lanes[i], waves[i], &hits, &ms);
            settle_wave(h, waves[i], s, hits, ms, active);
        }
    }
    for (hss_t* lane : h->lanes)
        if (lane) cudaStreamSynchronize(lane->stream);
}

int request_info(hss_t* h, Request* r, hss_request_info* info, hss_hit* hits, uint32_t cap) {
    if (info) {
        info->first = r->first;
        info->last = r->last;
        info->submitted_ns = r->submitted_ns;
        info->admitted_ns = r->admitted_ns;
        info->finished_ns = r->finished_ns;
        info->counts = r->counts;
        info->nhits = (uint32_t)r->hits.size();
        info->status = r->status;
    }
    if (hits && r->status == HSS_OK) copy_hits(r->hits, hits, cap);
    (void)h;
    return r->status == HSS_ERR_BUSY ? HSS_ERR_BUSY : HSS_OK;
}

}  // namespace

extern "C" {

int hss_serve_start(hss_t* h, uint32_t max_active, uint32_t wave_mpairs) {
    if (!h) return HSS_ERR_ARGUMENT;
    std::lock_guard<std::mutex> lock(h->serve_mu);
    if (h->serving) return HSS_OK;
    HSS_CUDA(h, cudaSetDevice(h->device));
    // device state arena: opts.serve_state_kb, else 1/16 of free HBM up to 256 MiB
    size_t free_b = 0, total_b = 0;
    HSS_CUDA(h, cudaMemGetInfo(&free_b, &total_b));
    size_t bytes = h->opts.serve_state_kb ? (size_t)h->opts.serve_state_kb << 10
                                          : std::min<size_t>(free_b / 16, (size_t)256 << 20);
    const uint32_t rows = (uint32_t)std::min<size_t>(bytes / sizeof(RowCounts), UINT32_MAX);
    if (rows == 0) return fail(h, HSS_ERR_ARGUMENT, "serving state arena holds no row");
    if (int s = device_alloc(h, &h->d_state, rows)) return s;
    for (int i = 0; i < 2; ++i) {
        int s = HSS_OK;
        h->lanes[i] = make_lane(h, &s);
        if (s) {
            for (hss_t*& lane : h->lanes) {
                if (lane) hss_close(lane);
                lane = nullptr;
            }
            device_free(h, h->d_state);
            h->d_state = nullptr;
            return fail(h, s, "serving lane set-up failed");
        }
    }
    h->arena.reset(rows);
    h->max_active = max_active ? max_active : 64;
    h->wave_items = wave_mpairs ? wave_mpairs : 256;
    h->serve_stop = false;
    h->serving = true;
    h->serve_thread = std::thread(serve_loop, h);
    return HSS_OK;
}

int hss_submit(hss_t* h, uint64_t first, uint64_t last, uint64_t* request_id) {
    if (!h || !request_id) return HSS_ERR_ARGUMENT;
    if (first < 1 || first > last || last > h->limit) return fail(h, HSS_ERR_ARGUMENT, "need 1 <= first <= last <= limit");
    std::lock_guard<std::mutex> lock(h->serve_mu);
    if (!h->serving) return fail(h, HSS_ERR_ARGUMENT, "serving loop not started");
    if (last - first + 1 > h->arena.size)
        return fail(h, HSS_ERR_MEMORY, "request rows exceed the serving state arena");
    Request* r = new Request();
    r->id = h->next_id++;
    r->first = first;
    r->last = last;
    r->submitted_ns = now_ns();
    h->requests[r->id] = r;
    h->pending.push_back(r->id);
    *request_id = r->id;
    h->serve_cv.notify_all();
    return HSS_OK;
}

int hss_poll(hss_t* h, uint64_t request_id, hss_request_info* info, hss_hit* hits, uint32_t hit_cap) {
    if (!h) return HSS_ERR_ARGUMENT;
    std::lock_guard<std::mutex> lock(h->serve_mu);
    auto it = h->requests.find(request_id);
    if (it == h->requests.end()) return HSS_ERR_NOT_FOUND;
    return request_info(h, it->second, info, hits, hit_cap);
}

int hss_wait(hss_t* h, uint64_t request_id, hss_request_info* info, hss_hit* hits, uint32_t hit_cap) {
    if (!h) return HSS_ERR_ARGUMENT;
    std::unique_lock<std::mutex> lock(h->serve_mu);
    auto it = h->requests.find(request_id);
    if (it == h->requests.end()) return HSS_ERR_NOT_FOUND;
    Request* r = it->second;
    h->serve_cv.wait(lock, [&] { return r->status != HSS_ERR_BUSY || h->serve_stop; });
    return request_info(h, r, info, hits, hit_cap);
}

int hss_serve_stop(hss_t* h) {
    if (!h) return HSS_ERR_ARGUMENT;
    {
        std::lock_guard<std::mutex> lock(h->serve_mu);
        if (!h->serving) return HSS_OK;
        h->serve_stop = true;
        h->serve_cv.notify_all();
    }
    if (h->serve_thread.joinable()) h->serve_thread.join();
    std::lock_guard<std::mutex> lock(h->serve_mu);
    for (auto& kv : h->requests) delete kv.second;
    h->requests.clear();
    h->pending.clear();
    for (hss_t*& lane : h->lanes) {
        if (lane) hss_close(lane);
        lane = nullptr;
    }
    device_free(h, h->d_state);
    h->d_state = nullptr;
    h->serving = false;
    return HSS_OK;
}

}  // extern "C"
