// Searches that outgrow the small queues a handle starts with, with and
// without memory for larger ones: the queues a call gets are no larger than
// stated, and where there is no room the call runs in smaller launches.
#include "fake_runtime.h"

namespace {

struct Launch {
    uint64_t pairs;
    uint32_t rows;
};
std::vector<Launch> merged, plain;

void check_queues(const hss::LaunchBuffers& b) {
    CHECK(fake::holds(b.merged_queue, b.merged_cap) && b.merged_cap, "shared-prime queue");
    CHECK(fake::holds(b.pair_desc, b.desc_chunk, kBigEntryWords) && b.desc_chunk, "descriptors");
    CHECK(fake::holds(b.exact_queue, b.exact_cap) && b.exact_cap, "exact queue");
}

}  // namespace

namespace hss {

// Stand-ins for the launches, and for the row constants the planner reads.
int arc_max_ctas_per_sm(int) { return 1; }
cudaError_t launch_arc_values(const ArcCache&, uint32_t, const ArcBuffers&, cudaStream_t) { return cudaSuccess; }
cudaError_t launch_arc(const ArcCache&, const ArcItem*, uint32_t, const ArcConfig&, const ArcBuffers&, cudaStream_t) { return cudaSuccess; }
cudaError_t launch_arc_rest(const DeviceCache&, const ArcRest*, uint32_t, const LaunchBuffers&, int, cudaStream_t) { return cudaSuccess; }
cudaError_t launch_arc_exact(const ArcCache&, const ArcBuffers&, int, cudaStream_t) { return cudaSuccess; }
cudaError_t launch_exact(const DeviceCache&, const LaunchBuffers&, int, cudaStream_t) { return cudaSuccess; }
cudaError_t launch_plain(const DeviceCache&, uint64_t, uint32_t rows, uint32_t, const LaunchBuffers&, cudaStream_t) {
    plain.push_back({0, rows});
    return cudaSuccess;
}
cudaError_t launch_merged(const DeviceCache&, uint64_t pairs, const LaunchBuffers& b, int, cudaStream_t, uint32_t* n) {
    check_queues(b);
    CHECK(pairs <= b.merged_cap, "%llu pairs, room for %u", (unsigned long long)pairs, b.merged_cap);
    merged.push_back({pairs, 0});
    *n = 1;
    return cudaSuccess;
}
void fill_row_info(const uint32_t* spf, const uint32_t* seg_off, uint64_t n, uint64_t l, RowInfo* R) {
    *R = RowInfo{};
    R->l = l;
    R->l2 = l * l;
    R->l4 = (unsigned __int128)R->l2 * R->l2;
    R->n4 = (unsigned __int128)(n * n) * (n * n);
    R->l3 = l % 3 == 0;
    R->l5 = l % 5 == 0;
    R->free_l = seg_off[l + 1] - seg_off[l] - 1;
    const NumberFactors f = factor_number(spf, l);
    R->nsplit = f.count;
    for (uint32_t i = 0; i < f.count; ++i) {
        R->sp[i] = f.primes[i];
        R->se[i] = f.exps[i];
    }
}

}  // namespace hss

namespace {

HostCache cache;

hss_t* open_handle(uint64_t limit) {
    hss_t* h = new hss_t();
    h->limit = limit;
    h->sm_count = 152;
    h->spf = cache.spf;
    h->seg_off = cache.seg_off;
    h->dev.max_exponent = cache.max_exponent;
    auto plan = std::make_shared<ArcPlan>();  // no blocks: rows and rest lists alone
    for (auto& s : plan->start) s.assign(limit + 1, 0);
    h->plan = plan;
    CHECK(alloc_launch_buffers(h) == HSS_OK, "launch buffers");
    return h;
}

uint64_t total(const std::vector<Launch>& v) {
    uint64_t t = 0;
    for (const Launch& x : v) t += x.pairs;
    return t;
}

}  // namespace

int main() {
    const uint64_t limit = 100000;
    std::string err;
    CHECK(build_host_cache(limit, 8, &cache, &err) == HSS_OK, "host cache");
    std::vector<RowRef> rows;
    for (uint64_t l = 1; l <= 40000; ++l) rows.push_back(RowRef{l, (uint32_t)(l - 1)});

    // room for everything: the queues grow once, to what is stated beside them
    hss_t* h = open_handle(limit);
    const size_t small = fake::used;
    CHECK(begin_call(h, rows.size()) == HSS_OK && run_batched(h, rows) == HSS_OK, "batched: %s", h->err.c_str());
    const uint64_t pairs = total(merged);
    CHECK(pairs > kArcMergedStart, "the case is too small: %llu pairs", (unsigned long long)pairs);
    CHECK(h->merged_cap == kArcMergedCap && h->desc_chunk == kArcDescChunk, "%u entries, chunks of %u", h->merged_cap, h->desc_chunk);
    CHECK(begin_call(h, rows.size()) == HSS_OK && run_plain(h, 1, 40000) == HSS_OK, "plain: %s", h->err.c_str());
    const size_t plain_launches = plain.size();
    CHECK(plain_launches == (40000 + kPlainBatch - 1) / kPlainBatch, "%zu plain launches", plain_launches);
    hss_close(h);

    // no room for larger queues (the call's rows and values still fit)
    merged.clear();
    plain.clear();
    h = open_handle(limit);
    CHECK(fake::used == small, "same start");
    fake::room = small + (300u << 20);
    int s = begin_call(h, rows.size());
    if (!s) s = run_batched(h, rows);
    CHECK(s == HSS_OK, "batched without room: %d %s", s, h->err.c_str());
    CHECK(total(merged) == pairs, "%llu pairs of %llu", (unsigned long long)total(merged), (unsigned long long)pairs);
    CHECK(merged.size() > 2, "%zu launches", merged.size());
    merged.clear();
    // long calls of the plain form, whose batches hold more pairs than fit
    const uint64_t bound = [&] {
        uint64_t most = 0;
        for (uint64_t b = 1; b <= 40000; b += kPlainBatch) {
            uint64_t t = 0;
            for (uint64_t l = b; l < std::min<uint64_t>(b + kPlainBatch, 40001); ++l) t += merged_bound(h, l);
            most = std::max(most, t);
        }
        return most;
    }();
    CHECK(bound > kArcMergedStart, "the case is too small: %llu pairs", (unsigned long long)bound);
    fake::room = fake::used + (8u << 20);
    s = begin_call(h, rows.size());
    if (!s) s = run_plain(h, 1, 40000);
    CHECK(s == HSS_OK, "plain without room: %d %s", s, h->err.c_str());
    uint64_t n = 0;
    for (const Launch& x : plain) n += x.rows;
    CHECK(n == 40000 && plain.size() > plain_launches, "%llu rows in %zu launches", (unsigned long long)n, plain.size());
    hss_close(h);
    std::printf("ok\n");
    return 0;
}
