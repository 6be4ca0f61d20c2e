// The autotuner's settings and choice, with device times given here.
#include "fake_runtime.h"

#include <set>
#include <tuple>

namespace {
hss_t* g_handle = nullptr;
float g_automatic = 10.f, g_fixed = 10.f;  // ms of a call with and without the planner's own item weight
}

extern "C" {
cudaError_t cudaEventElapsedTime(float* ms, cudaEvent_t, cudaEvent_t) {
    *ms = (g_handle->opts.item_target ? g_fixed : g_automatic) + (g_handle->opts.block_threads == 512 ? 1.f : 0.f);
    return cudaSuccess;
}
cudaError_t cudaMemcpy(void*, const void*, size_t, cudaMemcpyKind) { return cudaSuccess; }
}

namespace hss {

void fill_row_info(const uint32_t*, const uint32_t*, uint64_t n, uint64_t l, RowInfo* R) {
    *R = RowInfo{};
    R->l = l;
    R->l2 = l * l;
    R->l4 = (unsigned __int128)R->l2 * R->l2;
    R->n4 = (unsigned __int128)(n * n) * (n * n);
}
int batched_max_ctas_per_sm(int, int, size_t) { return 1; }
size_t batched_smem_bytes(int, uint32_t) { return 0; }
int arc_max_ctas_per_sm(int) { return 1; }
cudaError_t launch_batched(const DeviceCache&, const WorkItem*, uint32_t, const BatchedConfig&, const LaunchBuffers&, cudaStream_t) { return cudaSuccess; }
cudaError_t launch_merged(const DeviceCache&, uint64_t, const LaunchBuffers&, int, cudaStream_t, uint32_t* n) {
    *n = 0;
    return cudaSuccess;
}
cudaError_t launch_exact(const DeviceCache&, const LaunchBuffers&, int, cudaStream_t) { return cudaSuccess; }
cudaError_t launch_arc_values(const ArcCache&, uint32_t, const ArcBuffers&, cudaStream_t) { return cudaSuccess; }
cudaError_t launch_arc(const ArcCache&, const ArcItem*, uint32_t, const ArcConfig&, const ArcBuffers&, cudaStream_t) { return cudaSuccess; }
cudaError_t launch_arc_rest(const DeviceCache&, const ArcRest*, uint32_t, const LaunchBuffers&, int, cudaStream_t) { return cudaSuccess; }
cudaError_t launch_arc_exact(const ArcCache&, const ArcBuffers&, int, cudaStream_t) { return cudaSuccess; }

}  // namespace hss

int main() {
    HostCache cache;
    std::string err;
    const uint64_t limit = 20000;
    CHECK(build_host_cache(limit, 8, &cache, &err) == HSS_OK, "host cache");
    for (bool arcs : {true, false}) {
        hss_t* h = new hss_t();
        g_handle = h;
        h->limit = limit;
        h->sm_count = 152;
        h->spf = cache.spf;
        h->seg_off = cache.seg_off;
        if (arcs) {
            auto plan = std::make_shared<ArcPlan>();
            for (auto& s : plan->start) s.assign(limit + 1, 0);
            h->plan = plan;
        }
        CHECK(alloc_launch_buffers(h) == HSS_OK, "launch buffers");
        h->opts.use_graph = 0;
        hss_tune_trial trials[64];
        uint32_t n = 0;
        hss_opts best{};
        // weights within the noise of the planner's own
        g_automatic = 10.f;
        g_fixed = 9.9f;
        CHECK(hss_autotune(h, 1000, 1099, &best, trials, 64, &n) == HSS_OK, "%s", h->err.c_str());
        std::set<std::tuple<uint32_t, uint32_t, uint32_t>> kinds;
        bool automatic = false;
        for (uint32_t i = 0; i < n; ++i) {
            // by arcs only 512 threads or not, and the weight, make a difference
            if (arcs) kinds.insert({trials[i].block_threads == 512, 0, trials[i].item_target});
            else kinds.insert({trials[i].block_threads, trials[i].ctas_per_sm, trials[i].item_target});
            automatic |= trials[i].item_target == 0;
        }
        CHECK(kinds.size() == n, "%u trials of %zu settings (arcs %d)", n, kinds.size(), arcs);
        CHECK(best.block_threads == 128 || best.block_threads == 256 || best.block_threads == 512, "%u", best.block_threads);
        if (arcs) {
            CHECK(automatic && best.item_target == 0 && best.block_threads != 512, "noise chose weight %u", best.item_target);
            CHECK(h->opts.item_target == 0, "the handle's options");
            // a weight that is worth it
            g_fixed = 9.f;
            CHECK(hss_autotune(h, 1000, 1099, &best, nullptr, 0, nullptr) == HSS_OK && best.item_target != 0, "a faster weight");
        }
        // the handle's own setting is among them: tuning makes nothing slower
        h->opts.item_target = 12345678;
        h->opts.block_threads = 256;
        h->opts.ctas_per_sm = 2;
        CHECK(hss_autotune(h, 1000, 1099, &best, trials, 64, &n) == HSS_OK, "%s", h->err.c_str());
        bool own = false;
        for (uint32_t i = 0; i < n; ++i) own |= trials[i].item_target == 12345678 && trials[i].block_threads == 256;
        CHECK(own, "the handle's own setting was not tried");
        hss_close(h);
    }
    std::printf("ok\n");
    return 0;
}
