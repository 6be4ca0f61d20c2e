// Opening a handle as device memory gets short: with room for the cache and the
// product path's queues a handle opens, without the sorted layout where that
// (or the queues beside it) does not fit, and searches by products.
#include "fake_runtime.h"

namespace {
constexpr size_t kCacheBytes = 10u << 20, kLayoutBytes = (size_t)12 << 30;
HostCache cache;
bool by_products = false, by_arcs = false;
}  // namespace

extern "C" {
cudaError_t cudaGetDeviceCount(int* n) {
    *n = 1;
    return cudaSuccess;
}
cudaError_t cudaGetDeviceProperties(cudaDeviceProp* p, int) {
    *p = cudaDeviceProp{};
    p->major = 10;
    p->minor = 3;
    p->multiProcessorCount = 152;
    return cudaSuccess;
}
cudaError_t cudaMemcpy(void*, const void*, size_t, cudaMemcpyKind) { return cudaSuccess; }
}

namespace hss {

void build_residue_tables(uint8_t*) {}
void build_arc_tables(uint8_t*) {}
void fill_row_info(const uint32_t*, const uint32_t*, uint64_t, uint64_t l, RowInfo* R) {
    *R = RowInfo{};
    R->l = l;
}
int batched_max_ctas_per_sm(int, int, size_t) { return 1; }
size_t batched_smem_bytes(int, uint32_t) { return 0; }
int arc_max_ctas_per_sm(int) { return 1; }
cudaError_t launch_batched(const DeviceCache&, const WorkItem*, uint32_t, const BatchedConfig&, const LaunchBuffers& b, cudaStream_t) {
    by_products = true;
    CHECK(fake::holds(b.merged_queue, b.merged_cap) && b.merged_cap == kMergedCap, "%u entries", b.merged_cap);
    return cudaSuccess;
}
cudaError_t launch_merged(const DeviceCache&, uint64_t, const LaunchBuffers&, int, cudaStream_t, uint32_t* n) {
    *n = 0;
    return cudaSuccess;
}
cudaError_t launch_exact(const DeviceCache&, const LaunchBuffers&, int, cudaStream_t) { return cudaSuccess; }
cudaError_t launch_arc_values(const ArcCache&, uint32_t, const ArcBuffers&, cudaStream_t) {
    by_arcs = true;
    return cudaSuccess;
}
cudaError_t launch_arc(const ArcCache&, const ArcItem*, uint32_t, const ArcConfig&, const ArcBuffers&, cudaStream_t) { return cudaSuccess; }
cudaError_t launch_arc_exact(const ArcCache&, const ArcBuffers&, int, cudaStream_t) { return cudaSuccess; }

int build_device_cache(uint64_t, int, CUstream_st*, DeviceBuild* out, std::string*, const std::function<int()>& on_records) {
    void* p = nullptr;
    if (cudaMalloc(&p, kCacheBytes) != cudaSuccess) {
        cudaGetLastError();
        return HSS_ERR_CUDA;
    }
    out->owned.push_back(p);
    out->records = cache.records;
    out->max_exponent = cache.max_exponent;
    out->spf_host = cache.spf;
    out->seg_off_host = cache.seg_off;
    if (on_records)
        if (int s = on_records()) {
            cudaFree(p);
            out->owned.clear();
            return s;
        }
    return HSS_OK;
}
int plan_arc_blocks(const uint32_t*, uint64_t limit, cudaStream_t, ArcPlan* plan, std::string*) {
    for (auto& s : plan->start) s.assign(limit + 1, 0);
    return HSS_OK;
}
int build_arc_layout(const DeviceCache&, uint64_t, const ArcPlan&, cudaStream_t, ArcBuild* out, std::string*) {
    void* p = nullptr;
    if (cudaMalloc(&p, kLayoutBytes) != cudaSuccess) {
        cudaGetLastError();
        return HSS_ERR_MEMORY;
    }
    out->blocks = static_cast<ArcBlock*>(p);
    out->owned.push_back(p);
    return HSS_OK;
}

}  // namespace hss

int main() {
    std::string err;
    const uint64_t limit = 20000;
    CHECK(build_host_cache(limit, 8, &cache, &err) == HSS_OK, "host cache");
    // what the product path asks for at open, and an allowance for its call
    const size_t queues = (size_t)kMergedCap * 16 + (size_t)kDescChunk * 192 + ((size_t)1 << 20) * 192 + ((size_t)1 << 24) * 32;
    const size_t least = kCacheBytes + queues + (8u << 20);
    for (size_t room : {least, least + kLayoutBytes / 2, kCacheBytes + kLayoutBytes + (1u << 20), kCacheBytes + kLayoutBytes + queues}) {
        fake::room = room;
        hss_t* h = nullptr;
        const int s = hss_open(limit, 0, nullptr, &h);
        CHECK(s == HSS_OK, "room for %zu MB: status %d", room >> 20, s);
        by_products = by_arcs = false;
        std::vector<RowRef> rows;
        for (uint32_t l = 1000; l < 1100; ++l) rows.push_back(RowRef{l, l - 1000});
        CHECK(begin_call(h, rows.size()) == HSS_OK && run_batched(h, rows) == HSS_OK, "room for %zu MB: %s", room >> 20, h->err.c_str());
        const bool layout = room >= kCacheBytes + kLayoutBytes + queues;
        CHECK(by_arcs == layout && by_products == !layout, "room for %zu MB: wrong path", room >> 20);
        hss_close(h);
        CHECK(fake::used == 0, "%zu bytes left", fake::used);
    }
    fake::room = kCacheBytes / 2;
    hss_t* h = nullptr;
    CHECK(hss_open(limit, 0, nullptr, &h) != HSS_OK && !h && fake::used == 0, "no room for the cache");
    std::printf("ok\n");
    return 0;
}
