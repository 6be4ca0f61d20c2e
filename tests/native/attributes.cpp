// Two threads that launch the same kernel with different amounts of dynamic
// shared memory: between one's setting of the kernel's limit and its launch
// (here: inside the first's call of cudaFuncSetAttribute) the other sets its
// own and launches.  Links the library's objects with a runtime that keeps the
// limits and checks launches against them; nothing runs.
#include <cuda_runtime.h>

#include <cstdio>
#include <cstdlib>
#include <functional>
#include <map>
#include <string>

#include "../../heronian-square-search_gb300/csrc/hss_blocks.h"
#include "../../heronian-square-search_gb300/csrc/hss_kernels.h"

#define CHECK(cond, ...)                                            \
    do {                                                            \
        if (!(cond)) {                                              \
            std::printf("%s:%d: %s: ", __FILE__, __LINE__, #cond);  \
            std::printf(__VA_ARGS__);                               \
            std::printf("\n");                                      \
            std::exit(1);                                           \
        }                                                           \
    } while (0)

namespace {

constexpr int kOptIn = 227 * 1024, kStatic = 20 * 1024;
std::map<const void*, int> limits;
std::function<void()> other;  // the other thread, run once inside cudaFuncSetAttribute
cudaError_t last = cudaSuccess;
int launches = 0;
struct {
    dim3 grid, block;
    size_t smem;
    cudaStream_t stream;
} pushed;

cudaError_t launch(const void* fn, size_t smem) {
    ++launches;
    const auto it = limits.find(fn);
    const size_t most = it == limits.end() ? 48 * 1024 - kStatic : (size_t)it->second;
    return smem <= most ? cudaSuccess : (last = cudaErrorInvalidValue);
}

}  // namespace

extern "C" {
cudaError_t cudaFuncSetAttribute(const void* fn, cudaFuncAttribute, int value) {
    if (value > kOptIn - kStatic) return last = cudaErrorInvalidValue;
    limits[fn] = value;
    if (other) {
        auto run = other;
        other = nullptr;
        run();
    }
    return cudaSuccess;
}
cudaError_t cudaFuncGetAttributes(cudaFuncAttributes* a, const void*) {
    *a = cudaFuncAttributes{};
    a->sharedSizeBytes = kStatic;
    return cudaSuccess;
}
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessor(int* n, const void* fn, int, size_t smem) {
    *n = 1;
    return limits.count(fn) && smem <= (size_t)limits[fn] ? cudaSuccess : cudaErrorInvalidValue;
}
cudaError_t cudaLaunchKernel(const void* fn, dim3, dim3, void**, size_t smem, cudaStream_t) { return launch(fn, smem); }
cudaError_t cudaGetLastError(void) {
    const cudaError_t e = last;
    last = cudaSuccess;
    return e;
}
const char* cudaGetErrorString(cudaError_t) { return "an error"; }
cudaError_t cudaMalloc(void** p, size_t) {
    *p = std::malloc(1);
    return cudaSuccess;
}
cudaError_t cudaFree(void* p) {
    std::free(p);
    return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void*, const void*, size_t, cudaMemcpyKind, cudaStream_t) { return cudaSuccess; }
// what the compiler's launch syntax calls
unsigned __cudaPushCallConfiguration(dim3 grid, dim3 block, size_t smem, cudaStream_t stream) {
    pushed = {grid, block, smem, stream};
    return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3* grid, dim3* block, size_t* smem, void* stream) {
    *grid = pushed.grid;
    *block = pushed.block;
    *smem = pushed.smem;
    *(cudaStream_t*)stream = pushed.stream;
    return cudaSuccess;
}
cudaError_t __cudaGetKernel(cudaKernel_t* k, const void* fn) {
    *k = (cudaKernel_t)fn;
    return cudaSuccess;
}
cudaError_t __cudaLaunchKernel(cudaKernel_t k, dim3, dim3, void**, size_t smem, cudaStream_t) { return launch(k, smem); }
void** __cudaRegisterFatBinary(void*) {
    static void* handle;
    return &handle;
}
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
void __cudaRegisterFunction(void**, const char*, char*, const char*, int, uint3*, uint3*, dim3*, dim3*, int*) {}
void __cudaRegisterVar(void**, char*, char*, const char*, int, size_t, int, int) {}
}

using namespace hss;

int main() {
    auto layout = [](uint32_t entries) {
        ArcPlan plan;
        plan.blocks.push_back(ArcBlock{});
        plan.blocks[0].n = plan.cap = entries;
        plan.entries = (entries + 15) & ~15u;
        ArcBuild build;
        std::string err;
        const int s = build_arc_layout(DeviceCache{}, entries, plan, nullptr, &build, &err);
        for (void* p : build.owned) cudaFree(p);
        return s;
    };
    auto plain = [](uint32_t alpha) { return launch_plain(DeviceCache{}, 1, 1, alpha, LaunchBuffers{}, nullptr); };
    auto batched = [](uint32_t alpha) {
        BatchedConfig c;
        c.threads = 256;
        c.min_blocks = 2;
        c.alpha_cap = alpha;
        c.ctas = batched_max_ctas_per_sm(c.threads, c.min_blocks, batched_smem_bytes(c.threads, alpha));
        return launch_batched(DeviceCache{}, nullptr, 1, c, LaunchBuffers{}, nullptr);
    };
    other = [&] { CHECK(layout(128) == 0, "a small layout"); };
    CHECK(layout(kBlockEntries) == 0, "a large layout while a small one is built");
    other = [&] { CHECK(plain(2) == cudaSuccess, "plain, light rows"); };
    CHECK(plain(2000) == cudaSuccess, "plain, heavy rows beside light ones");
    other = [&] { CHECK(batched(2) == cudaSuccess, "products, light rows"); };
    CHECK(batched(2000) == cudaSuccess, "products, heavy rows beside light ones");
    CHECK(launches == 6, "%d launches", launches);
    std::printf("ok\n");
    return 0;
}
