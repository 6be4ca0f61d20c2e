// The host side of the library (csrc/hss_api.cpp) over a CUDA runtime that only
// keeps books: allocations are recorded and can be made to fail, copies and
// launches do nothing.  For checks of what the host does when memory is short;
// nothing here runs on a GPU.  Built with unresolved symbols allowed: a call
// that has no stand-in here must not be reached.
#pragma once
#include "../../heronian-square-search_gb300/csrc/hss_api.cpp"

#include <cstdio>
#include <cstdlib>
#include <map>

namespace fake {

std::map<const void*, size_t> live;  // device and pinned allocations with their sizes
size_t used = 0;                     // of the device
size_t room = ~size_t(0);            // bytes the device has
int fail_from = -1, fail_count = 0;  // the allocations to refuse, counted from now on (-1: none)
int calls = 0;                       // allocations asked for since reset()
cudaError_t last = cudaSuccess;      // as cudaGetLastError keeps it

void reset() {
    fail_from = -1;
    fail_count = 0;
    calls = 0;
}

cudaError_t take(void** p, size_t bytes, bool device) {
    const int i = calls++;
    const bool refused = fail_from >= 0 && i >= fail_from && i < fail_from + fail_count;
    if (refused || (device && used + bytes > room)) {
        *p = nullptr;
        return last = cudaErrorMemoryAllocation;
    }
    *p = std::malloc(device ? 1 : bytes);  // device memory is never touched
    live[*p] = bytes;
    if (device) used += bytes;
    return cudaSuccess;
}

bool give(void* p, bool device) {
    auto it = live.find(p);
    if (it == live.end()) return p == nullptr;
    if (device) used -= it->second;
    live.erase(it);
    std::free(p);
    return true;
}

// An array of `cap` elements is really there.
template <class T>
bool holds(const T* p, size_t cap, size_t per = 1) {
    if (cap == 0) return true;
    auto it = live.find(p);
    return it != live.end() && it->second >= cap * per * sizeof(T);
}

}  // namespace fake

extern "C" {
cudaError_t cudaMalloc(void** p, size_t n) { return fake::take(p, n, true); }
cudaError_t cudaMallocHost(void** p, size_t n) { return fake::take(p, n, false); }
cudaError_t cudaHostAlloc(void** p, size_t n, unsigned int) { return fake::take(p, n, false); }
cudaError_t cudaFree(void* p) { return fake::give(p, true) ? cudaSuccess : cudaErrorInvalidValue; }
cudaError_t cudaFreeHost(void* p) { return fake::give(p, false) ? cudaSuccess : cudaErrorInvalidValue; }
const char* cudaGetErrorString(cudaError_t e) { return e == cudaSuccess ? "no error" : "an error"; }
cudaError_t cudaGetLastError(void) {
    const cudaError_t e = fake::last;
    fake::last = cudaSuccess;
    return e;
}
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned int) {
    *s = nullptr;
    return cudaSuccess;
}
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventCreate(cudaEvent_t* e) {
    *e = nullptr;
    return cudaSuccess;
}
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned int) {
    *e = nullptr;
    return cudaSuccess;
}
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventRecordWithFlags(cudaEvent_t, cudaStream_t, unsigned int) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaMemsetAsync(void*, int, size_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaMemcpyAsync(void*, const void*, size_t, cudaMemcpyKind, cudaStream_t) { return cudaSuccess; }
}

#define CHECK(cond, ...)                                            \
    do {                                                            \
        if (!(cond)) {                                              \
            std::printf("%s:%d: %s: ", __FILE__, __LINE__, #cond);  \
            std::printf(__VA_ARGS__);                               \
            std::printf("\n");                                      \
            std::exit(1);                                           \
        }                                                           \
    } while (0)
