// hss_blocks.h - the arc layout of the factor cache (hss_blocks.cu).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include <string>
#include <vector>

#include "hss_internal.h"

namespace hss {

// Blocks of every type, type by type in increasing m (host side: n, base,
// roots and ranks; the list bounds are filled on the device).
struct ArcPlan {
    std::vector<ArcBlock> blocks;
    uint32_t type_first[kTypes + 1] = {};  // blocks of type t: [type_first[t], type_first[t + 1])
    std::vector<uint32_t> start[kTypes];   // the first block of the type that reaches m >> start_shift
    uint32_t start_shift = 0;
    uint32_t cap = 0;                      // entries of the largest block
    uint64_t entries = 0;                  // of the sorted arrays, padding included
};

// Cuts the roots 1..limit of every type into blocks of at most kBlockEntries
// records (on the device, from its segment offsets; waits for the stream).
// This and build_arc_layout return HSS_ERR_MEMORY where the device has no room.
int plan_arc_blocks(const uint32_t* d_seg_off, uint64_t limit, cudaStream_t stream, ArcPlan* plan, std::string* err);

// Device arrays of the arc layout; `owned` lists the allocations.
struct ArcBuild {
    ArcBlock* blocks = nullptr;
    uint32_t* w[kFields] = {};
    uint32_t* ang = nullptr;
    uint8_t* part = nullptr;
    uint32_t* src = nullptr;
    uint32_t* m = nullptr;
    float2* xy = nullptr;
    uint32_t* index = nullptr;
    uint32_t* mask = nullptr;
    uint16_t* pos = nullptr;
    std::vector<void*> owned;
};

// Sorts the records of every block on the device (enqueued on `stream`).
int build_arc_layout(const DeviceCache& cache, uint64_t records, const ArcPlan& plan, cudaStream_t stream,
                     ArcBuild* out, std::string* err);

}  // namespace hss
