// hss_blocks.cu - the arc layout: the factor cache's records again, block by
// block, sorted so that the terms a row counts are contiguous runs.
//
// A term of a row (l, P) - see hss_arc.cuh - is a pair of Gaussian values
// gamma (row side) and beta (root side) whose product's argument lies in an
// arc, and whose area 4A = Im(gamma beta) passes the divisibility test.  That
// test depends only on classes of the two values:
//   * 3 does not divide the root: beta has norm = 1 mod 3, so beta = +-1 (b3 =
//     0) or +-i (b3 = 1) mod 3, and 3 | Im(gamma beta) exactly when the two
//     bits agree;
//   * 5 does not divide the root: likewise mod 5 (b5);
//   * odd roots: Re beta is odd and 4 | Im beta, and Re beta = +-1 mod 8; s8 =
//     (Re beta = -1 mod 8) decides z mod 16.
// So the records of the roots of one type (divisibility by 2, 4, 3, 5) are
// grouped into up to eight lists by (s8, b3, b5), each sorted by the argument
// of the representative with positive imaginary part, and a ninth list holds
// the central values (x^2, 0) in root order.
//
// Arguments are stored as 2^32 / (2 pi) units with the low three bits clear
// (the sort key is list << 28 | argument >> 3); atan2f is within 3 units in
// the last place, so a stored argument is within kAngleSlack (hss_arc.cuh).
#include <math.h>

#include <algorithm>
#include <type_traits>

#include "hss_api_status.h"
#include "hss_blocks.h"

namespace hss {
namespace {

constexpr uint32_t kBlockThreads = 512;
constexpr uint32_t kBlockLeast = 128;
constexpr float kBlockScale = 3.f;

constexpr TypeTables kTypeTables = make_type_tables();
__constant__ TypeTables c_types = make_type_tables();

__device__ __forceinline__ uint32_t residue_i64(int64_t v, uint32_t m) {
    const int64_t r = v % (int64_t)m;
    return (uint32_t)(r < 0 ? r + m : r);
}

// Cuts the roots of every type into blocks: a warp per kCutRoots consecutive
// roots of one type, 32 at a time, a block closed before the root that would
// take it over its size (the warp's boundary closes one too).  The size: a row
// pays for every run it starts in a block (less the larger the block) and for
// every term between the tightest and the widest window of the block's roots (as
// the square of the size over the root and the type's share of all roots), so the
// best size grows as the square root of root times share (a factor of 3: 16,384
// rows at LIMIT 10^5 132 ms, root 6,325,815 at 10^7 23.2; of 2: 147 and 22.5, of 4.5:
// 129 and 23.7).  Without `blocks` the warp's count is left in at[task], with
// them they are written from there on.  0.2 ms each time at N = 10^7, where host
// threads took 14 ms.
constexpr uint32_t kCutRoots = 8192;
constexpr uint32_t kCutWarps = 4;
struct CutTasks {
    uint32_t roots[kTypes];      // of the type, up to the limit
    uint32_t first[kTypes + 1];  // first task of the type
};

__global__ void __launch_bounds__(kCutWarps * 32) block_cut_kernel(const uint32_t* __restrict__ seg_off, CutTasks tasks,
                                                                  uint32_t* at, ArcBlock* blocks) {
    const uint32_t lane = threadIdx.x & 31, task = blockIdx.x * kCutWarps + threadIdx.x / 32;
    if (task >= tasks.first[kTypes]) return;
    uint32_t type = 0;
    while (task >= tasks.first[type + 1]) ++type;
    const uint32_t rank = (task - tasks.first[type]) * kCutRoots;
    const uint32_t end = min(tasks.roots[type], rank + kCutRoots);
    uint32_t out = blocks ? at[task] : 0u, target = 0;
    ArcBlock b{};
    auto close = [&] {
        if (!b.n_m) return;
        if (blocks && lane == 0) blocks[out] = b;
        ++out;
        b = ArcBlock{};
    };
    for (uint32_t r0 = rank; r0 < end; r0 += 32) {
        const uint32_t have = min(32u, end - r0);
        const uint32_t m = nth_root(c_types, type, r0 + min(lane, have - 1));
        const uint32_t len = lane < have ? seg_off[m + 1] - seg_off[m] : 0u;
        uint32_t upto = len;
#pragma unroll
        for (uint32_t d = 1; d < 32; d <<= 1) {
            const uint32_t t = __shfl_up_sync(0xFFFFFFFFu, upto, d);
            if (lane >= d) upto += t;
        }
        const uint32_t plain = __ballot_sync(0xFFFFFFFFu, len == 1);
        uint32_t from = 0, used = 0;  // roots of these 32 taken so far, and their records
        while (from < have) {
            if (!b.n_m) {
                b.m_lo = __shfl_sync(0xFFFFFFFFu, m, from);
                b.rank0 = r0 + from;
                b.type = type;
                target = min(kBlockEntries, max(kBlockLeast, (uint32_t)(kBlockScale * sqrtf((float)(c_types.count[type] * b.m_lo)))));
            }
            const bool over = lane < have && lane >= from + (b.n_m == 0) && b.n + (upto - used) > target;
            const uint32_t stop = __ballot_sync(0xFFFFFFFFu, over);
            const uint32_t to = stop ? __ffs(stop) - 1 : have;
            if (to > from) {
                const uint32_t sum = __shfl_sync(0xFFFFFFFFu, upto, to - 1);
                b.m_hi = __shfl_sync(0xFFFFFFFFu, m, to - 1);
                b.n += sum - used;
                b.n_m += to - from;
                b.n_plain += __popc(plain >> from & (0xFFFFFFFFu >> (32 - (to - from))));
                used = sum;
                from = to;
            }
            if (stop) close();
        }
    }
    close();
    if (!blocks && lane == 0) at[task] = out;
}

// One CTA per block, three passes over its records (one key of 32 bits each):
//   1. keys, 32 roots per warp, a lane per record (the records of a root lie
//      together, its neighbours of the same type do not), counted into
//      kFine buckets of equal angle per list;
//   2. the keys' places by bucket;
//   3. a thread per key: its place inside its bucket by counting the smaller
//      keys there (angles spread evenly: a bucket of a full block holds less
//      than one key on average, and equal ones are ordered by record), then the
//      sorted arrays' entry.  Central values need no sort: their place is the
//      root's rank.
// 36 bytes read and 35 written per value, 1.2 TB/s: what bounds it is its barriers
// and chains of shared-memory accesses (26 % of the DRAM rate, 35 % of the issue
// slots, at N = 10^6), two CTAs per SM.  A
// bitonic sort of (key, record) pairs in shared memory, with a thread per root
// for the keys, took 11.5 ms at N = 10^7; this form takes 5.5 ms.
constexpr uint32_t kFine = 1024;
constexpr uint32_t kFineShift = 28 - 10;
constexpr uint32_t kHist = 8 * kFine;
static_assert(kFine % kBuckets == 0 && kBucketShift - 3 >= kFineShift, "the index is read off the histogram");

// A counter's place: one word of padding per 16, so that a thread's 16 counters
// in the scan lie 17 words from its neighbour's.
__device__ __forceinline__ uint32_t hist_at(uint32_t b) { return b + (b >> 4); }
constexpr uint32_t kHistWords = kHist + kHist / 16;

inline size_t block_sort_smem(uint32_t cap) { return kHistWords * 4 + (size_t)cap * 10 + 16; }

__global__ void __launch_bounds__(kBlockThreads) block_sort_kernel(
    ArcBlock* blocks, uint32_t cap, const uint32_t* __restrict__ seg_off, const HotRec* __restrict__ hot,
    const ExactRec* __restrict__ exact, const uint32_t* __restrict__ owner, uint32_t* w0, uint32_t* w1, uint32_t* w2,
    uint32_t* ang, uint8_t* part, uint32_t* src, uint32_t* root, float2* xy, uint32_t* index, uint32_t* mask, uint16_t* pos) {
    extern __shared__ __align__(16) unsigned char smem[];
    uint32_t* s_hist = reinterpret_cast<uint32_t*>(smem);
    uint32_t* s_key = s_hist + kHistWords;
    uint32_t* s_rec = s_key + cap;
    uint16_t* s_order = reinterpret_cast<uint16_t*>(s_rec + cap);
    __shared__ uint32_t s_fill;
    __shared__ uint32_t s_warp[kBlockThreads / 32];
    const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid / 32;
    const ArcBlock B = blocks[blockIdx.x];
    const uint32_t sorted = B.n - B.n_m;  // one central value per root
    if (tid == 0) s_fill = 0;
    for (uint32_t i = tid; i < kHistWords; i += kBlockThreads) s_hist[i] = 0;
    __syncthreads();
    for (uint32_t r0 = warp * 32; r0 < B.n_m; r0 += kBlockThreads) {
        const uint32_t r = r0 + lane;
        uint32_t m = 0, s0 = 0, len = 0;
        if (r < B.n_m) {
            m = nth_root(c_types, B.type, B.rank0 + r);
            s0 = seg_off[m];
            len = seg_off[m + 1] - s0;
        }
        uint32_t first = len;
#pragma unroll
        for (uint32_t d = 1; d < 32; d <<= 1) {
            const uint32_t t = __shfl_up_sync(0xFFFFFFFFu, first, d);
            if (lane >= d) first += t;
        }
        const uint32_t total = __shfl_sync(0xFFFFFFFFu, first, 31);
        first -= len;
        uint32_t at = lane == 0 ? atomicAdd(&s_fill, total) : 0u;
        at = __shfl_sync(0xFFFFFFFFu, at, 0);
        for (uint32_t q0 = 0; q0 < total; q0 += 32) {
            const uint32_t q = q0 + lane;
            uint32_t o = 0;  // the last of the warp's roots whose records start at or before q
#pragma unroll
            for (uint32_t step = 16; step; step >>= 1) {
                const uint32_t f = __shfl_sync(0xFFFFFFFFu, first, o + step);
                if (f <= q) o += step;
            }
            const uint32_t x = __shfl_sync(0xFFFFFFFFu, m, o);
            const uint32_t j = __shfl_sync(0xFFFFFFFFu, s0, o) + (q - __shfl_sync(0xFFFFFFFFu, first, o));
            if (q >= total || at + q >= B.n) continue;
            const HotRec h = hot[j];
            uint32_t k;
            if (h.rre & kCentralBit) {
                k = 8u << 28 | (r0 + o);
            } else {
                const uint32_t ra = h.rre & kMaskA, ia = h.rim & kMaskA;
                const uint32_t b3 = x % 3u != 0 && ia % 3u != 0;
                const uint32_t b5 = x % 5u != 0 && ia % 5u != 0;
                const uint32_t s8 = (x & 1u) && (ra & 7u) == 7u;
                const float th = atan2f(fabsf(h.im), h.re);
                uint32_t a = __float2uint_rn(th * 6.8356528e8f);  // 2^32 / (2 pi)
                if (a > 0x7FFFFFF8u) a = 0x7FFFFFF8u;
                k = (s8 << 2 | b3 << 1 | b5) << 28 | a >> 3;
                atomicAdd(&s_hist[hist_at(k >> kFineShift)], 1u);
            }
            s_key[at + q] = k;
            s_rec[at + q] = j;
        }
    }
    __syncthreads();
    // exclusive scan of the histogram
    constexpr uint32_t kEach = kHist / kBlockThreads;
    static_assert(kHist % kBlockThreads == 0 && kBlockEntries % kBlockThreads == 0, "whole rounds");
    uint32_t sum = 0;
    for (uint32_t i = 0; i < kEach; ++i) sum += s_hist[hist_at(tid * kEach + i)];
    uint32_t incl = sum;
#pragma unroll
    for (uint32_t d = 1; d < 32; d <<= 1) {
        const uint32_t t = __shfl_up_sync(0xFFFFFFFFu, incl, d);
        if (lane >= d) incl += t;
    }
    if (lane == 31) s_warp[warp] = incl;
    __syncthreads();
    if (warp == 0) {
        const uint32_t v = lane < kBlockThreads / 32 ? s_warp[lane] : 0u;
        uint32_t w = v;
#pragma unroll
        for (uint32_t d = 1; d < 32; d <<= 1) {
            const uint32_t t = __shfl_up_sync(0xFFFFFFFFu, w, d);
            if (lane >= d) w += t;
        }
        if (lane < kBlockThreads / 32) s_warp[lane] = w - v;
    }
    __syncthreads();
    uint32_t run = s_warp[warp] + incl - sum;
    for (uint32_t i = 0; i < kEach; ++i) {
        const uint32_t c = s_hist[hist_at(tid * kEach + i)];
        s_hist[hist_at(tid * kEach + i)] = run;
        run += c;
    }
    __syncthreads();
    // a bucket's counter ends at the start of the next one
    for (uint32_t i = tid; i < B.n; i += kBlockThreads) {
        const uint32_t k = s_key[i];
        const uint32_t p = (k >> 28) == 8u ? sorted + (k & 0x0FFFFFFFu) : atomicAdd(&s_hist[hist_at(k >> kFineShift)], 1u);
        if (p < B.n) s_order[p] = (uint16_t)i;
    }
    __syncthreads();
    for (uint32_t p = tid; p < B.n; p += kBlockThreads) {
        const uint32_t i = s_order[p], k = s_key[i], j = s_rec[i];
        uint32_t place = p;
        if (p < sorted) {
            const uint32_t b = k >> kFineShift, end = s_hist[hist_at(b)];
            place = b ? s_hist[hist_at(b - 1)] : 0u;
            for (uint32_t q = place, q1 = end; q < q1; ++q) {
                const uint32_t o = s_order[q], ok = s_key[o];
                place += ok < k || (ok == k && s_rec[o] < j);
            }
        }
        const uint32_t m = owner[j];
        const ExactRec e = exact[j];
        const HotRec h = hot[j];
        const int64_t im = e.im < 0 ? -e.im : e.im;
        uint32_t w[kFields];
#pragma unroll
        for (uint32_t f = 0; f < kFields; ++f) {
            const uint32_t M = field_mod(f);
            const uint32_t q = m % M, q2 = q * q % M;
            w[f] = residue_i64(e.re, M) | residue_i64(im, M) << 10 | (q2 * q2 % M) << 20;
        }
        const uint32_t at = B.base + place;
        w0[at] = w[0];
        w1[at] = w[1];
        w2[at] = w[2];
        ang[at] = (k >> 28) == 8u ? m : (k & 0x0FFFFFFFu) << 3;
        part[at] = (uint8_t)((m - B.m_lo) / part_step(B.m_lo, B.m_hi));
        src[at] = j;
        root[at] = m;
        xy[at] = make_float2(h.re, fabsf(h.im));
        pos[j] = (uint16_t)place;
    }
    __syncthreads();
    // the small primes' bit sets, a word per warp at a time
    uint32_t* sets = mask + (size_t)blockIdx.x * (kMaskPrimes * kMaskWords);
    for (uint32_t i = tid; i < kBlockEntries; i += kBlockThreads) {
        const uint32_t m = i < B.n ? root[B.base + i] : 1u;
        uint32_t word = 0;
#pragma unroll
        for (uint32_t q = 0; q < kMaskPrimes; ++q) {
            const uint32_t set = __ballot_sync(0xFFFFFFFFu, m % mask_prime(q) == 0);
            if (lane == q) word = set;
        }
        if (lane < kMaskPrimes) sets[lane * kMaskWords + i / 32] = word;
    }
    // list bounds and the angle index
    auto bucket_start = [&](uint32_t b) { return b ? s_hist[hist_at(b - 1)] : 0u; };
    if (tid <= kLists)
        blocks[blockIdx.x].list[tid] = (uint16_t)(tid == kLists ? B.n : tid == 8 ? sorted : bucket_start(tid * kFine));
    uint16_t* idx = reinterpret_cast<uint16_t*>(index + (size_t)blockIdx.x * kIndexWords);
    for (uint32_t t = tid; t < 8 * (kBuckets + 2); t += kBlockThreads) {
        const uint32_t s = t / (kBuckets + 2), x = t % (kBuckets + 2);
        idx[t] = (uint16_t)bucket_start(s * kFine + min(x, kBuckets) * (kFine / kBuckets));
    }
}

}  // namespace

int plan_arc_blocks(const uint32_t* d_seg_off, uint64_t limit, cudaStream_t stream, ArcPlan* plan, std::string* err) {
    CutTasks tasks{};
    for (uint32_t t = 0; t < kTypes; ++t) {
        tasks.roots[t] = roots_upto(kTypeTables, t, (uint32_t)limit);
        tasks.first[t + 1] = tasks.first[t] + (tasks.roots[t] + kCutRoots - 1) / kCutRoots;
    }
    const uint32_t n_tasks = tasks.first[kTypes];
    std::vector<uint32_t> at(n_tasks + 1);
    uint32_t* d_at = nullptr;
    ArcBlock* d_blocks = nullptr;
    auto cut = [&](ArcBlock* blocks) {
        block_cut_kernel<<<(n_tasks + kCutWarps - 1) / kCutWarps, kCutWarps * 32, 0, stream>>>(d_seg_off, tasks, d_at,
                                                                                               blocks);
        return cudaGetLastError();
    };
    cudaError_t e = cudaMalloc((void**)&d_at, (n_tasks + 1) * sizeof(uint32_t));
    if (e == cudaSuccess) e = cut(nullptr);
    if (e == cudaSuccess)
        e = cudaMemcpyAsync(at.data(), d_at, n_tasks * sizeof(uint32_t), cudaMemcpyDeviceToHost, stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(stream);
    if (e == cudaSuccess) {
        uint32_t run = 0;
        for (uint32_t& x : at) {
            const uint32_t c = x;
            x = run;
            run += c;
        }
        plan->blocks.resize(at[n_tasks]);
        e = cudaMalloc((void**)&d_blocks, (plan->blocks.size() + 1) * sizeof(ArcBlock));
    }
    if (e == cudaSuccess)
        e = cudaMemcpyAsync(d_at, at.data(), n_tasks * sizeof(uint32_t), cudaMemcpyHostToDevice, stream);
    if (e == cudaSuccess) e = cut(d_blocks);
    if (e == cudaSuccess)
        e = cudaMemcpyAsync(plan->blocks.data(), d_blocks, plan->blocks.size() * sizeof(ArcBlock),
                            cudaMemcpyDeviceToHost, stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(stream);
    cudaFree(d_at);
    cudaFree(d_blocks);
    if (e != cudaSuccess) {
        cudaGetLastError();  // not left for the next launch's check
        *err = cudaGetErrorString(e);
        return e == cudaErrorMemoryAllocation ? HSS_ERR_MEMORY : HSS_ERR_CUDA;
    }
    uint64_t base = 0;
    plan->cap = 0;
    uint32_t next = 0;
    for (uint32_t t = 0; t < kTypes; ++t) {
        plan->type_first[t] = next;
        for (; next < at[tasks.first[t + 1]]; ++next) {
            ArcBlock& b = plan->blocks[next];
            b.base = (uint32_t)base;
            base += (b.n + 15) & ~15u;
            plan->cap = std::max(plan->cap, b.n);
        }
    }
    plan->type_first[kTypes] = next;
    plan->entries = base;
    while ((limit >> plan->start_shift) > 4096) ++plan->start_shift;
    for (uint32_t t = 0; t < kTypes; ++t) {
        std::vector<uint32_t>& start = plan->start[t];
        start.resize((limit >> plan->start_shift) + 1);
        uint32_t b = plan->type_first[t];
        for (size_t i = 0; i < start.size(); ++i) {
            while (b < plan->type_first[t + 1] && plan->blocks[b].m_hi < (uint64_t)i << plan->start_shift) ++b;
            start[i] = b;
        }
    }
    return HSS_OK;
}

int build_arc_layout(const DeviceCache& cache, uint64_t records, const ArcPlan& plan, cudaStream_t stream,
                     ArcBuild* out, std::string* err) {
    if (plan.entries + 16 > UINT32_MAX || plan.cap > kBlockEntries) {
        *err = "arc layout beyond its indexing";
        return HSS_ERR_LIMIT;
    }
    // one allocation for all arrays, each from a 256-byte boundary
    size_t bytes = 0;
    unsigned char* slab = nullptr;
    auto place = [&](auto** p, size_t count) {
        if (slab) *p = reinterpret_cast<std::remove_reference_t<decltype(*p)>>(slab + bytes);
        bytes += (count * sizeof(**p) + 255) & ~(size_t)255;
    };
    auto lay_out = [&] {
        bytes = 0;
        place(&out->blocks, plan.blocks.size());
        for (uint32_t f = 0; f < kFields; ++f) place(&out->w[f], plan.entries + 16);
        place(&out->ang, plan.entries + 16);
        place(&out->part, plan.entries + 16);
        place(&out->src, plan.entries + 16);
        place(&out->m, plan.entries + 16);
        place(&out->xy, plan.entries + 16);
        place(&out->index, plan.blocks.size() * kIndexWords);
        place(&out->mask, plan.blocks.size() * kMaskPrimes * kMaskWords);
        place(&out->pos, records + 1);
    };
    lay_out();
    cudaError_t e = cudaMalloc((void**)&slab, bytes);
    if (e == cudaSuccess) {
        out->owned.push_back(slab);
        lay_out();
    }
    if (e == cudaSuccess)
        e = cudaMemcpyAsync(out->blocks, plan.blocks.data(), plan.blocks.size() * sizeof(ArcBlock),
                            cudaMemcpyHostToDevice, stream);
    if (e == cudaSuccess && !plan.blocks.empty()) {
        const size_t smem = block_sort_smem(plan.cap);
        // (the limit is the kernel's, for every thread of the process: the same at every launch)
        e = cudaFuncSetAttribute((const void*)block_sort_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)block_sort_smem(kBlockEntries));
        if (e == cudaSuccess) {
            block_sort_kernel<<<(unsigned)plan.blocks.size(), kBlockThreads, smem, stream>>>(
                out->blocks, plan.cap, cache.seg_off, cache.hot, cache.exact, cache.owner, out->w[0], out->w[1], out->w[2],
                out->ang, out->part, out->src, out->m, out->xy, out->index, out->mask, out->pos);
            e = cudaGetLastError();
        }
    }
    if (e != cudaSuccess) {
        for (void* p : out->owned) cudaFree(p);
        out->owned.clear();
        cudaGetLastError();
        *err = cudaGetErrorString(e);
        return e == cudaErrorMemoryAllocation ? HSS_ERR_MEMORY : HSS_ERR_CUDA;
    }
    return HSS_OK;
}

}  // namespace hss
