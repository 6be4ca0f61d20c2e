// hss_devprep.cu - the factor cache built on the device.
//
// The same arrays, layout and values as build_host_cache (hss_prep.cpp, which
// follows src/gpu_search_v42.cu:354-391, :525-594), made by sm_103a kernels
// instead of host threads, so that opening a handle needs no host pass over
// 10^7 integers and no upload of the 3.4 GB cache:
//   1. spf[x]: a sieve in shared-memory tiles over the primes up to sqrt(N)
//      (those few hundred primes come from a host sieve);
//   2. prime-power table: per split prime p its block size (sum over a of
//      4a+1, a <= 2 log_p N), an exclusive scan for pp_base, then a thread per
//      p finds pi = u + iv (smallest u, as the host) and a warp per p writes
//      pi^r conj(pi)^(4a-r) for every a and r, exact and hot;
//   3. segment sizes (W(x)-1)/2 + 1 from the factorisation of x, an exclusive
//      scan for seg_off;
//   4. one thread per record decodes its free vector (or the central value)
//      from its place in x's segment, in the host's order (64-bit products:
//      every partial product divides x^2 in the Gaussian integers, so its
//      coordinates are at most x^2 < 2^50).
// The host keeps copies of spf and seg_off (the item builder reads them).
#include <cuda_runtime.h>
#include <math.h>

#include <chrono>
#include <vector>

#include "hss_api_status.h"
#include "hss_prep.h"

namespace hss {
namespace {

constexpr int kThreads = 256;

__device__ __forceinline__ uint32_t residue64(int64_t v, uint32_t m) {
    const int64_t r = v % (int64_t)m;
    return (uint32_t)(r < 0 ? r + m : r);
}

__device__ __forceinline__ uint32_t pack64(int64_t v) {
    return residue64(v, kModA) | (residue64(v, kModD) << kShiftD);
}

// Number of powers p^j <= n (j >= 1), as the host's power_count.
__device__ __forceinline__ uint32_t power_count(uint64_t p, uint64_t n) {
    uint32_t k = 0;
    for (uint64_t q = p; q <= n; q *= p) {
        ++k;
        if (q > n / p) break;
    }
    return k;
}

struct Factors {
    uint32_t primes[8];
    uint32_t exps[8];
    uint32_t count;
    uint64_t fixed;
};

__device__ Factors factor(const uint32_t* spf, uint32_t x) {
    Factors f;
    f.count = 0;
    f.fixed = 1;
    while (x > 1) {
        const uint32_t p = spf[x];
        uint32_t a = 0;
        do {
            x /= p;
            ++a;
        } while (x % p == 0);
        if (p % 4 == 1) {
            f.primes[f.count] = p;
            f.exps[f.count] = a;
            ++f.count;
        } else {
            for (uint32_t i = 0; i < 2 * a; ++i) f.fixed *= p;
        }
    }
    return f;
}

// Smallest prime factors, kSieveTile integers per CTA in shared memory: the
// primes below 32 by trial (a thread per integer, most integers end there), the
// others a thread per prime over its multiples in the tile from p^2 on, the
// smallest kept by atomicMin.  Trial division of every integer by every prime up to
// its root spent 3.36 ms at N = 10^7 on the few integers that need all of them;
// this form takes 0.16 ms.
constexpr uint32_t kSieveTile = 8192;
constexpr uint32_t kTrialPrimes = 11;  // 2 .. 31

__global__ void __launch_bounds__(kThreads) sieve_kernel(uint32_t* spf, uint32_t n, const uint32_t* primes,
                                                         uint32_t nprimes) {
    __shared__ uint32_t s[kSieveTile];
    const uint32_t tiles = n / kSieveTile + 1;
    for (uint32_t tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
        const uint32_t x0 = tile * kSieveTile, count = min(kSieveTile, n - x0 + 1);
        for (uint32_t i = threadIdx.x; i < count; i += kThreads) {
            const uint32_t x = x0 + i;
            uint32_t f = x;  // spf[0] = 0, spf[1] = 1, spf[p] = p
            for (uint32_t k = 0; k < kTrialPrimes && k < nprimes; ++k) {
                const uint32_t p = primes[k];
                if (p * p > x) break;
                if (x % p == 0) {
                    f = p;
                    break;
                }
            }
            s[i] = f;
        }
        __syncthreads();
        for (uint32_t k = kTrialPrimes + threadIdx.x; k < nprimes; k += kThreads) {
            const uint32_t p = primes[k];
            if (p * p >= x0 + count) break;  // (p <= sqrt(3e7): 32 bits)
            uint32_t m = max(p * p, (x0 + p - 1) / p * p);
            for (; m < x0 + count; m += p) atomicMin(&s[m - x0], p);
        }
        __syncthreads();
        for (uint32_t i = threadIdx.x; i < count; i += kThreads) spf[x0 + i] = s[i];
        __syncthreads();
    }
}

// Block sizes of the prime-power table (0 unless p is a split prime) and
// the largest exponent covered.
__global__ void pp_size_kernel(const uint32_t* spf, uint32_t n, uint64_t* size, unsigned int* max_exp) {
    for (uint32_t p = blockIdx.x * blockDim.x + threadIdx.x; p <= n; p += gridDim.x * blockDim.x) {
        uint64_t s = 0;
        if (p >= 5 && p % 4 == 1 && spf[p] == p) {
            const uint32_t max_a = 2 * power_count(p, n);
            s = 2ull * max_a * max_a + 3ull * max_a;  // sum_{a=1}^{max_a} (4a+1)
            atomicMax(max_exp, max_a);
        }
        size[p] = s;
    }
}

struct Gauss {
    __int128 re, im;
};

__device__ __forceinline__ Gauss gmul(Gauss a, Gauss b) {
    return {a.re * b.re - a.im * b.im, a.re * b.im + a.im * b.re};
}

// Exact floor(sqrt(r)) for r < 2^26 (float estimate, integer correction).
__device__ __forceinline__ uint32_t isqrt32(uint32_t r) {
    uint32_t v = (uint32_t)sqrtf((float)r);
    while (v * v > r) --v;
    while ((v + 1) * (v + 1) <= r) ++v;
    return v;
}

// a b mod p for a, b < p < 2^32 by Barrett's reduction, inv = floor((2^64 - 1) / p):
// the quotient is at most one short.
__device__ __forceinline__ uint32_t mul_mod(uint32_t a, uint32_t b, uint32_t p, uint64_t inv) {
    const uint64_t x = (uint64_t)a * b;
    const uint64_t r = x - __umul64hi(x, inv) * p;
    return (uint32_t)(r >= p ? r - p : r);
}

// The smaller u of p = u^2 + v^2 for every split prime p, left in pp_base[p],
// by Cornacchia's method: r = a^((p - 1) / 4) is a square root of -1 for every
// non-residue a (about every second one), and the first remainder of Euclid's
// algorithm on (p, r) at or below sqrt(p) is one of the two.  A thread per
// integer, bound by the chain of modular products on the one lane in 30 that has a
// prime: 0.94 ms at N = 10^7 (2.77 ms with a 64-bit division per product).  With
// pp_fill_kernel (1.06 ms) it replaces a search for u by a warp per prime (3.17 ms).
__global__ void pp_root_kernel(const uint32_t* spf, uint32_t n, uint32_t* pp_base) {
    for (uint32_t p = blockIdx.x * blockDim.x + threadIdx.x; p <= n; p += gridDim.x * blockDim.x) {
        if (!(p >= 5 && p % 4 == 1 && spf[p] == p)) continue;
        uint32_t r = 0;
        const uint64_t inv = ~0ull / p;
        for (uint32_t a = 2; a < p; ++a) {
            uint32_t base = a, e = (p - 1) / 4;
            r = 1;
            for (; e; e >>= 1) {
                if (e & 1u) r = mul_mod(r, base, p, inv);
                base = mul_mod(base, base, p, inv);
            }
            if (mul_mod(r, r, p, inv) == p - 1) break;
        }
        uint32_t x = p, y = r;
        while ((uint64_t)y * y > p) {
            const uint32_t t = x % y;
            x = y;
            y = t;
        }
        const uint32_t v = isqrt32(p - y * y);
        pp_base[p] = min(y, v);
    }
}

// A warp takes 32 integers at a time and, for each split prime p among them,
// shares the block's entries (a, r): pi^r conj(pi)^(4a-r) by repeated products
// (at most 4a <= 8 log_5 N of them, no per-thread arrays), pi = u + iv with the
// u that pp_root_kernel left in pp_base.
__global__ void pp_fill_kernel(const uint32_t* spf, uint32_t n, const uint64_t* offs, uint32_t* pp_base,
                               HotRec* pp_hot, __int128* pp_exact) {
    const uint32_t lane = threadIdx.x & 31;
    const uint32_t warps = gridDim.x * blockDim.x / 32;
    for (uint32_t p0 = (blockIdx.x * blockDim.x + threadIdx.x) / 32 * 32; p0 <= n; p0 += warps * 32) {
        const uint32_t mine = p0 + lane;
        const bool split = mine <= n && mine >= 5 && mine % 4 == 1 && spf[mine] == mine;
        const uint32_t root = split ? pp_base[mine] : 0u;
        if (mine <= n) pp_base[mine] = split ? (uint32_t)offs[mine] : 0xFFFFFFFFu;
        for (uint32_t todo = __ballot_sync(0xFFFFFFFFu, split); todo; todo &= todo - 1) {
            const uint32_t src = __ffs(todo) - 1, p = p0 + src;
            const uint32_t u = __shfl_sync(0xFFFFFFFFu, root, src), v = isqrt32(p - u * u);
            const uint32_t max_a = 2 * power_count(p, n);
            const uint64_t base = offs[p];
            const Gauss pi{(__int128)u, (__int128)v}, pc{(__int128)u, -(__int128)v};
            const uint32_t total = 2 * max_a * max_a + 3 * max_a;
            for (uint32_t k = lane; k < total; k += 32) {
                uint32_t a = 1, r = k;
                while (r >= 4 * a + 1) {
                    r -= 4 * a + 1;
                    ++a;
                }
                Gauss val{1, 0};
                for (uint32_t j = 0; j < r; ++j) val = gmul(val, pi);
                for (uint32_t j = 0; j < 4 * a - r; ++j) val = gmul(val, pc);
                pp_exact[2 * (base + k)] = val.re;
                pp_exact[2 * (base + k) + 1] = val.im;
                HotRec h;
                h.re = i128_to_float(val.re);
                h.im = i128_to_float(val.im);
                h.rre = pack_residues(val.re) | (r == 2 * a ? kCentralBit : 0u);
                h.rim = pack_residues(val.im);
                pp_hot[base + k] = h;
            }
        }
    }
}

// Segment lengths (free set + central value), the reference's cached-value
// count (free + central + raw per x) and the longest segment.
__global__ void seg_size_kernel(const uint32_t* spf, uint32_t n, uint64_t* len, unsigned long long* ref_cached,
                                unsigned int* longest) {
    unsigned long long local = 0;
    uint32_t lmax = 0;
    for (uint32_t x = blockIdx.x * blockDim.x + threadIdx.x; x <= n + 1; x += gridDim.x * blockDim.x) {
        if (x == 0 || x == n + 1) {
            len[x] = 0;
            continue;
        }
        const Factors f = factor(spf, x);
        uint64_t w = 1;
        for (uint32_t i = 0; i < f.count; ++i) w *= 4u * f.exps[i] + 1;
        len[x] = (w - 1) / 2 + 1;
        local += (w - 1) / 2 + 1 + w;
        lmax = max(lmax, (uint32_t)((w - 1) / 2 + 1));
    }
    for (int d = 16; d > 0; d >>= 1) {
        local += __shfl_down_sync(0xFFFFFFFFu, local, d);
        lmax = max(lmax, __shfl_down_sync(0xFFFFFFFFu, lmax, d));
    }
    if ((threadIdx.x & 31) == 0) {
        atomicAdd(ref_cached, local);
        atomicMax(longest, lmax);
    }
}

__global__ void narrow_kernel(const uint64_t* in, uint32_t* out, uint32_t count) {
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < count; i += gridDim.x * blockDim.x)
        out[i] = (uint32_t)in[i];
}

__device__ __forceinline__ void cmul64(int64_t ar, int64_t ai, int64_t br, int64_t bi, int64_t& re, int64_t& im) {
    re = ar * br - ai * bi;
    im = ar * bi + ai * br;
}

// Free set of x, then its central value: for the first non-central index i
// and r_i < 2e_i, every digit combination of the later primes with the
// earlier digit most significant (the host's recursion order).
//
// A CTA takes kFillRoots consecutive x: a thread factors each, then all threads
// share the tile's records, one at a time and in order, so that the 36 bytes of a
// record are written coalesced; a record's x is found among the tile's offsets,
// its digits from its place in the segment.  (A thread per x that walked its own
// segment took 10.7 ms at N = 10^7: 94.8 M records, stores of a warp to 32 segments; this
// form takes 3.2 ms, 3.4 GB written.)
constexpr uint32_t kFillRoots = 128;

struct FillRoot {
    uint64_t fixed;
    uint32_t base[8];  // first prime-power value of the term
    uint8_t e[8];
    uint32_t count;
    uint32_t pad;
};

__global__ void __launch_bounds__(kThreads) seg_fill_kernel(const uint32_t* spf, uint32_t n, const uint32_t* seg_off,
                                                            const uint32_t* pp_base, const __int128* pp_exact,
                                                            HotRec* hot, ExactRec* exact, uint32_t* owner,
                                                            unsigned int* err) {
    __shared__ FillRoot s_root[kFillRoots];
    __shared__ uint32_t s_off[kFillRoots + 1];
    const uint32_t tiles = n / kFillRoots + 1;
    for (uint32_t tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
        const uint32_t x0 = tile * kFillRoots;
        __syncthreads();
        for (uint32_t i = threadIdx.x; i <= kFillRoots; i += kThreads) s_off[i] = seg_off[min(x0 + i, n + 1)];
        for (uint32_t i = threadIdx.x; i < kFillRoots; i += kThreads) {
            const uint32_t x = x0 + i;
            FillRoot r;
            r.count = 0;
            if (x >= 1 && x <= n) {
                const Factors f = factor(spf, x);
                uint32_t w = 1;
                r.fixed = f.fixed;
                r.count = f.count;
                for (uint32_t j = 0; j < f.count; ++j) {
                    r.base[j] = pp_base[f.primes[j]] + pp_exponent_offset(f.exps[j]);
                    r.e[j] = (uint8_t)f.exps[j];
                    w *= 4u * f.exps[j] + 1;
                }
                if (seg_off[x + 1] - seg_off[x] != (w - 1) / 2 + 1) atomicOr(err, 1u);  // segment size invariant
            }
            s_root[i] = r;
        }
        __syncthreads();
        const uint32_t first = s_off[0], records = s_off[kFillRoots] - first;
        for (uint32_t q = threadIdx.x; q < records; q += kThreads) {
            const uint32_t pos = first + q;
            uint32_t i = 0;  // the last root whose segment starts at or before pos
#pragma unroll
            for (uint32_t step = kFillRoots / 2; step; step >>= 1)
                if (s_off[i + step] <= pos) i += step;
            const FillRoot& R = s_root[i];
            const uint32_t x = x0 + i, count = R.count;
            uint32_t k = pos - s_off[i];
            int64_t re = (int64_t)R.fixed, im = 0;
            bool central = false;
            uint32_t below = 1;  // values of the terms after the first non-central one
            for (uint32_t j = 1; j < count; ++j) below *= 4u * R.e[j] + 1;
            uint32_t t = 0;
            for (;; ++t) {
                if (t >= count) {
                    central = true;
                    break;
                }
                const uint32_t block = 2u * R.e[t] * below;
                if (k < block) break;
                k -= block;
                re *= (int64_t)pp_exact[2 * ((uint64_t)R.base[t] + 2u * R.e[t])];  // p^(2e)
                if (t + 1 < count) below /= 4u * R.e[t + 1] + 1;
            }
            if (central) {
                re = (int64_t)x * x;
            } else {
                for (; t < count; ++t) {
                    const uint32_t d = k / below;
                    k -= d * below;
                    if (t + 1 < count) below /= 4u * R.e[t + 1] + 1;
                    const __int128* v = pp_exact + 2 * ((uint64_t)R.base[t] + d);
                    int64_t nr, ni;
                    cmul64(re, im, (int64_t)v[0], (int64_t)v[1], nr, ni);
                    re = nr;
                    im = ni;
                }
            }
            HotRec h;
            h.re = (float)re;
            h.im = (float)im;
            h.rre = pack64(re) | (central ? kCentralBit : 0u);
            h.rim = pack64(im);
            hot[pos] = h;
            exact[pos] = ExactRec{re, im};
            owner[pos] = x;
        }
    }
}

// Exclusive scan of count 64-bit values (in place allowed): tile sums, a
// single-block scan of the tile sums, then each tile scanned with its offset.
constexpr uint32_t kScanTile = 4 * kThreads;

__device__ __forceinline__ uint64_t block_exclusive(uint64_t v, uint64_t* s_warp, uint64_t* total) {
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x / 32;
    uint64_t incl = v;
    for (int d = 1; d < 32; d <<= 1) {
        const uint64_t t = __shfl_up_sync(0xFFFFFFFFu, incl, d);
        if (lane >= (uint32_t)d) incl += t;
    }
    if (lane == 31) s_warp[warp] = incl;
    __syncthreads();
    if (warp == 0) {
        uint64_t ws = lane < kThreads / 32 ? s_warp[lane] : 0;
        uint64_t wi = ws;
        for (int d = 1; d < 32; d <<= 1) {
            const uint64_t t = __shfl_up_sync(0xFFFFFFFFu, wi, d);
            if (lane >= (uint32_t)d) wi += t;
        }
        if (lane < kThreads / 32) s_warp[lane] = wi - ws;
        if (lane == kThreads / 32 - 1) *total = wi;
    }
    __syncthreads();
    const uint64_t r = s_warp[warp] + incl - v;
    __syncthreads();
    return r;
}

__global__ void scan_tiles_kernel(const uint64_t* in, uint64_t count, uint64_t* tile_sums) {
    __shared__ uint64_t s_warp[kThreads / 32];
    __shared__ uint64_t total;
    const uint64_t base = (uint64_t)blockIdx.x * kScanTile + 4ull * threadIdx.x;
    uint64_t v = 0;
    for (uint32_t k = 0; k < 4; ++k)
        if (base + k < count) v += in[base + k];
    block_exclusive(v, s_warp, &total);
    if (threadIdx.x == 0) tile_sums[blockIdx.x] = total;
}

__global__ void scan_sums_kernel(uint64_t* tile_sums, uint32_t tiles, uint64_t* grand) {
    __shared__ uint64_t s_warp[kThreads / 32];
    __shared__ uint64_t total;
    uint64_t carry = 0;
    for (uint32_t b = 0; b < tiles; b += kThreads) {
        const uint64_t v = b + threadIdx.x < tiles ? tile_sums[b + threadIdx.x] : 0;
        const uint64_t e = block_exclusive(v, s_warp, &total);
        if (b + threadIdx.x < tiles) tile_sums[b + threadIdx.x] = carry + e;
        carry += total;
        __syncthreads();
    }
    if (threadIdx.x == 0) *grand = carry;
}

__global__ void scan_apply_kernel(const uint64_t* in, uint64_t count, const uint64_t* tile_sums, uint64_t* out) {
    __shared__ uint64_t s_warp[kThreads / 32];
    __shared__ uint64_t total;
    const uint64_t base = (uint64_t)blockIdx.x * kScanTile + 4ull * threadIdx.x;
    uint64_t v[4], sum = 0;
    for (uint32_t k = 0; k < 4; ++k) {
        v[k] = base + k < count ? in[base + k] : 0;
        sum += v[k];
    }
    __syncthreads();  // in and out may alias: every read of the tile precedes its writes
    uint64_t run = tile_sums[blockIdx.x] + block_exclusive(sum, s_warp, &total);
    for (uint32_t k = 0; k < 4; ++k) {
        if (base + k < count) out[base + k] = run;
        run += v[k];
    }
}

// Exclusive scan of in[0 .. count) into out; *grand (device) receives the total.
cudaError_t exclusive_scan(const uint64_t* in, uint64_t* out, uint64_t count, uint64_t* tile_sums, uint64_t* grand,
                           cudaStream_t st) {
    const uint32_t tiles = (uint32_t)((count + kScanTile - 1) / kScanTile);
    scan_tiles_kernel<<<tiles, kThreads, 0, st>>>(in, count, tile_sums);
    scan_sums_kernel<<<1, kThreads, 0, st>>>(tile_sums, tiles, grand);
    scan_apply_kernel<<<tiles, kThreads, 0, st>>>(in, count, tile_sums, out);
    return cudaGetLastError();
}

template <class T>
cudaError_t dalloc(T** p, size_t count, std::vector<void*>* owned) {
    cudaError_t e = cudaMalloc((void**)p, (count ? count : 1) * sizeof(T));
    if (e == cudaSuccess) owned->push_back(*p);
    return e;
}

}  // namespace

int build_device_cache(uint64_t n, int sm_count, CUstream_st* st, DeviceBuild* out, std::string* err,
                       const std::function<int()>& on_records) {
    auto t0 = std::chrono::steady_clock::now();
    if (n < 1 || n > kMaxLimit) {
        *err = "limit out of range";
        return HSS_ERR_ARGUMENT;
    }
    DeviceBuild& b = *out;
    b.limit = n;
    std::vector<void*> scratch;
    struct Copies {
        cudaStream_t stream = nullptr;
        cudaEvent_t ready = nullptr;
        ~Copies() {
            if (stream) {
                cudaStreamSynchronize(stream);
                cudaStreamDestroy(stream);
            }
            if (ready) cudaEventDestroy(ready);
        }
    } copies;
    auto cleanup = [&]() {
        for (void* p : scratch) cudaFree(p);
        scratch.clear();
    };
    auto release = [&]() {  // on failure the cache arrays go too
        cleanup();
        for (void* p : b.owned) cudaFree(p);
        b.owned.clear();
    };
    auto fail = [&](cudaError_t e) {
        release();
        cudaGetLastError();  // a refused allocation's error is not left for the next launch's check
        *err = cudaGetErrorString(e);
        return HSS_ERR_CUDA;
    };
#define DEV(call)                          \
    do {                                   \
        cudaError_t e_ = (call);           \
        if (e_ != cudaSuccess) return fail(e_); \
    } while (0)
    // primes up to sqrt(n) for the sieve (a few hundred)
    uint32_t root = (uint32_t)sqrt((double)n);
    while ((uint64_t)(root + 1) * (root + 1) <= n) ++root;
    while ((uint64_t)root * root > n) --root;
    std::vector<uint32_t> small_primes;
    {
        std::vector<uint8_t> comp(root + 1, 0);
        for (uint32_t i = 2; i <= root; ++i) {
            if (comp[i]) continue;
            small_primes.push_back(i);
            for (uint64_t j = (uint64_t)i * i; j <= root; j += i) comp[j] = 1;
        }
    }
    const int grid = sm_count * 8;
    uint32_t* d_primes = nullptr;
    uint64_t *d_u64 = nullptr, *d_tiles = nullptr, *d_grand = nullptr;
    unsigned int* d_flags = nullptr;  // [0] max exponent, [1] longest segment, [2] fill error
    unsigned long long* d_refc = nullptr;
    DEV(dalloc(&d_primes, small_primes.size(), &scratch));
    DEV(dalloc(&d_u64, n + 2, &scratch));
    DEV(dalloc(&d_tiles, (n + 2 + kScanTile - 1) / kScanTile + 1, &scratch));
    DEV(dalloc(&d_grand, 1, &scratch));
    DEV(dalloc(&d_flags, 4, &scratch));
    DEV(dalloc(&d_refc, 1, &scratch));
    DEV(cudaMemsetAsync(d_flags, 0, 4 * sizeof(unsigned int), st));
    DEV(cudaMemsetAsync(d_refc, 0, sizeof(unsigned long long), st));
    if (!small_primes.empty())
        DEV(cudaMemcpyAsync(d_primes, small_primes.data(), small_primes.size() * sizeof(uint32_t),
                            cudaMemcpyHostToDevice, st));

    // 1. smallest prime factors
    DEV(dalloc(&b.spf, n + 1, &b.owned));
    sieve_kernel<<<grid, kThreads, 0, st>>>(b.spf, (uint32_t)n, d_primes, (uint32_t)small_primes.size());
    DEV(cudaGetLastError());

    // 2. prime-power table
    pp_size_kernel<<<grid, kThreads, 0, st>>>(b.spf, (uint32_t)n, d_u64, d_flags + 0);
    DEV(cudaGetLastError());
    DEV(exclusive_scan(d_u64, d_u64, n + 1, d_tiles, d_grand, st));
    uint64_t pp_total = 0;
    DEV(cudaMemcpyAsync(&pp_total, d_grand, sizeof pp_total, cudaMemcpyDeviceToHost, st));
    DEV(cudaStreamSynchronize(st));
    if (pp_total >= UINT32_MAX) {
        release();
        *err = "prime-power table exceeds 32-bit indexing";
        return HSS_ERR_LIMIT;
    }
    b.reference_flattened = pp_total;
    b.pp_count = pp_total;
    DEV(dalloc(&b.pp_base, n + 1, &b.owned));
    DEV(dalloc(&b.pp_hot, pp_total, &b.owned));
    DEV(dalloc(&b.pp_exact, 2 * pp_total, &b.owned));
    pp_root_kernel<<<grid, kThreads, 0, st>>>(b.spf, (uint32_t)n, b.pp_base);
    DEV(cudaGetLastError());
    pp_fill_kernel<<<grid, kThreads, 0, st>>>(b.spf, (uint32_t)n, d_u64, b.pp_base, b.pp_hot, b.pp_exact);
    DEV(cudaGetLastError());


    // 3. segment offsets
    seg_size_kernel<<<grid, kThreads, 0, st>>>(b.spf, (uint32_t)n, d_u64, d_refc, d_flags + 1);
    DEV(cudaGetLastError());
    DEV(exclusive_scan(d_u64, d_u64, n + 2, d_tiles, d_grand, st));
    uint64_t records = 0;
    unsigned int flags[4];
    unsigned long long refc = 0;
    DEV(cudaMemcpyAsync(&records, d_grand, sizeof records, cudaMemcpyDeviceToHost, st));
    DEV(cudaMemcpyAsync(flags, d_flags, sizeof flags, cudaMemcpyDeviceToHost, st));
    DEV(cudaMemcpyAsync(&refc, d_refc, sizeof refc, cudaMemcpyDeviceToHost, st));
    DEV(cudaStreamSynchronize(st));
    if (records >= UINT32_MAX) {
        release();
        *err = "factor cache exceeds 32-bit indexing";
        return HSS_ERR_LIMIT;
    }
    b.records = records;
    b.max_exponent = flags[0];
    b.longest = flags[1];
    b.reference_cached = refc;
    DEV(dalloc(&b.seg_off, n + 2, &b.owned));
    narrow_kernel<<<grid, kThreads, 0, st>>>(d_u64, b.seg_off, (uint32_t)(n + 2));
    DEV(cudaGetLastError());
    DEV(cudaStreamCreateWithFlags(&copies.stream, cudaStreamNonBlocking));
    DEV(cudaEventCreateWithFlags(&copies.ready, cudaEventDisableTiming));
    DEV(cudaEventRecord(copies.ready, st));
    DEV(cudaStreamWaitEvent(copies.stream, copies.ready, 0));

    // 4. records
    DEV(dalloc(&b.hot, records, &b.owned));
    DEV(dalloc(&b.exact, records, &b.owned));
    DEV(dalloc(&b.owner, records, &b.owned));
    seg_fill_kernel<<<grid, kThreads, 0, st>>>(b.spf, (uint32_t)n, b.seg_off, b.pp_base, b.pp_exact, b.hot, b.exact,
                                               b.owner, d_flags + 2);
    DEV(cudaGetLastError());

    if (on_records)
        if (int s = on_records()) {
            cudaStreamSynchronize(st);
            release();
            return s;
        }
    // Host copies the item builder reads, on a stream of their own: the memory
    // is touched and filled while the records and their layout are written (behind
    // them the copies took 2.3 of 15.3 ms of an open at N = 10^7).
    b.spf_host.resize(n + 1);
    b.seg_off_host.resize(n + 2);
    DEV(cudaMemcpyAsync(b.spf_host.data(), b.spf, (n + 1) * sizeof(uint32_t), cudaMemcpyDeviceToHost, copies.stream));
    DEV(cudaMemcpyAsync(b.seg_off_host.data(), b.seg_off, (n + 2) * sizeof(uint32_t), cudaMemcpyDeviceToHost,
                        copies.stream));
    DEV(cudaStreamSynchronize(copies.stream));
    DEV(cudaMemcpyAsync(flags, d_flags, sizeof flags, cudaMemcpyDeviceToHost, st));
    DEV(cudaStreamSynchronize(st));
#undef DEV
    if (flags[2]) {
        release();
        *err = "device cache build: a segment's size disagrees with its enumeration";
        return HSS_ERR_LIMIT;
    }
    cleanup();
    b.seconds = std::chrono::duration<double>(std::chrono::steady_clock::now() - t0).count();
    return HSS_OK;
}

}  // namespace hss
