// hss_arc.cuh - the arc path: the batched search by sorted runs (included by
// hss_kernels.cu, inside namespace hss's anonymous namespace).
//
// The reference multiplies out every product of a pair (l, m) and tests it.
// A counted term is a signed D = +-Re or +-Im of a product with
//     w = l^4 + m^4 - N^4 <= D <= l^4   and   area 4A (the other part) divisible.
// With gamma = 2 i^u alpha or its conjugate (alpha a value of l, u = 0..3) and
// beta a value of m with positive imaginary part, the terms are exactly the
// pairs (gamma, beta) with D = Re(gamma beta) in the window: each product's
// two orientations and two signs are the four u.  |gamma beta| = 2 l^2 m^2 is
// fixed, so the window is an arc of arg gamma + arg beta, namely +-[phi0, phi1]
// with cos phi0 = l^2 / (2 m^2), cos phi1 = w / (2 l^2 m^2); the area test and
// z = l^4 + m^4 - D mod 16 depend only on the classes of the two values
// (hss_blocks.cu).  So for one gamma and one block of roots the counted terms
// of a class list, sorted by argument, are a contiguous run: their number is a
// difference of two positions, and only the runs whose z = 0, 1 mod 16 have to
// be read, by the residue filter alone.  The windows of a block's roots differ
// a little: the run between the tightest bounds is certain, the terms between
// the tightest and the widest are decided one by one against their own root's
// window (in float with an error bound, by the exact kernel when within it).
//
// Pairs that share split primes are rows too: with P the common part of m
// (m = P m', m' prime to l's split primes) the value set of (l, m) is that of
// l P times that of m' (the exponents add), so (l, P) is a row against m'.
//
// Roots m' that an odd prime >= 7 of l divides are not the row's (skipped
// pairs for an inert prime, another row's for a split one).  Their records
// are marked in a bit set per row and block and subtracted from the run
// lengths by rank; the filter reads them along (about 6 %), and an event
// drops them.  2, 3 and 5 are handled by the block types.
//
// What bounds it: instruction issue (64 rows at LIMIT 10^6: 68 % of the issue
// slots while an SM is busy, 27 of 32 lanes; DRAM under 1 %: a block is read
// once per item, 17 bytes an entry, for a million tests and more).  One CTA of
// 24 warps per SM, since the block of 6144 entries and the warps' own staging
// fill its shared memory; two CTAs of 8 or 12 warps with smaller blocks were
// slower (more runs per row).  Warps work on rows by themselves, with no barrier
// but at a change of block.  In place of one test of every product (512 rows at
// LIMIT 10^7, l = 7.5 10^6: 778 ms) the batch takes 106 ms; root 6,325,815 (branch
// weight 625) takes 22 ms (87), 37 roots near the limit 1.35 ms (14.7).
// Of the batch's 86 G warp instructions some 29 G are the filter (1.03 G tests of 32
// terms) and 9 G the starts of its 0.19 G runs.

__constant__ TypeTables c_arc_types = make_type_tables();

constexpr uint32_t kAngleSlack = 4096;       // 6e-6 rad: both arguments and the arc bounds
constexpr uint32_t kArcMax = 0x7FFFFFFFu;    // last angle of the upper half turn
// more undecided terms than this and a run is checked term by term (24: 2 % more time)
constexpr uint32_t kArcWide = 48;
constexpr uint32_t kArcOpen = 64;             // terms of a warp awaiting their own root's window
constexpr uint32_t kStageWords = 12;          // per lane: a staged run
constexpr uint32_t kArcQueue = 96;           // events per warp: under 32 kept, up to 64 of one round of the filter

// Shared memory of the kernel: a block's three residue words and arguments (a
// stride that every block fits, so that one register addresses all four), its
// bucket index, the filter's tables, and per warp the staged runs, the bit set of
// marked entries with ranks, and the event queue.
constexpr uint32_t kArcCap = kBlockEntries + 32;  // the filter's last round reads past a run's end
constexpr uint32_t kArcWords = kArcCap / 32;
static_assert(kIndexWords % 4 == 0 && sizeof(ArcBlock) % 16 == 0, "prefetched in 16-byte pieces");
static_assert(kArcCap % 32 == 0 && kArcCap < 65536, "whole words, 16-bit positions");
// The filter's 12 constants of one gamma: per field the multipliers of the
// packed word, of it >> 10 and of it >> 20, and the row's term.  With
// w = re + 2^10 im + 2^20 m4, the sum is scale * (l^4 + P^4 m^4 - Re(gamma beta))
// mod 2^32 without unpacking a field.
struct ArcFilter {
    uint32_t c0[kFields], c1[kFields], c2[kFields], c3[kFields];
};

__device__ __forceinline__ void arc_variant(uint32_t var, uint32_t& a, uint32_t& b) {
    if (var & 4u) b = 0u - b;
    if (var & 1u) {
        const uint32_t t = a;
        a = 0u - b;
        b = t;
    }
    if (var & 2u) {
        a = 0u - a;
        b = 0u - b;
    }
}

__device__ __forceinline__ void arc_variant(uint32_t var, float& a, float& b) {
    if (var & 4u) b = -b;
    if (var & 1u) {
        const float t = a;
        a = -b;
        b = t;
    }
    if (var & 2u) {
        a = -a;
        b = -b;
    }
}

__device__ __forceinline__ ArcFilter arc_filter(const ArcValue& g, uint32_t var, const ArcRow& row) {
    ArcFilter c;
#pragma unroll
    for (uint32_t f = 0; f < kFields; ++f) {
        uint32_t a = g.re[f], b = g.im[f];
        arc_variant(var, a, b);
        // z = l^4 + P^4 m4 - a re + b im
        c.c0[f] = row.c0[f];
        c.c1[f] = 0u - a;
        c.c2[f] = b + (a << 10);
        c.c3[f] = row.c3[f] - (b << 10);
    }
    return c;
}

// Whether z passes field f (1 or 0); the top 11 bits of the scaled residue index
// the field's table.
__device__ __forceinline__ uint32_t arc_pass(uint32_t f, uint32_t x, const ArcFilter& c, const uint8_t* tab) {
    const uint32_t z = imad(x, c.c1[f], imad(x >> 10, c.c2[f], imad(x >> 20, c.c3[f], c.c0[f])));
    return tab[(f << 11) + (z >> 21)];
}

// All three fields of the entry at x (its words kArcCap apart).
__device__ __forceinline__ uint32_t arc_test(const uint32_t* x, const ArcFilter& c, const uint8_t* tab) {
    return arc_pass(0, x[0], c, tab) & arc_pass(1, x[kArcCap], c, tab) & arc_pass(2, x[2 * kArcCap], c, tab);
}

// A staged run: words 0..2 and 4..6 the first two multipliers of the fields,
// word 8 its value and form (kRunId) and these marks, 9 its angle, 10 and 11 its bounds
// p0 | c0 << 16 and c1 | p1 << 16.
static_assert(kArcValuesMost << 3 == 1ull << 28, "a value and its form fit kRunId");
constexpr uint32_t kRunId = 0x0FFFFFFFu, kRunCentral = 1u << 28, kRunLower = 1u << 29, kRunKeep = 1u << 30;

// A row against the CTA's block, as one warp works on it.
struct ArcSlot {
    ArcRow row;
    uint32_t phi[4];  // phi0 certain, phi0 possible, phi1 certain, phi1 possible: the block's tightest and widest
};

// What one warp keeps in shared memory, behind one base register.
struct __align__(16) ArcWarp {
    uint32_t stage[32 * kStageWords];
    uint4 range[kParts];
    ArcSlot slot;
    unsigned long long cand, r16;  // of the unit
    uint32_t open_at[kArcOpen], open_id[kArcOpen];
    uint32_t ev_at[kArcQueue], ev_row[kArcQueue], ev_id[kArcQueue];
    uint32_t bits[kArcWords];
    uint16_t rank[kArcWords + 2];
};

template <int WARPS>
struct ArcSmem {
    uint32_t w0[kArcCap], w1[kArcCap], w2[kArcCap], ang[kArcCap];
    uint8_t part[kArcCap];
    uint8_t tab[kArcTabBytes];
    uint32_t index[kIndexWords];
    ArcWarp warp[WARPS];
};

struct ArcShared {
    uint32_t item, ahead, next;
    uint32_t pad;
    ArcBlock block;
    ArcItem rec;  // read from here by the units, not kept in registers
};

// Asks for a block's arrays in L2 (sizes and addresses are multiples of 16 bytes).
__device__ __forceinline__ void arc_prefetch(const uint32_t* p, uint32_t quads) {
    asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(p), "r"(16u * quads) : "memory");
}

// m^4 in two floats (m < 2^25), the second exact to about 2^-45 of the first:
// m = a + b with a even, so both fit a float.
__device__ __forceinline__ float m4_float(uint32_t m, float& lo) {
    const float a = (float)(m & ~1u), b = (float)(m & 1u);
    const float x = __fmul_rn(a, a);
    const float y = fmaf(2.f * a, b, fmaf(a, a, -x) + b);  // m^2 = x + y
    const float h = __fadd_rn(x, y), l = __fadd_rn(y, -__fadd_rn(h, -x));
    const float p = __fmul_rn(h, h);
    lo = fmaf(2.f * h, l, fmaf(h, h, -p));
    return p;
}

// w = l^4 + m^4 - N^4 in float, within |w| 2^-22 + m^4 2^-43.
__device__ __forceinline__ float window_low(const ArcRow& r, uint32_t m, float& m4) {
    float lo;
    m4 = m4_float(m, lo);
    const float s = __fadd_rn(m4, r.lw_hi);
    const float t = __fadd_rn(s, -m4);
    const float e = __fadd_rn(__fadd_rn(m4, -__fadd_rn(s, -t)), __fadd_rn(r.lw_hi, -t));
    return s + (e + (lo + r.lw_lo));
}

// Marked entries before entry i.
__device__ __forceinline__ uint32_t arc_rank(const uint32_t* bits, const uint16_t* rank, uint32_t i) {
    const uint32_t part = i & 31u;
    return rank[i >> 5] + (part ? __popc(bits[i >> 5] & ((1u << part) - 1u)) : 0u);
}

// The lane whose run of a warp's items, laid end to end, holds item s: the
// first lane whose inclusive sum exceeds it.
__device__ __forceinline__ uint32_t arc_owner(uint32_t incl, uint32_t s) {
    uint32_t own = 0;
#pragma unroll
    for (uint32_t step = 16; step >= 1; step >>= 1) {
        const uint32_t x = __shfl_sync(kFull, incl, own + step - 1);
        if (x <= s) own += step;
    }
    return own & 31u;
}

__device__ __forceinline__ uint32_t arc_scan(uint32_t v, uint32_t lane) {
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const uint32_t t = __shfl_up_sync(kFull, v, d);
        if (lane >= (uint32_t)d) v += t;
    }
    return v;
}

// One warp prepares a row: arc bounds, marked entries with their ranks, and
// the counts that need no term (processed pairs, records, the all-central
// products).  The block is in shared memory (s_ang of a central entry is its
// root).  Returns false when the row has no root in the block.
struct ArcCounts {
    uint32_t processed, records, cc;
    bool excl;
};

__device__ __forceinline__ bool arc_prepare(const ArcCache& cache, const ArcBuffers& buf, const ArcBlock& B, uint32_t block,
                                            const uint32_t* s_ang, ArcSlot& S, uint32_t* bits,
                                            uint16_t* rank, uint4* range, uint32_t lane, ArcCounts& out) {
    const ArcRow& row = S.row;
    const RowInfo& R = buf.row_info[row.row];
    const uint32_t lo = max(B.m_lo, row.m_lo), hi = min(B.m_hi, row.m_hi);
    if (lo > hi) return false;
    // odd primes of l, one per lane
    const uint32_t p = lane < R.nodd ? inverse_odd(R.pinv[lane]) : 0u;
    // lane j: the bounds of the block's j-th range of roots.  phi0 grows and
    // phi1 falls with m, so the tightest are at its end, the widest at its start.
    {
        const uint32_t step = part_step(B.m_lo, B.m_hi);
        const uint32_t m0 = max(B.m_lo + lane * step, lo), m1 = min(B.m_lo + (lane + 1) * step - 1, hi);
        uint32_t a[4] = {0xFFFFFFFFu, 0xFFFFFFFFu, 0u, 0u};  // a range without roots of the row
        if (m0 <= m1) {
#pragma unroll
            for (uint32_t h = 0; h < 2; ++h) {
                const uint32_t m = h ? m0 : m1;
                const float mf = (float)m, m2f = mf * mf;
                float m4;
                const float w = window_low(row, m * row.p, m4);
                const float z = row.zscale * m2f;
                const float slack = (2e-6f * fabsf(w) + 0x1p-40f * m4) / z + 1e-7f;
                const float c0 = row.q0 / m2f * (h ? 1.000001f : 0.999999f), c1 = w / z + (h ? -slack : slack);
                const uint32_t t0 = (uint32_t)(acosf(fminf(c0, 1.f)) * 6.8356528e8f);  // 2^32 / (2 pi); below 2^30
                const float f1 = acosf(fminf(fmaxf(c1, -1.f), 1.f)) * 6.8356528e8f;
                const uint32_t t1 = f1 >= 2147483392.f ? kArcMax : (uint32_t)f1;
                if (h) {
                    a[1] = t0 < kAngleSlack ? 0u : t0 - kAngleSlack;
                    a[3] = t1 > kArcMax - kAngleSlack ? kArcMax : t1 + kAngleSlack;
                } else {
                    a[0] = t0 + kAngleSlack;
                    a[2] = t1 < kAngleSlack ? 0u : t1 - kAngleSlack;
                }
                if (c1 <= -1.f) a[h ? 3 : 2] = kArcMax;  // every D >= -|z| is inside
            }
        }
        range[lane] = make_uint4(a[0], a[1], a[2], a[3]);
        const bool some = m0 <= m1;
        const uint32_t b0 = __reduce_max_sync(kFull, some ? a[0] : 0u), b1 = __reduce_min_sync(kFull, a[1]);
        const uint32_t b2 = __reduce_min_sync(kFull, some ? a[2] : kArcMax), b3 = __reduce_max_sync(kFull, a[3]);
        if (lane == 0) {
            S.phi[0] = b0;
            S.phi[1] = b1;
            S.phi[2] = b2;
            S.phi[3] = b3;
        }
    }
    // entries that are not the row's: roots outside [m_lo, m_hi], or multiples
    // of an odd prime >= 7 of l
    const bool trim = B.m_lo < row.m_lo || B.m_hi > row.m_hi;
    // (p is prime to 60, so its multiples of the block's type are p times the
    // integers of that type)
    uint32_t r0 = 0, multiples = 0;
    if (p >= 7) {
        r0 = roots_upto(c_arc_types, B.type, (lo - 1) / p);
        multiples = roots_upto(c_arc_types, B.type, hi / p) - r0;
    }
    // Small primes have their bit sets ready, so that most rows gather little or
    // nothing: three rows at LIMIT 10^7 (l = 160,000) 8.1 ms without them and 5.1 ms
    // with, 37 near the limit 1.5 and 1.35; 512 rows, before their items were cut as
    // now, 125 and 121.
    uint32_t small = __ballot_sync(kFull, multiples != 0 && p <= mask_prime(kMaskPrimes - 1));
    const bool masks = small != 0;
    uint32_t pick = 0, picked = 0;  // which of them, four bits each
    for (; small; small &= small - 1) pick |= mask_of(__shfl_sync(kFull, p, __ffs(small) - 1)) << (4 * picked++);
    if (p <= mask_prime(kMaskPrimes - 1)) multiples = 0;
    const uint32_t incl_p = arc_scan(multiples, lane), all = __shfl_sync(kFull, incl_p, 31);
    const uint32_t words = (B.n + 31) / 32;
    const bool excl = trim || masks || all != 0;
    uint32_t marked = 0, marked_roots = 0;
    if (excl) {
        if (trim) {
            const uint32_t* m_at = cache.arc_m + B.base;
            for (uint32_t w0 = 0; w0 < words; w0 += 8) {
                uint32_t m[8];
#pragma unroll
                for (uint32_t q = 0; q < 8; ++q) {
                    const uint32_t i = 32 * (w0 + q) + lane;
                    m[q] = i < B.n ? m_at[i] : lo;
                }
#pragma unroll
                for (uint32_t q = 0; q < 8; ++q) {
                    const uint32_t word = __ballot_sync(kFull, m[q] < lo || m[q] > hi);
                    if (lane == q && w0 + q < words) bits[w0 + q] = word;
                }
            }
        } else {
            for (uint32_t i = lane; i < words; i += 32) bits[i] = 0;
        }
        __syncwarp();
        const uint32_t* mask = cache.arc_mask + (size_t)block * (kMaskPrimes * kMaskWords);
        for (uint32_t k = 0; k < picked; ++k) {
            const uint32_t* set = mask + ((pick >> (4 * k)) & 15u) * kMaskWords;
#pragma unroll
            for (uint32_t q = 0; q < kMaskWords / 32; ++q)
                if (32 * q + lane < words) bits[32 * q + lane] |= set[32 * q + lane];
        }
        __syncwarp();
        // multiples of the larger primes, 32 roots at a time; their records laid end to end
        for (uint32_t b0 = 0; b0 < all; b0 += 32) {
            const uint32_t own = arc_owner(incl_p, b0 + lane);
            const uint32_t q = __shfl_sync(kFull, p, own), k0 = __shfl_sync(kFull, r0, own);
            const uint32_t k = b0 + lane - __shfl_sync(kFull, incl_p - multiples, own);
            uint32_t s0 = 0, len = 0;
            if (b0 + lane < all) {
                const uint32_t m = q * nth_root(c_arc_types, B.type, k0 + k);
                s0 = cache.seg_off[m];
                len = cache.seg_off[m + 1] - s0;
            }
            const uint32_t incl = arc_scan(len, lane), total = __shfl_sync(kFull, incl, 31), ex = incl - len;
            for (uint32_t t0 = 0; t0 < total; t0 += 64) {
                uint32_t at[2];
#pragma unroll
                for (uint32_t h = 0; h < 2; ++h) {
                    const uint32_t t = t0 + 32 * h + lane, o = arc_owner(incl, t);
                    const uint32_t j = __shfl_sync(kFull, s0, o) + t - __shfl_sync(kFull, ex, o);
                    at[h] = t < total ? cache.pos[j] : 0xFFFFFFFFu;
                }
#pragma unroll
                for (uint32_t h = 0; h < 2; ++h)
                    if (at[h] != 0xFFFFFFFFu && index_ok(at[h], B.n, buf.error_flags))
                        atomicOr(&bits[at[h] >> 5], 1u << (at[h] & 31u));
            }
        }
        __syncwarp();
        // rank of the marked entries, per word of the bit set
        const uint32_t per = (words + 31) / 32, w0 = min(lane * per, words), w1 = min(w0 + per, words);
        uint32_t sum = 0;
        for (uint32_t i = w0; i < w1; ++i) sum += __popc(bits[i]);
        uint32_t at = arc_scan(sum, lane) - sum;
        for (uint32_t i = w0; i < w1; ++i) {
            rank[i] = (uint16_t)at;
            at += __popc(bits[i]);
        }
        if (lane == 31) rank[words] = (uint16_t)at;
        __syncwarp();
        marked = rank[words];
        marked_roots = arc_rank(bits, rank, B.list[9]) - arc_rank(bits, rank, B.list[8]);
    }
    // processed pairs: a root without a split prime only counts when l has one
    const bool bare = row.na == 1;
    uint32_t plain = 0;  // of the row's roots, those without a split prime
    if (bare) {
        plain = B.n_plain;
        if (excl) {
            uint32_t gone = 0;
            for (uint32_t i = B.list[8] + lane; i < B.list[9]; i += 32) {
                const uint32_t m = s_ang[i];
                if ((bits[i >> 5] >> (i & 31u)) & 1u) gone += cache.seg_off[m + 1] - cache.seg_off[m] == 1;
            }
            plain -= __reduce_add_sync(kFull, gone);
        }
    }
    out.processed = B.n_m - marked_roots - plain;
    out.records = B.n - marked - plain;
    // the all-central product (2 l^2 m^2, 0): its orientation D = 0 is counted
    // when 0 is in the window and the area 2 l^2 m^2 passes; z = l^4 + m^4 = 1 mod 16
    const bool three = (row.l_class & 4u) || (B.type & 2u), five = (row.l_class & 8u) || (B.type & 1u);
    const bool even = (row.l_class & 3u) || B.type >= 4;
    uint32_t cc = 0;
    if (three && five && even && row.cc_hi >= lo) {
        if (row.cc_hi >= hi) {
            cc = out.processed;
        } else {
            for (uint32_t i = B.list[8] + lane; i < B.list[9]; i += 32) {
                const uint32_t m = s_ang[i];
                if (m > row.cc_hi || (excl && ((bits[i >> 5] >> (i & 31u)) & 1u))) continue;
                cc += !(bare && cache.seg_off[m + 1] - cache.seg_off[m] == 1);
            }
            cc = __reduce_add_sync(kFull, cc);
        }
    }
    out.cc = cc;
    out.excl = excl;
    __syncwarp();
    return true;
}

// Events: terms that passed the filter, 32 at a time.  The lane forms its
// term's exact residues mod 9360 and 45917 and z's float bounds; the warp
// scans the candidate roots of all lanes together, and possible hits go to
// the exact kernel.
// Inlined at the kernel's two drains: no call in the kernel.
__device__ __forceinline__ void arc_events(uint32_t at, uint32_t v, uint32_t ev, bool live, const ArcCache& cache,
                                           const ArcBuffers& buf) {
    const uint32_t lane = threadIdx.x & 31, var = ev & 7u, ent = ev >> 3;
    uint32_t nlo = 1, nhi = 0, zres = 0, j = 0, m1 = 0, row_id = 0, m = 0, l = 0;
    if (live) {
        const ArcRow& row = buf.arc_rows[v];
        const RowInfo& R = buf.row_info[row.row];
        j = cache.arc_src[at];
        m1 = cache.arc_m[at];
        row_id = row.row;
        l = row.l;
        m = m1 * row.p;
        bool mine = m1 >= row.m_lo && m1 <= row.m_hi;
        // (3 and 5 are left to the block types)
        for (uint32_t t = 0; t < R.nodd; ++t) mine &= !divides(R.pinv[t], R.pthr[t], m1) || R.pthr[t] > 0xFFFFFFFFu / 7;
        if (mine) {
            const HotRec h = cache.hot[j], g = buf.arc_hot[ent];
            float gr = g.re, gi = g.im;
            arc_variant(var, gr, gi);
            const bool flip = h.im < 0.f;
            const float d = gr * h.re - gi * (flip ? -h.im : h.im);
            uint32_t z[2];
#pragma unroll
            for (uint32_t f = 0; f < 2; ++f) {
                const uint32_t M = f ? kModD : kModA, mask = f ? kMaskD : kMaskA, shift = f ? kShiftD : 0u;
                const uint32_t br = (h.rre >> shift) & mask, bi = (h.rim >> shift) & mask;
                uint32_t a = (g.rre >> shift) & mask, b = (g.rim >> shift) & mask;
                // variant of (a, b) with residues kept in [0, M)
                if (var & 4u) b = b ? M - b : 0u;
                if (var & 1u) {
                    const uint32_t t = a;
                    a = b ? M - b : 0u;
                    b = t;
                }
                if (var & 2u) {
                    a = a ? M - a : 0u;
                    b = b ? M - b : 0u;
                }
                const uint32_t im = flip && bi ? M - bi : bi;
                const uint32_t x = (a * br + M * M - b * im) % M;
                const uint32_t s = ((f ? R.lmodD : R.lmodA) + pow4_mod(m % M, M)) % M;
                z[f] = s >= x ? s - x : s + M - x;
            }
            zres = z[0] | z[1] << kShiftD;
            const uint8_t tab = buf.tables[kTabA + z[0]];
            const bool need5 = R.l % 5 != 0 && m % 5u != 0;
            if ((tab & (need5 ? 4u : 2u)) && tab_d(tab_d_bits(buf.tables, kTabD), z[1])) {
                const uint64_t m2 = (uint64_t)m * m;
                PairCtx c;
                c.sf = u128_to_float(R.l4 + (u128)m2 * m2);
                const float mf = (float)m1;
                c.eps = row.zscale * (mf * mf) * 0x1p-20f;
                c.m = m;
                root_window(c.sf - d, c, (uint32_t)cache.limit, nlo, nhi);
            }
        }
    }
    const uint32_t n0 = root_first(nlo, zres);
    const uint32_t mine = n0 <= nhi ? (nhi - n0) / 2 + 1 : 0u;
    uint32_t incl = mine;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const uint32_t t = __shfl_up_sync(kFull, incl, d);
        if (lane >= (uint32_t)d) incl += t;
    }
    const uint32_t total = __shfl_sync(kFull, incl, 31), excl = incl - mine;
    bool passed = false;
    for (uint32_t base = 0; base < total; base += 32) {
        const uint32_t s = base + lane;
        uint32_t owner = 0;
#pragma unroll
        for (uint32_t step = 16; step >= 1; step >>= 1) {
            const uint32_t t = __shfl_sync(kFull, incl, owner + step - 1);
            if (t <= s) owner += step;
        }
        owner &= 31u;
        const uint32_t from = __shfl_sync(kFull, n0, owner), z = __shfl_sync(kFull, zres, owner);
        const uint32_t off = s - __shfl_sync(kFull, excl, owner);
        uint32_t mm = __ballot_sync(kFull, s < total && root_match(from + 2u * off, z));
        while (mm) {  // rare: a possible root
            const uint32_t src = __ffs(mm) - 1;
            mm &= mm - 1;
            passed |= lane == __shfl_sync(kFull, owner, src);
        }
    }
    if (passed) {
        const unsigned int idx = atomicAdd(buf.exact_count, 1u);
        if (idx < buf.exact_cap)
            buf.exact_queue[idx] = ExactItem{kExHit | 32u, ent, j, l, m, row_id, v, var};
        else
            atomicOr(buf.error_flags, 4u);
    }
}

__device__ __forceinline__ uint32_t lower_bound_u32(const uint32_t* a, uint32_t lo, uint32_t hi, uint32_t x) {
    uint32_t n = hi - lo;
    while (n) {
        const uint32_t half = n >> 1;
        if (a[lo + half] < x) {
            lo += half + 1;
            n -= half + 1;
        } else {
            n = half;
        }
    }
    return lo;
}

// First entry of the list [first, end) at or after angle x (x < 2^31), from the
// list's bucket index.  The clamps keep every access inside the list whatever
// the bounds hold.
__device__ __forceinline__ uint32_t arc_find(const uint32_t* s_ang, const uint16_t* index, uint32_t first, uint32_t end,
                                             uint32_t x) {
    const uint32_t b = min(x >> kBucketShift, kBuckets - 1);
    const uint32_t lo = max((uint32_t)index[b], first), hi = min((uint32_t)index[b + 1], end);
    return lower_bound_u32(s_ang, min(lo, end), max(hi, min(lo, end)), x);
}

// The part of the arc start .. start + len (mod a turn) in the upper half turn.
__device__ __forceinline__ bool arc_piece(uint32_t start, uint32_t len, uint32_t& x, uint32_t& y) {
    const uint32_t end = start + len;
    if (start <= kArcMax) {
        x = start;
        y = end < start || end > kArcMax ? kArcMax : end;
        return true;
    }
    x = 0;
    y = end;
    return end < start;  // wrapped into the upper half
}

template <int NT>
__global__ void __launch_bounds__(NT, 1) arc_kernel(const __grid_constant__ ArcCache cache,
                                                       const ArcItem* __restrict__ items, uint32_t n_items,
                                                       const __grid_constant__ ArcBuffers buf) {
    constexpr uint32_t kWarps = NT / 32;
    extern __shared__ __align__(16) unsigned char smem[];
    ArcSmem<kWarps>& M = *reinterpret_cast<ArcSmem<kWarps>*>(smem);
    __shared__ ArcShared S;

    const uint32_t tid = threadIdx.x, lane = tid & 31;
    ArcWarp& W = M.warp[tid / 32];
    ArcSlot& T = W.slot;
    const uint32_t* s_ang = M.ang;
    const uint8_t* s_tab = M.tab;
    const uint16_t* index = reinterpret_cast<const uint16_t*>(M.index);
    uint32_t qn = 0;
    for (uint32_t i = tid; i < kArcTabBytes / 4; i += NT)
        reinterpret_cast<uint32_t*>(M.tab)[i] = reinterpret_cast<const uint32_t*>(buf.arc_tabs)[i];

    // processes the first n events, one per lane, and moves the rest up
    auto drain = [&](uint32_t n) {
        __syncwarp();
        const bool live = lane < n;
        const uint32_t a = live ? W.ev_at[lane] : 0u, b = live ? W.ev_row[lane] : 0u, c = live ? W.ev_id[lane] : 0u;
        const uint32_t rest = qn - n;  // at most 64
        uint32_t t[2][3] = {};
#pragma unroll
        for (uint32_t h = 0; h < 2; ++h)
            if (32 * h + lane < rest) {
                t[h][0] = W.ev_at[n + 32 * h + lane];
                t[h][1] = W.ev_row[n + 32 * h + lane];
                t[h][2] = W.ev_id[n + 32 * h + lane];
            }
        __syncwarp();
#pragma unroll
        for (uint32_t h = 0; h < 2; ++h)
            if (32 * h + lane < rest) {
                W.ev_at[32 * h + lane] = t[h][0];
                W.ev_row[32 * h + lane] = t[h][1];
                W.ev_id[32 * h + lane] = t[h][2];
            }
        __syncwarp();
        qn = rest;
        arc_events(a, b, c, live, cache, buf);
        __syncwarp();
    };
    // queues the lanes' events (all 32 lanes call it)
    auto push = [&](bool has, uint32_t at, uint32_t v, uint32_t id) {
        const uint32_t mask = __ballot_sync(kFull, has);
        if (has) {
            const uint32_t q = qn + __popc(mask & ((1u << lane) - 1u));
            W.ev_at[q] = at;
            W.ev_row[q] = v;
            W.ev_id[q] = id;
        }
        qn += __popc(mask);
    };

    if (tid == 0) S.ahead = atomicAdd(buf.next_item, 1u);
    for (;;) {
        __syncthreads();
        if (tid == 0) {
            S.item = S.ahead;
            S.next = 0;
        }
        __syncthreads();
        const uint32_t it = S.item;
        if (it >= n_items) break;
        const ArcItem w = items[it];
        if (tid < sizeof(ArcItem) / 4)
            reinterpret_cast<uint32_t*>(&S.rec)[tid] = reinterpret_cast<const uint32_t*>(items + it)[tid];
        if (tid < sizeof(ArcBlock) / 4)
            reinterpret_cast<uint32_t*>(&S.block)[tid] = reinterpret_cast<const uint32_t*>(cache.blocks + w.block)[tid];
        {
            // the block's four arrays, 16 bytes per asynchronous copy
            const uint32_t base = w.base, quads = (w.n + 15u) / 16 * 4;
#pragma unroll
            for (uint32_t arr = 0; arr < 4; ++arr) {
                const uint32_t* src = arr < 3 ? cache.arc_w[arr] : cache.arc_ang;
                for (uint32_t k = tid; k < quads; k += NT) {
                    const uint32_t dst = (uint32_t)__cvta_generic_to_shared(M.w0 + arr * kArcCap + 4 * k);
                    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src + base + 4 * k) : "memory");
                }
            }
            for (uint32_t k = tid; k < quads / 4; k += NT) {
                const uint32_t dst = (uint32_t)__cvta_generic_to_shared(M.part + 16 * k);
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(cache.arc_part + base + 16 * k) : "memory");
            }
            asm volatile("cp.async.commit_group;" ::: "memory");
            for (uint32_t k = tid; k < kIndexWords; k += NT)
                M.index[k] = cache.arc_index[(size_t)w.block * kIndexWords + k];
        }
        // the next item, and its block towards L2 while this one runs
        if (tid == NT - 1) {
            const uint32_t ahead = atomicAdd(buf.next_item, 1u);
            S.ahead = ahead;
            if (ahead < n_items) {
                const ArcItem x = items[ahead];
                const uint32_t quads = (x.n + 3u) / 4;
                if (x.block != w.block && quads) {
                    // (whole quads: 16-byte sizes, from 16-byte boundaries)
#pragma unroll
                    for (uint32_t f = 0; f < kFields; ++f) arc_prefetch(cache.arc_w[f] + x.base, quads);
                    arc_prefetch(cache.arc_ang + x.base, quads);
                    arc_prefetch(reinterpret_cast<const uint32_t*>(cache.arc_part + x.base), (x.n + 15u) / 16);
                    arc_prefetch(cache.arc_mask + (size_t)x.block * (kMaskPrimes * kMaskWords), kMaskPrimes * kMaskWords / 4);
                    arc_prefetch(cache.arc_index + (size_t)x.block * kIndexWords, kIndexWords / 4);
                    arc_prefetch(reinterpret_cast<const uint32_t*>(cache.blocks + x.block), sizeof(ArcBlock) / 16);
                }
            }
        }
        asm volatile("cp.async.wait_all;" ::: "memory");
        __syncthreads();
        const ArcBlock& B = S.block;
        const uint32_t type = B.type, block0 = B.base;
        // warps take rows (or parts of rows) on their own
        const uint32_t shared = S.rec.split * S.rec.parts, units = (shared + S.rec.nv - S.rec.split) * S.rec.share;
        for (;;) {
            uint32_t unit = 0;
            if (lane == 0) unit = atomicAdd(&S.next, 1u);
            unit = __shfl_sync(kFull, unit, 0);
            if (unit >= units) break;
            // of the runs of a group, this warp's: lanes = turn mod share
            const uint32_t turn = unit % S.rec.share;
            const uint32_t mask_mine = kFull / ((S.rec.share < 32 ? 1u << S.rec.share : 0u) - 1u) << turn;  // share a power of two
            unit /= S.rec.share;
            const bool whole = unit >= shared;
            const uint32_t parts = whole ? 1u : S.rec.of, part = whole ? 0u : S.rec.from + unit % S.rec.parts;
            const uint32_t v = S.rec.v0 + (whole ? unit - shared + S.rec.split : unit / S.rec.parts);
            __syncwarp();
            if (lane < sizeof(ArcRow) / 4)
                reinterpret_cast<uint32_t*>(&T.row)[lane] = reinterpret_cast<const uint32_t*>(buf.arc_rows + v)[lane];
            __syncwarp();
            // class rules of the row against the block's type; l and m' have no
            // common factor 2, 3 or 5
            const uint32_t lc = T.row.l_class;
            if (((lc & 3u) && type >= 4) || ((lc & 4u) && (type & 2u)) || ((lc & 8u) && (type & 1u))) continue;
            {
                const uint32_t defined = (type < 4 ? 4u : 0u) | ((type & 2u) ? 0u : 2u) | ((type & 1u) ? 0u : 1u);
                const uint32_t match = defined & (((lc & 4u) ? 0u : 2u) | ((lc & 8u) ? 0u : 1u));
                const bool odd = type < 4 && (lc & 3u) == 0;
                const bool always = (lc & 3u) == 2u || type >= 8u;  // even pairs: z = 1 mod 16 whatever D
                const uint32_t lu = odd ? 1u : 2u, lt = __popc(defined & ~match) + 2u + lu;
                const uint32_t runs1 = T.row.na << lt, runs2 = (T.row.na - 1) << lu;
                if (32 * part >= runs1 + runs2) continue;  // no runs left for this part
                // (kept in shared memory, away from the filter's registers)
                if (lane == 0) T.row.rules = match | (defined & ~match) << 3 | (odd ? 64u : 0u) | (always ? 128u : 0u) | lt << 8;
            }
            ArcCounts counts;
            if (!arc_prepare(cache, buf, B, S.rec.block, s_ang, T, W.bits, W.rank, W.range, lane, counts)) continue;
            const bool excl = counts.excl;
            const uint32_t k0[kFields] = {T.row.c0[0], T.row.c0[1], T.row.c0[2]};
            auto marked = [&](uint32_t i) { return ((W.bits[i >> 5] >> (i & 31u)) & 1u) != 0; };
            if (lane == 0) W.cand = W.r16 = 0;
            uint32_t open_n = 0;  // the unit's terms awaiting their own root's window
            auto await = [&](bool has, uint32_t i, uint32_t id) {
                const uint32_t mask = __ballot_sync(kFull, has);
                if (has) {
                    const uint32_t e = open_n + __popc(mask & ((1u << lane) - 1u));
                    W.open_at[e] = i;
                    W.open_id[e] = id;
                }
                open_n += __popc(mask);
            };
            auto runs_of_row = [&] { return (T.row.na << (T.row.rules >> 8)) + ((T.row.na - 1) << ((T.row.rules & 64u) ? 1 : 2)); };
            for (uint32_t t0 = 32 * part; t0 < runs_of_row(); t0 += 32 * parts) {
                uint32_t t = t0 + lane;
                const uint32_t rules = T.row.rules, na = T.row.na, ent0 = T.row.ent;
                const uint32_t match = rules & 7u, open = (rules >> 3) & 7u, lt = rules >> 8;
                const bool odd = (rules & 64u) != 0, always = (rules & 128u) != 0;
                const uint32_t lu = odd ? 1u : 2u, runs1 = na << lt;
                // the lane's run: possible [p0, p1), certain [c0, c1)
                uint32_t p0 = 0, p1 = 0, c0 = 0, c1 = 0, id = 0, ang0 = 0;
                bool keep = false;  // z = 0, 1 mod 16
                if (t < runs1) {
                    uint32_t sub = 0;
                    {
                        uint32_t bitsel = open;
                        while (bitsel) {
                            const uint32_t b = bitsel & (0u - bitsel);
                            if (t & 1u) sub |= b;
                            t >>= 1;
                            bitsel &= bitsel - 1;
                        }
                    }
                    const uint32_t lower = t & 1u, conj = (t >> 1) & 1u;
                    t >>= 2;
                    const uint32_t u = odd ? (t & 1u) * 2u : t & 3u;
                    const uint32_t k = t >> lu;
                    if (k + 1 < na || !conj) {
                        const uint2 g = *reinterpret_cast<const uint2*>(buf.arc_values + ent0 + k);
                        const uint32_t cls = g.y ^ ((u & 1u) ? 3u : 0u) ^ ((u & 2u) ? 4u : 0u);
                        sub |= cls & match;
                        keep = odd ? ((cls ^ sub) & 4u) == 0 : (always || (u & 1u) != 0);
                        const uint32_t ga = (conj ? 0u - g.x : g.x) + (u << 30);
                        id = (ent0 + k) << 3 | conj << 2 | u;
                        ang0 = lower ? ~ga : ga;  // an entry of angle a is at ang0 -+ a
                        if (lower) id |= kRunLower;
                        const uint16_t* ix = index + sub * (kBuckets + 2);
                        const uint32_t lo = B.list[sub], hi = B.list[sub + 1];
                        const uint32_t p0c = T.phi[0], p0p = T.phi[1], p1c = T.phi[2], p1p = T.phi[3];
                        uint32_t x, y;
                        const uint32_t startp = lower ? (p1p == kArcMax ? 0x80000000u : 0u - p1p) : p0p;
                        if (hi > lo && p1p >= p0p && arc_piece(startp - ga, p1p - p0p, x, y)) {
                            p0 = arc_find(s_ang, ix, lo, hi, x);
                            p1 = y >= kArcMax ? hi : max(p0, arc_find(s_ang, ix, lo, hi, y + 1u));
                            c0 = c1 = p0;
                            uint32_t cx, cy;
                            if (p1 > p0 && p1c >= p0c &&
                                arc_piece((lower ? (p1c == kArcMax ? 0x80000000u : 0u - p1c) : p0c) - ga, p1c - p0c, cx, cy)) {
                                c0 = s_ang[p0] >= cx ? p0 : min(p1, max(p0, arc_find(s_ang, ix, lo, hi, cx)));
                                c1 = s_ang[p1 - 1] <= cy ? p1 : min(p1, max(c0, arc_find(s_ang, ix, lo, hi, cy + 1u)));
                            }
                        }
                    }
                } else if (t < runs_of_row()) {
                    t -= runs1;
                    const uint32_t u = odd ? (t & 1u) * 2u : t & 3u, k = t >> lu;
                    const uint32_t cls = buf.arc_values[ent0 + k].cls ^ ((u & 1u) ? 3u : 0u) ^ ((u & 2u) ? 4u : 0u);
                    if ((cls & match & 3u) == 0) {
                        keep = odd ? (cls & 4u) == 0 : (always || (u & 1u) != 0);
                        const uint32_t ga = buf.arc_values[ent0 + k].ang + (u << 30);
                        ang0 = min((int32_t)ga < 0 ? 0u - ga : ga, kArcMax);
                        id = (ent0 + k) << 3 | u | kRunCentral;
                        if (ang0 >= T.phi[1] && ang0 <= T.phi[3]) {
                            p0 = c0 = c1 = B.list[8];
                            p1 = B.list[9];
                            if (ang0 >= T.phi[0] && ang0 <= T.phi[2]) c1 = p1;
                        }
                    }
                }
                // A run with many undecided terms is checked term by term;
                // else its certain part counts by position, and the filter
                // reads it without a check.
                const uint32_t doubt = (p1 - p0) - (c1 - c0);
                const bool wide = keep && doubt > kArcWide;
                uint32_t n = wide ? 0u : c1 - c0;
                if (excl && n) n -= arc_rank(W.bits, W.rank, c1) - arc_rank(W.bits, W.rank, c0);
                if (turn != 0) n = 0;  // counted by the first of the sharing warps
                uint32_t cand32 = __reduce_add_sync(kFull, n), r32 = __reduce_add_sync(kFull, keep ? n : 0u);
                // Each lane lays its run out in shared memory, so that starting
                // a run costs the warp a few broadcast loads.
                __syncwarp();
                if (p1 > p0) {
                    uint4* st = reinterpret_cast<uint4*>(W.stage + lane * kStageWords);
                    if (keep) {
                        const ArcFilter f = arc_filter(buf.arc_values[(id & kRunId) >> 3], id & 7u, T.row);
                        st[0] = make_uint4(f.c1[0], f.c1[1], f.c1[2], 0u);
                        st[1] = make_uint4(f.c2[0], f.c2[1], f.c2[2], 0u);
                    }
                    if (keep) id |= kRunKeep;
                    st[2] = make_uint4(id, ang0, p0 | c0 << 16, c1 | p1 << 16);
                }
                __syncwarp();
                uint32_t todo = __ballot_sync(kFull, keep && (wide || c1 > c0)) & mask_mine;
                const uint32_t checked = __ballot_sync(kFull, wide);
                const uint32_t mine = wide || turn != 0 ? 0u : doubt;  // the lane's other undecided terms
                uint32_t incl = mine, total = 0;
                if (__any_sync(kFull, mine != 0)) {
                    incl = arc_scan(mine, lane);
                    total = __shfl_sync(kFull, incl, 31);
                }
                const uint32_t ex = incl - mine;
                // the multipliers of a staged run
                auto staged = [&](uint32_t src) {
                    const uint4* st = reinterpret_cast<const uint4*>(W.stage + src * kStageWords);
                    const uint4 x = st[0], y = st[1];
                    ArcFilter f{{k0[0], k0[1], k0[2]}, {x.x, x.y, x.z}, {y.x, y.y, y.z}, {}};
#pragma unroll
                    for (uint32_t q = 0; q < kFields; ++q) f.c3[q] = T.row.c3[q] - ((f.c2[q] + (f.c1[q] << 10)) << 10);
                    return f;
                };
                // an entry's place in the row's arc (0 .. kArcMax: the half turn
                // of its run), against the bounds of its root's range
                auto place = [&](uint32_t i, uint32_t tag, uint32_t a0, bool& in, bool& doubtful) {
                    const uint32_t a = (tag & kRunCentral) ? 0u : M.ang[i];
                    const uint32_t x = (tag & kRunLower) ? a0 - a : a0 + a;
                    const uint4 r = W.range[M.part[i]];
                    in = x >= r.x && x <= r.z;
                    doubtful = !in && x >= r.y && x <= r.w;
                };
                const bool final = t0 + 32 * parts >= runs_of_row();  // the unit's last runs
                uint32_t at = 0, end = 0, tag = 0, ang_run = 0, base = 0;
                bool check = false;
                ArcFilter c{};
                for (;;) {
                    const bool runs = at < end || todo != 0, last = !runs && base >= total;
                    if (open_n >= 32 || (last && final && open_n != 0)) {
                        // terms that their range leaves open, each against its own root's window
                        const uint32_t take = min(open_n, 32u), rest = open_n - take;
                        __syncwarp();
                        const uint32_t i = lane < take ? W.open_at[lane] : 0u, fid = lane < take ? W.open_id[lane] : 0u;
                        const uint32_t more_at = lane < rest ? W.open_at[32 + lane] : 0u, more_id = lane < rest ? W.open_id[32 + lane] : 0u;
                        __syncwarp();
                        if (lane < rest) {
                            W.open_at[lane] = more_at;
                            W.open_id[lane] = more_id;
                        }
                        __syncwarp();
                        open_n = rest;
                        bool in = false, has = false;
                        if (lane < take && !(excl && marked(i))) {
                            const float2 b = cache.arc_xy[block0 + i];
                            const uint32_t m1 = cache.arc_m[block0 + i], m = m1 * T.row.p;
                            const float2 g = *reinterpret_cast<const float2*>(buf.arc_hot + ((fid & kRunId) >> 3));
                            float gr = g.x, gi = g.y;
                            arc_variant(fid & 7u, gr, gi);
                            const float l4 = T.row.q0 * T.row.zscale;  // l^4
                            const float mf = (float)m1, eps = T.row.zscale * (mf * mf) * 0x1p-20f;
                            const float d = gr * b.x - gi * b.y;
                            float m4;
                            const float lowf = window_low(T.row, m, m4);
                            const float e1 = eps + l4 * 0x1p-21f, e2 = eps + fabsf(lowf) * 0x1p-21f + m4 * 0x1p-42f;
                            in = d <= l4 - e1 && d >= lowf + e2;
                            if (!in && d <= l4 + e1 && d >= lowf - e2) {
                                const unsigned int x = atomicAdd(buf.exact_count, 1u);
                                if (x < buf.exact_cap)
                                    buf.exact_queue[x] = ExactItem{kExCount | 32u, (fid & kRunId) >> 3, cache.arc_src[block0 + i],
                                                                   T.row.l, m, T.row.row, v, fid & 7u};
                                else
                                    atomicOr(buf.error_flags, 4u);
                            }
                            if (in && (fid & kRunKeep)) {
                                const ArcFilter f = arc_filter(buf.arc_values[(fid & kRunId) >> 3], fid & 7u, T.row);
                                has = arc_test(M.w0 + i, f, s_tab) != 0;
                            }
                        }
                        cand32 += __popc(__ballot_sync(kFull, in));
                        r32 += __popc(__ballot_sync(kFull, in && (fid & kRunKeep)));
                        if (__any_sync(kFull, has)) push(has, block0 + i, v, fid & kRunId);
                    } else if (runs) {
                        if (at >= end) {  // the next run
                            const uint32_t run = __ffs(todo) - 1;
                            todo &= todo - 1;
                            check = ((checked >> run) & 1u) != 0;
                            const uint4 z = reinterpret_cast<const uint4*>(W.stage + run * kStageWords)[2];
                            tag = z.x;
                            ang_run = z.y;
                            at = check ? z.z & 0xFFFFu : z.z >> 16;
                            end = check ? z.w >> 16 : z.w & 0xFFFFu;
                            c = staged(run);
                        }
                        if (!check) {
                            // rounds of 64 terms, the last with its end checked
                            const uint32_t* w = M.w0 + lane;
                            bool h0 = false, h1 = false, any = false;
                            uint32_t from = at;
                            while (at < end) {
                                from = at;
                                const uint32_t* x = w + at;
                                uint32_t q0 = arc_test(x, c, s_tab), q1 = 0;
                                if (at + 32 < end) q1 = arc_test(x + 32, c, s_tab);
                                at += 64;
                                h0 = q0 != 0 && from + lane < end;
                                h1 = q1 != 0 && from + lane + 32 < end;
                                any = __any_sync(kFull, h0 || h1);
                                if (any) break;
                            }
                            if (any) {
                                push(h0, block0 + from + lane, v, tag & kRunId);
                                push(h1, block0 + from + lane + 32, v, tag & kRunId);
                            }
                        } else {
                            bool has = false, any = false;
                            uint32_t i = 0;
                            while (at < end) {
                                i = at + lane;
                                bool in = false, doubtful = false;
                                if (i < end && !(excl && marked(i))) place(i, tag, ang_run, in, doubtful);
                                const uint32_t q = arc_test(M.w0 + i, c, s_tab);
                                at += 32;
                                const uint32_t inside = __popc(__ballot_sync(kFull, in));
                                cand32 += inside;
                                r32 += inside;
                                has = in && q != 0;
                                any = __any_sync(kFull, has);
                                await(doubtful, i, tag);
                                if (any || open_n >= 32) break;
                            }
                            if (any) push(has, block0 + i, v, tag & kRunId);
                        }
                    } else if (base < total) {
                        // undecided terms of the other runs, all lanes' end to end
                        const uint32_t q = base + lane;
                        base += 32;
                        const uint32_t own = arc_owner(incl, q), off = q - __shfl_sync(kFull, ex, own);
                        bool in = false, doubtful = false, has = false;
                        uint32_t i = 0, fid = 0;
                        if (q < total) {
                            const uint4 z = reinterpret_cast<const uint4*>(W.stage + own * kStageWords)[2];
                            fid = z.x;
                            i = (z.z & 0xFFFFu) + off;
                            if (i >= z.z >> 16) i += (z.w & 0xFFFFu) - (z.z >> 16);  // past the certain part
                            if (!(excl && marked(i))) place(i, fid, z.y, in, doubtful);
                            if (in && (fid & kRunKeep)) has = arc_test(M.w0 + i, staged(own), s_tab) != 0;
                        }
                        cand32 += __popc(__ballot_sync(kFull, in));
                        r32 += __popc(__ballot_sync(kFull, in && (fid & kRunKeep)));
                        await(doubtful, i, fid);
                        if (__any_sync(kFull, has)) push(has, block0 + i, v, fid & kRunId);
                    } else {
                        break;
                    }
                    while (qn >= 32) drain(32);
                }
                if (lane == 0) {
                    W.cand += cand32;
                    W.r16 += r32;
                }
            }
            if (lane == 0) {
                unsigned long long cand = W.cand, r16 = W.r16;
                RowCounts* rc = &buf.rows[T.row.row];
                const bool shared_prime = T.row.p != 1;
                if (part == 0 && turn == 0) {
                    cand += counts.cc;
                    r16 += counts.cc;
                    const unsigned long long products =
                        (2ull * T.row.na - 1) * counts.records - (unsigned long long)(T.row.na - 1) * counts.processed;
                    if (counts.processed) {
                        atomicAdd(&rc->processed, (unsigned long long)counts.processed);
                        atomicAdd(&rc->products, products);
                        if (shared_prime) {
                            atomicAdd(&rc->merged, (unsigned long long)counts.processed);
                            atomicAdd(&rc->mproducts, products);
                        }
                    }
                }
                if (cand) {
                    atomicAdd(&rc->candidates, cand);
                    if (shared_prime) atomicAdd(&rc->mcandidates, cand);
                }
                if (r16) {
                    atomicAdd(&rc->r16, r16);
                    if (shared_prime) atomicAdd(&rc->mr16, r16);
                }
            }
        }
    }
    while (qn) drain(qn < 32 ? qn : 32);
}

// The values of one arc row per CTA: the free set of l P and its central
// value, exact from the prime-power table.
__device__ void arc_group(const DeviceCache& cache, const RowInfo& R, uint32_t p, Group& g) {
    g.count = R.nsplit;
    uint32_t rest = p;
    for (uint32_t i = 0; i < R.nsplit; ++i) {
        uint32_t e = R.se[i];
        while (rest % R.sp[i] == 0) {
            rest /= R.sp[i];
            ++e;
        }
        g.e[i] = e;
        g.base[i] = cache.pp_base[R.sp[i]] + pp_exponent_offset(e);
    }
    group_finish(g);
    g.scale = (i128)2 * (i128)R.fixed;
}

__global__ void __launch_bounds__(64) arc_value_kernel(const DeviceCache cache, const ArcBuffers buf) {
    __shared__ Group g;
    const ArcRow row = buf.arc_rows[blockIdx.x];
    const RowInfo& R = buf.row_info[row.row];
    if (threadIdx.x == 0) {
        arc_group(cache, R, row.p, g);
        if (g.free_count + 1 != row.na) atomicOr(buf.error_flags, kErrIndex);
    }
    __syncthreads();
    for (uint32_t k = threadIdx.x; k < row.na; k += blockDim.x) {
        i128 re, im;
        group_value(cache, g, k, re, im);
        ArcValue a;
        HotRec h;
        h.re = i128_to_float(re);
        h.im = i128_to_float(im);
        h.rre = pack_residues(re) | (k + 1 == row.na ? kCentralBit : 0u);
        h.rim = pack_residues(im);
        const float th = atan2f(h.im, h.re);
        a.ang = (uint32_t)(int32_t)__float2int_rn(th * 6.8356528e8f);
        // classes of alpha = value / 2 (odd rows for s8): 3 and 5 see the
        // doubled value alike, mod 8 the half is taken mod 16
        const uint32_t re16 = (h.rre & kMaskA) & 15u;
        a.cls = ((re16 >> 1) == 7u ? 4u : 0u) | ((h.rim & kMaskA) % 3u ? 2u : 0u) | ((h.rim & kMaskA) % 5u ? 1u : 0u);
#pragma unroll
        for (uint32_t f = 0; f < kFields; ++f) {
            a.re[f] = field_scale(f) * mod_i128(re, field_mod(f));
            a.im[f] = field_scale(f) * mod_i128(im, field_mod(f));
        }
        buf.arc_values[row.ent + k] = a;
        buf.arc_hot[row.ent + k] = h;
    }
}

// Shared-prime pairs of the rest list: the skip rules of the reference
// (both even, a common inert prime), the common part exactly P.
__global__ void __launch_bounds__(128) arc_rest_kernel(const DeviceCache cache, const ArcRest* __restrict__ rest,
                                                       uint32_t n, const LaunchBuffers buf) {
    for (uint32_t i = blockIdx.x; i < n; i += gridDim.x) {
        const ArcRest e = rest[i];
        const RowInfo& R = buf.row_info[e.row];
        for (uint32_t m = e.m_lo + threadIdx.x; m <= e.m_hi; m += blockDim.x) {
            if (R.leven && (m & 1u) == 0) continue;
            bool mine = true;
            for (uint32_t t = 0; t < R.nodd; ++t) mine &= !divides(R.pinv[t], R.pthr[t], m);
            if (!mine) continue;
            push_merged(buf, e.l, e.p * m, e.row);
            RowCounts* rc = &buf.rows[e.row];
            atomicAdd(&rc->processed, 1ull);
            atomicAdd(&rc->merged, 1ull);
        }
    }
}

// Exact evaluation of one term of an arc row.
__device__ __noinline__ void arc_exact_term(const DeviceCache& cache, const ArcBuffers& buf, const ExactItem& it,
                                            const uint8_t* tab, uint32_t* cand, uint32_t* r16) {
    const ArcRow row = buf.arc_rows[it.arc_row];
    Group g;
    arc_group(cache, buf.row_info[row.row], row.p, g);
    i128 gr, gi;
    group_value(cache, g, it.a - row.ent, gr, gi);
    if (it.variant & 4u) gi = -gi;
    if (it.variant & 1u) {
        const i128 t = gr;
        gr = -gi;
        gi = t;
    }
    if (it.variant & 2u) {
        gr = -gr;
        gi = -gi;
    }
    const ExactRec b = cache.exact[it.b];
    const i128 br = b.re, bi = b.im < 0 ? -(i128)b.im : (i128)b.im;
    const i128 d = gr * br - gi * bi, area4 = gr * bi + gi * br;
    const ExactPair p = exact_pair(it.l, it.m, cache.limit, it.row);
    uint32_t c = 0, r = 0;
    if (d >= p.lower && d <= p.upper && area4 != 0) exact_test_d(p, d, area4, c, r, tab, buf);
    *cand = c;
    *r16 = r;
}
