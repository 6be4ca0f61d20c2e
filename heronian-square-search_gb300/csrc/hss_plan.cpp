// hss_plan.cpp - rows and work items of the arc path (host side).
#include "hss_plan.h"

#include <math.h>

#include <algorithm>

namespace hss {
namespace {

constexpr size_t kMergedRows = 64;  // most rows of an item of several groups
constexpr uint64_t kSmallItem = 300;    // items are not cut below this cost for balance alone (100: 2 % and up to 30 % at small limits)
constexpr uint64_t kMergedCost = 1000;  // and their cost at most (400 and 4,000: within 2 %)

using u128 = unsigned __int128;
using i128 = __int128;

uint64_t fourth_root(u128 x) {
    uint64_t r = (uint64_t)sqrt(sqrt((double)x));
    while (r > 0 && (u128)r * r * r * r > x) --r;
    while ((u128)(r + 1) * (r + 1) * (r + 1) * (r + 1) <= x) ++r;
    return r;
}

}  // namespace

// A row (l, P) costs its value list and a visit to every block of its range; the
// shared-prime kernels set every pair up by itself, and cost three launches
// that wait for one another.  Few rows: no shared-prime launch at all (37 roots at
// LIMIT 10^7 1.34 ms against 1.81 ms with 48 roots, one at 70,000 0.15 against 0.22 ms).
// Many: 48 (512 roots at 10^7 106.1 ms, against 109.6 ms with 1 and 106.3 with 150), at small
// limits, whose blocks hold fewer roots each, 150 (2,001 roots at 20,000 5.4 ms against 5.8 ms with 48).
uint64_t min_roots(uint64_t limit, size_t rows) { return rows <= 64 ? 1 : limit < 1000000 ? 150 : 48; }

void ArcPlanner::clear() {
    rows.clear();
    rest.clear();
    items.clear();
    keys_.clear();
    entries = rest_pairs = 0;
}

void ArcPlanner::add(const RowInfo& R, uint32_t row, uint64_t limit, uint32_t max_exponent, uint64_t m0, uint64_t m1,
                     uint64_t least) {
    const uint64_t l = R.l;
    m0 = std::max(m0, l);
    m1 = std::min(m1, limit);
    if (m0 > m1) return;
    const uint64_t zero_hi = R.n4 > R.l4 ? fourth_root(R.n4 - R.l4) : 0;  // largest m with w <= 0
    const i128 lw = (i128)R.l4 - (i128)R.n4;
    const float lw_hi = i128_to_float(lw), lw_lo = i128_to_float(lw - (i128)lw_hi);
    uint32_t c0[kFields];
    for (uint32_t f = 0; f < kFields; ++f) {
        const uint32_t M = field_mod(f), r = (uint32_t)(l % M), r2 = r * r % M;
        c0[f] = field_scale(f) * (r2 * r2 % M);
    }
    const uint32_t l_class = ((l & 1) ? 0u : (l & 3) ? 1u : 2u) | (R.l3 ? 4u : 0u) | (R.l5 ? 8u : 0u);
    // every P, depth first over the split primes: (P, number of values, prime)
    struct Part {
        uint64_t p, w;
        uint32_t i;
        bool fits;
    };
    Part stack[64];
    int top = 0;
    stack[top++] = Part{1, 2ull * R.free_l + 1, 0, true};
    while (top) {
        const Part s = stack[--top];
        if (s.i < R.nsplit) {
            const uint64_t p = R.sp[s.i], e = R.se[s.i];
            stack[top++] = Part{s.p, s.w, s.i + 1, s.fits};
            uint64_t q = s.p;
            for (uint64_t a = 1; q <= limit / p; ++a) {
                q *= p;
                if (q > m1) break;
                // no room for a multiple of q in [m0, m1] does not exclude a
                // further power: every q <= m1 is visited
                stack[top++] = Part{q, s.w / (4 * e + 1) * (4 * (e + a) + 1), s.i + 1, s.fits && e + a <= max_exponent};
            }
            continue;
        }
        const uint64_t lo = (m0 + s.p - 1) / s.p, hi = m1 / s.p;
        if (lo > hi) continue;
        if (s.p != 1 && (!s.fits || hi - lo + 1 < least)) {
            rest.push_back(ArcRest{row, (uint32_t)l, (uint32_t)s.p, (uint32_t)lo, (uint32_t)hi});
            rest_pairs += hi - lo + 1;
            continue;
        }
        ArcRow a{};
        a.row = row;
        a.p = (uint32_t)s.p;
        a.m_lo = (uint32_t)lo;
        a.m_hi = (uint32_t)hi;
        a.na = (uint32_t)((s.w + 1) / 2);
        a.cc_hi = (uint32_t)(zero_hi / s.p);
        a.l = (uint32_t)l;
        const double p2 = (double)s.p * (double)s.p, l2 = (double)R.l2;
        a.q0 = (float)(l2 / (2.0 * p2));
        a.zscale = (float)(2.0 * l2 * p2);
        a.lw_hi = lw_hi;
        a.lw_lo = lw_lo;
        a.l_class = l_class;
        for (uint32_t f = 0; f < kFields; ++f) {
            const uint32_t M = field_mod(f), p1 = (uint32_t)s.p % M, p2m = p1 * p1 % M;
            a.c0[f] = c0[f];
            a.c3[f] = field_scale(f) * (p2m * p2m % M);
        }
        entries += a.na;
        keys_.push_back((uint64_t)s.p << 3 | ((l_class & 3) ? 4u : 0u) | (R.l3 ? 2u : 0u) | (R.l5 ? 1u : 0u));
        rows.push_back(a);
    }
}

// Rows by (P, parity, divisibility by 3 and 5), those of many values first.
bool ArcPlanner::sort() {
    const size_t n = rows.size();
    order_.clear();
    sorted_.clear();
    order_.resize(n);
    sorted_.resize(n);
    if (order_.over() || sorted_.over() || keys_.over()) return false;
    for (size_t i = 0; i < n; ++i) order_[i] = Order{keys_[i], (uint64_t)(UINT32_MAX - rows[i].na) << 32 | i};
    std::sort(order_.begin(), order_.end(),
              [](const Order& x, const Order& y) { return x.key != y.key ? x.key < y.key : x.rest < y.rest; });
    for (size_t i = 0; i < n; ++i) {
        sorted_[i] = rows[(uint32_t)order_[i].rest];
        keys_[i] = order_[i].key;
    }
    rows.swap(sorted_);
    return true;
}

void ArcPlanner::take(const ArcPlanner& from, size_t i0, size_t i1) {
    clear();
    for (size_t i = i0; i < i1; ++i) {
        rows.push_back(from.rows[i]);
        keys_.push_back(from.keys_[i]);
        entries += from.rows[i].na;
    }
}

bool ArcPlanner::finish(const ArcPlan& plan, uint32_t ctas, uint64_t item_target) {
    items.clear();
    groups_.clear();
    if (rows.over() || keys_.over() || rest.over() || entries > kArcValuesMost) return false;
    if (rows.empty()) return true;
    if (!sort()) return false;
    uint32_t ent = 0;
    for (size_t i = 0; i < rows.size(); ++i) {
        rows[i].ent = ent;
        ent += rows[i].na;
    }
    const Store<uint64_t>& keys = keys_;
    // the blocks of a type whose roots meet [lo, hi]
    auto range_of = [&](uint32_t t, uint32_t lo, uint32_t hi, uint32_t* b0, uint32_t* b1) {
        const uint32_t end = plan.type_first[t + 1];
        const uint32_t* start = plan.start[t].data();
        uint32_t x = start[lo >> plan.start_shift], y;
        while (x < end && plan.blocks[x].m_hi < lo) ++x;
        y = std::max(x, start[hi >> plan.start_shift]);
        while (y < end && plan.blocks[y].m_lo <= hi) ++y;
        *b0 = x;
        *b1 = y;
    };
    auto type_allowed = [](uint64_t key, uint32_t t) {
        return !((key & 4u) && t >= 4) && !((key & 2u) && (t & 2u)) && !((key & 1u) && (t & 1u));
    };
    auto cost = [](const ArcRow& r) { return (uint64_t)r.na + 16; };
    uint64_t total = 0;
    for (size_t g0 = 0; g0 < rows.size();) {
        size_t g1 = g0;
        uint64_t w = 0;
        uint32_t lo = rows[g0].m_lo, hi = 0;
        while (g1 < rows.size() && keys[g1] == keys[g0]) {
            w += cost(rows[g1]);
            lo = std::min(lo, rows[g1].m_lo);
            hi = std::max(hi, rows[g1].m_hi);
            ++g1;
        }
        Group g{};
        g.g0 = g0;
        g.g1 = g1;
        g.cost = w;
        for (uint32_t t = 0; t < kTypes; ++t) {
            if (!type_allowed(keys[g0], t)) continue;
            range_of(t, lo, hi, &g.b0[t], &g.b1[t]);
            total += w * (g.b1[t] - g.b0[t]);
        }
        groups_.push_back(g);
        g0 = g1;
    }
    if (groups_.over()) return false;
    // Item size: the caller's, or a sixty-fourth of a CTA's work, but not below
    // kSmallItem unless that leaves a CTA fewer than twelve items.  With twelve items
    // in every call the last ones ran alone, and CTAs worked 77 % of the time of 64 rows
    // at LIMIT 10^6 (15.1 ms, now 11.4), 81 % of 16,384 rows' at 10^5 (154 ms, 128), 83 % of
    // root 6,325,815's (branch weight 625) at 10^7 (25 ms, 22).
    const uint64_t share12 = total / ((uint64_t)ctas * 12), share64 = total / ((uint64_t)ctas * 64);
    // A caller's size is not followed below a 2^17th of the launch's work: each
    // item is 32 bytes of host and device memory (3,000 rows at LIMIT 10^5 would make
    // 480,000 of cost 16), and callers without the power to allocate have room for 2^18.
    const uint64_t target = std::max<uint64_t>(
        16, item_target ? std::max(item_target, total >> 17) : std::max(share64, std::min<uint64_t>(share12, kSmallItem)));
    const uint64_t merged = std::min(std::max(target, std::min<uint64_t>(total / ctas, 400)), kMergedCost);
    Store<ArcItem>& cut = cut_;
    Store<uint32_t>& cut_lo = cut_lo_;
    auto emit = [&](ArcItem item, uint32_t b) {
        item.block = b;
        item.base = plan.blocks[b].base;
        item.n = (uint16_t)plan.blocks[b].n;
        items.push_back(item);
    };
    for (size_t x = 0; x < groups_.size();) {
        // Groups that fit one item together share it: a block is loaded and waited
        // for once for all of them.  With an item per group, three rows at LIMIT 10^7
        // spent 43 to 79 % of their time on loads and barriers; when this came they went from
        // 4.5 to 2.4 ms (l = 331,000) and 10.8 to 8.1 ms (l = 160,000), 8 rows at 7.5 10^6
        // from 4.8 to 2.9 ms, 37 near the limit from 1.75 to 1.5 ms.  Groups above kMergedCost hold enough
        // work per block by themselves.
        size_t y = x + 1;
        uint64_t w = groups_[x].cost;
        while (y < groups_.size() && w + groups_[y].cost <= merged && groups_[y].g1 - groups_[x].g0 <= kMergedRows)
            w += groups_[y++].cost;
        if (y - x > 1) {
            for (uint32_t t = 0; t < kTypes; ++t) {
                // between the ends of the groups' ranges the groups that meet a block stay the same
                uint32_t edge[2 * kMergedRows];
                size_t n = 0;
                for (size_t i = x; i < y; ++i) {
                    if (groups_[i].b0[t] == groups_[i].b1[t]) continue;
                    edge[n++] = groups_[i].b0[t];
                    edge[n++] = groups_[i].b1[t];
                }
                std::sort(edge, edge + n);
                for (size_t k = 0; k + 1 < n; ++k) {
                    if (edge[k] == edge[k + 1]) continue;
                    size_t first = y, last = x;
                    uint64_t units = 0, sum = 0;
                    uint32_t most = 1;
                    for (size_t i = x; i < y; ++i) {
                        if (groups_[i].b0[t] > edge[k] || groups_[i].b1[t] <= edge[k]) continue;
                        first = std::min(first, i);
                        last = i;
                    }
                    if (first == y) continue;
                    const size_t v0 = groups_[first].g0, nv = groups_[last].g1 - v0;
                    for (size_t i = 0; i < nv; ++i) {
                        most = std::max(most, rows[v0 + i].na);
                        sum += cost(rows[v0 + i]);
                    }
                    // rows in up to `parts` parts (a part holds at least 32 runs; what
                    // is past a row's last run is passed over), so that there is a
                    // unit per warp and none holds more than a forty-eighth
                    const uint64_t want = std::max<uint64_t>(24 / nv, ((most + 16) * 48 + sum - 1) / sum);
                    const uint32_t parts = (uint32_t)std::max<uint64_t>(1, std::min<uint64_t>({want, 24, (most + 1) / 2}));
                    for (size_t i = 0; i < nv; ++i) units += std::min(parts, (rows[v0 + i].na + 1) / 2);
                    uint32_t share = 1;
                    for (; units < 16 && share < 8; units *= 2) share *= 2;
                    const ArcItem item{0, 0, (uint32_t)v0, (uint16_t)nv, (uint16_t)nv, (uint16_t)parts, 0, (uint16_t)parts, 0, share, 0};
                    for (uint32_t b = edge[k]; b < edge[k + 1]; ++b) emit(item, b);
                }
            }
            x = y;
            if (items.over()) return false;
            continue;
        }
        const Group& g = groups_[x++];
        cut.clear();
        cut_lo.clear();
        for (size_t i = g.g0; i < g.g1;) {
            // a row above one and a half items by itself, over several (24 parts each)
            const uint64_t several = std::min({cost(rows[i]) / target, (uint64_t)rows[i].na / 48, (uint64_t)512});
            if (cost(rows[i]) * 2 > target * 3 && several > 1) {
                for (uint64_t k = 0; k < several; ++k) {
                    cut.push_back(ArcItem{0, 0, (uint32_t)i, 1, 1, 24, (uint16_t)(24 * k), (uint16_t)(24 * several), 0, 1, 0});
                    cut_lo.push_back(rows[i].m_lo);
                }
                ++i;
                continue;
            }
            uint64_t w = 0;
            size_t e = i;
            uint32_t lo = UINT32_MAX;
            for (; e < g.g1 && e - i < 512 && (e == i || w + cost(rows[e]) <= target); ++e) {
                w += cost(rows[e]);
                lo = std::min(lo, rows[e].m_lo);
            }
            // rows above a forty-eighth of the chunk are shared by warps
            uint32_t split = 0;
            while (i + split < e && cost(rows[i + split]) * 48 > w) ++split;
            // (a part holds at least a few groups of 32 runs)
            const uint64_t parts =
                split ? std::max<uint64_t>(1, std::min({(uint64_t)24, (cost(rows[i]) * 48 + w - 1) / w, (uint64_t)rows[i].na / 2})) : 1;
            ArcItem item{0, 0, (uint32_t)i, (uint16_t)(e - i), (uint16_t)split, (uint16_t)parts, 0, (uint16_t)parts, 0, 1, 0};
            // fewer units than warps: the runs of a group are shared too
            uint64_t units = split * parts + (e - i - split);
            for (; units < 16 && item.share < 8; units *= 2) item.share *= 2;
            cut.push_back(item);
            cut_lo.push_back(lo);
            i = e;
        }
        for (uint32_t t = 0; t < kTypes; ++t)
            for (uint32_t b = g.b0[t]; b < g.b1[t]; ++b)
                for (size_t c = 0; c < cut.size(); ++c)
                    if (cut_lo[c] <= plan.blocks[b].m_hi) emit(cut[c], b);
        if (items.over() || cut.over() || cut_lo.over()) return false;
    }
    return true;
}

}  // namespace hss
