// The planner of the arc path on the host: rows and items over a block plan cut
// here, in equal pieces, from the segment offsets.
#include "../../heronian-square-search_gb300/csrc/hss_plan.h"

#include <cstdio>
#include <cstdlib>
#include <new>

#include "../../heronian-square-search_gb300/csrc/hss_prep.h"

using namespace hss;

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
size_t g_largest = ~size_t(0);  // allocations beyond this are refused
}
void* operator new(size_t n) {
    void* p = n > g_largest ? nullptr : std::malloc(n);
    if (!p) throw std::bad_alloc();
    return p;
}
void operator delete(void* p) noexcept { std::free(p); }
void operator delete(void* p, size_t) noexcept { std::free(p); }

namespace {

constexpr uint64_t kLimit = 100000;
constexpr uint32_t kCtas = 152;
HostCache cache;

ArcPlan make_plan() {
    const TypeTables types = make_type_tables();
    ArcPlan plan;
    for (uint32_t t = 0; t < kTypes; ++t) {
        plan.type_first[t] = (uint32_t)plan.blocks.size();
        const uint32_t roots = roots_upto(types, t, (uint32_t)kLimit);
        for (uint32_t r0 = 0; r0 < roots; r0 += 400) {
            const uint32_t r1 = std::min(roots, r0 + 400);
            ArcBlock b{};
            b.type = t;
            b.rank0 = r0;
            b.n_m = r1 - r0;
            b.m_lo = nth_root(types, t, r0);
            b.m_hi = nth_root(types, t, r1 - 1);
            for (uint32_t r = r0; r < r1; ++r) {
                const uint32_t m = nth_root(types, t, r);
                b.n += cache.seg_off[m + 1] - cache.seg_off[m];
            }
            plan.blocks.push_back(b);
        }
    }
    plan.type_first[kTypes] = (uint32_t)plan.blocks.size();
    while ((kLimit >> plan.start_shift) > 4096) ++plan.start_shift;
    for (uint32_t t = 0; t < kTypes; ++t) {
        uint32_t b = plan.type_first[t];
        for (uint64_t i = 0; i <= kLimit >> plan.start_shift; ++i) {
            while (b < plan.type_first[t + 1] && plan.blocks[b].m_hi < i << plan.start_shift) ++b;
            plan.start[t].push_back(b);
        }
    }
    return plan;
}

// The constants of a root that the planner reads.
RowInfo row_info(uint64_t l) {
    RowInfo R{};
    R.l = l;
    R.l2 = l * l;
    R.l4 = (unsigned __int128)R.l2 * R.l2;
    R.n4 = (unsigned __int128)(kLimit * kLimit) * (kLimit * kLimit);
    R.l3 = l % 3 == 0;
    R.l5 = l % 5 == 0;
    R.free_l = cache.seg_off[l + 1] - cache.seg_off[l] - 1;
    const NumberFactors f = factor_number(cache.spf.data(), l);
    R.nsplit = f.count;
    for (uint32_t i = 0; i < f.count; ++i) {
        R.sp[i] = f.primes[i];
        R.se[i] = f.exps[i];
    }
    return R;
}

void add(ArcPlanner& p, uint64_t first, uint64_t last) {
    for (uint64_t l = first; l <= last; ++l)
        p.add(row_info(l), (uint32_t)(l - first), kLimit, cache.max_exponent, 1, kLimit, min_roots(kLimit, last - first + 1));
}

// A term's id holds its value's number in 28 bits, beside three of its form.
void check_value_ids(const ArcPlan& plan) {
    ArcPlanner p;
    add(p, 1000, 1010);
    p.entries = (uint64_t)1 << 25;
    CHECK(p.finish(plan, kCtas, 0), "2^25 values have ids");
    p.entries += 1;
    CHECK(!p.finish(plan, kCtas, 0), "one more has none");
}

// However small an item the caller asks for, their number stays within what
// a launch's host and device memory hold.
void check_item_weight(const ArcPlan& plan) {
    ArcPlanner coarse, fine, fit;
    add(coarse, 10000, 12999);
    add(fine, 10000, 12999);
    CHECK(coarse.finish(plan, kCtas, (uint64_t)1 << 40) && fine.finish(plan, kCtas, 1), "two weights");
    CHECK(fine.items.size() > coarse.items.size(), "%zu and %zu items", fine.items.size(), coarse.items.size());
    CHECK(fine.items.size() <= coarse.items.size() + ((size_t)1 << 18), "%zu items, %zu at least", fine.items.size(),
          coarse.items.size());
    // a caller without the power to allocate has room for 2^18: a heavy root fits
    static ArcPlanner::Arena<8192, 1 << 18> arena;
    fit.use(arena);
    add(fit, 32045, 32045);
    CHECK(fit.finish(plan, kCtas, 1), "a heavy root's items");
}

// Host memory that runs out, at any size of the planner's arrays, is an answer
// and no exception; the planner works again with memory.
void check_memory(const ArcPlan& plan) {
    ArcPlanner p;
    for (size_t most = 64; most < (1u << 24); most *= 2) {
        bool planned = false;
        g_largest = most;
        try {
            p = ArcPlanner();
            p.clear();
            add(p, 10000, 10999);
            planned = p.finish(plan, kCtas, 0);
        } catch (const std::bad_alloc&) {
            g_largest = ~size_t(0);
            CHECK(false, "an exception with arrays of at most %zu bytes", most);
        }
        g_largest = ~size_t(0);
        CHECK(!planned || most > 64, "planned in %zu bytes", most);
    }
    p.clear();
    add(p, 10000, 10999);
    CHECK(p.finish(plan, kCtas, 0), "with memory");
}

}  // namespace

int main() {
    std::string err;
    CHECK(build_host_cache(kLimit, 8, &cache, &err) == 0, "host cache");
    const ArcPlan plan = make_plan();
    check_value_ids(plan);
    check_item_weight(plan);
    check_memory(plan);
    std::printf("ok\n");
    return 0;
}
