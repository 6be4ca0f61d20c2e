// Every buffer that grows on demand, its growth refused at each allocation in
// turn: the call reports the failure, no capacity claims more than its array
// holds, and the next call finds every buffer again.
#include "fake_runtime.h"

namespace {

constexpr size_t kSmall = 100, kBig = 5000000;

hss_t* open_handle() {
    hss_t* h = new hss_t();
    h->limit = 100000;
    h->sm_count = 152;
    h->plan = std::make_shared<ArcPlan>();
    CHECK(alloc_launch_buffers(h) == HSS_OK, "launch buffers");
    return h;
}

void check_buffers(hss_t* h, const char* what, int k) {
    CHECK(fake::holds(h->d_rows, h->rows_cap), "%s, refusal %d", what, k);
    CHECK(fake::holds(h->h_rows, h->h_rows_cap), "%s, refusal %d", what, k);
    CHECK(fake::holds(h->d_merged, h->merged_cap), "%s, refusal %d", what, k);
    CHECK(fake::holds(h->d_big, h->big_cap, kBigEntryWords), "%s, refusal %d", what, k);
    CHECK(fake::holds(h->d_desc, h->desc_chunk, kBigEntryWords), "%s, refusal %d", what, k);
    CHECK(fake::holds(h->d_exact, h->exact_cap), "%s, refusal %d", what, k);
    CHECK(fake::holds(h->d_items, h->items_cap), "%s, refusal %d", what, k);
    CHECK(fake::holds(h->h_items, h->h_items_cap), "%s, refusal %d", what, k);
    CHECK(fake::holds(h->d_row_info, h->row_info_cap), "%s, refusal %d", what, k);
    CHECK(fake::holds(h->h_row_info, h->h_row_info_cap), "%s, refusal %d", what, k);
    CHECK(fake::holds(h->d_slots, h->slots_cap), "%s, refusal %d", what, k);
    CHECK(fake::holds(h->h_slots, h->h_slots_cap), "%s, refusal %d", what, k);
    CHECK(fake::holds(h->d_group, h->group_cap), "%s, refusal %d", what, k);
    for (unsigned char* p : h->h_group) CHECK(fake::holds(p, h->group_cap), "%s, refusal %d", what, k);
    CHECK(fake::holds(h->d_values, h->values_cap), "%s, refusal %d", what, k);
    CHECK(fake::holds(h->d_value_hot, h->values_cap), "%s, refusal %d", what, k);
}

template <class Grow>
void check_growth(const char* what, Grow grow) {
    // one allocation refused, or all from there on
    for (int count : {1, 1000})
        for (int k = 0; k < 4; ++k) {
            hss_t* h = open_handle();
            CHECK(grow(h, kSmall) == HSS_OK, "%s: first growth", what);
            fake::reset();
            fake::fail_from = k;
            fake::fail_count = count;
            const int s = grow(h, kBig);
            CHECK(s == HSS_OK || s == HSS_ERR_MEMORY || s == HSS_ERR_CUDA, "%s: status %d", what, s);
            if (k == 0 && count == 1000) CHECK(s != HSS_OK, "%s: a refused growth reported as done", what);
            check_buffers(h, what, k);
            CHECK(fake::last == cudaSuccess, "%s, refusal %d: the next launch's check would meet its error", what, k);
            fake::reset();
            CHECK(begin_call(h, kSmall) == HSS_OK, "%s: the next call", what);
            CHECK(h->d_merged && h->merged_cap && h->d_big && h->big_cap && h->d_desc && h->desc_chunk && h->d_exact && h->exact_cap,
                  "%s, refusal %d: a queue is missing in the next call", what, k);
            CHECK(grow(h, kSmall) == HSS_OK, "%s: a small call after the refusal", what);
            check_buffers(h, what, k);
            CHECK(grow(h, kBig) == HSS_OK, "%s: the growth tried again", what);
            check_buffers(h, what, k);
            hss_close(h);
        }
}

}  // namespace

int main() {
    check_growth("row counters", [](hss_t* h, size_t n) { return ensure_rows(h, n); });
    check_growth("shared-prime queue", [](hss_t* h, size_t n) { return ensure_merged(h, 100 * n); });
    check_growth("items", [](hss_t* h, size_t n) { return ensure_items(h, n); });
    check_growth("row constants", [](hss_t* h, size_t n) { return ensure_row_info(h, n); });
    check_growth("serving slots", [](hss_t* h, size_t n) { return ensure_slots(h, n); });
    check_growth("launch group", [](hss_t* h, size_t n) { return ensure_group(h, 16 * n, n); });
    check_growth("exact queue", [](hss_t* h, size_t n) {
        if (n == kSmall) return HSS_OK;
        h->exact_overflow = true;
        return grow_overflowed(h);
    });
    check_growth("big-pair queue", [](hss_t* h, size_t n) {
        if (n == kSmall) return HSS_OK;
        h->big_overflow = true;
        return grow_overflowed(h);
    });
    std::printf("ok\n");
    return 0;
}
