// hss_plan.h - rows and work items of the arc path (host side).
#pragma once
#include <stdint.h>

#include <vector>

#include "hss_blocks.h"
#include "hss_kernels.h"

namespace hss {

// Roots m' below which the pairs of a common part P are handed to the
// shared-prime kernels, for a call of `rows` roots.
uint64_t min_roots(uint64_t limit, size_t rows);

// Collects the rows of one launch group: for every root l the rows (l, P) -
// P = 1 and every product P of powers of l's split primes with a multiple in
// [l, N] - that hold enough roots m' to be worth a row, and a rest list of
// the others; then cuts rows x blocks into work items.
class ArcPlanner {
  public:
    void clear();
    // Adds root R.l (RowInfo index `row`) against m in [m0, m1]; a (l, P) of
    // fewer than `least` roots m' goes to the rest list.
    void add(const RowInfo& R, uint32_t row, uint64_t limit, uint32_t max_exponent, uint64_t m0, uint64_t m1,
             uint64_t least);
    // Orders the rows, assigns their values' entries and builds the items.
    void finish(const ArcPlan& plan, uint32_t ctas, uint64_t item_target);

    std::vector<ArcRow> rows;
    std::vector<ArcRest> rest;
    std::vector<ArcItem> items;
    uint64_t entries = 0;     // values of all rows
    uint64_t rest_pairs = 0;  // pairs of the rest list at most

  private:
    std::vector<uint64_t> keys;  // sort key of rows[i]
};

}  // namespace hss
