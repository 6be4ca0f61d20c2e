// hss_plan.h - rows and work items of the arc path (host side).
#pragma once
#include <stdint.h>

#include <algorithm>
#include <exception>
#include <vector>

#include "hss_blocks.h"
#include "hss_kernels.h"

namespace hss {

// The planner's arrays: grown as needed, or over memory that is given once and
// never exceeded.  over() tells that an entry found no room (in the given memory, or
// in the host's: no exception leaves the planner, which C callers reach).
template <class T>
class Store {
  public:
    void fix(T* p, size_t cap) {
        p_ = p;
        cap_ = cap;
        fixed_ = true;
    }
    void push_back(const T& x) {
        if (n_ == cap_ && !grow(n_ + 1)) return;
        p_[n_++] = x;
    }
    void resize(size_t n) {
        if (n > cap_ && !grow(n)) n = cap_;
        n_ = n;
    }
    void clear() {
        n_ = 0;
        over_ = false;
    }
    void swap(Store& o) {
        own_.swap(o.own_);
        std::swap(p_, o.p_);
        std::swap(n_, o.n_);
        std::swap(cap_, o.cap_);
        std::swap(fixed_, o.fixed_);
        std::swap(over_, o.over_);
    }
    size_t size() const { return n_; }
    bool empty() const { return n_ == 0; }
    bool over() const { return over_; }
    T* data() { return p_; }
    T* begin() { return p_; }
    T* end() { return p_ + n_; }
    T& back() { return p_[n_ - 1]; }
    T& operator[](size_t i) { return p_[i]; }
    const T& operator[](size_t i) const { return p_[i]; }

  private:
    bool grow(size_t n) {
        if (fixed_) {
            over_ = true;
            return false;
        }
        try {
            own_.resize(std::max(n, 2 * cap_));
        } catch (const std::exception&) {  // bad_alloc, length_error
            over_ = true;
            return false;
        }
        p_ = own_.data();
        cap_ = own_.size();
        return true;
    }
    std::vector<T> own_;
    T* p_ = nullptr;
    size_t n_ = 0, cap_ = 0;
    bool fixed_ = false, over_ = false;
};

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
    // False when an array had no room, or for more values than kArcValuesMost.
    bool finish(const ArcPlan& plan, uint32_t ctas, uint64_t item_target);
    // Orders the rows as finish does (false without room for it), and takes rows
    // [i0, i1) of another planner.
    bool sort();
    void take(const ArcPlanner& from, size_t i0, size_t i1);

    // Arrays over given memory, for callers that may not allocate.
    struct Order {
        uint64_t key, rest;  // rest: values descending, then the order of addition
    };
    struct Group {
        size_t g0, g1;            // rows of one key
        uint64_t cost;
        uint32_t b0[kTypes], b1[kTypes];  // its blocks of every type
    };
    template <size_t ROWS, size_t ITEMS>
    struct Arena {
        ArcRow rows[ROWS], sorted[ROWS];
        ArcItem items[ITEMS], cut[ROWS];
        uint64_t keys[ROWS];
        uint32_t cut_lo[ROWS];
        Order order[ROWS];
        Group groups[ROWS];
    };
    template <size_t ROWS, size_t ITEMS>
    void use(Arena<ROWS, ITEMS>& a) {
        rows.fix(a.rows, ROWS);
        sorted_.fix(a.sorted, ROWS);
        items.fix(a.items, ITEMS);
        cut_.fix(a.cut, ROWS);
        keys_.fix(a.keys, ROWS);
        cut_lo_.fix(a.cut_lo, ROWS);
        order_.fix(a.order, ROWS);
        groups_.fix(a.groups, ROWS);
        rest.fix(nullptr, 0);
    }

    Store<ArcRow> rows;
    Store<ArcRest> rest;
    Store<ArcItem> items;
    uint64_t entries = 0;     // values of all rows
    uint64_t rest_pairs = 0;  // pairs of the rest list at most

  private:
    Store<uint64_t> keys_;  // sort key of rows[i]
    Store<ArcRow> sorted_;
    Store<Order> order_;
    Store<Group> groups_;
    Store<ArcItem> cut_;  // the group's chunks of rows, without a block
    Store<uint32_t> cut_lo_;
};

}  // namespace hss
