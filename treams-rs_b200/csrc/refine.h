// Host side of the iterative refinement of dense solves: which columns take another sweep.
#pragma once

#include <algorithm>
#include <cmath>
#include <cstddef>
#include <vector>

namespace tcu {

// Refinement state of the columns of one solve in groups of 8 that converge separately: a group
// takes another sweep while its worst relative residual is above the target, the last sweep
// halved it and sweeps are left; afterwards its columns and their residuals stay as they are.
// settle: a group that has met the target with less than a factor 10 to spare takes one sweep more
// if its sweeps still gain a factor 16 each. Factors of the bfloat16 split start at a residual of 2e-7 and meet
// 1e-13 at 6e-14 in two sweeps; the third ends at the rounding level (1e-16 to 9e-15), as the three sweeps of
// the two-pass TF32 split (from 2e-6) do, for one product and one pair of sweeps. A line at a factor 64
// cost adjoint solves (rounding level 7e-15) a fourth sweep: 18.8 against 16.4 ms for 17 columns each way
// at 9600 modes.
// The columns of the groups that still sweep are kept packed, in their order, so that a sweep and its residual
// cost what those columns cost: of 128 columns of which one group of 8 converges slowly, the other 120 would
// take every one of its sweeps with it (each an application of the operator).
struct RefineGroups {
    static constexpr int WIDTH = 8;
    struct Group {
        bool active = true, settled = false;
        int sweeps = 1, left = 0;
        double prev = INFINITY;
    };
    std::vector<Group> g;
    std::vector<size_t> live;  // groups whose columns are packed, ascending
    std::vector<double> rn;    // residual norms of the columns' current solutions
    int p;
    double target;
    bool settle;
    RefineGroups(int p_, double target_, int max_sweeps, bool settle_)
        : g((p_ + WIDTH - 1) / WIDTH), rn(p_), p(p_), target(target_), settle(settle_) {
        for (Group& q : g) q.left = max_sweeps;
        for (size_t q = 0; q < g.size(); ++q) live.push_back(q);
    }
    size_t first(size_t q) const { return q * WIDTH; }
    int width(size_t q) const { return std::min(WIDTH, p - (int)q * WIDTH); }
    int columns() const {  // packed ones
        int c = 0;
        for (size_t q : live) c += width(q);
        return c;
    }
    // norms of the packed columns to their places among all columns
    void scatter(const std::vector<double>& packed, std::vector<double>& all) const {
        size_t from = 0;
        for (size_t q : live)
            for (int c = 0; c < width(q); ++c) all[first(q) + c] = packed[from++];
    }
    // The groups that sweep no more leave the packed columns: done(q, from) for each of them, then
    // shift(from, to, width) for those that close the gaps (to + width <= from: only the last group is narrower).
    template <class Done, class Shift>
    void compact(Done done, Shift shift) {
        int from = 0;
        for (size_t q : live) {
            if (!g[q].active) done(q, from);
            from += width(q);
        }
        std::vector<size_t> next;
        int to = from = 0;
        for (size_t q : live) {
            if (g[q].active) {
                if (from != to) shift(from, to, width(q));
                to += width(q);
                next.push_back(q);
            }
            from += width(q);
        }
        live.swap(next);
    }
    // worst relative residual of a group: infinite where a correction made a residual that is no number, so that
    // the group stops and a mixed factor's goes on to the fallback factor (a maximum would pass a NaN over as
    // converged). Columns whose right-hand side is none have nothing to gain from another factor.
    double worst(size_t q, const std::vector<double>& r, const std::vector<double>& bn) const {
        double w = 0.0;
        for (int c = (int)first(q); c < (int)first(q) + width(q); ++c) {
            if (!std::isfinite(bn[c])) continue;
            const double rel = bn[c] > 0 ? r[c] / bn[c] : r[c];
            if (!std::isfinite(rel)) return INFINITY;
            w = std::max(w, rel);
        }
        return w;
    }
    // r: norms after the latest sweep; true while a group takes another one
    bool advance(const std::vector<double>& r, const std::vector<double>& bn) {
        bool any = false;
        for (size_t q = 0; q < g.size(); ++q) {
            if (!g[q].active) continue;
            for (int c = (int)first(q); c < (int)first(q) + width(q); ++c) rn[c] = r[c];
            const double w = worst(q, r, bn);
            bool stop = g[q].left == 0 || !(w < 0.5 * g[q].prev);
            if (!stop && w <= target) {
                stop = !settle || g[q].settled || w <= target / 10 || !(w < g[q].prev / 16);
                g[q].settled = true;
            }
            if (stop) {
                g[q].active = false;
                continue;
            }
            g[q].prev = w;
            --g[q].left;
            ++g[q].sweeps;
            any = true;
        }
        return any;
    }
    bool any_above(const std::vector<double>& bn, double limit) const {
        for (size_t q = 0; q < g.size(); ++q)
            if (!(worst(q, rn, bn) <= limit)) return true;
        return false;
    }
};

}  // namespace tcu
