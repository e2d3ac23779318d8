// window_plan.cpp -- which columns may step side by side in the windowed sweep.
//
// Two columns that share no row read and write different state, so taking
// their steps together gives the sequential result.  The sweep keeps kWindow
// consecutive positions in flight and needs, for each position, which of the
// kWindow - 1 before it share a row with it.  One walk over the entries finds
// this: every row remembers the last position that touched it and, as a bit
// mask, the ones just before that.
#include "window.h"

#include <algorithm>

namespace ccdb {

namespace {

struct RowHistory {
    int32_t last = -1;   // the last position that touched the row
    uint32_t mask = 0;   // bit b: position last - b touched it
};

constexpr uint32_t kDistances = (1u << (kWindow - 1)) - 1;  // bit d - 1: distance d = 1 .. kWindow - 1

// bit d - 1 (distance d) -> bit kWindow - 1 - d
uint16_t by_position(uint32_t distances) {
    uint32_t r = 0;
    for (int d = 1; d < kWindow; ++d)
        if (distances >> (d - 1) & 1u) r |= 1u << (kWindow - 1 - d);
    return (uint16_t)r;
}

}  // namespace

WindowPlan build_window_plan(int64_t K, int32_t J, const int64_t* col_start, const int32_t* rows,
                             const int64_t* val_start, const uint8_t* fmt, const uint8_t* fixed, int C,
                             int64_t short_entries, int64_t long_entries) {
    WindowPlan w;
    int32_t n_active = 0;
    for (int32_t j = 0; j < J; ++j) n_active += (fixed && fixed[j]) ? 0 : 1;
    w.cols.reserve(n_active);
    w.slices.resize((size_t)C * n_active);
    std::vector<RowHistory> seen((size_t)std::max<int64_t>(K, 1));
    // bit d - 1: the column d positions back holds every row, or any row
    uint32_t all_rows = 0, any_row = 0;
    for (int32_t j = 0; j < J; ++j) {
        if (fixed && fixed[j]) continue;
        const int32_t q = (int32_t)w.cols.size();
        const uint8_t f = fmt[j];
        const bool has_rows = (f == F_SPARSE || f == F_INDICATOR);
        const int64_t b = col_start[j], n = has_rows ? col_start[j + 1] - b : K;
        WinCol c{};
        c.cb = b;
        c.vb = val_start[j];
        c.j = j;
        c.n = (int32_t)n;
        c.flags = (has_rows ? 1 : 0) | ((f == F_SPARSE || f == F_DENSE) ? 2 : 0) |
                  ((f == F_INDICATOR || f == F_INTERCEPT) ? 4 : 0);
        int64_t longest = 0;
        const int32_t* at = rows + b;
        for (int r = 0; r < C; ++r) {
            WinSlice s;
            if (has_rows) {
                s.lo = (int32_t)(at - (rows + b));
                at = (r == C - 1) ? rows + b + n : std::lower_bound(at, rows + b + n, window_row(K, r + 1, C));
                s.hi = (int32_t)(at - (rows + b));
            } else {
                s.lo = (int32_t)window_row(K, r, C);
                s.hi = (int32_t)window_row(K, r + 1, C);
            }
            w.slices[(size_t)r * n_active + q] = s;
            longest = std::max<int64_t>(longest, s.hi - s.lo);
        }
        uint32_t dist = n > 0 ? all_rows : 0;
        bool holds_all = false;
        if (longest > short_entries) c.flags |= 16;
        if (longest > long_entries) {
            c.flags |= 8;  // never in flight beside another column: its conflicts are not needed
        } else if (!has_rows) {
            dist = any_row;
            holds_all = true;
        } else {
            for (int64_t p = b; p < b + n; ++p) {
                if (p + 16 < b + n) __builtin_prefetch(&seen[rows[p + 16]], 1);
                RowHistory& h = seen[rows[p]];
                const int32_t d = q - h.last;
                if (h.last >= 0 && d < kWindow) {
                    dist |= h.mask << (d - 1);
                    h.mask = h.mask << d | 1u;
                } else {
                    h.mask = 1u;
                }
                h.last = q;
            }
        }
        c.conflict = by_position(dist & kDistances);
        all_rows = (all_rows << 1 | (holds_all ? 1u : 0u)) & kDistances;
        any_row = (any_row << 1 | (n > 0 ? 1u : 0u)) & kDistances;
        w.cols.push_back(c);
    }
    return w;
}

}  // namespace ccdb
