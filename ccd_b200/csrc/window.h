// window.h -- the windowed sweep of independent-row fits (window.cu) and the
// plan that it walks (window_plan.cpp).
#pragma once

#include <cstddef>
#include <cstdint>
#include <vector>

#include "types.h"

namespace ccdb {

constexpr int kWindow = 16;         // consecutive positions in flight, one per warp
constexpr int kWindowCluster = 16;  // most CTAs that share the rows

// By the most entries that one CTA holds of it, a column is short, medium (more
// than kWindowShort: alone when it is likely to move) or long (more than
// kWindowLong: always alone, on every warp).
constexpr int64_t kWindowShort = 128;
constexpr int64_t kWindowLong = 512;

// One active column in visiting order.  flags: bit 0 row ids, bit 1 values,
// bit 2 indicator or intercept, bit 3 long, bit 4 medium.  conflict: bit b tells that
// the column shares a row with the one 15 - b positions before it (b = 0..14).
struct WinCol {
    int64_t cb, vb;  // offsets of its row ids and values
    int32_t j, n;    // column and entry count
    uint16_t conflict, flags;
    int32_t pad;
};
static_assert(sizeof(WinCol) == 32 && offsetof(WinCol, conflict) % 4 == 0 &&
                  offsetof(WinCol, flags) == offsetof(WinCol, conflict) + 2, "WinCol layout");

// Half-open range of a column's entries (of rows, for DENSE and INTERCEPT
// columns) that one CTA owns.
struct WinSlice {
    int32_t lo, hi;
};

struct WindowPlan {
    std::vector<WinCol> cols;      // active columns in visiting order
    std::vector<WinSlice> slices;  // [CTA][position]
};

// Rows [K r / C, K (r + 1) / C) belong to CTA r.
constexpr int64_t window_row(int64_t K, int r, int C) { return K * r / C; }

WindowPlan build_window_plan(int64_t K, int32_t J, const int64_t* col_start, const int32_t* rows,
                             const int64_t* val_start, const uint8_t* fmt, const uint8_t* fixed, int C,
                             int64_t short_entries = kWindowShort, int64_t long_entries = kWindowLong);

}  // namespace ccdb
