// batch_route.h -- which engine runs a batch of fits, and how (host code).
#pragma once

#include <algorithm>
#include <cstdint>

namespace ccdb {

// Mean entries of the columns that a batch steps, the longest one (an intercept
// usually) and an offset in column 0 left out.
template <typename Entries>
int64_t batch_mean_entries(int J, bool offset_col0, Entries&& entries) {
    int64_t sum = 0, longest = 0, n = 0;
    for (int j = offset_col0 ? 1 : 0; j < J; ++j, ++n) {
        const int64_t e = entries(j);
        sum += e;
        longest = std::max(longest, e);
    }
    return n > 1 ? (sum - longest) / (n - 1) : longest;
}

// The team of warps that a column of the windowed batch engine has, by that mean:
// one warp up to kBatchOneWarp, four above, since a warp walks a column 32 entries
// at a time but four columns in flight find fewer to take than sixteen.  200 fits,
// 300 columns, B200, one warp against four: mean 16, 0.58 against 1.45 ms; 48, 1.1
// against 1.6; 80, 5.2 against 3.9; 200, 12.5 against 7.6.
// A column is medium or long (window.h) above the entries given here.
constexpr int64_t kBatchOneWarp = 64;
struct BatchTeam {
    int warps;
    int64_t short_entries, long_entries;
};
constexpr BatchTeam batch_team(int64_t mean) {
    return mean <= kBatchOneWarp ? BatchTeam{1, 128, 512} : BatchTeam{4, 320, 2048};
}
// Above this mean the sweeps that take one column at a time are the faster ones:
// their gathers fill the memory pipe, and the lockstep groups read a row once for
// four fits.  200 fits of 100,000 rows, windowed against one column at a time: mean
// 200, FP64 7.4 against 14.1 ms and mixed 6.9 against 14.8; 500, 17.0 against 19.4
// and 15.6 against 19.3; 1,000, 35.4 against 33.4 and 31.4 against 25.5.
constexpr int64_t kBatchWindowMean = 640;

}  // namespace ccdb
