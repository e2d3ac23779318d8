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
// A batch as the choice between the engines sees it.
struct BatchSize {
    bool mixed;
    bool share_in_shared;  // the rows' shares fit a CTA's shared memory
    int64_t K, mean;
    int n, n_sm;
};

// Lockstep group size of the mixed-precision batched engine.  G = 4 packs the
// group's state for one row into one 32-byte sector (a quarter of the DRAM
// sectors G = 1 moves per instance), but gives one CTA G times the per-column
// arithmetic and leaves ceil(n / G) CTAs for the SMs.  Take the largest G that
// still gives every third SM a CTA.
constexpr int batch_group_size(int n, int n_sm) {
    const int want = std::max(1, n_sm / 3);
    for (int G : {4, 2})
        if ((n + G - 1) / G >= want) return G;
    return 1;
}
// The group, and the waves of CTAs when a cluster of up to eight gives every SM one.
struct LockstepShape {
    int group, cluster, waves;
};
constexpr LockstepShape lockstep_shape(int n, int n_sm) {
    const int G = batch_group_size(n, n_sm), groups = (n + G - 1) / G;
    int C = 1;
    while (C < 8 && groups * C < n_sm) C *= 2;
    return {G, C, (groups * C + n_sm - 1) / n_sm};
}

// Whether the windowed engine is the faster one.  It takes time like the columns'
// mean and like n / SMs (a CTA takes the next fit when one ends); the sweeps that
// step one column at a time fill the memory pipe with a long column's gathers, the
// mixed ones read a row once for the up to four fits of a group, and their time
// goes in whole waves.  So the line is a mean: 300 where the shares lie in global
// memory, 480 in shared memory, for a wave of each, times the waves and what a group
// costs more (of two 1.12; of four 1.45, 2 without a cluster), over n / SMs.
// Up to 500 and 640 whatever the waves: above 508 entries a column is not all
// copied ahead.  Time of the mixed engine over the windowed one, 600 columns:
//   rows, fits: mean 200   300   350   450   500   560
//   40,000,   4     2.25  1.38  1.16  1.11  0.99  0.83
//   40,000, 450     2.28  1.55  1.30  1.20  1.03  0.85
//   40,000, 1000    1.46  0.97  0.81  0.78  0.67  0.55
//   100,000,   4    1.92  1.06  0.83  0.77  0.68  0.57
//   100,000,  60    3.74  2.06  1.61  1.48  1.27  1.01
//   100,000, 250    2.52  1.61  1.27  1.11  0.98  0.80
//   100,000, 600    1.33  0.88  0.70  0.64  0.56  0.46
// FP64 has one CTA a fit in both.  With the rows in shared memory the windowed one
// is faster to the end (20,000 rows, mean 560: 1.13 to 1.67).  Else, up to one fit
// an SM, the two are even from 360 to 450 and it loses above (100,000 rows, 148
// fits: mean 300 1.11, 400 0.92; 40,000 rows: 400 1.07, 500 1.00, 560 0.87).  With
// more fits it gains from the fits that end early while the running ones' state
// fits L2 (40,000 rows, 200 fits: mean 500 1.27, 560 1.07), and less beyond (100,000
// rows: 400 1.14, 500 1.02; 250,000 rows: 300 1.22, 400 1.00, 500 0.91).
constexpr int64_t kBatchWindowMean = 640;  // above it never (100,000 rows, 200 fits, mean 1,000: 0.94, mixed 0.72)
constexpr int64_t kBatchL2 = 100 << 20;    // of the 126 MB of L2, what the fits' rows may take

constexpr bool batch_prefers_window(const BatchSize& b) {
    if (b.mean > kBatchWindowMean) return false;
    if (b.mixed) {
        const LockstepShape s = lockstep_shape(b.n, b.n_sm);
        const double turns = std::max(1.0, (double)b.n / b.n_sm);
        const double group = s.group == 1 ? 1.0 : s.group == 2 ? 1.12 : s.cluster > 1 ? 1.45 : 2.0;
        const double line = (b.share_in_shared ? 480 : 300) * s.waves * group / turns;
        return b.mean <= std::min(line, b.share_in_shared ? 640.0 : 500.0);
    }
    if (b.share_in_shared) return true;
    if (b.n <= b.n_sm) return b.mean <= 360;
    return 16 * b.K * b.n_sm <= kBatchL2 || b.mean <= 450;
}

}  // namespace ccdb
