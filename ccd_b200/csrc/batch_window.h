// batch_window.h -- parameters and launcher of the windowed sweep over many
// fits of one matrix (batch_window.cu).
#pragma once

#include <cuda_runtime.h>

#include "batch.h"
#include "window_sweep.h"

namespace ccdb {

// The team of warps that a column has, by the mean entries of the columns (the
// longest one, an intercept usually, left out): one warp up to kBatchOneWarp, four
// above, since a warp walks a column 32 entries at a time but four columns in
// flight find fewer to take than sixteen.  200 fits, 300 columns, B200, one warp
// against four: mean 16, 0.58 against 1.45 ms; 48, 1.1 against 1.6; 80, 5.2
// against 3.9; 200, 12.5 against 7.6.
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

struct BatchWindowParams {
    BatchParams P;          // matrix, outcomes, instances, results
    const WinCol* cols;     // n_active
    const WinSlice* slices;  // n_active, the whole columns
    const int32_t* longs;   // positions of the long columns
    double* beta_out;       // n_inst x J
    WinScal* scal;          // ctas x n_active, written by the kernel
    double2* bh;            // ctas x n_active {beta, bound}, written by the kernel
    double* xbeta;          // ctas x K, where it is not in shared memory
    double* share;          // ctas x K (floats in mixed precision), where it is not in shared memory
    int64_t entries;        // of the active columns
    int32_t n_active, n_long;
    int32_t any_vals;       // some active column has values
    int32_t vals_at;        // where the staged values lie in shared memory (the launcher's)
    int32_t mixed;
    int32_t ctas;           // instances that run at once
    int32_t team;           // warps to a column: 1 or 4
    int32_t pad;
};

// What of a row's state does not fit in shared memory: bit 0 its xBeta, bit 1 its share.
cudaError_t batch_window_spill(int64_t K, bool mixed, bool vals, int* spill);
cudaError_t launch_batch_window(const BatchWindowParams& R, cudaStream_t stream);

}  // namespace ccdb
