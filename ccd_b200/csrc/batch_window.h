// batch_window.h -- parameters and launcher of the windowed sweep over many
// fits of one matrix (batch_window.cu).
#pragma once

#include <cuda_runtime.h>

#include "batch.h"
#include "batch_route.h"
#include "window_sweep.h"

namespace ccdb {

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
    uint32_t step;          // what a copy under way adds to a helper's phase (the launcher's)
};

// What of a row's state does not fit in shared memory: bit 0 its xBeta, bit 1 its share.
cudaError_t batch_window_spill(int64_t K, bool mixed, bool vals, int* spill);
cudaError_t launch_batch_window(const BatchWindowParams& R, cudaStream_t stream);

}  // namespace ccdb
