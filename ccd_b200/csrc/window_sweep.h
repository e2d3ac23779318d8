// window_sweep.h -- parameters and launcher of the windowed sweep (window.cu).
#pragma once

#include <cuda_runtime.h>

#include "indep.h"
#include "window.h"

namespace ccdb {

// A round of a traced sweep (CTA 0's SM clock): its beginning, its steps known, its
// end; the first position in flight, the columns in flight, taken, and moved, and
// whether one ran alone.
struct RoundStamp {
    int64_t begin, steps, end, base, flying, taken, moved, alone;
};
constexpr int kTracedRounds = 4096;  // the first ones of a sweep

// What a column's step needs beside its entries, by position.
struct WinScal {
    double xjy, pvar, lambda, inv_var;  // sqrt(2 / pvar) of a Laplace prior, 1 / pvar of a normal one
    int32_t ptype, pad0;
    int64_t pad1;
};

struct WindowParams {
    IndepParams P;           // matrix, row and column state, convergence (no schedule)
    const WinCol* cols;      // n_active
    const WinSlice* slices;  // cluster x n_active
    WinScal* scal;           // n_active, written by the kernel
    double2* bh;             // n_active {beta, bound}, written by the kernel
    double* share;           // K: each row's share of a gradient, where it is not in shared memory
    int32_t n_active;
    int32_t weighted;        // 0: every row weight is 1.0 and is not read
    int32_t any_vals;        // some active column has values
    int32_t vals_at;         // where the staged values lie in shared memory (the launcher's)
    int32_t cluster;         // CTAs
    int32_t weights_shared;  // the weights lie beside the rest of a row (the launcher's)
    RoundStamp* trace;       // kTracedRounds, of a traced launch
};

// The largest cluster (16, 8, 4, 2, 1) that can be resident with the most
// shared memory a CTA may hold, and that memory's bytes; 0 if none.
cudaError_t window_limits(int* cluster, int64_t* smem);
// Whether the shares of `rows` rows fit in `smem` bytes beside what is staged
// (then `share` may be nullptr).
bool window_share_fits(int64_t rows, bool vals, int64_t smem);
cudaError_t launch_window_sweep(const WindowParams& R, int64_t smem, cudaStream_t stream);
// with R.trace filled (window_trace.cu)
cudaError_t launch_window_sweep_traced(const WindowParams& R, int64_t smem, cudaStream_t stream);

}  // namespace ccdb
