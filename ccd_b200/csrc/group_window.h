// group_window.h -- the windowed sweep of the group models (group_window.cu):
// Breslow Cox and the grouped models (conditional logistic / Poisson), one launch
// per findMode.
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

#include "cox.h"
#include "types.h"
#include "window_sweep.h"

namespace ccdb {

constexpr int kGroupWindowCtas = 160;  // most CTAs of the grid form
constexpr int64_t kGroupLong = 512;    // a column with a larger slice may run alone

// What one CTA owns: rows [row0, next row0) and groups [g0, next g0); a sentinel
// follows the last CTA's.  Strata (Cox): `first` and `last` are those of its
// first and last group; bit 0 of flags: `first` began in the CTA before it, bit 1:
// all its groups lie in one stratum.  Its accumulated denominators take in the
// tail sums of the CTAs [lo, itself), its suffix sums the head sums of (itself, hi].
struct GroupCut {
    int32_t row0, g0, flags, first, last, lo, hi, pad;
};

struct GroupWindowParams {
    CoxParams P;
    int32_t cox;       // 1: Breslow Cox (accumulated denominators and suffix sums)
    int32_t n_active;  // columns visited per cycle
    const WinCol* cols;
    const WinSlice* slices;  // [CTA][position]
    WinScal* scal;           // n_active, written by the kernel
    double2* bh;             // n_active {beta, bound}, written by the kernel
    const GroupCut* cuts;    // ctas + 1
    double* beta;
    double* hdelta;
    const int32_t* ptype;
    const double* pvar;
    int32_t J;
    int32_t conv;
    int32_t max_iter;
    int32_t ctas;
    double tol;
    double ll_fixed;
    int32_t any_vals;  // some active column has values
    int32_t any_long;  // some may be marked long
    int32_t meet;      // Cox: a stratum spans CTAs, which then exchange tail and head sums
    int32_t chain;     // lanes that a carry may pass over (1 + the CTAs within one stratum in a row)
    int32_t vals_at;   // where the staged values lie in shared memory (the launcher's)
    DevStatus* st;
    // grid form: what CTAs send each other, in two buffers by exchange parity
    double2* part;   // 2 x kWindow x ctas x 3
    double* tails;   // 2 x ctas
    double2* heads;  // 2 x ctas
    double2* red;    // 2 x ctas: objective partials
    unsigned* grid_bar;
    long long wait_limit_ns;  // bound on any single wait for the other CTAs
    RoundStamp* trace;  // kTracedRounds, of a traced launch
};

// The largest cluster (16, 8, 4, 2, 1) that can be resident (0 if none), and the
// shared memory a CTA may hold: grid form, cluster of a grouped model, of Cox.
struct GroupWindowLimits {
    int cluster;
    int64_t smem[3];
};
cudaError_t group_window_limits(GroupWindowLimits* w);
// Whether the groups that one of `ctas` CTAs owns fit in `smem` bytes.
bool group_window_fits(bool cox, int64_t groups, int ctas, bool vals, int64_t smem);
// Entry ranges of every column that each CTA owns, from the CTAs' first rows; with
// `mark_long`, a column of which a CTA owns more than kGroupLong entries is marked.
cudaError_t launch_window_slices(const int32_t* rows, WinCol* cols, int32_t n_active, const GroupCut* cuts,
                                 int ctas, bool mark_long, WinSlice* slices, cudaStream_t stream);
// `most_rows`, `most_groups`: the most that one CTA owns.
cudaError_t launch_group_window(const GroupWindowParams& Q, bool cluster, int64_t most_rows, int64_t most_groups,
                                cudaStream_t stream);
// Cox with Q.any_long (group_window_long.cu)
cudaError_t launch_group_window_long(const GroupWindowParams& Q, bool cluster, int64_t most_rows, int64_t most_groups,
                                     cudaStream_t stream);
// with Q.trace filled (group_window_trace.cu)
cudaError_t launch_group_window_traced(const GroupWindowParams& Q, bool cluster, int64_t most_rows, int64_t most_groups,
                                       cudaStream_t stream);

}  // namespace ccdb
