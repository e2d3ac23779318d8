// mm.cu -- the MM algorithm's step over every coordinate at once
// (CyclicCoordinateDescent::mmUpdateAllBeta, CyclicCoordinateDescent.cpp:1354-1391,
// over ModelSpecifics::computeMMGradientAndHessian(Impl), ModelSpecifics.hpp:776-889).
//
// Every free column's (g, h) comes from the same state, so the J columns are
// independent.  A row's part in a sum, events x exp(xBeta) / denominator of its
// group, is worked out once per row; one CTA per column then gathers that one
// word per entry (four dependent words and a division before) and reduces in a
// fixed order, and its thread 0 applies the clamp h < 0 -> (0, 0) and the
// prior's closed-form step (JointPrior::getDelta), with no trust-region bound
// (the reference's MM cycle leaves applyBounds out, .cpp:984-987).  xBeta is
// then recomputed from beta by the row-major product (launch_xbeta_csr).
#include "common.cuh"
#include "mm.h"

namespace ccdb {
namespace {

constexpr int kMT = 256;

__device__ __forceinline__ double mm_share(const MMParams& P, int32_t grp, int64_t k) {
    return P.nEv[grp] * P.xbe[k].y / P.denom[grp];
}

__global__ void __launch_bounds__(kMT) mm_share_kernel(MMParams P) {
    for (int64_t k = (int64_t)blockIdx.x * kMT + threadIdx.x; k < P.K; k += (int64_t)gridDim.x * kMT) {
        const int32_t grp = P.grp[k];
        P.share[k] = mm_share(P, grp, k);
    }
}

// Small calls, and matrices with few entries for their rows, work the share out for
// each entry: the launch before costs 3 us of some 30 (8 columns of 200 entries,
// 20,000 rows: 28 us, with it 33; of 30,000 entries, 300,000 rows: 137 and 100).
// incrementMMGradientAndHessian of the Survival models (ModelSpecifics.h:499-516,
// the conditional and Cox models): weight = hNWeight and denominator =
// denomPid of the row's group; indicator columns drop x.  Latency of the gathers:
// 2.6 million entries over 130,000 rows 25 us and the shares 4, 41 before.
template <bool SHARES>
__global__ void __launch_bounds__(kMT) mm_gh_kernel(MMParams P) {
    __shared__ double2 s_red[kMT / 32];
    const int j = blockIdx.x;
    if (P.fixed && P.fixed[j]) {
        if (threadIdx.x == 0) P.gh[j] = make_double2(0.0, 0.0);
        return;
    }
    const uint8_t f = P.fmt[j];
    const bool has_rows = (f == F_SPARSE || f == F_INDICATOR);
    const bool has_vals = (f == F_SPARSE || f == F_DENSE);
    const bool ind = (f == F_INDICATOR || f == F_INTERCEPT);
    const int64_t cb = P.col_ptr[j], vb = P.val_ptr[j];
    const int64_t n = has_rows ? (P.col_ptr[j + 1] - cb) : P.K;
    double g = 0.0, h = 0.0;
#pragma unroll 4
    for (int64_t p = threadIdx.x; p < n; p += kMT) {
        const int64_t k = has_rows ? (int64_t)__ldg(P.rows + cb + p) : p;
        const double r = SHARES ? P.share[k] : mm_share(P, P.grp[k], k);
        if (ind) {
            g += r;
            h += r;
        } else {
            const double x = has_vals ? __ldg(P.vals + vb + p) : 1.0;
            g += r * x;
            h += r * x * x;
        }
    }
    const double2 t = block_sum2<kMT / 32>(make_double2(g, h), s_red);
    if (threadIdx.x == 0) {
        const double gj = t.x - P.xjy[j];  // precomputeGradient
        P.gh[j] = make_double2(gj, t.y);
        if (P.step) {
            const double b = P.beta[j];
            const double delta = newton_prior_delta(gj, t.y, b, P.ptype[j], P.pvar[j]);
            if (delta != 0.0) P.beta[j] = b + delta;
        }
    }
}

}  // namespace

cudaError_t launch_mm_gradient_hessian(const MMParams& P, cudaStream_t s) {
    if (P.J <= 0) return cudaSuccess;
    const int64_t blocks = (P.K + kMT - 1) / kMT;
    if (P.share) {
        mm_share_kernel<<<(unsigned)(blocks < 1184 ? blocks : 1184), kMT, 0, s>>>(P);
        mm_gh_kernel<true><<<P.J, kMT, 0, s>>>(P);
    } else {
        mm_gh_kernel<false><<<P.J, kMT, 0, s>>>(P);
    }
    return cudaGetLastError();
}

}  // namespace ccdb
