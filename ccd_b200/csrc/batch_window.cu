// batch_window.cu -- many fits over one matrix in one launch (the
// cross-validation grid: folds x prior variances), each fit on one CTA with the
// next four or sixteen columns in flight.
//
// An instance has its own row weights (0 on its held-out fold, as
// CrossValidationSelector::getWeights sets them, drivers/CrossValidationSelector.cpp:72-130),
// prior variance, coefficients and bounds.  CTAs take instances from a queue,
// weakest priors first, and never wait for one another.  The sweep is the one of
// window.cu on one CTA: sixteen warps, in teams of one or four with a column
// each, gather gradients against the same state, and in visiting order a step
// stands unless an earlier column in flight that shares a row with it moves or is
// itself held back; four helper warps copy ahead and decide what is in flight
// next.  The instance therefore takes exactly the steps of the sequential cycle
// (CyclicCoordinateDescent.cpp:1008-1021).  After convergence it reports the
// predictive log-likelihood of its held-out rows (ModelSpecifics.hpp:652-690).
//
// State of a row: xBeta in FP64 and its share of a gradient, from which a
// gather makes an entry's terms.  FP64: p = exp(xBeta) / (1 + exp(xBeta)) or
// exp(xBeta), eight bytes.  Mixed precision (FP32 terms, compensated sums, FP64
// from the warp's sum on): exp(-|xBeta|) with the sign of xBeta, or exp(xBeta),
// four bytes.  A row of the held-out fold is marked in its share, so a gather
// needs no weight: FP64 and Poisson by the sign, logistic in mixed precision by a
// magnitude above one.
//
// A round is a chain of latencies, about 4,300 SM clocks with teams of four
// (gather 1,150, sums 740, step 610, update 700, two barriers and the decision
// between them the rest), and the launch lasts as long as the fit with the most
// cycles.  What shortens it: no exp and no division in a gather; the two entries
// that a thread of a team has stay in registers from the gather to the update;
// xBeta, when it is in global memory, is loaded with the gather where the step is
// going to stand; the bounds are settled by a helper.  With one warp a column,
// seven entries a lane, the mixed grid below takes 53 ms where teams of four took
// 27.  Measured on a B200: 200 mixed fits of 40,000 x 1,001 in 22 ms, in lockstep
// groups with a cluster exchange a column 82; 100 FP64 fits of 8,000 x 301 in 3.5
// ms, one column at a time with exp and division in the gather 12.1.
//
// The helpers' copies go through the copy engine and are awaited with a bound; a
// wait that runs out is reported as a timeout of the instance.
#include <algorithm>
#include <cstdint>
#include <type_traits>

#include "batch_common.cuh"
#include "batch_window.h"
#include "window_device.cuh"

namespace ccdb {

namespace {

using namespace win;
using bm::two_sum;

constexpr int kLane = 4;  // staged entries per lane
// A copy under way in a helper's `phase`: 2, and this too where the bound is below one
// sleep of a wait, so that the test for a copy is the test for such a bound (one more
// in front of each wait had cost 0.5 %).
constexpr unsigned kBriefStep = 1u << 16;

// A column has a team of T warps, so kWindow / T columns are in flight.
template <int T>
struct Team {
    static constexpr int kCols = kWindow / T;
    static constexpr int kLanes = 32 * T;
    static constexpr int kStaged = kLane * kLanes;  // room for a column's first entries, copied ahead
    static constexpr unsigned kSlots = (1u << kCols) - 1;
    static constexpr int kCopy = 8 * T;  // lanes of a helper that copy for a column
};

// What shared memory holds of a row: everything; the share alone; nothing
enum Where : int { kBoth = 0, kShare = 1, kNone = 2 };

template <int MODEL, bool MX>
using Share = std::conditional_t<MX, float, double>;

// A row's share at xBeta; a held-out row's is marked and gives no terms.
template <int MODEL, bool MX>
__device__ __forceinline__ Share<MODEL, MX> share_of(double xb, bool held) {
    if constexpr (MX) {
        const float xf = (float)xb;
        if (MODEL == M_LOGISTIC) {
            const float a = expf(-fabsf(xf));
            return held ? 2.0f : (xf >= 0.0f) ? a : -a;
        }
        return held ? -1.0f : expf(xf);
    } else {
        const double e = exp(xb);
        const double p = (MODEL == M_LOGISTIC) ? e / (1.0 + e) : e;
        // the sign marks the row; a share that is not finite keeps its effect on the sums
        const long long b = __double_as_longlong(held ? 0.0 * p : p);
        return __longlong_as_double(held ? b | (1ll << 63) : b & ~(1ll << 63));
    }
}
template <int MODEL, bool MX>
__device__ __forceinline__ bool is_held(Share<MODEL, MX> s) {
    if constexpr (MX) return MODEL == M_LOGISTIC ? s > 1.0f : s < 0.0f;
    else return __double_as_longlong(s) < 0;
}

// the share of no row: no terms
template <int MODEL, bool MX>
__device__ __forceinline__ Share<MODEL, MX> no_share() {
    if constexpr (MX) return MODEL == M_LOGISTIC ? 2.0f : -1.0f;
    else return -0.0;
}

template <bool MX>
struct Sums {
    double g = 0.0, h = 0.0;
};
template <>
struct Sums<true> {
    float g = 0.f, gc = 0.f, h = 0.f, hc = 0.f;
};

// One entry's gradient and Hessian terms from its row's share
// (ModelSpecifics.h:541-568 logistic, :1509-1530 Poisson).
template <int MODEL, bool MX>
__device__ __forceinline__ void add_entry(bool ind, double x, Share<MODEL, MX> s, Sums<MX>& a) {
    if constexpr (MX) {
        const float xf = ind ? 1.0f : (float)x;
        float t, ht;
        if (MODEL == M_LOGISTIC) {
            const float e = fabsf(s);
            const float r = __frcp_rn(1.0f + e), er = e * r;
            const bool up = __float_as_int(s) >= 0;  // xBeta >= 0
            t = up ? r : er;
            ht = t * (up ? er : r);
        } else {
            t = ht = s;
        }
        const bool held = is_held<MODEL, MX>(s);
        float gt = ind ? t : t * xf;
        ht = ind ? ht : ht * (xf * xf);
        two_sum(a.g, a.gc, held ? 0.0f : gt);
        two_sum(a.h, a.hc, held ? 0.0f : ht);
    } else {
        const double t = ind ? s : s * x;
        a.g += t;
        if (MODEL == M_LOGISTIC) a.h += ind ? t * (1.0 - t) : t * x - t * t;
        else a.h += ind ? t : t * x;
    }
}

// Sums of g over the warp in lanes 0..15 and of h in lanes 16..31.
template <bool MX>
__device__ __forceinline__ double warp_pair_sum(const Sums<MX>& a) {
    double g, h;
    if constexpr (MX) {
        g = (double)a.g + (double)a.gc;
        h = (double)a.h + (double)a.hc;
    } else {
        g = a.g;
        h = a.h;
    }
    const bool upper = threadIdx.x & 16;
    double mine = upper ? h : g;
    const double other = upper ? g : h;
    mine += __shfl_xor_sync(kFull, other, 16);
#pragma unroll
    for (int o = 8; o > 0; o >>= 1) mine += __shfl_xor_sync(kFull, mine, o);
    return mine;
}

template <int MODEL, bool MX, int WHERE, int T>
__global__ void __launch_bounds__(kT, 1) batch_window_kernel(BatchWindowParams R) {
    using S = Share<MODEL, MX>;
    constexpr int W = Team<T>::kCols, L = Team<T>::kLanes, kStaged = Team<T>::kStaged, kCopy = Team<T>::kCopy;
    __shared__ Rec s_rec[4][W];  // by position: (position / W) & 3, slot
    __shared__ double s_red[kWindow][2];
    __shared__ double4 s_red4[kWarps];
    __shared__ double s_delta[2][W];  // by round parity: the column's step
    __shared__ unsigned s_holders[W];  // the slots that hold the column back if they move
    __shared__ Turn s_turn;
    __shared__ unsigned long long s_count[2];  // nonzero steps and their entries
    __shared__ int s_next, s_failed;
    __shared__ uint64_t s_bar[kHelpers];
    extern __shared__ __align__(16) unsigned char s_dyn[];

    const BatchParams& P = R.P;
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    const int n_active = R.n_active, n_rows = (int)P.K;
    // dynamic shared memory: the staged rows, the state, the staged values (where there are any)
    int32_t* const s_rows = reinterpret_cast<int32_t*>(s_dyn);
    unsigned char* const s_state = s_dyn + 2 * W * kStaged * sizeof(int32_t);
    double* const s_vals = reinterpret_cast<double*>(s_dyn + R.vals_at);
    double* const xb = (WHERE == kBoth) ? reinterpret_cast<double*>(s_state) : R.xbeta + (size_t)blockIdx.x * n_rows;
    S* const share = (WHERE == kNone)   ? reinterpret_cast<S*>(R.share) + (size_t)blockIdx.x * n_rows
                     : (WHERE == kBoth) ? reinterpret_cast<S*>(s_state + sizeof(double) * n_rows)
                                        : reinterpret_cast<S*>(s_state);
    WinScal* const scal = R.scal + (size_t)blockIdx.x * n_active;
    double2* const bh = R.bh + (size_t)blockIdx.x * n_active;

    auto update = [&](int k, double x0, double delta_x) {
        const double x = x0 + delta_x;
        xb[k] = x;
        share[k] = share_of<MODEL, MX>(x, is_held<MODEL, MX>(share[k]));
    };
    // what the helpers copy ahead: records two columns ahead of a warp, entries one
    auto rec_of = [&](int at) -> Rec& { return s_rec[(at / W) & 3][at & (W - 1)]; };
    const Ahead ahead{R.cols, scal, bh, R.slices, P.rows, P.vals, n_active};
    auto fetch = [&](int at, int l8) { ahead.record(at, rec_of(at), l8); };
    // a column's first entries, from the 16-byte boundary at or before them: the lane
    // that copies for a column calls begin, then each copy of the warp is awaited
    auto stage = [&](int at, bool leads, unsigned& phase) {
        unsigned nr = 0, nv = 0;
        const Rec& r = rec_of(at);
        if (leads && at < n_active && !(r.c.flags & 8)) {
            const int n = min(r.c.n, kStaged - 4);
            if (r.c.flags & 1) nr = ((n + (int)(r.c.cb & 3)) * 4 + 15) & ~15;
            if (r.c.flags & 2) nv = ((n + (int)(r.c.vb & 1)) * 8 + 15) & ~15;
        }
        const unsigned total = __reduce_add_sync(kFull, nr + nv);
        if (total == 0) return;
        uint64_t* const bar = &s_bar[wid - kWindow];
        if (lane == 0) expect_bytes(bar, total);
        __syncwarp();
        const int to = stage_at<kStaged, W>(at);
        if (nr) bulk_copy(s_rows + to, P.rows + (r.c.cb & ~int64_t(3)), nr, bar);
        if (nv) bulk_copy(s_vals + to, P.vals + (r.c.vb & ~int64_t(1)), nv, bar);
        phase += R.step;  // bit 0: the parity to wait for; above: copies under way
    };
    auto staged_all = [&](unsigned& phase) {
        bool ok;
        if (phase - 2 < kBriefStep - 2) ok = wait_sleeping(&s_bar[wid - kWindow], phase & 1, P.xch_wait_ns);
        else if (phase < 2) return true;
        else ok = wait_looking(&s_bar[wid - kWindow], phase & 1, P.xch_wait_ns);
        if (!ok) drain(&s_bar[wid - kWindow], phase & 1);  // what is under way lands before the CTA leaves
        phase = (phase & 1) ^ 1;
        return ok;
    };

    unsigned phase = 0;  // of a helper's copies
    if (tid == 0) {
        s_failed = 0;
        init_bars(s_bar, kHelpers);
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    for (;;) {
        if (tid == 0) s_next = atomicAdd(P.queue, 1);
        __syncthreads();
        const int turn_no = s_next;
        if (turn_no >= P.n_inst) break;
        const int inst = P.order[turn_no];
        const int hold = P.holdout[inst];
        const double var = P.variance[inst];
        if (tid < 2) s_count[tid] = 0;

        // ---- the instance's xBeta, XjY (ModelSpecifics.hpp:486-524), coefficients and shares
#pragma unroll 1
        for (int k = tid; k < n_rows; k += kT) {
            xb[k] = P.offset_vals ? 0.0 + 1.0 * P.offset_vals[k] : 0.0;
            const bool held = hold >= 0 && P.row_fold && P.row_fold[k] == hold;
            share[k] = held ? share_of<MODEL, MX>(0.0, true) : share_of<MODEL, MX>(xb[k], false);
        }
        __syncthreads();
        auto xy_part = [&](const WinCol& c, int from, int by) {
            double v = 0.0;
#pragma unroll 4
            for (int e = from; e < c.n; e += by) {
                const int k = (c.flags & 1) ? __ldg(P.rows + c.cb + e) : e;
                const double x = (c.flags & 2) ? __ldg(P.vals + c.vb + e) : 1.0;
                v += x * P.y[k] * (is_held<MODEL, MX>(share[k]) ? 0.0 : 1.0);
            }
            return v;
        };
        auto begin_column = [&](int q, int j, double xjy) {
            const int pt = P.ptype[j];
            const double pv = pt == 0 ? 1.0 : var;
            scal[q] = WinScal{xjy, pv, pt == 1 ? sqrt(2.0 / pv) : 0.0, pt == 2 ? 1.0 / pv : 0.0, pt, 0, 0};
            bh[q] = make_double2(0.0, P.initial_bound);
        };
#pragma unroll 1
        for (int q = wid; q < n_active; q += kWarps) {
            const WinCol c = R.cols[q];
            if (c.flags & 8) continue;
            double v = xy_part(c, lane, 32);
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(kFull, v, o);
            if (lane == 0) begin_column(q, c.j, v);
        }
#pragma unroll 1
        for (int i = 0; i < R.n_long; ++i) {
            const int q = R.longs[i];
            const WinCol c = R.cols[q];
            const double4 v = block_sum4<kWarps>(make_double4(xy_part(c, tid, kT), 0.0, 0.0, 0.0), s_red4);
            if (tid == 0) begin_column(q, c.j, v.x);
        }
        __syncthreads();

        // ---- the objective (ModelSpecifics.hpp:103-120, 605-650; JointPrior.h:121-128)
        auto objective = [&](double& ll) {
            double4 acc = make_double4(0.0, 0.0, 0.0, 0.0);
#pragma unroll 1
            for (int k = tid; k < n_rows; k += kT) {
                const double x = xb[k], yk = P.y[k];
                const double w = is_held<MODEL, MX>(share[k]) ? 0.0 : 1.0;
                acc.z += x * yk * w;
                if (P.conv != C_GRADIENT) {
                    const double e = exp(x);
                    acc.x += (double)((int)yk) * x * w;
                    acc.y += w * ((MODEL == M_LOGISTIC) ? log(1.0 + e) : e);
                }
            }
            if (P.conv == C_LANGE) {
#pragma unroll 1
                for (int q = tid; q < n_active; q += kT) acc.w += log_prior_one(bh[q].x, scal[q].ptype, scal[q].pvar);
                // a column that is not stepped (the offset) keeps its coefficient of one
                if (tid == 0 && P.offset_vals) acc.w += log_prior_one(1.0, P.ptype[0], P.ptype[0] == 0 ? 1.0 : var);
            }
            acc = block_sum4<kWarps>(acc, s_red4);
            ll = (acc.x - acc.y) + ((MODEL == M_POISSON && P.ll_fixed) ? P.ll_fixed[inst] : 0.0);
            return (P.conv == C_GRADIENT) ? acc.z : (P.conv == C_MITTAL ? ll : ll + acc.w);
        };

        double ll, last = 0.0;
        int iteration = 0, flag = R_FAIL;
        for (;; ++iteration) {
            // ---- a cycle is complete: convergence (findMode, CyclicCoordinateDescent.cpp:541-558, 839-906)
            const double cur = objective(ll);
            const double before = last;
            last = cur;
            if (iteration > 0) {
                const bool ill = cur != cur;
                const double conv = ill ? 0.0 : fabs(cur - before) / (fabs(cur) + 1.0);
                if (P.tol > 0 && conv < P.tol) {
                    flag = ill ? R_ILLCONDITIONED : R_SUCCESS;
                    break;
                }
                if (iteration == P.max_iter) {
                    flag = R_MAX_ITERATIONS;
                    break;
                }
            } else if (P.max_iter <= 0 && !(MX && P.tol > 0)) {
                break;  // no cycle at all; mixed fits without a limit end by the tolerance
            }
            if (wid >= kWindow) {
                // ================ a helper: lane l follows slot l; the lanes of all share out the copies
                const int me = wid - kWindow;
                unsigned long long moved = 0, entries = 0;  // nonzero steps, their entries
                int q = lane < W ? lane : 0x7fffffff;  // the slot's position
                const int l8 = lane & (kCopy - 1), mine = me + kHelpers * (lane / kCopy);  // kCopy lanes a slot
                for (int i = 0; i < 3; ++i) fetch(mine + i * W, l8);
                ahead.done();
                bool ok = true;
                for (int i = 0; i < 2; ++i) {
                    stage(mine + i * W, l8 == 0, phase);
                    ok = staged_all(phase) && ok;
                }
                if (!ok) s_failed = 1;
                unsigned moved_on = 0;  // the slots that took up a new column in the last round
                int par = 0;
                // the bound of a column whose step was taken in the last round, and its
                // coefficient where the step moved it (lane l: slot l), off the warps' path
                auto settle = [&]() {
                    if (me != kHelpers - 1 || !(moved_on >> lane & 1u)) return;
                    const Rec& r = rec_of(q - W);
                    const double d = s_delta[par ^ 1][lane];
                    double hd = r.bh.y;
                    apply_bounds(d, hd);
                    bh[q - W] = make_double2(d != 0.0 ? r.bh.x + d : r.bh.x, hd);
                    if (d != 0.0) {
                        ++moved;
                        entries += r.c.n;
                    }
                };
                Turn t{0, 0, 0, 0};
                // what is in flight next: a column runs alone when it is long, or medium and
                // expected to move (nothing holds it at zero, or a warp has found its step)
                bool found = false;  // lane l: slot l is medium and its step is not zero
                auto next_turn = [&]() {
                    bool alone = found;
                    if (q < n_active && !found) {
                        const Rec& r = rec_of(q);
                        alone = (r.c.flags & 8) || ((r.c.flags & 16) && (r.s.ptype != 1 || r.bh.x != 0.0));
                    }
                    t.base = __reduce_min_sync(kFull, q);
                    const int first_alone = __reduce_min_sync(kFull, alone ? q : 0x7fffffff);
                    t.alone = t.base == first_alone;
                    t.limit = t.alone ? t.base + 1 : min(min(t.base + W, first_alone), n_active);
                    if (me == 0 && lane == 0) s_turn = t;
                };
                __syncthreads();  // every helper's records
                next_turn();
                __syncthreads();
                while (t.base < n_active && !s_failed) {
                    const bool flying = q < t.limit;
                    const unsigned slots = __ballot_sync(kFull, flying);
                    const int turn = t.base & (W - 1);
                    if (me == 0) {
                        // the earlier columns in flight that hold a column back if they move: those
                        // it shares a row with, and those that may hold one of these back
                        unsigned holders = 0;
                        if (flying && !t.alone) {
                            const unsigned rel = (slots >> turn | slots << (W - turn)) & Team<T>::kSlots;
                            holders = ((unsigned)rec_of(q).c.conflict >> (kWindow - 1 - (q - t.base))) & rel;
                        }
#pragma unroll
                        for (int i = 0; i < W - 1; ++i) {
                            const unsigned more = __shfl_sync(kFull, holders, (turn + i) & (W - 1));
                            if (holders >> i & 1u) holders |= more;
                        }
                        // from positions relative to base to slots
                        if (lane < W) s_holders[lane] = (holders << turn | holders >> (W - turn)) & Team<T>::kSlots;
                    }
                    const int at = __shfl_sync(kFull, q, mine);
                    const bool moved_mine = moved_on >> mine & 1u;
                    stage(at + W, moved_mine && l8 == 0, phase);
                    if (moved_mine) fetch(at + 2 * W, l8);
                    settle();
                    __syncthreads();
                    // ---- which steps stand, and what is in flight next
                    const unsigned moves = __ballot_sync(kFull, flying && s_delta[par][lane & (W - 1)] != 0.0);
                    bool stands = flying && (s_holders[lane & (W - 1)] & moves) == 0;
                    found = stands && !t.alone && (moves >> lane & 1u) && (rec_of(q).c.flags & 16);
                    stands = stands && !found;
                    const unsigned taken = __ballot_sync(kFull, stands);
                    if (taken >> lane & 1u) q += W;
                    moved_on = taken;
                    par ^= 1;
                    next_turn();
                    ahead.done();
                    if (!staged_all(phase)) s_failed = 1;
                    __syncthreads();
                }
                settle();
                if (moved) {
                    atomicAdd(&s_count[0], moved);
                    atomicAdd(&s_count[1], entries);
                }
            } else {
                // ================ a warp with a column
                const int team = wid / T, me = tid & (L - 1);  // its slot, the thread's place in it
                int pos = team;
                bool fresh = true;  // the column's first round
                int par = 0;
                __syncthreads();
                __syncthreads();
                for (;;) {
                    const Turn now = s_turn;
                    if (now.base >= n_active || s_failed) break;
                    const bool alone = now.alone != 0, mine = alone || pos < now.limit;
                    const int slot = alone ? now.base & (W - 1) : team;
                    const int at = alone ? now.base : pos;
                    const Rec& r = rec_of(at);
                    const int n = r.c.n, flags = r.c.flags;
                    const bool ind = flags & 4, has_vals = flags & 2;
                    const int staged = (flags & 8) ? 0 : min(n, kStaged - 4);
                    const int32_t* const kr = s_rows + stage_at<kStaged, W>(at) + (int)(r.c.cb & 3);
                    const double* const xr = s_vals + stage_at<kStaged, W>(at) + (int)(r.c.vb & 1);
                    // entry e of the column, whether copied ahead or not
                    auto entry_row = [&](int e) {
                        return !(flags & 1) ? e : e < staged ? kr[e] : __ldg(P.rows + r.c.cb + e);
                    };
                    auto entry_val = [&](int e) {
                        return !has_vals ? 1.0 : e < staged ? xr[e] : __ldg(P.vals + r.c.vb + e);
                    };
                    // a column that is all copied ahead, by its own team: the first two entries of a
                    // thread stay in registers from the gather to the update (nothing touches a row of
                    // a column whose step stands in between)
                    const bool quick = !alone && (flags & 1) && n <= kStaged - 4;
                    const int first = alone ? tid : me, stride = alone ? kWorkers : L;
                    const bool second = (me & ~31) + L < n;  // some thread of the warp has a second entry
                    int k0 = 0, k1 = 0;
                    double x0 = 0.0, x1 = 0.0;
                    S s0 = no_share<MODEL, MX>(), s1 = s0;
                    bool loaded = false;
                    double d = 0.0;
                    if (mine) {
                        Sums<MX> a;
                        const double b0 = r.bh.x, hd = r.bh.y;
                        const double xjy = r.s.xjy, lambda = r.s.lambda, inv_var = r.s.inv_var, pvar = r.s.pvar;
                        const int pt = r.s.ptype;
                        if (quick) {
                            // xBeta from global memory: early where the step will stand (no earlier column
                            // in flight shares a row) and likely move
                            loaded = WHERE == kBoth || ((b0 != 0.0 || !fresh || pt != 1) &&
                                                        ((unsigned)r.c.conflict >> (kWindow - 1 - (pos - now.base))) == 0);
                            if (me < n) {
                                k0 = kr[me];
                                s0 = share[k0];
                                if (me + L < n) {
                                    k1 = kr[me + L];
                                    s1 = share[k1];
                                }
                                if (loaded) {
                                    x0 = xb[k0];
                                    if (me + L < n) x1 = xb[k1];
                                }
                                if (has_vals) {
                                    add_entry<MODEL, MX>(false, xr[me], s0, a);
                                    if (me + L < n) add_entry<MODEL, MX>(false, xr[me + L], s1, a);
                                } else {
                                    add_entry<MODEL, MX>(true, 1.0, s0, a);
                                    if (second) add_entry<MODEL, MX>(true, 1.0, s1, a);
                                }
                            }
#pragma unroll 1
                            for (int e = me + 2 * L; e < n; e += L)
                                add_entry<MODEL, MX>(ind, has_vals ? xr[e] : 1.0, share[kr[e]], a);
                        } else {
#pragma unroll 4
                            for (int e = first; e < n; e += stride)
                                add_entry<MODEL, MX>(ind, entry_val(e), share[entry_row(e)], a);
                        }
                        double v = warp_pair_sum<MX>(a);
                        if (alone || T > 1) {
                            if ((lane & 15) == 0) s_red[wid][lane >> 4] = v;
                            if (alone) {
                                workers_barrier();
                                v = s_red[lane & 15][lane >> 4];
#pragma unroll
                                for (int o = 8; o >= T; o >>= 1) v += __shfl_xor_sync(kFull, v, o);
                            } else {
                                asm volatile("bar.sync %0, %1;" ::"r"(2 + team), "n"(L) : "memory");
                                v = s_red[team * T + (lane & (T - 1))][lane >> 4];
                            }
#pragma unroll
                            for (int o = T / 2; o > 0; o >>= 1) v += __shfl_xor_sync(kFull, v, o);
                        }
                        const double b_var = pt == 2 ? b0 / pvar : 0.0;
                        double2 t = make_double2(__shfl_sync(kFull, v, 0), __shfl_sync(kFull, v, 16));
                        if (n > 0) t.x -= xjy;
                        else t = make_double2(0.0, 0.0);  // an empty column gives (0, 0) (ModelSpecifics.hpp:720-723)
                        d = newton_quotient_step(t.x, t.y, b0, pt, pvar, lambda, inv_var, b_var);
                        d = (d < -hd) ? -hd : (d > hd ? hd : d);  // apply_bounds; its new bound is not needed yet
                        if (me == 0) s_delta[par][team] = d;
                    }
                    fresh = false;
                    __syncthreads();
                    const unsigned moves = __ballot_sync(kFull, s_delta[par][lane & (W - 1)] != 0.0) & Team<T>::kSlots;
                    par ^= 1;
                    // does the step stand (a medium column's waits until it runs alone)
                    if (mine && (alone || ((s_holders[team] & moves) == 0 && !((flags & 16) && d != 0.0)))) {
                        if (d != 0.0) {
                            int e = first;
                            if (quick) {
                                if (!loaded) {
                                    if (me < n) x0 = xb[k0];
                                    if (me + L < n) x1 = xb[k1];
                                }
                                x0 += has_vals && me < n ? d * xr[me] : d;
                                const S n0 = share_of<MODEL, MX>(x0, is_held<MODEL, MX>(s0));
                                if (second) {
                                    x1 += has_vals && me + L < n ? d * xr[me + L] : d;
                                    const S n1 = share_of<MODEL, MX>(x1, is_held<MODEL, MX>(s1));
                                    if (me + L < n) {
                                        xb[k1] = x1;
                                        share[k1] = n1;
                                    }
                                }
                                if (me < n) {
                                    xb[k0] = x0;
                                    share[k0] = n0;
                                }
                                e += 2 * L;
                            }
#pragma unroll 2
                            for (; e < n; e += stride) {
                                const int k = entry_row(e);
                                update(k, xb[k], d * entry_val(e));
                            }
                        }
                        if (team == slot) {  // pos is the position of this column
                            pos += W;
                            fresh = true;
                        }
                    }
                    __syncthreads();
                }
            }
            __syncthreads();
            if (s_failed) break;
        }
        if (s_failed) {  // a copy did not come within its time
            if (tid == 0) {
                BatchResult r{};
                r.flag = kBatchTimeoutFlag;
                P.results[inst] = r;
            }
            break;
        }
        // ---- the log-likelihoods of the training and of the held-out rows, the coefficients
        double4 acc = make_double4(0.0, 0.0, 0.0, 0.0);
#pragma unroll 1
        for (int k = tid; k < n_rows; k += kT) {
            const double x = xb[k], yk = P.y[k], e = exp(x);
            const double w = is_held<MODEL, MX>(share[k]) ? 0.0 : 1.0, wo = 1.0 - w;
            acc.x += (double)((int)yk) * x * w;
            if (MODEL == M_LOGISTIC) {
                const double lg = log(1.0 + e);
                acc.y += w * lg;
                acc.z += yk * wo * (x - lg);
            } else {
                acc.y += w * e;
                acc.z += (yk * x - e) * wo;
            }
        }
        acc = block_sum4<kWarps>(acc, s_red4);
        double* const out = R.beta_out + (size_t)inst * P.J;
#pragma unroll 1
        for (int q = tid; q < n_active; q += kT) out[R.cols[q].j] = bh[q].x;
        if (tid == 0) {
            if (P.offset_vals) out[0] = 1.0;
            BatchResult r;
            r.flag = flag;
            r.iterations = iteration;
            r.loglik = (acc.x - acc.y) + ((MODEL == M_POISSON && P.ll_fixed) ? P.ll_fixed[inst] : 0.0);
            r.objective = last;
            r.pred_loglik = acc.z;
            r.steps = (long long)iteration * n_active;
            r.updates = (long long)s_count[0];
            r.update_entries = (long long)s_count[1];
            r.sweep_entries = (long long)iteration * R.entries;
            P.results[inst] = r;
        }
        __syncthreads();
    }
}

// Static shared memory of the kernel stays below this.
constexpr int64_t kStaticSmem = 12288;
constexpr int64_t kStagedRows = 2 * kWindow * 32 * kLane * sizeof(int32_t);  // whatever the team
constexpr int64_t kStagedVals = 2 * kWindow * 32 * kLane * sizeof(double);

using Kernel = void (*)(BatchWindowParams);

template <int MODEL, bool MX, int T>
Kernel pick(int where) {
    return where == kBoth    ? batch_window_kernel<MODEL, MX, kBoth, T>
           : where == kShare ? batch_window_kernel<MODEL, MX, kShare, T>
                             : batch_window_kernel<MODEL, MX, kNone, T>;
}
template <int T>
Kernel pick(int model, bool mixed, int where) {
    if (model == M_LOGISTIC) return mixed ? pick<M_LOGISTIC, true, T>(where) : pick<M_LOGISTIC, false, T>(where);
    return mixed ? pick<M_POISSON, true, T>(where) : pick<M_POISSON, false, T>(where);
}
Kernel pick(int model, bool mixed, int where, int team) {
    return team == 1 ? pick<1>(model, mixed, where) : pick<4>(model, mixed, where);
}

cudaError_t smem_limit(int64_t* bytes) {
    int dev = 0, optin = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
    *bytes = std::max<int64_t>(0, (int64_t)optin - kStaticSmem);
    return e;
}

// where the rows' state lies, and its bytes of shared memory
cudaError_t placement(int64_t K, bool mixed, bool vals, int* where, int64_t* state) {
    int64_t smem = 0;
    const cudaError_t e = smem_limit(&smem);
    smem -= kStagedRows + (vals ? kStagedVals : 0);
    const int64_t share = (mixed ? 4 : 8) * K;
    *where = 8 * K + share <= smem - 16 ? kBoth : share <= smem - 16 ? kShare : kNone;
    *state = *where == kBoth ? 8 * K + share : *where == kShare ? share : 0;
    *state = (*state + 15) & ~int64_t(15);
    return e;
}

}  // namespace

cudaError_t batch_window_spill(int64_t K, bool mixed, bool vals, int* spill) {
    int where = kNone;
    int64_t state = 0;
    const cudaError_t e = placement(K, mixed, vals, &where, &state);
    *spill = where == kBoth ? 0 : where == kShare ? 1 : 3;
    return e;
}

cudaError_t launch_batch_window(const BatchWindowParams& R, cudaStream_t stream) {
    int where = kNone;
    int64_t state = 0;
    cudaError_t e = placement(R.P.K, R.mixed != 0, R.any_vals != 0, &where, &state);
    if (e != cudaSuccess) return e;
    if ((where != kBoth && !R.xbeta) || (where == kNone && !R.share)) return cudaErrorInvalidValue;
    BatchWindowParams Q = R;
    Q.step = 2 + (R.P.xch_wait_ns < win::kLookNs ? kBriefStep : 0);
    Q.vals_at = (int32_t)(kStagedRows + state);
    const size_t smem = (size_t)(Q.vals_at + (R.any_vals ? kStagedVals : 0));
    static std::atomic<uint64_t> done{0};
    e = once_per_device(done, [] {  // of all kernels (why: window.cu)
        int64_t dyn = 0;
        cudaError_t r = smem_limit(&dyn);
        for (int model : {(int)M_LOGISTIC, (int)M_POISSON})
            for (int team : {1, 4})
                for (int v = 0; v < 6 && r == cudaSuccess; ++v)
                    r = cudaFuncSetAttribute(pick(model, v & 1, v >> 1, team), cudaFuncAttributeMaxDynamicSharedMemorySize,
                                             (int)dyn);
        return r;
    });
    if (e != cudaSuccess) return e;
    pick(R.P.model, R.mixed != 0, where, R.team)<<<R.ctas, kT, smem, stream>>>(Q);
    return cudaGetLastError();
}

}  // namespace ccdb
