// window.cu -- one findMode of an independent-row fit (logistic, Poisson) in
// one thread-block cluster whose CTAs share out the rows.
//
// The sweep is the sequential cycle (CyclicCoordinateDescent.cpp:1008-1021) with
// the next kWindow columns in flight at once, one per warp.  In a round every
// warp gathers its column's gradient and Hessian against the same state and
// takes the step; then, in visiting order, a column's step is taken unless an
// earlier column in flight that shares a row with it (the plan's conflict masks)
// moves or is itself held back.  A step that is taken saw exactly the state
// that the sequential cycle shows it: every earlier column that touches its
// rows is behind it, zero steps leave the state as it is, and columns without a
// common row touch different state.  The others stay in flight for the next
// round.  The bound (hDelta) changes with every visited coordinate, as
// applyBounds does, when its step is taken.  A column too long for one warp
// (the intercept, dense columns) runs alone, on every warp.
//
// Each CTA owns the rows [K r / C, K (r + 1) / C) and walks only their entries.
// The state of its rows stays with it, so the only thing that crosses CTAs is
// one (g, h) pair per column, CTA and round, sent to every CTA's shared memory
// by st.async and counted by the receiver's mbarrier; every CTA then adds the C
// pairs in the same order and takes the same decision.  There is no cluster
// barrier and no fence on global memory inside a cycle.
//
// State of a row: xBeta, exp(xBeta), the denominator, and its share of a
// gradient -- p = exp(xBeta) / denominator (logistic) or exp(xBeta) (Poisson).
// The share is all that a gradient gathers: one 8-byte word, no exp and no
// division per entry, computed once where the row changes.  It lives in shared
// memory when the CTA's rows fit (8 bytes a row), with xBeta and the
// denominator beside it when they fit too (24 bytes a row, 32 of a logistic fit, which
// keeps exp(xBeta) as well), and the weights when there is room for these besides (8
// more); otherwise they stay in global memory, where only their CTA touches them.
//
// Beside the sixteen warps with columns, four helper warps take everything that
// looks ahead off the round's path: they copy a warp's next entries and records
// into shared memory, close the conflict masks transitively and decide what is in
// flight next.
//
// A round is a chain of latencies (gather, warp sum, exchange, FP64 division,
// exp): nothing in it is bound by bandwidth, so what counts is how many dependent
// instructions it has and how many columns it takes.  Measured on a B200 at
// 1,965 MHz, a round is about 3,200 SM clocks (gather and warp sum 900, exchange
// 500, sums and step 550, update 750, two barriers and skew the rest) and takes
// 5.7 columns of the 10,000 x 1,001 L1 logistic fit: 4.2 ms a fit, where
// speculative batches on one CTA that recomputed exp and divided for every
// gathered entry took 9.3 ms.  60,000 x 2,501 L1 logistic: 45 ms; Poisson, 50,000
// x 4,002, every step nonzero: 136 ms; both ran one cluster barrier per
// dependency level before, at 217 and 398 ms.  Short straight code counts: with
// the CTAs' pairs added four at a time in every lane, bounds settled by the warps
// with columns and the gather unrolled, these took 4.5, 53 and 154 ms.
//
// The wait for the other CTAs' pairs is bounded (the fit's limit).  A CTA whose wait runs out
// steps and sends no more; at the end of the cycle the CTAs learn of it from one
// another and all leave, each once what was sent to it has landed (sweep_exit.h).
#include <algorithm>
#include <cstdint>

#include "window_device.cuh"

namespace ccdb {

namespace {

using namespace win;

// What shared memory holds of a row: everything; the share alone; nothing; or, on
// one CTA, xBeta and the denominator, from which a gather works the share out
enum Where : int { kAllShared = 0, kShareShared = 1, kGlobal = 2, kPairShared = 3 };

// One entry's gradient and Hessian terms from its row's share
// (ModelSpecifics.h:541-568 logistic, ModelSpecifics.h:1509-1530 Poisson).
template <int MODEL>
__device__ __forceinline__ void add_terms(bool ind, bool weighted, double x, double p, double w, double& g, double& h) {
    const double t = ind ? p : p * x;
    const double wt = weighted ? w * t : t;
    g += wt;
    if (MODEL == M_LOGISTIC) {
        if (ind) h += wt * (1.0 - t);
        else h += weighted ? w * (t * x - t * t) : t * x - t * t;
    } else {
        // the weight last, as in the reference: a row of weight zero whose term overflows
        // is not a number there either
        h += ind ? wt : weighted ? w * (t * x) : t * x;
    }
}

// Sums of g over the warp in lanes 0..15 and of h in lanes 16..31.
__device__ __forceinline__ double warp_pair_sum(double g, double h) {
    const bool upper = threadIdx.x & 16;
    double mine = upper ? h : g;
    const double other = upper ? g : h;
    mine += __shfl_xor_sync(kFull, other, 16);
#pragma unroll
    for (int o = 8; o > 0; o >>= 1) mine += __shfl_xor_sync(kFull, mine, o);
    return mine;
}

// The rows [r0, r0 + n) that a CTA owns.
template <int MODEL, int WHERE, bool WT>
struct Rows {
    double* share;   // by local row, in shared or global memory
    double* ex;      // exp(xBeta), shared form of a logistic fit (a Poisson share is it)
    double2* xd;     // {xBeta, denominator}, shared form
    double2* row;    // the engine's row words of the CTA's first row
    const double* wt;  // weights, wt_step words apart: beside the state, or in the row words
    int wt_step;

    static constexpr bool kPair = WHERE == kAllShared || WHERE == kPairShared;  // xd holds the row
    __device__ __forceinline__ double p(int k) const {
        if (WHERE != kPairShared) return share[k];
        const double2 s = xd[k];
        const double e = exp(s.x);
        return (MODEL == M_LOGISTIC) ? e / s.y : e;
    }
    // In shared memory where they fit beside the rest (8 bytes a row): read from the row
    // words, a second cache line an entry, they cost weighted fits whose columns nearly all
    // move more than the windows gave them (1,500 rows, 70 columns of 450 entries, normal
    // prior: logistic 4.51 ms, from shared memory 4.40, Poisson 4.16 and 4.06; 3,000 rows,
    // columns of 1,800: 6.3 and 5.7).
    __device__ __forceinline__ double weight(int k) const { return WT ? wt[(int64_t)k * wt_step] : 1.0; }
    // the row words that an update will read, on their way to L1 ahead of it
    __device__ __forceinline__ void expect(int k) const {
        if (!kPair) asm volatile("prefetch.global.L1 [%0];" ::"l"(row + 2 * (int64_t)k));
    }
    // xBeta += delta x, then exp, denominator and share (ModelSpecifics.hpp:1548-1571)
    __device__ __forceinline__ void update(int k, double delta_x) const {
        double2 s;
        double e0;
        if (kPair) {
            s = xd[k];
            e0 = (WHERE == kPairShared) ? exp(s.x) : (MODEL == M_LOGISTIC) ? ex[k] : share[k];
        } else {
            const double2 a = row[2 * (int64_t)k];
            s = make_double2(a.x, row[2 * (int64_t)k + 1].x);
            e0 = a.y;
        }
        s.x += delta_x;
        const double e = exp(s.x);
        s.y += e - e0;
        if (WHERE != kPairShared) share[k] = (MODEL == M_LOGISTIC) ? e / s.y : e;
        if (kPair) {
            xd[k] = s;
            if (WHERE == kAllShared && MODEL == M_LOGISTIC) ex[k] = e;
        } else {
            row[2 * (int64_t)k] = make_double2(s.x, e);
            row[2 * (int64_t)k + 1].x = s.y;
        }
    }
    __device__ __forceinline__ double2 xb_denominator(int k) const {
        if (kPair) return xd[k];
        return make_double2(row[2 * (int64_t)k].x, row[2 * (int64_t)k + 1].x);
    }
};

// FEW: no more columns than there are records in the buffers, 64; they stay there from
// cycle to cycle, and the entries of up to 32 columns beside them (a cycle of 30
// columns of a 1,000-row fit took 25.2 us, now 23.1; chosen when the kernel runs, it
// cost the fits with more columns 1.5 %).
template <int MODEL, int WHERE, bool CL, bool WT, bool FEW>
__global__ void __launch_bounds__(kT, 1) window_sweep_kernel(WindowParams R) {
    __shared__ Rec s_rec[4][kWindow];  // by position: (position / kWindow) & 3, slot
    __shared__ double2 s_pair[2][kWindow][kWindowCluster];  // (g, h) by round parity, column and CTA
    __shared__ double s_red[kWindow][2];
    __shared__ double4 s_red4[kWarps];
    // by cycle parity and CTA: a CTA that gave up may be a cycle ahead of one that reads them
    __shared__ double4 s_obj[CL ? 2 : 1][kWindowCluster];
    __shared__ CycleReport s_report[CL ? 2 : 1][kWindowCluster];
    __shared__ unsigned s_sent[2];  // bytes to each CTA, by exchange parity
    __shared__ double s_delta[2][kWindow];  // by round parity: the column's step
    __shared__ unsigned s_holders[kWindow];  // the slots that hold the column back if they move
    __shared__ Turn s_turn;
    __shared__ uint64_t s_bar[2];
    __shared__ int s_abort;
    extern __shared__ __align__(16) unsigned char s_dyn[];

    const IndepParams& P = R.P;
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    const int C = CL ? R.cluster : 1, rank = CL ? (int)blockIdx.x : 0;
    const int n_active = R.n_active;
    const int64_t r0 = window_row(P.K, rank, C);
    const int n_rows = (int)(window_row(P.K, rank + 1, C) - r0);
    Rows<MODEL, WHERE, WT> rows;
    rows.row = P.row + 2 * r0;
    // dynamic shared memory: the staged rows, the state, the staged values (where there are any)
    int32_t* const s_rows = reinterpret_cast<int32_t*>(s_dyn);
    double* const s_state = reinterpret_cast<double*>(s_rows + 2 * kWindow * kStage);
    double* const s_vals = reinterpret_cast<double*>(s_dyn + R.vals_at);
    rows.share = (WHERE == kGlobal) ? R.share + r0 : s_state;
    const int even = (n_rows + 1) & ~1;
    rows.ex = s_state + even;
    rows.xd = reinterpret_cast<double2*>(s_state + (WHERE == kPairShared ? 0 : MODEL == M_LOGISTIC ? 2 : 1) * even);
    const bool own_wt = WT && WHERE == kAllShared && R.weights_shared;
    double* const s_wt = reinterpret_cast<double*>(rows.xd + n_rows);
    rows.wt = own_wt ? s_wt : &rows.row[1].y;
    rows.wt_step = own_wt ? 1 : 4;
    const WinSlice* const slices = R.slices + (int64_t)rank * n_active;

    // ---- the state of the rows, the records of the columns
#pragma unroll 1
    for (int k = tid; k < n_rows; k += kT) {
        const double2 a = rows.row[2 * (int64_t)k];
        const double d = rows.row[2 * (int64_t)k + 1].x;
        if (WHERE != kPairShared) rows.share[k] = (MODEL == M_LOGISTIC) ? a.y / d : a.y;
        if (rows.kPair) rows.xd[k] = make_double2(a.x, d);
        if (WHERE == kAllShared && MODEL == M_LOGISTIC) rows.ex[k] = a.y;
        if (own_wt) s_wt[k] = rows.row[2 * (int64_t)k + 1].y;
    }
#pragma unroll 1
    for (int q = rank * kT + tid; q < n_active; q += C * kT) {
        const int j = R.cols[q].j;
        const double var = P.pvar[j];
        const int pt = P.ptype[j];
        R.scal[q] = WinScal{P.xjy[j], var, pt == 1 ? sqrt(2.0 / var) : 0.0, pt == 2 ? 1.0 / var : 0.0, pt, 0, 0};
        R.bh[q] = make_double2(P.beta[j], P.hdelta[j]);
    }
    if (tid == 0) {
        s_abort = 0;
        if (CL) {
            for (int i = 0; i < 2 * kWindow * kWindowCluster; ++i) (&s_pair[0][0][0])[i] = make_double2(0.0, 0.0);
            init_bars(s_bar, 2);
        }
    }
    if (CL) cluster_barrier();
    __syncthreads();

    // ---- exchange of one (g, h) pair per column between the CTAs
    unsigned n_xch = 0;  // exchanges so far: parity picks the buffer and its mbarrier
    // where this warp's pair goes: lane l sends to CTA l
    unsigned to_pair = 0, to_bar = 0;
    if (CL && lane < C) {
        to_pair = peer_u32(&s_pair[0][wid][rank], lane);
        to_bar = peer_u32(&s_bar[0], lane);
    }
    // lanes 0..15 hold g, lanes 16..31 h
    auto send_pair = [&](double v) {
        const double h = __shfl_xor_sync(kFull, v, 16);
        const unsigned par = n_xch & 1;
        if (lane < C) send16(to_pair + par * (unsigned)sizeof(s_pair[0]), to_bar + par * (unsigned)sizeof(s_bar[0]), v, h);
    };
    auto expect_pairs = [&](int columns) {
        expect_bytes(&s_bar[n_xch & 1], (unsigned)(columns * C * 2 * sizeof(double)));
    };
    auto wait_pairs = [&]() {
        if (!wait_bytes(&s_bar[n_xch & 1], (n_xch >> 1) & 1, P.wait_limit_ns)) s_abort = 1;
    };
    // the column's sums over the CTAs, the same bits in every lane and CTA (the
    // pairs of CTAs that there are not stay zero): lane l takes CTA l & 15, its g
    // below lane 16 and its h above
    auto pair_sum = [&](int c) {
        const double* from = &s_pair[n_xch & 1][c][lane & 15].x;
        double v = from[lane >> 4];
#pragma unroll
        for (int o = 8; o > 0; o >>= 1) v += __shfl_xor_sync(kFull, v, o);
        return v;
    };

    // ---- the objective terms {LL numerator, LL denominator, gradient objective,
    // log prior} (ModelSpecifics.hpp:103-120, 605-650; JointPrior.h:121-128); false
    // when a CTA gave up in this cycle
    auto objective = [&](int cycle, bool gave_up, double& obj, double& ll, double& lp) {
        double4 acc = make_double4(0.0, 0.0, 0.0, 0.0);
#pragma unroll 1
        for (int k = tid; k < n_rows; k += kT) {
            const double2 s = rows.xb_denominator(k);
            const double w = rows.weight(k), yk = P.y[r0 + k];
            acc.x += (double)((int)yk) * s.x * w;
            acc.y += w * ((MODEL == M_LOGISTIC) ? log(s.y) : s.y);
            acc.z += s.x * yk * w;
        }
        if (rank == 0)  // the CTA that writes the coefficients
#pragma unroll 1
            for (int j = tid; j < P.J; j += kT) acc.w += log_prior_one(P.beta[j], P.ptype[j], P.pvar[j]);
        acc = block_sum4<kWarps>(acc, s_red4);
        if (CL) {
            if (tid < C) {
                const unsigned a = peer_u32(&s_obj[cycle & 1][rank], tid);
                asm volatile("st.shared::cluster.v2.f64 [%0], {%1, %2};" ::"r"(a), "d"(acc.x), "d"(acc.y) : "memory");
                asm volatile("st.shared::cluster.v2.f64 [%0], {%1, %2};" ::"r"(a + 16), "d"(acc.z), "d"(acc.w) : "memory");
                tell(&s_report[cycle & 1][rank], tid, CycleReport{gave_up ? 1u : 0u, n_xch, {s_sent[0], s_sent[1]}});
            }
            cluster_barrier();  // also: rank 0's coefficients and bounds are seen by the next cycle
            acc = make_double4(0.0, 0.0, 0.0, 0.0);
            unsigned any = 0;
#pragma unroll 1
            for (int c = 0; c < C; ++c) {
                const double4 o = s_obj[cycle & 1][c];
                acc.x += o.x;
                acc.y += o.y;
                acc.z += o.z;
                acc.w += o.w;
                any |= s_report[cycle & 1][c].gave_up;
            }
            if (any) return false;
        }
        ll = (acc.x - acc.y) + P.ll_fixed;
        lp = acc.w;
        obj = (P.conv == C_GRADIENT) ? acc.z : (P.conv == C_MITTAL ? ll : ll + lp);
        return true;
    };

    // ---- what the helpers copy ahead: records two columns ahead of a warp, entries one
    auto rec_of = [&](int at) -> Rec& { return s_rec[(at / kWindow) & 3][at & (kWindow - 1)]; };
    const Ahead ahead{R.cols, R.scal, R.bh, slices, P.rows, P.vals, n_active};
    auto fetch = [&](int at, int l8) { ahead.record(at, rec_of(at), l8); };
    auto stage = [&](int at, int l8) { ahead.entries(at, rec_of(at), s_rows + stage_at(at), s_vals + stage_at(at), l8); };

    double last = 0.0;
    unsigned long long moved = 0;
    Tracer tracer{R.trace, rank == 0 && tid == kWorkers + 32, &s_turn.base};
    bool gave_up = false;  // a wait of this CTA ran out

    for (int iteration = 0;; ++iteration) {
        // ---- a cycle is complete: convergence (findMode, CyclicCoordinateDescent.cpp:1023-1056)
        double cur, ll, lp;
        if (!objective(iteration, gave_up, cur, ll, lp)) {  // every CTA leaves
            if (gave_up && tid == 0) {
                if (atomicCAS(&P.st->error, 0, E_WAIT_CLUSTER) == 0) P.st->error_where = rank;
                land_all(s_bar, s_report[iteration & 1], C, rank);
            }
            return;
        }
        if (iteration > 0) {
            const bool ill = cur != cur;
            const double conv = ill ? 0.0 : fabs(cur - last) / (fabs(cur) + 1.0);
            const bool met = P.tol > 0 && conv < P.tol, done = met || iteration == P.max_iter;
            if (rank == 0 && tid == 0) {
                P.st->iterations = iteration;
                P.st->objective = cur;
                P.st->loglik = ll;
                P.st->log_prior = lp;
                if (done) P.st->flag = !met ? R_MAX_ITERATIONS : (ill ? R_ILLCONDITIONED : R_SUCCESS);
            }
            if (done) break;
        }
        if (P.max_iter <= 0) break;  // no cycle at all
        last = cur;
        if (wid >= kWindow) {
            // ================ a helper: lane l follows slot l; each warp copies for a quarter of the slots
            const int me = wid - kWindow;
            int q = lane < kWindow ? lane : 0x7fffffff;  // the slot's position
            const int l8 = lane & 7, mine = me + kHelpers * (lane >> 3);  // eight lanes a slot
            const bool fetches = !FEW || iteration == 0;
            const bool stages = !FEW || iteration == 0 || n_active > 2 * kWindow;
            if (fetches) {
                for (int i = 0; i < 3; ++i) fetch(mine + i * kWindow, l8);
                ahead.done();
            }
            if (stages) {
                stage(mine, l8);
                stage(mine + kWindow, l8);
                ahead.done();
            }
            unsigned moved_on = 0;  // the slots that took up a new column in the last round
            int par = 0;
            // the bound of a column whose step was taken in the last round, and its
            // coefficient where the step moved it (lane l: slot l), off the warps' path
            auto settle = [&]() {
                if ((rank != 0 && !FEW) || me != kHelpers - 1 || !(moved_on >> lane & 1u)) return;
                Rec& r = rec_of(q - kWindow);
                const double d = s_delta[par ^ 1][lane];
                double2 bh = r.bh;
                apply_bounds(d, bh.y);
                if (d != 0.0) bh.x += d;
                if (FEW) r.bh = bh;
                if (rank != 0) return;
                if (d != 0.0) P.beta[r.c.j] = bh.x;
                R.bh[q - kWindow] = bh;
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
                t.limit = t.alone ? t.base + 1 : min(min(t.base + kWindow, first_alone), n_active);
                if (me == 0 && lane == 0) s_turn = t;
            };
            __syncthreads();  // every helper's records
            next_turn();
            __syncthreads();
            for (;;) {
                if (t.base >= n_active || t.stop) break;
                const bool flying = q < t.limit;
                const unsigned slots = __ballot_sync(kFull, flying);
                tracer.begin(t.base, __popc(slots), t.alone);
                const int turn = t.base & (kWindow - 1);
                if (me == 0) {
                    if (CL && lane == 0) {
                        expect_pairs(__popc(slots));
                        s_sent[n_xch & 1] = (unsigned)(__popc(slots) * 2 * sizeof(double));
                    }
                    // the earlier columns in flight that hold a column back if they move: those
                    // it shares a row with, and those that may hold one of these back
                    unsigned holders = 0;
                    if (flying && !t.alone) {
                        const unsigned rel = (slots >> turn | slots << (kWindow - turn)) & 0xffffu;
                        holders = ((unsigned)rec_of(q).c.conflict >> (kWindow - 1 - (q - t.base))) & rel;
                    }
#pragma unroll
                    for (int i = 0; i < kWindow - 1; ++i) {
                        const unsigned more = __shfl_sync(kFull, holders, (turn + i) & (kWindow - 1));
                        if (holders >> i & 1u) holders |= more;
                    }
                    // from positions relative to base to slots
                    if (lane < kWindow) s_holders[lane] = (holders << turn | holders >> (kWindow - turn)) & 0xffffu;
                }
                const int at = __shfl_sync(kFull, q, mine);
                if (moved_on >> mine & 1u) {
                    if (stages) stage(at + kWindow, l8);
                    if (fetches) fetch(at + 2 * kWindow, l8);
                }
                settle();
                if (CL) ++n_xch;
                __syncthreads();
                tracer.steps();
                // ---- which steps stand, and what is in flight next
                const unsigned moves = __ballot_sync(kFull, flying && s_delta[par][lane & (kWindow - 1)] != 0.0);
                bool stands = flying && (s_holders[lane & (kWindow - 1)] & moves) == 0;
                found = stands && !t.alone && (moves >> lane & 1u) && (rec_of(q).c.flags & 16);
                stands = stands && !found;
                const unsigned taken = __ballot_sync(kFull, stands);
                if (me == 0 && lane == 0) moved += __popc(taken & moves);
                if (taken >> lane & 1u) q += kWindow;
                moved_on = taken;
                par ^= 1;
                t.stop = CL ? s_abort : 0;
                next_turn();
                ahead.done();
                __syncthreads();
                tracer.end(__popc(taken), __popc(taken & moves));
            }
            settle();
        } else {
            // ================ a warp with a column
            int pos = wid;
            bool fresh = true;  // the column's first round
            int par = 0;
            __syncthreads();
            __syncthreads();
            for (;;) {
                const Turn now = s_turn;
                if (now.base >= n_active || now.stop) break;
                const bool alone = now.alone != 0, mine = alone || pos < now.limit;
                const int slot = alone ? now.base & (kWindow - 1) : wid;
                const Rec& r = rec_of(alone ? now.base : pos);
                const int n = r.e.hi - r.e.lo, flags = r.c.flags;
                const bool ind = flags & 4, has_vals = flags & 2;
                const int32_t* const kr = s_rows + stage_at(pos);
                const double* const xr = s_vals + stage_at(pos);
                // entry e of the slice, from global memory: local row and value
                auto entry_row = [&](int e) { return ((flags & 1) ? __ldg(P.rows + r.c.cb + r.e.lo + e) : r.e.lo + e) - (int)r0; };
                auto entry_val = [&](int e) { return has_vals ? __ldg(P.vals + r.c.vb + r.e.lo + e) : 1.0; };
                const int first = alone ? tid : lane + kStage, stride = alone ? kWorkers : 32;
                double d = 0.0;
                if (mine) {
                    double g = 0.0, h = 0.0;
                    if (!alone) {
#pragma unroll 1
                        for (int e = lane; e < min(n, kStage); e += 32) {
                            const int k = kr[e] - (int)r0;
                            add_terms<MODEL>(ind, WT, has_vals ? xr[e] : 1.0, rows.p(k), rows.weight(k), g, h);
                            if (fresh) rows.expect(k);
                        }
                    }
                    if (alone || n > kStage) {
#pragma unroll 4
                        for (int e = first; e < n; e += stride) {
                            const int k = entry_row(e);
                            add_terms<MODEL>(ind, WT, entry_val(e), rows.p(k), rows.weight(k), g, h);
                        }
                    }
                    double v = warp_pair_sum(g, h);
                    if (alone) {
                        if ((lane & 15) == 0) s_red[wid][lane >> 4] = v;
                        workers_barrier();
                        v = s_red[lane & 15][lane >> 4];
#pragma unroll
                        for (int o = 8; o > 0; o >>= 1) v += __shfl_xor_sync(kFull, v, o);
                    }
                    if (CL && (!alone || wid == slot)) send_pair(v);
                    const double b0 = r.bh.x, hd = r.bh.y;
                    const double b_var = r.s.ptype == 2 ? b0 / r.s.pvar : 0.0;
                    if (CL) {
                        wait_pairs();
                        v = pair_sum(slot);
                    }
                    double2 t = make_double2(__shfl_sync(kFull, v, 0), __shfl_sync(kFull, v, 16));
                    if (r.c.n > 0) t.x -= r.s.xjy;
                    else t = make_double2(0.0, 0.0);  // an empty column gives (0, 0) (ModelSpecifics.hpp:720-723)
                    d = newton_quotient_step(t.x, t.y, b0, r.s.ptype, r.s.pvar, r.s.lambda, r.s.inv_var, b_var);
                    d = (d < -hd) ? -hd : (d > hd ? hd : d);  // apply_bounds; its new bound is not needed yet
                    if (lane == 0) s_delta[par][wid] = d;
                }
                fresh = false;
                if (CL) ++n_xch;
                __syncthreads();
                const unsigned moves = __ballot_sync(kFull, s_delta[par][lane & (kWindow - 1)] != 0.0);
                par ^= 1;
                // does the step stand (a medium column's waits until it runs alone)
                if (mine && (alone || ((s_holders[wid] & moves) == 0 && !((flags & 16) && d != 0.0)))) {
                    if (d != 0.0) {
                        if (alone) {
#pragma unroll 2
                            for (int e = tid; e < n; e += kWorkers) rows.update(entry_row(e), d * entry_val(e));
                        } else {
#pragma unroll(CL ? 1 : 2)
                            for (int e = lane; e < n; e += 32) rows.update(kr[e] - (int)r0, has_vals ? d * xr[e] : d);
                        }
                    }
                    if (wid == slot) {  // pos is the position of this column
                        pos += kWindow;
                        fresh = true;
                    }
                }
                __syncthreads();
            }
        }
        __syncthreads();  // the last round's bounds and coefficients
        gave_up = CL && s_abort;
    }
    if (CL) cluster_barrier();  // no CTA leaves while another may still send to it
    // the state back to where the other calls read it
    if (rows.kPair)
#pragma unroll 1
        for (int k = tid; k < n_rows; k += kT) {
            const double2 s = rows.xd[k];
            const double e = (WHERE == kPairShared) ? exp(s.x) : (MODEL == M_LOGISTIC) ? rows.ex[k] : rows.share[k];
            rows.row[2 * (int64_t)k] = make_double2(s.x, e);
            rows.row[2 * (int64_t)k + 1].x = s.y;
        }
    if (rank == 0) {
        __syncthreads();
        for (int p = tid; p < n_active; p += kT) P.hdelta[R.cols[p].j] = R.bh[p].y;
    }
    if (rank == 0 && moved) P.st->nonzero_steps = moved;
}

// Static shared memory of the kernel stays below this.
constexpr int64_t kStaticSmem = 18432;
constexpr int64_t kStagedRows = 2 * kWindow * kStage * sizeof(int32_t);
constexpr int64_t kStagedVals = 2 * kWindow * kStage * sizeof(double);

using Kernel = void (*)(WindowParams);

// Few columns have a kernel of their own where the rows are few too and have no
// weights: a process's first fit loads them all, 0.3 ms each.
template <int MODEL, int WHERE>
Kernel pick(bool cl, bool wt, bool few) {
    if constexpr (WHERE == kAllShared) {
        if (few && !wt) return cl ? window_sweep_kernel<MODEL, WHERE, true, false, true> : window_sweep_kernel<MODEL, WHERE, false, false, true>;
    }
    if constexpr (WHERE != kPairShared) {
        if (cl) return wt ? window_sweep_kernel<MODEL, WHERE, true, true, false> : window_sweep_kernel<MODEL, WHERE, true, false, false>;
    }
    return wt ? window_sweep_kernel<MODEL, WHERE, false, true, false> : window_sweep_kernel<MODEL, WHERE, false, false, false>;
}
template <int MODEL>
Kernel pick(int where, bool cl, bool wt, bool few) {
    switch (where) {
    case kAllShared: return pick<MODEL, kAllShared>(cl, wt, few);
    case kShareShared: return pick<MODEL, kShareShared>(cl, wt, few);
    case kGlobal: return pick<MODEL, kGlobal>(cl, wt, few);
    default: return pick<MODEL, kPairShared>(false, wt, few);
    }
}
Kernel pick(int model, int where, bool cl, bool wt, bool few) {
    return model == M_LOGISTIC ? pick<M_LOGISTIC>(where, cl, wt, few) : pick<M_POISSON>(where, cl, wt, few);
}

cudaError_t smem_limit(int64_t* bytes) {
    int dev = 0, optin = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
    *bytes = std::max<int64_t>(0, (int64_t)optin - kStaticSmem);
    return e;
}

// The attributes of all kernels at the first launch on a device: one that is set, and
// its kernel loaded, while other contexts' sweeps run waits for them (a replay of 200
// requests: p50 8 ms, 340 to 760 with each kernel's at its own first launch).
cudaError_t kernel_attrs() {
    static std::atomic<uint64_t> done{0};
    return once_per_device(done, [] {
        int64_t dyn = 0;
        cudaError_t e = smem_limit(&dyn);
        for (int model : {(int)M_LOGISTIC, (int)M_POISSON})
            for (int where : {(int)kAllShared, (int)kShareShared, (int)kGlobal, (int)kPairShared})
                for (int v = 0; v < 8 && e == cudaSuccess; ++v) {
                    const Kernel fn = pick(model, where, v & 1, v & 2, v & 4);
                    e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)dyn);
                    if (e == cudaSuccess) e = cudaFuncSetAttribute(fn, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
                }
        return e;
    });
}

cudaLaunchConfig_t config(int C, size_t smem, cudaStream_t stream, cudaLaunchAttribute* at) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(C);
    cfg.blockDim = dim3(kT);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = C;
    at[0].val.clusterDim.y = 1;
    at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    return cfg;
}

int64_t all_bytes(int model, int64_t rows) { return (model == M_LOGISTIC ? 16 : 8) * ((rows + 1) & ~int64_t(1)) + 16 * rows; }

}  // namespace

#ifndef CCDB_TRACE_ROUNDS
bool window_share_fits(int64_t rows, bool vals, int64_t smem) {
    return kStagedRows + 8 * ((rows + 1) & ~int64_t(1)) + (vals ? kStagedVals : 0) <= smem;
}

cudaError_t window_limits(int* cluster, int64_t* smem) {
    *cluster = 0;
    // one for all: they have the same threads, and their shared memory is asked for in full
    const Kernel fn = pick(M_LOGISTIC, kAllShared, true, false, false);
    cudaError_t e = smem_limit(smem);
    if (e == cudaSuccess) e = kernel_attrs();
    if (e != cudaSuccess) return e;
    for (int C = kWindowCluster; C >= 1; C /= 2) {
        cudaLaunchAttribute at[1];
        const cudaLaunchConfig_t cfg = config(C, (size_t)*smem, 0, at);
        int n = 0;
        const bool fits = cudaOccupancyMaxActiveClusters(&n, fn, &cfg) == cudaSuccess && n >= 1;
        cudaGetLastError();  // a size the device rejects is not an error here: try the next
        if (fits) {
            *cluster = C;
            return cudaSuccess;
        }
    }
    return cudaSuccess;
}

cudaError_t launch_window_sweep(const WindowParams& R, int64_t smem, cudaStream_t stream) {
#else
cudaError_t launch_window_sweep_traced(const WindowParams& R, int64_t smem, cudaStream_t stream) {
#endif
    const int C = R.cluster;
    if (C < 1 || C > kWindowCluster) return cudaErrorInvalidValue;
    const int64_t rows = (R.P.K + C - 1) / C;  // the most a CTA owns
    const int64_t vals = R.any_vals ? kStagedVals : 0;
    int where = kGlobal;
    int64_t state = 0;
    bool weights_shared = false;
    if (kStagedRows + all_bytes(R.P.model, rows) + vals <= smem) {
        where = kAllShared;
        state = all_bytes(R.P.model, rows);
        const int64_t weights = 8 * ((rows + 1) & ~int64_t(1));
        weights_shared = R.weighted && kStagedRows + state + weights + vals <= smem;
        if (weights_shared) state += weights;
    } else if (C == 1 && kStagedRows + 16 * rows + vals <= smem) {
        where = kPairShared;
        state = 16 * rows;
    } else if (ccdb::window_share_fits(rows, R.any_vals != 0, smem)) {
        where = kShareShared;
        state = 8 * ((rows + 1) & ~int64_t(1));
    }
    if (where == kGlobal && !R.share) return cudaErrorInvalidValue;
    const Kernel fn = pick(R.P.model, where, C > 1, R.weighted != 0, R.n_active <= 4 * kWindow);
    const cudaError_t e = kernel_attrs();
    if (e != cudaSuccess) return e;
    WindowParams Q = R;
    Q.vals_at = (int32_t)(kStagedRows + state);
    Q.weights_shared = weights_shared ? 1 : 0;
    cudaLaunchAttribute at[1];
    const cudaLaunchConfig_t cfg = config(C, (size_t)(Q.vals_at + vals), stream, at);
    return cudaLaunchKernelEx(&cfg, fn, Q);
}

}  // namespace ccdb
