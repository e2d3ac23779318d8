// group_window.cu -- one findMode of a group model (Breslow Cox, conditional
// logistic / Poisson) in one launch, its rows and groups shared out over CTAs.
//
// The sweep is the sequential cycle (CyclicCoordinateDescent.cpp:1008-1021).  Up
// to kWindow consecutive columns are in flight, one per warp; all of them are
// evaluated against one state, every step up to the first that is not zero is
// taken (zero steps leave the state as it is), and the columns behind it stay in
// flight.  Rows of one column touch most strata, so nearly any two columns
// meet: no step is taken past one that moves.
//
// Each CTA owns whole groups (risk-set tie groups, or strata) and their rows.
// Every warp sums its column over the CTA's slice of it; the CTAs send each other
// these partial sums and every CTA adds them in CTA order, so all take the same
// decision.  A step that moves updates each CTA's own rows and group
// denominators, without a barrier between CTAs.
//
// Grouped models (GroupedData, ModelSpecifics.hpp:1101-1179): a stratum's run of
// entries contributes t = numerator / denominator; a CTA's strata are whole, so a
// column's partial sums are just (g, h).  A column with a slice of over kGroupLong
// entries runs alone, on every warp: one warp that walked it was slower than the
// kernel before this one where few CTAs shared the rows (300,000 rows, six dense
// columns, on 1, 4, 8 CTAs: 197, 49, 22 ms; on every warp 30, 8.0, 3.9).  Alone
// against one warp, 60 columns on 16 CTAs, slices of 600: 1.19 and 2.45 ms (L1), 1.46
// and 4.23 (every step moves); of 300, on one CTA with hardly a step that moves, where
// it gives up columns in flight: 0.64 and 0.42.
//
// Cox (cox.cu): g = sum n1 S1, h = sum n2 S1 - sum S2 (A^2 - A'^2) with A the
// running sum of n1 within the stratum and A' the one before the entry.  A stratum
// may span CTAs: a CTA's running sums then miss a carry c, the sum of n1 over the
// stratum's entries before it, and (c + A)^2 - (c + A')^2 = A^2 - A'^2 + 2 c n1.
// So a CTA sends G = sum n1 S1, H2, HQ = sum S2 (A^2 - A'^2), B = sum S2 n1 over
// its first stratum and T, the sum of n1 over its last one; c follows from the T
// of the CTAs before it.  After a step the accumulated denominators D (prefix sums
// within strata, computeAccumlatedDenominator, ModelSpecifics.hpp:1670-1715) and
// the suffix sums S1 = sum nEv / D, S2 = sum nEv / D^2 are rebuilt from the group
// denominators: each thread takes a contiguous run of the CTA's groups, and the
// CTAs exchange one tail sum, then one pair of head sums.
//
// Long columns run alone there too, but only while steps move (the last round's did, or
// the column is not held at zero): a Cox column at rest is cheaper beside fifteen others
// on one warp.  A warp's part of a slice misses a carry as a CTA's does.  And the rows of
// a long column fall into one tie group by the hundred, whose changes its first entry
// added one by one: a warp of one group, rows that a zero weight drops aside, hands its
// sum over (440,351 rows, 20 % of weight zero, 14 dense columns of 44: 119 ms; before the
// windows 530, with every change added by itself 1,981).  150,637 rows, one stratum,
// days as ties, 50 columns up to dense, 9 cycles: 43 ms; one warp a column 539, the kernel
// before this one 203.  18,498 rows, 18 columns, six dense: 2.25 ms, 5.14, 7.7; 150,000
// rows, 198 sparse columns and two dense: 3.10, 3.77, 42.7.
//
// Cox works on blocks, runs of groups up to one with events or to their stratum's
// end: D counts only where there are events and S1, S2 change only there (cox_host.cu
// builds them).  "Group" below is a block.
//
// Groups' state lives in shared memory (36 bytes a group for Cox, 16 otherwise)
// and the rows' too when they fit (20 bytes a row).  Two forms share the code: a
// thread-block cluster whose CTAs exchange by st.async on each other's mbarriers,
// and a cooperative grid that exchanges through global memory with a counter.
//
// A round is a chain of latencies, as in window.cu; so is a rebuild.  Measured on
// a B200 at 1,965 MHz, a step that moves takes 6.1 us on the 20,000 x 400 Cox fit
// (gather 1,700 SM clocks, each of the three exchanges 1,300 to 1,800 with the
// CTAs' skew, step 1,100, rows and denominators 1,400, prefix 800, D and suffix
// 1,500), 9.2 us at 400,000 rows, 14.9 us at 1,000,000 (grid), 2.2 us on the
// 26,000 x 500 conditional logistic fit; the grid barriers, per-entry buffers in
// global memory and the rebuild over every group that it replaces took 27, 38, 60
// and 11 us.
//
// The waits of both forms are bounded.  In the grid form one that runs out raises
// the launch's abort word and every CTA leaves at its next wait.  In a cluster the
// CTA steps and sends no more, and all leave together at the end of the cycle, each
// once what was sent to it has landed (sweep_exit.h).  Within a CTA the warps pass
// the same barriers: a wait marks the half of the round that it lies in, and every
// warp reads the mark in the other half.
#include <algorithm>
#include <cstdint>

#include "group_window.h"
#include "window_device.cuh"

namespace ccdb {

namespace {

using namespace win;

// what shared memory holds: rows and groups, groups, neither
enum Where : int { kRowsShared = 0, kGroupsShared = 1, kGlobal = 2 };

// Cox: a Hessian below this part of the moment that it is left of is what rounding
// leaves of zero: a column that is constant within every risk set carries no
// information and gives (0, 0), which the reference's quotients have exactly and which
// ends an unpenalised fit as ill-conditioned.
constexpr double kCoxNoise = 256 * 2.220446049250313e-16;

constexpr int kNarrow = 4;  // columns in flight after a step that moved; zero rounds double them

// exp of a row's xBeta: FP64, or in the mixed precision of the Cox engine FP32.
template <bool MX>
__device__ __forceinline__ double row_exp(double xb) {
    return MX ? (double)expf((float)xb) : exp(xb);
}

// Knuth's TwoSum: s + c carries the running FP32 sum with its rounding errors.
__device__ __forceinline__ void two_sum_f(float& s, float& c, float v) {
    const float t = s + v, bp = t - s;
    c += (s - (t - bp)) + (v - bp);
    s = t;
}

// Which elements end a segmented scan's reach does not change during a fit, so a
// scan carries values only: `from` is the lowest lane that a lane's prefix takes in,
// `to` the highest that its suffix does.
__device__ __forceinline__ int reach_down(unsigned starts, int lane) {  // starts: lanes that begin a segment
    const unsigned m = starts & (kFull >> (31 - lane));
    return m ? 31 - __clz(m) : 0;
}
__device__ __forceinline__ int reach_up(unsigned ends, int lane) {
    const unsigned m = ends >> lane;
    return m ? lane + __ffs(m) - 1 : 31;
}
// inclusive scans over the first `width` lanes, ascending and descending
__device__ __forceinline__ double scan_up(double x, int from, int width) {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        if (o >= width) break;
        const double y = __shfl_up_sync(kFull, x, o);
        if (lane - o >= from) x += y;
    }
    return x;
}
__device__ __forceinline__ double2 scan_down(double2 x, int to, int width) {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        if (o >= width) break;
        const double ya = __shfl_down_sync(kFull, x.x, o), yb = __shfl_down_sync(kFull, x.y, o);
        if (lane + o <= to) {
            x.x += ya;
            x.y += yb;
        }
    }
    return x;
}

// Sums over the warp: lanes 0..7 a, 8..15 b, 16..23 c, 24..31 d.
__device__ __forceinline__ double warp_sum_of_four(double a, double b, double c, double d) {
    const bool hi = threadIdx.x & 16, odd = threadIdx.x & 8;
    double u = hi ? c : a, v = hi ? d : b;
    u += __shfl_xor_sync(kFull, hi ? a : c, 16);
    v += __shfl_xor_sync(kFull, hi ? b : d, 16);
    double s = odd ? v : u;
    s += __shfl_xor_sync(kFull, odd ? u : v, 8);
#pragma unroll
    for (int o = 4; o > 0; o >>= 1) s += __shfl_xor_sync(kFull, s, o);
    return s;
}

// Sums of g and h over the warp, in every lane.
__device__ __forceinline__ double2 warp_sum_of_two(double g, double h) {
    const bool hi = threadIdx.x & 16;
    double s = hi ? h : g;
    s += __shfl_xor_sync(kFull, hi ? g : h, 16);
#pragma unroll
    for (int o = 8; o > 0; o >>= 1) s += __shfl_xor_sync(kFull, s, o);
    return make_double2(__shfl_sync(kFull, s, 0), __shfl_sync(kFull, s, 16));
}

// A CTA's rows and groups, by local index.
template <bool COX, int WHERE>
struct Owned {
    const CoxParams* P;
    int64_t row0, g0;
    int n_rows, n_groups;
    double *e_, *xb_;  // rows
    int32_t* grp_;
    double *den_, *nev_, *s1_, *s2_;  // groups
    int32_t* strat_;                  // stratum << 2 | last group of it << 1 | first

    __device__ __forceinline__ double ex(int k) const { return WHERE == kRowsShared ? e_[k] : P->xbe[row0 + k].y; }
    __device__ __forceinline__ double xb(int k) const { return WHERE == kRowsShared ? xb_[k] : P->xbe[row0 + k].x; }
    __device__ __forceinline__ void set_row(int k, double x, double e) const {
        if (WHERE == kRowsShared) {
            xb_[k] = x;
            e_[k] = e;
        } else {
            P->xbe[row0 + k] = make_double2(x, e);
        }
    }
    // local group of a row, -1 for a row that a zero weight drops
    __device__ __forceinline__ int read_group(int k) const {
        const int32_t g = P->grp[row0 + k];
        return g == P->N ? -1 : (int)(g - g0);
    }
    __device__ __forceinline__ int group(int k) const { return WHERE == kRowsShared ? grp_[k] : read_group(k); }
    __device__ __forceinline__ int stratum(int k, int g) const {
        return (WHERE != kGlobal && g >= 0) ? strat_[g] >> 2 : P->rstrat[row0 + k];
    }
    __device__ __forceinline__ double& den(int g) const { return WHERE != kGlobal ? den_[g] : P->denom[g0 + g]; }
    __device__ __forceinline__ double nev(int g) const { return WHERE != kGlobal ? nev_[g] : P->nEv[g0 + g]; }
    __device__ __forceinline__ double& s1(int g) const { return WHERE != kGlobal ? s1_[g] : P->S1[g0 + g]; }
    __device__ __forceinline__ double& s2(int g) const { return WHERE != kGlobal ? s2_[g] : P->S2[g0 + g]; }
    __device__ __forceinline__ bool first(int g) const { return WHERE != kGlobal ? strat_[g] & 1 : P->gfirst[g0 + g]; }
    __device__ __forceinline__ bool last(int g) const { return WHERE != kGlobal ? strat_[g] & 2 : P->glast[g0 + g]; }
};

// MX: the mixed precision of the Cox engine.  LONG: a column may be long; without it the
// code of one costs the others (26,000 x 500 conditional logistic, no long column: 3.17
// ms, 3.4 with it; Cox, 12,000 x 60: 3.09 and 3.17).
template <bool COX, int WHERE, bool CL, bool MX, bool LONG>
__global__ void __launch_bounds__(kT, 1) group_window_kernel(GroupWindowParams Q) {
    __shared__ Rec s_rec[4][kWindow];  // by position: (position / kWindow) & 3, slot
    // cluster form, by exchange parity, column and CTA: Cox {G, HQ}, {B, T}, {H2, 0}, else {g, h}
    __shared__ double2 s_part[CL ? 2 : 1][CL ? kWindow : 1][COX ? 3 : 1][CL ? kWindowCluster : 1];
    constexpr int kSumBuffers = CL && COX ? 2 : 1, kSumCtas = CL && COX ? kWindowCluster : 1;
    __shared__ double s_tail[kSumBuffers][kSumCtas];
    __shared__ double2 s_head[kSumBuffers][kSumCtas];
    __shared__ double4 s_red4[kWarps];
    // by cycle parity and CTA: a CTA that gave up may be a cycle ahead of one that reads them
    __shared__ double4 s_obj[CL ? 2 : 1][kWindowCluster];
    __shared__ CycleReport s_report[CL ? 2 : 1][kWindowCluster];
    __shared__ unsigned s_sent[2];  // bytes to each CTA, by exchange parity
    __shared__ double s_dd[kWorkers];    // an update's changes of exp, by entry
    __shared__ int32_t s_dg[kWorkers];   // and their groups
    __shared__ double s_run[kWindow];    // the worker warps' prefix sums
    __shared__ double2 s_run2[kWindow];  // and suffix sums
    __shared__ int s_first[kWindow], s_last[kWindow];  // a stratum begins, ends among a worker warp's groups
    // the steps of the columns in flight; behind them, not zero: a wait for their sums ran
    // out (before the round's first barrier, and read behind it; one of an update is in
    // s_turn.stop, before the second barrier and read behind that)
    __shared__ double s_delta[kWindow + 1];
    __shared__ Turn s_turn;
    __shared__ uint64_t s_bar[2];
    __shared__ int32_t s_fail;
    __shared__ uint8_t s_flags[kGroupWindowCtas];  // GroupCut::flags of every CTA
    extern __shared__ __align__(16) unsigned char s_dyn[];

    const CoxParams& P = Q.P;
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    const int C = Q.ctas, rank = (int)blockIdx.x, n_active = Q.n_active;
    const GroupCut cut = Q.cuts[rank];
    const WinSlice* const slices = Q.slices + (int64_t)rank * n_active;
    Owned<COX, WHERE> own;
    own.P = &Q.P;
    own.row0 = cut.row0;
    own.g0 = cut.g0;
    own.n_rows = Q.cuts[rank + 1].row0 - cut.row0;
    own.n_groups = Q.cuts[rank + 1].g0 - cut.g0;
    // dynamic shared memory: the staged rows, the groups, the rows, the staged values
    int32_t* const s_rows = reinterpret_cast<int32_t*>(s_dyn);
    double* const s_vals = reinterpret_cast<double*>(s_dyn + Q.vals_at);
    {
        double* at = reinterpret_cast<double*>(s_rows + 2 * kWindow * kStage);
        if (WHERE != kGlobal) {
            own.den_ = at;
            own.nev_ = own.den_ + own.n_groups;
            at = own.nev_ + own.n_groups;
            if (COX) {
                own.s1_ = at;
                own.s2_ = own.s1_ + own.n_groups;
                at = own.s2_ + own.n_groups;
            }
        }
        if (WHERE == kRowsShared) {
            own.e_ = at;
            own.xb_ = own.e_ + own.n_rows;
            at = own.xb_ + own.n_rows;
        }
        int32_t* ints = reinterpret_cast<int32_t*>(at);
        own.strat_ = ints;
        own.grp_ = ints + (COX && WHERE != kGlobal ? own.n_groups : 0);
    }
    // ---- the state of the rows and groups, the records of the columns
#pragma unroll 1
    for (int g = tid; WHERE != kGlobal && g < own.n_groups; g += kT) {
        own.den_[g] = P.denom[own.g0 + g];
        own.nev_[g] = P.nEv[own.g0 + g];
        if (COX) {
            own.s1_[g] = P.S1[own.g0 + g];
            own.s2_[g] = P.S2[own.g0 + g];
            own.strat_[g] = P.rstrat[P.grow[own.g0 + g]] << 2 | (P.glast[own.g0 + g] ? 2 : 0) | (P.gfirst[own.g0 + g] ? 1 : 0);
        }
    }
#pragma unroll 1
    for (int k = tid; WHERE == kRowsShared && k < own.n_rows; k += kT) {
        const double2 a = P.xbe[own.row0 + k];
        own.set_row(k, a.x, a.y);
        own.grp_[k] = own.read_group(k);
    }
#pragma unroll 1
    for (int q = rank * kT + tid; q < n_active; q += C * kT) {
        const int j = Q.cols[q].j;
        const double var = Q.pvar[j];
        const int pt = Q.ptype[j];
        Q.scal[q] = WinScal{P.xjy[j], var, pt == 1 ? sqrt(2.0 / var) : 0.0, pt == 2 ? 1.0 / var : 0.0, pt, 0, 0};
        Q.bh[q] = make_double2(Q.beta[j], Q.hdelta[j]);
    }
    for (int c = tid; c < C; c += kT) s_flags[c] = (uint8_t)Q.cuts[c].flags;
    if (tid == 0) {
        s_delta[kWindow] = 0.0;
        s_turn.stop = 0;
        if (CL) init_bars(s_bar, 2);
    }
    // sums of CTAs that there are not stay zero
    if (CL && COX && tid < 2 * kWindowCluster) {
        (&s_tail[0][0])[tid] = 0.0;
        (&s_head[0][0])[tid] = make_double2(0.0, 0.0);
    }
    for (int i = tid; CL && i < (int)(sizeof(s_part) / sizeof(double2)); i += kT)
        (&s_part[0][0][0][0])[i] = make_double2(0.0, 0.0);
    unsigned epoch = 0;  // grid barriers passed (thread 0)
    if (CL) cluster_barrier();
    __syncthreads();

    // ---- exchange between the CTAs
    unsigned n_xch = 0;  // exchanges so far: parity picks the buffers and the mbarrier
    // cluster form: the base of each peer's shared variables, lane l for CTA l
    unsigned to_part = 0, to_bar = 0, to_tail = 0, to_head = 0;
    if (CL && lane < C) {
        to_tail = peer_u32(&s_tail[0][COX ? rank : 0], lane);
        to_head = peer_u32(&s_head[0][COX ? rank : 0], lane);
        to_part = peer_u32(&s_part[0][0][0][0], lane);
        to_bar = peer_u32(&s_bar[0], lane);
    }
    constexpr unsigned kColumnBytes = sizeof(s_part[0][0]), kSumBytes = sizeof(double2) * kWindowCluster;
    // bytes that a column's partial sums of one CTA take in an exchange
    auto pair_bytes = [&](int pos, const Rec& r) { return COX ? ((r.c.flags & 4) ? 32u : 48u) : 16u; };
    // workers, grid form: everything written before is seen by every CTA after it
    auto grid_wait = [&](auto& quit) {
        workers_barrier();
        if (tid == 0) {
            ++epoch;
            red_release_gpu_add(Q.grid_bar, 1u);
            if (!wait_geq(Q.grid_bar, epoch * (unsigned)C, Q.wait_limit_ns, Q.st, E_WAIT_GRID, -1)) quit = 1;
        }
        workers_barrier();
    };
    // this exchange's bytes have come to this thread (cluster form)
    auto wait_sums = [&](auto& quit) {
        const bool ok = wait_bytes(&s_bar[n_xch & 1], (n_xch >> 1) & 1, Q.wait_limit_ns);
        if (!ok) quit = 1;
        return ok;
    };
    // announce an exchange in which every CTA sends `bytes` to every other (cluster form)
    auto expect_sums = [&](unsigned bytes) {
        expect_bytes(&s_bar[n_xch & 1], bytes * (unsigned)C);
        s_sent[n_xch & 1] = bytes;
    };

    // ---- the objective terms {LL numerator, LL denominator, gradient objective,
    // log prior} (ModelSpecifics.hpp:103-120, 605-650; JointPrior.h:121-128); false
    // when a wait ran out, of any CTA of a cluster
    auto objective = [&](int cycle, bool gave_up, double& obj, double& ll, double& lp) {
        double4 acc = make_double4(0.0, 0.0, 0.0, 0.0);
#pragma unroll 1
        for (int k = tid; k < own.n_rows; k += kT) {
            const double xb = own.xb(k), yk = P.y[own.row0 + k], w = P.weighted ? P.w[own.row0 + k] : 1.0;
            const int yi = (int)yk;
            const double c = COX ? ((yi != 1) ? 0.0 : xb) : yi * xb;
            acc.x += P.weighted ? c * w : c;
            acc.z += P.weighted ? xb * yk * w : xb * yk;
        }
#pragma unroll 1
        for (int g = tid; g < own.n_groups; g += kT) acc.y += own.nev(g) * log(COX ? __ldcg(P.D + own.g0 + g) : own.den(g));
        if (rank == 0)  // the CTA that writes the coefficients
#pragma unroll 1
            for (int j = tid; j < Q.J; j += kT) acc.w += log_prior_one(Q.beta[j], Q.ptype[j], Q.pvar[j]);
        acc = block_sum4<kWarps>(acc, s_red4);
        double4 t = make_double4(0.0, 0.0, 0.0, 0.0);
        if (CL) {
            if (tid < C) {
                const unsigned a = peer_u32(&s_obj[cycle & 1][rank], tid);
                asm volatile("st.shared::cluster.v2.f64 [%0], {%1, %2};" ::"r"(a), "d"(acc.x), "d"(acc.y) : "memory");
                asm volatile("st.shared::cluster.v2.f64 [%0], {%1, %2};" ::"r"(a + 16), "d"(acc.z), "d"(acc.w) : "memory");
                tell(&s_report[cycle & 1][rank], tid, CycleReport{gave_up ? 1u : 0u, n_xch, {s_sent[0], s_sent[1]}});
            }
            cluster_barrier();  // also: rank 0's coefficients and bounds are seen by the next cycle
            unsigned any = 0;
#pragma unroll 1
            for (int c = 0; c < C; ++c) {
                const double4 o = s_obj[cycle & 1][c];
                t.x += o.x;
                t.y += o.y;
                t.z += o.z;
                t.w += o.w;
                any |= s_report[cycle & 1][c].gave_up;
            }
            if (any) return false;
        } else {
            if (tid == 0) {
                __stcg(Q.red + 2 * rank, make_double2(acc.x, acc.y));
                __stcg(Q.red + 2 * rank + 1, make_double2(acc.z, acc.w));
            }
            if (!grid_barrier(Q.grid_bar, epoch, Q.wait_limit_ns, Q.st, &s_fail)) return false;
#pragma unroll 4
            for (int c = 0; c < C; ++c) {
                const double2 u = __ldcg(Q.red + 2 * c), v = __ldcg(Q.red + 2 * c + 1);
                t.x += u.x;
                t.y += u.y;
                t.z += v.x;
                t.w += v.y;
            }
            // every CTA has read the partials before any of them writes the next ones
            if (!grid_barrier(Q.grid_bar, epoch, Q.wait_limit_ns, Q.st, &s_fail)) return false;
        }
        ll = (t.x - t.y) + Q.ll_fixed;
        lp = t.w;
        obj = (Q.conv == C_GRADIENT) ? t.z : (Q.conv == C_MITTAL ? ll : ll + t.w);
        return true;
    };

    auto rec_of = [&](int at) -> Rec& { return s_rec[(at / kWindow) & 3][at & (kWindow - 1)]; };
    const Ahead ahead{Q.cols, Q.scal, Q.bh, slices, P.rows, P.vals, n_active};
    auto fetch = [&](int at, int l8) { ahead.record(at, rec_of(at), l8); };
    auto stage = [&](int at, int l8) { ahead.entries(at, rec_of(at), s_rows + stage_at(at), s_vals + stage_at(at), l8); };
    // a column that runs alone, on every warp (grouped models); it is not copied ahead
    auto long_column = [&](const Rec& r) { return LONG && (r.c.flags & 8); };
    // entry e of a record's slice: local row and value
    auto entry_row = [&](const Rec& r, int at, int e) {
        if (e < kStage && !long_column(r)) return s_rows[stage_at(at) + e] - (int)own.row0;
        return ((r.c.flags & 1) ? __ldg(P.rows + r.c.cb + r.e.lo + e) : r.e.lo + e) - (int)own.row0;
    };
    auto entry_val = [&](const Rec& r, int at, int e) {
        if (!(r.c.flags & 2)) return 1.0;
        return e < kStage && !long_column(r) ? s_vals[stage_at(at) + e] : __ldg(P.vals + r.c.vb + r.e.lo + e);
    };

    // Grouped models: the sums of a long column over this CTA's slice, by all workers, in
    // the warp that `takes` them.  Each warp walks sixteenths of the slice, whole passes of
    // 32 entries; a run of entries that goes over its ends (a stratum met from both sides)
    // is handed on in parts and put together at the end.
    auto gather_alone = [&](const Rec& r, int at, bool takes) {
        const int n = r.e.hi - r.e.lo, share = ((n + 32 * kWindow - 1) / (32 * kWindow)) * 32;
        const int c0 = min(wid * share, n), c1 = min(c0 + share, n);
        const bool ind = r.c.flags & 4;
        // by warp: {g, h}, the part of a run that began before it, the part of one that goes on
        // behind it; s_dg: 1 the former ends here, 2 it goes on, 4 there is a latter; and its stratum
        double* const mine = s_dd + 6 * wid;
        double g = 0.0, h = 0.0, run1 = 0.0, run2 = 0.0;
        auto add_run = [&](int key, double a, double b) {
            const double dn = own.den(key), ne = own.nev(key), t = a / dn, gg = ne * t;
            g += gg;
            h += ind ? gg * (1.0 - t) : ne * (b / dn - t * t);
        };
        int run_key = c0 > 0 && c0 < n ? own.group(entry_row(r, at, c0 - 1)) : -1;
        bool joined = true;  // no run has begun in this warp's part so far
        int parts = 0;
#pragma unroll 1
        for (int e0 = c0; e0 < c1; e0 += 32) {
            const int e = e0 + lane;
            const bool in = e < n;
            int key = 0x7fffffff;
            double a = 0.0, b = 0.0;
            if (in) {
                const int k = entry_row(r, at, e);
                const double x = entry_val(r, at, e), ex = own.ex(k);
                key = own.group(k);
                a = ex * x;
                if (!ind) b = ex * x * x;
            }
            int next = __shfl_down_sync(kFull, key, 1);
            if (lane == 31) next = e + 1 < n ? own.group(entry_row(r, at, e + 1)) : -1;
            int prev = __shfl_up_sync(kFull, key, 1);
            if (lane == 0) prev = run_key;
            const unsigned all_starts = __ballot_sync(kFull, key != prev);
            const unsigned starts = all_starts & (kFull >> (31 - lane));
            const int start = reach_down(all_starts, lane);
#pragma unroll 1
            for (int o = 1; o < 32; o <<= 1) {
                const bool more = lane - o >= start;
                if (!__any_sync(kFull, in && more)) break;  // no run is longer than o
                const double y = __shfl_up_sync(kFull, a, o), z = __shfl_up_sync(kFull, b, o);
                if (more) {
                    a += y;
                    b += z;
                }
            }
            if (!starts) {
                a += run1;
                b += run2;
            }
            const bool ends = next != key || e + 1 >= n, before = joined && !starts;
            const bool goes_on = !ends && e + 1 == c1;
            if (__any_sync(kFull, in && before && ends)) parts |= 1;
            if (__any_sync(kFull, in && before && goes_on)) parts |= 2;
            if (__any_sync(kFull, in && !before && goes_on)) parts |= 4;
            if (in && before && (ends || goes_on)) {
                mine[2] = a;
                mine[3] = b;
                if (ends) s_dg[2 * wid + 1] = key;
            } else if (in && ends) {
                add_run(key, a, b);
            } else if (in && goes_on) {
                mine[4] = a;
                mine[5] = b;
            }
            joined = joined && all_starts == 0;
            run1 = __shfl_sync(kFull, a, 31);
            run2 = __shfl_sync(kFull, b, 31);
            run_key = __shfl_sync(kFull, key, 31);
        }
        const double2 gh = warp_sum_of_two(g, h);
        if (lane == 0) {
            mine[0] = gh.x;
            mine[1] = gh.y;
            s_dg[2 * wid] = parts;
        }
        workers_barrier();
        if (!takes) return gh;
        g = h = 0.0;
        if (lane < kWindow) {  // lane w: warp w
            if (s_dg[2 * lane] & 1) {
                double a = s_dd[6 * lane + 2], b = s_dd[6 * lane + 3];
                for (int w = lane - 1; w >= 0; --w) {
                    const bool on = s_dg[2 * w] & 2;
                    a += s_dd[6 * w + (on ? 2 : 4)];
                    b += s_dd[6 * w + (on ? 3 : 5)];
                    if (!on) break;
                }
                add_run(s_dg[2 * lane + 1], a, b);
            }
            g += s_dd[6 * lane];
            h += s_dd[6 * lane + 1];
        }
        return warp_sum_of_two(g, h);
    };

    // A column's partial sums of this CTA, Cox, from the warp that has them to every CTA.
    auto send_cox = [&](double2 gq, double2 bt, double h2, bool ind) {
        if (CL) {
            if (lane < C) {
                const unsigned par = n_xch & 1, bar = to_bar + par * 8u;
                const unsigned a = to_part + (par * kWindow + wid) * kColumnBytes + rank * (unsigned)sizeof(double2);
                send16(a, bar, gq.x, gq.y);
                send16(a + kSumBytes, bar, bt.x, bt.y);
                if (!ind) send16(a + 2 * kSumBytes, bar, h2, 0.0);
            }
        } else if (lane == 0) {
            double2* to = Q.part + ((size_t)((n_xch & 1) * kWindow + wid) * C + rank) * 3;
            __stcg(to, gq);
            __stcg(to + 1, bt);
            __stcg(to + 2, make_double2(h2, 0.0));
        }
    };

    // Cox: the same of a long column, by all workers, sent by the warp that `takes` it.
    // Each warp walks a part of whole passes of 32 entries with running sums that begin at
    // its own first entry; what they miss of a stratum that the warps before it have begun
    // is a carry, as it is from CTA to CTA: HQ grows by 2 c times the sum of S2 n1 over that
    // stratum's entries here.
    auto cox_alone = [&](const Rec& r, int at, bool takes) {
        const int n = r.e.hi - r.e.lo, share = ((n + 32 * kWindow - 1) / (32 * kWindow)) * 32;
        const int c0 = min(wid * share, n), c1 = min(c0 + share, n);
        const bool ind = r.c.flags & 4;
        const int first = (cut.flags & 1) ? cut.first : -2;
        auto key_of = [&](int e) {
            const int k = entry_row(r, at, e);
            return own.stratum(k, own.group(k));
        };
        const int before = c0 > 0 && c0 < c1 ? key_of(c0 - 1) : -1;  // the stratum that the warp below ends in
        double G = 0.0, H2 = 0.0, HQ = 0.0, B = 0.0, BW = 0.0, run = 0.0, A = 0.0;
        float gs = 0.f, gc = 0.f, hs = 0.f, hc = 0.f;  // mixed: FP32 TwoSum partials of G and H2
        int run_key = -1, key = -1;
        bool joined = false;
#pragma unroll 1
        for (int e0 = c0; e0 < c1; e0 += 32) {
            const int e = e0 + lane;
            const bool in = e < c1;
            double n1 = 0.0, n2 = 0.0, s1 = 0.0, s2 = 0.0;
            float n1f = 0.f, n2f = 0.f;
            key = 0x7fffffff;
            if (in) {
                const int k = entry_row(r, at, e), gr = own.group(k);
                const double x = entry_val(r, at, e), ex = own.ex(k), w = P.weighted ? P.w[own.row0 + k] : 1.0;
                key = own.stratum(k, gr);
                if (gr >= 0) {
                    s1 = own.s1(gr);
                    s2 = own.s2(gr);
                }
                if (MX) {
                    const float xf = (float)x, ef = (float)ex;
                    n1f = P.weighted ? (float)w * (ef * xf) : ef * xf;
                    if (!ind) n2f = n1f * xf;
                    n1 = (double)n1f;
                } else {
                    n1 = P.weighted ? w * (ex * x) : ex * x;
                    if (!ind) n2 = P.weighted ? w * (ex * x * x) : ex * x * x;
                }
            }
            int prev = __shfl_up_sync(kFull, key, 1);
            if (lane == 0) prev = run_key;
            const unsigned starts = __ballot_sync(kFull, key != prev);
            A = scan_up(n1, reach_down(starts, lane), 32);
            if (!(starts & (kFull >> (31 - lane)))) A += run;
            const double before_it = A - n1;
            if (MX) {
                const float s1f = (float)s1;
                two_sum_f(gs, gc, n1f * s1f);
                two_sum_f(hs, hc, n2f * s1f);
            } else {
                G += n1 * s1;
                H2 += n2 * s1;
            }
            if (in) HQ += s2 * (A * A - before_it * before_it);  // risk-set sums: FP64
            if (key == first) B += s2 * n1;
            if (key == before) BW += s2 * n1;
            if (e0 == c0) joined = __shfl_sync(kFull, key, 0) == before;
            if (e0 + 32 < c1) {
                run = __shfl_sync(kFull, A, 31);
                run_key = __shfl_sync(kFull, key, 31);
            }
        }
        if (MX) {
            G = (double)gs + (double)gc;
            H2 = (double)hs + (double)hc;
        }
        const int end = (c1 - c0 + 31) & 31;  // the part's last entry's lane
        const double T = c0 < c1 ? __shfl_sync(kFull, A, end) : 0.0;
        const int last_key = __shfl_sync(kFull, key, end);
        const double s = warp_sum_of_four(G, H2, HQ, B), bw = warp_sum_of_two(BW, 0.0).x;
        // by warp: G, H2, HQ, B, BW, T; s_dg: 1 the part begins within a stratum, 2 it lies in it; the last key
        double* const mine = s_dd + 6 * wid;
        if ((lane & 7) == 0) mine[lane >> 3] = s;
        if (lane == 0) {
            mine[4] = bw;
            mine[5] = T;
            s_dg[2 * wid] = joined ? (last_key == before ? 3 : 1) : 0;
            s_dg[2 * wid + 1] = last_key;
        }
        workers_barrier();
        if (!takes) return;
        // lane w: warp w; what a part passes on, and what comes in to it
        const double* const of = s_dd + 6 * (lane & (kWindow - 1));
        const int fl = lane < kWindow ? s_dg[2 * lane] : 0, parts = n > 0 ? (n - 1) / share : 0;  // the last part
        const unsigned starts = __ballot_sync(kFull, fl != 3);
        const double pass = scan_up(of[5], reach_down(starts, lane), kWindow);
        const double in = __shfl_up_sync(kFull, pass, 1), t = __shfl_sync(kFull, pass, parts);
        const double carry = (fl & 1) ? in : 0.0;
        const bool have = lane < kWindow;
        const double u = warp_sum_of_four(have ? of[0] : 0.0, have ? of[1] : 0.0, have ? of[2] + 2.0 * carry * of[4] : 0.0,
                                          have ? of[3] : 0.0);
        const double2 gq = make_double2(__shfl_sync(kFull, u, 0), __shfl_sync(kFull, u, 16));
        const double2 bt = make_double2(__shfl_sync(kFull, u, 24), n > 0 && s_dg[2 * parts + 1] == cut.last ? t : 0.0);
        send_cox(gq, bt, __shfl_sync(kFull, u, 8), ind);
    };

    // a worker's groups [ga, gz), and how far the scans over them reach
    const int per_worker = ((own.n_groups + kWorkers - 1) / kWorkers) | 1;  // odd: no bank conflicts
    const int ga = min(tid * per_worker, own.n_groups), gz = wid < kWindow ? min(ga + per_worker, own.n_groups) : ga;
    int lane_from = 0, lane_to = 31, warp_from = 0, warp_to = 0;
    bool lane_open = false, warp_open = false, lane_open_up = false, warp_open_up = false;
    if (COX) {
        bool any_first = false, any_last = false;
        for (int i = ga; i < gz; ++i) {
            any_first |= own.first(i);
            any_last |= own.last(i);
        }
        const unsigned firsts = __ballot_sync(kFull, any_first), lasts = __ballot_sync(kFull, any_last);
        if (wid < kWindow && lane == 0) {
            s_first[wid] = firsts != 0;
            s_last[wid] = lasts != 0;
        }
        __syncthreads();
        const unsigned wf = __ballot_sync(kFull, lane < kWindow && s_first[lane & (kWindow - 1)]);
        const unsigned wl = __ballot_sync(kFull, lane < kWindow && s_last[lane & (kWindow - 1)]);
        lane_from = reach_down(firsts, lane);
        lane_to = reach_up(lasts, lane);
        warp_from = reach_down(wf, lane);
        warp_to = min(reach_up(wl, lane), kWindow - 1);
        lane_open = !(firsts & ((1u << lane) - 1));                       // no stratum begins in the lanes below,
        warp_open = !(wf & ((1u << (wid & (kWindow - 1))) - 1));          // in the warps below
        lane_open_up = !(lane < 31 && lasts >> (lane + 1));              // none ends in the lanes above,
        warp_open_up = !(wl >> ((wid & (kWindow - 1)) + 1));             // in the warps above
    }

    double last = 0.0;
    long long moved = 0, rounds = 0;
    Tracer tracer{Q.trace, rank == 0 && tid == kWorkers + 32, &s_turn.base};
    bool gave_up = false;  // a wait of this CTA ran out

    for (int iteration = 0;; ++iteration) {
        // ---- a cycle is complete: convergence (findMode, CyclicCoordinateDescent.cpp:1023-1056)
        double cur, ll, lp;
        if (!objective(iteration, gave_up, cur, ll, lp)) {  // every CTA leaves
            if (CL && gave_up && tid == 0) {
                if (atomicCAS(&Q.st->error, 0, E_WAIT_CLUSTER) == 0) Q.st->error_where = rank;
                land_all(s_bar, s_report[iteration & 1], C, rank);
            }
            return;
        }
        if (iteration > 0) {
            const bool ill = cur != cur;
            const double conv = ill ? 0.0 : fabs(cur - last) / (fabs(cur) + 1.0);
            const bool met = Q.tol > 0 && conv < Q.tol, done = met || iteration == Q.max_iter;
            if (rank == 0 && tid == 0) {
                Q.st->iterations = iteration;
                Q.st->objective = cur;
                Q.st->loglik = ll;
                Q.st->log_prior = lp;
                if (done) Q.st->flag = !met ? R_MAX_ITERATIONS : (ill ? R_ILLCONDITIONED : R_SUCCESS);
            }
            if (done) break;
        }
        if (Q.max_iter <= 0) break;  // no cycle at all
        last = cur;
        if (wid >= kWindow) {
            // ================ a helper: lane l follows slot l; each warp copies for a quarter of the slots
            const int me = wid - kWindow;
            int q = lane < kWindow ? lane : 0x7fffffff;  // the slot's position
            const int l8 = lane & 7, mine = me + kHelpers * (lane >> 3);  // eight lanes a slot
            for (int i = 0; i < 3; ++i) fetch(mine + i * kWindow, l8);
            ahead.done();
            stage(mine, l8);
            stage(mine + kWindow, l8);
            ahead.done();
            unsigned moved_on = 0;  // the slots that took up a new column in the last round
            int width = kNarrow;
            Turn t{0, 0, 0, 0};
            // what is in flight next, up to the next long column
            auto next_turn = [&]() {
                t.base = __reduce_min_sync(kFull, q);
                t.limit = min(t.base + width, n_active);
                if (LONG) {
                    bool alone = false;
                    if (q < n_active && long_column(rec_of(q))) {
                        const Rec& r = rec_of(q);
                        alone = !COX || width == kNarrow || r.s.ptype != 1 || r.bh.x != 0.0;
                    }
                    const int first = __reduce_min_sync(kFull, alone ? q : 0x7fffffff);
                    t.alone = first == t.base;
                    t.limit = t.alone ? t.base + 1 : min(t.limit, first);
                }
                if (me != 0 || lane != 0) return;
                s_turn.base = t.base;
                s_turn.limit = t.limit;
                if (LONG) s_turn.alone = t.alone;
            };
            if (LONG) __syncthreads();  // every helper's records
            next_turn();
            __syncthreads();
            for (;;) {
                if (t.base >= n_active) break;
                const bool flying = q < t.limit;
                tracer.begin(t.base, t.limit - t.base, t.alone);
                if (CL && me == 0) {
                    const unsigned bytes = __reduce_add_sync(kFull, flying ? pair_bytes(q, rec_of(q)) : 0u);
                    if (lane == 0) expect_sums(bytes);
                }
                const int at = __shfl_sync(kFull, q, mine);
                if (moved_on >> mine & 1u) {
                    stage(at + kWindow, l8);
                    fetch(at + 2 * kWindow, l8);
                }
                ++n_xch;
                __syncthreads();
                tracer.steps();
                const bool quit = s_delta[kWindow] != 0.0;
                // ---- every column up to the first that moves is behind us
                const unsigned to = __reduce_min_sync(kFull, flying && s_delta[lane & (kWindow - 1)] != 0.0 ? (unsigned)q : 0xffffffffu);
                const bool moves = to != 0xffffffffu;
                const bool taken = flying && (unsigned)q <= to;
                moved_on = __ballot_sync(kFull, taken);
                if (taken) q += kWindow;
                width = moves ? kNarrow : min(2 * width, kWindow);
                if (COX && moves && Q.meet) n_xch += 2;
                moved += moves;
                ++rounds;
                next_turn();
                ahead.done();
                __syncthreads();
                tracer.end(__popc(moved_on), moves);
                if (quit | (s_turn.stop != 0)) break;
            }
            ahead.done();
        } else {
            // ================ a warp with a column
            int pos = wid;
            // the lane's entry of the column's first 32: looked up once, while the column is in flight
            bool fresh = true;
            int ck = 0, cg = -1, ckey = 0x7fffffff;
            double cx = 1.0;
            if (LONG) __syncthreads();
            __syncthreads();
            for (;;) {
                const Turn now = s_turn;
                if (now.stop || now.base >= n_active) break;
                const bool mine = pos < now.limit;
                const Rec& r = rec_of(pos);
                double d = 0.0, hd = 0.0, b0 = 0.0, g = 0.0, h = 0.0;
                if (LONG && COX && now.alone) {
                    cox_alone(rec_of(now.base), now.base, mine);
                    if (mine) {
                        b0 = r.bh.x;
                        hd = r.bh.y;
                    }
                } else if (LONG && now.alone) {
                    const double2 gh = gather_alone(rec_of(now.base), now.base, mine);
                    if (mine) {
                        b0 = r.bh.x;
                        hd = r.bh.y;
                        if (CL) {
                            if (lane < C) {
                                const unsigned par = n_xch & 1;
                                send16(to_part + (par * kWindow + wid) * kColumnBytes + rank * (unsigned)sizeof(double2), to_bar + par * 8u,
                                       gh.x, gh.y);
                            }
                        } else if (lane == 0) {
                            __stcg(Q.part + ((size_t)((n_xch & 1) * kWindow + wid) * C + rank) * 3, gh);
                        }
                    }
                } else if (mine) {
                    // ---- the column's sums over this CTA's slice
                    const int n = r.e.hi - r.e.lo;
                    const bool ind = r.c.flags & 4;
                    b0 = r.bh.x;
                    hd = r.bh.y;
                    if (fresh) {
                        fresh = false;
                        cg = -1;
                        ckey = 0x7fffffff;
                        if (lane < n) {
                            ck = entry_row(r, pos, lane);
                            cx = entry_val(r, pos, lane);
                            cg = own.group(ck);
                            ckey = COX ? own.stratum(ck, cg) : cg;
                        }
                    }
                    if (COX) {
                        double G = 0.0, H2 = 0.0, HQ = 0.0, B = 0.0, run = 0.0, A = 0.0;
                        float gs = 0.f, gc = 0.f, hs = 0.f, hc = 0.f;  // mixed: FP32 TwoSum partials of G and H2
                        int run_key = -1, key = -1;
                        const int first = (cut.flags & 1) ? cut.first : -2;
#pragma unroll 1
                        for (int e0 = 0; e0 < n; e0 += 32) {
                            const int e = e0 + lane;
                            const bool in = e < n;
                            double n1 = 0.0, n2 = 0.0, s1 = 0.0, s2 = 0.0;
                            float n1f = 0.f, n2f = 0.f;
                            int k = ck, gr = cg;
                            double x = cx;
                            key = ckey;
                            if (e0 > 0) {
                                key = 0x7fffffff;
                                if (in) {
                                    k = entry_row(r, pos, e);
                                    gr = own.group(k);
                                    x = entry_val(r, pos, e);
                                    key = own.stratum(k, gr);
                                }
                            }
                            if (in) {
                                const double ex = own.ex(k);
                                const double w = P.weighted ? P.w[own.row0 + k] : 1.0;
                                if (gr >= 0) {
                                    s1 = own.s1(gr);
                                    s2 = own.s2(gr);
                                }
                                if (MX) {  // the per-entry terms in FP32
                                    const float xf = (float)x, ef = (float)ex;
                                    n1f = P.weighted ? (float)w * (ef * xf) : ef * xf;
                                    if (!ind) n2f = n1f * xf;
                                    n1 = (double)n1f;
                                } else {
                                    // incrementNumeratorForGradientImpl (ModelSpecifics.hpp:1433-1449)
                                    n1 = P.weighted ? w * (ex * x) : ex * x;
                                    if (!ind) n2 = P.weighted ? w * (ex * x * x) : ex * x * x;
                                }
                            }
                            // the running sum within the stratum
                            int prev = __shfl_up_sync(kFull, key, 1);
                            if (lane == 0) prev = run_key;
                            const unsigned starts = __ballot_sync(kFull, key != prev);
                            A = scan_up(n1, reach_down(starts, lane), n - e0);
                            if (!(starts & (kFull >> (31 - lane)))) A += run;
                            const double before_it = A - n1;
                            if (MX) {
                                const float s1f = (float)s1;
                                two_sum_f(gs, gc, n1f * s1f);
                                two_sum_f(hs, hc, n2f * s1f);
                            } else {
                                G += n1 * s1;
                                H2 += n2 * s1;
                            }
                            if (in) HQ += s2 * (A * A - before_it * before_it);  // risk-set sums: FP64
                            if (key == first) B += s2 * n1;
                            if (e0 + 32 < n) {
                                run = __shfl_sync(kFull, A, 31);
                                run_key = __shfl_sync(kFull, key, 31);
                            }
                        }
                        if (MX) {
                            G = (double)gs + (double)gc;
                            H2 = (double)hs + (double)hc;
                        }
                        const int end = (n + 31) & 31;  // the last entry's lane
                        double T = __shfl_sync(kFull, A, end);
                        if (n == 0 || __shfl_sync(kFull, key, end) != cut.last) T = 0.0;
                        const double s = warp_sum_of_four(G, H2, HQ, B);
                        // lanes 0..7 {G, HQ}, lanes 8..15 {H2, B}
                        const double other = __shfl_xor_sync(kFull, s, 16);
                        const double Bv = __shfl_sync(kFull, other, 8);
                        const double2 gq = make_double2(__shfl_sync(kFull, s, 0), __shfl_sync(kFull, other, 0));
                        const double h2 = __shfl_sync(kFull, s, 8);
                        send_cox(gq, make_double2(Bv, T), h2, ind);
                    } else {
                        double run1 = 0.0, run2 = 0.0;
                        int run_key = -1;
#pragma unroll 1
                        for (int e0 = 0; e0 < n; e0 += 32) {
                            const int e = e0 + lane;
                            const bool in = e < n;
                            int key = ckey, k = ck;
                            double a = 0.0, b = 0.0, x = cx;
                            if (e0 > 0) {
                                key = 0x7fffffff;
                                if (in) {
                                    k = entry_row(r, pos, e);
                                    x = entry_val(r, pos, e);
                                    key = own.group(k);
                                }
                            }
                            if (in) {
                                const double ex = own.ex(k);
                                a = ex * x;
                                if (!ind) b = ex * x * x;
                            }
                            // the next entry's stratum, and whether a run ends here
                            int next = __shfl_down_sync(kFull, key, 1);
                            if (lane == 31) next = e + 1 < n ? own.group(entry_row(r, pos, e + 1)) : -1;
                            int prev = __shfl_up_sync(kFull, key, 1);
                            if (lane == 0) prev = run_key;
                            const unsigned all_starts = __ballot_sync(kFull, key != prev);
                            const unsigned starts = all_starts & (kFull >> (31 - lane));
                            const int start = reach_down(all_starts, lane);
#pragma unroll 1
                            for (int o = 1; o < 32; o <<= 1) {
                                const bool takes = lane - o >= start;
                                if (!__any_sync(kFull, in && takes)) break;  // no run is longer than o
                                const double y = __shfl_up_sync(kFull, a, o), z = __shfl_up_sync(kFull, b, o);
                                if (takes) {
                                    a += y;
                                    b += z;
                                }
                            }
                            if (!starts) {
                                a += run1;
                                b += run2;
                            }
                            if (in && (next != key || e + 1 >= n)) {
                                const double dn = own.den(key), ne = own.nev(key), t = a / dn, gg = ne * t;
                                g += gg;
                                h += ind ? gg * (1.0 - t) : ne * (b / dn - t * t);
                            }
                            if (e0 + 32 < n) {
                                run1 = __shfl_sync(kFull, a, 31);
                                run2 = __shfl_sync(kFull, b, 31);
                                run_key = __shfl_sync(kFull, key, 31);
                            }
                        }
                        const double2 gh = warp_sum_of_two(g, h);
                        if (CL) {
                            if (lane < C) {
                                const unsigned par = n_xch & 1;
                                send16(to_part + (par * kWindow + wid) * kColumnBytes + rank * (unsigned)sizeof(double2), to_bar + par * 8u,
                                       gh.x, gh.y);
                            }
                        } else if (lane == 0) {
                            __stcg(Q.part + ((size_t)((n_xch & 1) * kWindow + wid) * C + rank) * 3, gh);
                        }
                    }
                }
                // ---- the column's sums over the CTAs, the same bits in every one, and its step
                if (!CL) grid_wait(s_delta[kWindow]);
                if (mine) {
                    const bool ind = r.c.flags & 4;
                    const double b_var = r.s.ptype == 2 ? b0 / r.s.pvar : 0.0;
                    if (CL) wait_sums(s_delta[kWindow]);
                    g = 0.0;
                    h = 0.0;
                    double second = 0.0;  // Cox, a column with values: the sum of H2
                    if (CL) {  // lane l: CTA l
                        const double2* const from = &s_part[n_xch & 1][wid][0][0];
                        if (COX) {
                            const int c = lane & (kWindowCluster - 1);
                            const double2 gq = from[c], bt = from[kWindowCluster + c], h2 = ind ? gq : from[2 * kWindowCluster + c];
                            const int fl = c < C ? s_flags[c] : 0;
                            // what the CTAs pass on, and what comes in to each of them
                            const unsigned starts = __ballot_sync(kFull, fl != 3);
                            const double pass = scan_up(bt.y, reach_down(starts, lane), Q.chain);
                            const double in = __shfl_up_sync(kFull, pass, 1);
                            const double carry = (fl & 1) ? in : 0.0;
                            if (lane < C) {
                                g = gq.x;
                                h = h2.x - (gq.y + 2.0 * carry * bt.x);
                                second = h2.x;
                            }
                        } else if (lane < C) {
                            g = from[lane].x;
                            h = from[lane].y;
                        }
                    } else {  // consecutive CTAs of a lane
                        const int per = (C + 31) / 32, c0 = min(lane * per, C), c1 = min(c0 + per, C);
                        const double2* const from = Q.part + (size_t)((n_xch & 1) * kWindow + wid) * C * 3;
                        double in = 0.0;
                        if (COX) {
                            double pass = 0.0;
                            bool starts = false;
#pragma unroll 5
                            for (int c = c0; c < c1; ++c) {
                                const double v = __ldcg(from + 3 * c + 1).y;
                                const bool go = s_flags[c] == 3;
                                pass = go ? pass + v : v;
                                starts |= !go;
                            }
                            pass = scan_up(pass, reach_down(__ballot_sync(kFull, starts), lane), 32);
                            in = __shfl_up_sync(kFull, pass, 1);
                            if (lane == 0) in = 0.0;
                        }
#pragma unroll 5
                        for (int c = c0; c < c1; ++c) {
                            const double2 gq = __ldcg(from + 3 * c);
                            if (COX) {
                                const double2 bt = __ldcg(from + 3 * c + 1);
                                const double h2 = ind ? gq.x : __ldcg(from + 3 * c + 2).x, carry = (s_flags[c] & 1) ? in : 0.0;
                                g += gq.x;
                                h += h2 - (gq.y + 2.0 * carry * bt.x);
                                second += h2;
                                in = s_flags[c] == 3 ? in + bt.y : bt.y;
                            } else {
                                g += gq.x;
                                h += gq.y;
                            }
                        }
                    }
                    const double2 gh = warp_sum_of_two(g, h);
                    g = gh.x;
                    h = gh.y;
                    bool noise = false;
                    if (COX && !MX) {
                        if (ind) second = g;
                        else second = warp_sum_of_two(second, 0.0).x;
                        noise = second > 0.0 && fabs(h) <= kCoxNoise * second && fabs(h) <= 1.7976931348623157e308;
                    }
                    if (noise) g = h = 0.0;
                    else if (r.c.n > 0) g -= r.s.xjy;
                    else g = h = 0.0;  // an empty column gives (0, 0) (ModelSpecifics.hpp:720-723)
                    d = newton_quotient_step(g, h, b0, r.s.ptype, r.s.pvar, r.s.lambda, r.s.inv_var, b_var);
                    d = (d < -hd) ? -hd : (d > hd ? hd : d);  // apply_bounds; its new bound is not needed yet
                    if (lane == 0) s_delta[wid] = d;
                }
                ++n_xch;
                __syncthreads();
                // ---- every step up to the first that is not zero stands
                int to;
                bool quit;
                {
                    const int slot = lane < kWindow ? (now.base + lane) & (kWindow - 1) : kWindow;
                    const bool here = lane < kWindow ? now.base + lane < now.limit : lane == kWindow;
                    const unsigned nz = __ballot_sync(kFull, here & (s_delta[slot] != 0.0));
                    quit = nz >> kWindow;
                    to = nz - 1 < (1u << kWindow) - 1 ? now.base + __ffs(nz) - 1 : 0x7fffffff;
                }
                if (mine && pos <= to) {
                    if (rank == 0 && lane == 0) {  // the bound, and the coefficient where the step moved it
                        apply_bounds(d, hd);
                        Q.bh[pos] = make_double2(d != 0.0 ? b0 + d : b0, hd);
                        if (d != 0.0) Q.beta[r.c.j] = b0 + d;
                    }
                    fresh = true;
                    pos += kWindow;
                }
                if (to != 0x7fffffff) {
                    // ---- the rows of the column that moves: xBeta += delta x, exp; each group's first
                    // entry adds the group's changes to its denominator in row order
                    // (ModelSpecifics.hpp:1548-1571); rows that a zero weight drops may lie between
                    const Rec& mv = rec_of(to);
                    const double delta = s_delta[to & (kWindow - 1)];
                    const int n = mv.e.hi - mv.e.lo;
                    if (n <= 32 && !P.weighted && !long_column(mv)) {  // the column's own warp, which has its entries at hand
                        if (wid == (to & (kWindow - 1))) {
                            double change = 0.0;
                            if (lane < n) {
                                const double old = own.ex(ck), xb = own.xb(ck) + delta * cx, en = row_exp<MX>(xb);
                                own.set_row(ck, xb, en);
                                change = en - old;
                            }
                            const int prev = __shfl_up_sync(kFull, cg, 1);
                            const bool head = lane < n && (lane == 0 || prev != cg);
                            double v = head ? own.den(cg) + change : 0.0;
                            for (int o = 1; o < n; ++o) {
                                const double y = __shfl_down_sync(kFull, change, o);
                                const bool same = __shfl_down_sync(kFull, cg, o) == cg && lane + o < n;
                                if (!__any_sync(kFull, head && same)) break;  // no longer run
                                if (same) v += y;
                            }
                            if (head) own.den(cg) = v;
                        }
                        if (COX) workers_barrier();
                    } else
#pragma unroll 1
                    for (int e0 = 0; e0 < n; e0 += kWorkers) {
                        const int e = e0 + tid;
                        int gr = -1;
                        if (e < n) {
                            const int k = entry_row(mv, to, e);
                            gr = own.group(k);
                            const double old = own.ex(k), xb = own.xb(k) + delta * entry_val(mv, to, e), en = row_exp<MX>(xb);
                            own.set_row(k, xb, en);
                            if (COX && P.weighted) {
                                const double w = P.w[own.row0 + k];
                                s_dd[tid] = w * en - w * old;
                            } else {
                                s_dd[tid] = en - old;
                            }
                        }
                        s_dg[tid] = gr;
                        if (LONG) {  // a warp within one group has its sum ready for the head of the run
                            const int g1 = __reduce_max_sync(kFull, gr);
                            const bool one = __all_sync(kFull, gr == g1 || gr < 0);
                            if (one) {
                                const double t = warp_sum_of_two(gr >= 0 ? s_dd[tid] : 0.0, 0.0).x;
                                if (lane == 0) s_run[wid] = t;
                            }
                            if (lane == 0) s_first[wid] = one ? g1 : -1;
                        }
                        workers_barrier();
                        if (gr >= 0) {
                            int b = tid - 1;
                            while (b >= 0 && s_dg[b] < 0) --b;
                            if (b < 0 || s_dg[b] != gr) {
                                double v = own.den(gr);
                                const int most = min(kWorkers, n - e0);
                                for (int i = tid; i < most; ++i) {
                                    if (LONG && (i & 31) == 0 && s_first[i >> 5] == gr) {
                                        v = v + s_run[i >> 5];
                                        i += 31;
                                        continue;
                                    }
                                    if (s_dg[i] < 0) continue;
                                    if (s_dg[i] != gr) break;
                                    v = v + s_dd[i];
                                }
                                own.den(gr) = v;
                            }
                        }
                        workers_barrier();
                    }
                    if (COX) {
                        // ---- the accumulated denominators: a worker's groups, its warp, the CTA
                        double sum = 0.0;
#pragma unroll 2
                        for (int i = ga; i < gz; ++i) sum = own.first(i) ? own.den(i) : sum + own.den(i);
                        sum = scan_up(sum, lane_from, 32);
                        double pre = __shfl_up_sync(kFull, sum, 1);
                        if (lane == 31) s_run[wid] = sum;
                        workers_barrier();
                        const double all = scan_up(s_run[lane & (kWindow - 1)], warp_from, kWindow);
                        const double below = __shfl_sync(kFull, all, wid ? wid - 1 : 0);
                        if (lane == 0) pre = 0.0;
                        if (lane_open && wid > 0) pre += below;
                        bool tails = true;  // they have come
                        if (Q.meet) {  // a stratum spans CTAs: the tail sums of the CTAs before
                            double carry = 0.0;
                            const double total = __shfl_sync(kFull, all, kWindow - 1);
                            if (CL) {
                                if (wid == 0 && lane < C)
                                    send8(to_tail + (n_xch & 1) * (unsigned)sizeof(s_tail[0]), to_bar + (n_xch & 1) * 8u, total);
                                if (tid == 0) expect_sums(8);
                                tails = __all_sync(kFull, wait_sums(s_turn.stop));
                                carry = (lane >= cut.lo && lane < rank) ? s_tail[n_xch & (kSumBuffers - 1)][lane & (kSumCtas - 1)] : 0.0;
                            } else {
                                if (tid == 0) __stcg(Q.tails + (n_xch & 1) * C + rank, total);
                                grid_wait(s_turn.stop);
                                for (int c = cut.lo + lane; c < rank; c += 32) carry += __ldcg(Q.tails + (n_xch & 1) * C + c);
                            }
#pragma unroll
                            for (int o = 16; o > 0; o >>= 1) carry += __shfl_xor_sync(kFull, carry, o);
                            ++n_xch;
                            if (lane_open && warp_open) pre += carry;
                        }
                        // ---- D of the groups, their terms of the suffix sums, and the suffix sums
                        double D = pre;
                        double2 suf = make_double2(0.0, 0.0);
                        bool ended = false;
#pragma unroll 2
                        for (int i = ga; i < gz; ++i) {
                            D = own.first(i) ? own.den(i) : D + own.den(i);
                            P.D[own.g0 + i] = D;
                            const double ne = own.nev(i), t1 = ne / D, t2 = ne / (D * D);
                            own.s1(i) = t1;
                            own.s2(i) = t2;
                            if (!ended) {
                                suf.x += t1;
                                suf.y += t2;
                                ended = own.last(i);
                            }
                        }
                        suf = scan_down(suf, lane_to, 32);
                        double2 nxt = make_double2(__shfl_down_sync(kFull, suf.x, 1), __shfl_down_sync(kFull, suf.y, 1));
                        if (lane == 0) s_run2[wid] = suf;
                        workers_barrier();
                        const double2 all2 = scan_down(s_run2[lane & (kWindow - 1)], warp_to, kWindow);
                        const int up = wid < kWindow - 1 ? wid + 1 : wid;
                        const double ax = __shfl_sync(kFull, all2.x, up), ay = __shfl_sync(kFull, all2.y, up);
                        if (lane == 31) nxt = make_double2(0.0, 0.0);
                        if (lane_open_up && wid < kWindow - 1) {
                            nxt.x += ax;
                            nxt.y += ay;
                        }
                        if (Q.meet && tails) {  // the head sums of the CTAs after
                            double c1 = 0.0, c2 = 0.0;
                            if (CL) {
                                if (wid == 0 && lane < C) {
                                    const double hx = __shfl_sync(kFull >> (32 - C), all2.x, 0), hy = __shfl_sync(kFull >> (32 - C), all2.y, 0);
                                    send16(to_head + (n_xch & 1) * (unsigned)sizeof(s_head[0]), to_bar + (n_xch & 1) * 8u, hx, hy);
                                }
                                if (tid == 0) expect_sums(16);
                                wait_sums(s_turn.stop);
                                if (lane > rank && lane <= cut.hi) {
                                    const double2 v = s_head[n_xch & (kSumBuffers - 1)][lane & (kSumCtas - 1)];
                                    c1 = v.x;
                                    c2 = v.y;
                                }
                            } else {
                                if (tid == 0) __stcg(Q.heads + (n_xch & 1) * C + rank, all2);
                                grid_wait(s_turn.stop);
                                for (int c = rank + 1 + lane; c <= cut.hi; c += 32) {
                                    const double2 v = __ldcg(Q.heads + (n_xch & 1) * C + c);
                                    c1 += v.x;
                                    c2 += v.y;
                                }
                            }
#pragma unroll
                            for (int o = 16; o > 0; o >>= 1) {
                                c1 += __shfl_xor_sync(kFull, c1, o);
                                c2 += __shfl_xor_sync(kFull, c2, o);
                            }
                            ++n_xch;
                            if (lane_open_up && warp_open_up) {
                                nxt.x += c1;
                                nxt.y += c2;
                            }
                        }
#pragma unroll 2
                        for (int i = gz - 1; i >= ga; --i) {
                            const bool end = own.last(i);
                            nxt.x = end ? own.s1(i) : own.s1(i) + nxt.x;
                            nxt.y = end ? own.s2(i) : own.s2(i) + nxt.y;
                            own.s1(i) = nxt.x;
                            own.s2(i) = nxt.y;
                        }
                    }
                }
                __syncthreads();
                if (quit) break;
            }
        }
        gave_up = s_delta[kWindow] != 0.0 || s_turn.stop;
        if (!CL && gave_up) return;
    }
    if (CL) cluster_barrier();  // no CTA leaves while another may still send to it
    // the state back to where the other calls read it
#pragma unroll 1
    for (int k = tid; WHERE == kRowsShared && k < own.n_rows; k += kT) P.xbe[own.row0 + k] = make_double2(own.xb(k), own.ex(k));
#pragma unroll 1
    for (int g = tid; WHERE != kGlobal && g < own.n_groups; g += kT) {
        P.denom[own.g0 + g] = own.den(g);
        if (COX) {
            P.S1[own.g0 + g] = own.s1(g);
            P.S2[own.g0 + g] = own.s2(g);
        }
    }
    if (rank == 0) {
        __syncthreads();
        for (int p = tid; p < n_active; p += kT) Q.hdelta[Q.cols[p].j] = Q.bh[p].y;
        if (wid == kWindow && lane == 0) {
            Q.st->nonzero_steps = (unsigned long long)moved;
            Q.st->rounds = (unsigned long long)rounds;
        }
    }
}

__global__ void window_slices_kernel(const int32_t* rows, WinCol* cols, int32_t n_active, const GroupCut* cuts, int ctas,
                                     int32_t mark_long, WinSlice* slices) {
    const int64_t total = (int64_t)n_active * ctas;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (int64_t)gridDim.x * blockDim.x) {
        const int r = (int)(i / n_active);
        const WinCol c = cols[i % n_active];
        const int32_t k0 = cuts[r].row0, k1 = cuts[r + 1].row0;
        WinSlice s{k0, k1};
        if (c.flags & 1) {
            auto find = [&](int32_t k) {  // the first entry at row k or after it
                int32_t lo = 0, hi = c.n;
                while (lo < hi) {
                    const int32_t mid = lo + (hi - lo) / 2;
                    if (__ldg(rows + c.cb + mid) < k) lo = mid + 1;
                    else hi = mid;
                }
                return lo;
            };
            s.lo = find(k0);
            s.hi = find(k1);
        }
        slices[i] = s;
        if (mark_long && s.hi - s.lo > kGroupLong)  // flags: the upper half of the word
            atomicOr(reinterpret_cast<unsigned*>(&cols[i % n_active].conflict), 8u << 16);
    }
}

using Kernel = void (*)(GroupWindowParams);

template <bool COX, bool CL, bool MX, bool LONG>
Kernel pick_where(int where) {
    switch (where) {
    case kRowsShared: return group_window_kernel<COX, kRowsShared, CL, MX, LONG>;
    case kGroupsShared: return group_window_kernel<COX, kGroupsShared, CL, MX, LONG>;
    default: return group_window_kernel<COX, kGlobal, CL, MX, LONG>;
    }
}
template <bool COX, bool MX, bool LONG>
Kernel pick_form(int where, bool cl) {
    return cl ? pick_where<COX, true, MX, LONG>(where) : pick_where<COX, false, MX, LONG>(where);
}
// `mixed`: the mixed precision of Cox; `longs`: a column may be long.  The kernels of Cox
// fits with long columns are a compilation of their own (group_window_long.cu): loaded
// with the others they cost every process's first group fit 12 ms.
Kernel pick(bool cox, int where, bool cl, bool mixed, bool longs) {
#ifndef CCDB_COX_LONG
    if (!cox) return longs ? pick_form<false, false, true>(where, cl) : pick_form<false, false, false>(where, cl);
    if (!longs) return mixed ? pick_form<true, true, false>(where, cl) : pick_form<true, false, false>(where, cl);
#endif
#if defined(CCDB_COX_LONG) || defined(CCDB_TRACE_ROUNDS)
    if (cox && longs) return mixed ? pick_form<true, true, true>(where, cl) : pick_form<true, false, true>(where, cl);
#endif
    return nullptr;
}

constexpr int64_t kStagedRows = 2 * kWindow * kStage * sizeof(int32_t);
constexpr int64_t kStagedVals = 2 * kWindow * kStage * sizeof(double);

int64_t group_bytes(bool cox, int64_t groups) { return (cox ? 36 : 16) * groups; }
int64_t row_bytes(int64_t rows) { return 20 * rows; }
int64_t even(int64_t b) { return (b + 15) & ~int64_t(15); }

// Dynamic shared memory that the kernels of a form may hold: grid, cluster of a
// grouped model, cluster of Cox.
cudaError_t smem_limits(int64_t smem[3]) {
    int dev = 0, optin = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
    // the kernels' static shared memory stays below these
    constexpr int64_t kStatic[3] = {16384, 24576, 45056};
    for (int c = 0; c < 3; ++c) smem[c] = std::max<int64_t>(0, optin - kStatic[c]);
    return e;
}

// The attributes of all kernels at the first launch on a device (why all: window.cu).
cudaError_t kernel_attrs(const int64_t smem[3]) {
    static std::atomic<uint64_t> done{0};
    return once_per_device(done, [&] {
        cudaError_t r = cudaSuccess;
        for (int cox = 0; cox < 2; ++cox)
            for (int where : {(int)kRowsShared, (int)kGroupsShared, (int)kGlobal})
                for (int v = 0; v < (cox ? 8 : 4) && r == cudaSuccess; ++v) {
                    const int cl = v & 1;
                    const Kernel fn = pick(cox != 0, where, cl != 0, (v & 4) != 0, (v & 2) != 0);
                    if (!fn) continue;
                    r = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem[cl ? 1 + cox : 0]);
                    if (r == cudaSuccess && cl) r = cudaFuncSetAttribute(fn, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
                }
        return r;
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

}  // namespace

#if !defined(CCDB_TRACE_ROUNDS) && !defined(CCDB_COX_LONG)
bool group_window_fits(bool cox, int64_t groups, int ctas, bool vals, int64_t smem) {
    return kStagedRows + even(group_bytes(cox, (groups + ctas - 1) / ctas)) + (vals ? kStagedVals : 0) <= smem;
}

cudaError_t group_window_limits(GroupWindowLimits* w) {
    w->cluster = 0;
    cudaError_t e = smem_limits(w->smem);
    // one for all: they have the same threads, and their shared memory is asked for in full
    const Kernel fn = pick(false, kRowsShared, true, false, false);
    if (e == cudaSuccess) e = kernel_attrs(w->smem);
    if (e != cudaSuccess) return e;
    for (int C = kWindowCluster; C >= 1; C /= 2) {
        cudaLaunchAttribute at[1];
        const cudaLaunchConfig_t cfg = config(C, (size_t)w->smem[1], 0, at);
        int n = 0;
        const bool fits = cudaOccupancyMaxActiveClusters(&n, fn, &cfg) == cudaSuccess && n >= 1;
        cudaGetLastError();  // a size the device rejects is not an error here: try the next
        if (fits) {
            w->cluster = C;
            return cudaSuccess;
        }
    }
    return cudaSuccess;
}

cudaError_t launch_window_slices(const int32_t* rows, WinCol* cols, int32_t n_active, const GroupCut* cuts, int ctas,
                                 bool mark_long, WinSlice* slices, cudaStream_t stream) {
    const int64_t total = (int64_t)n_active * ctas;
    window_slices_kernel<<<(unsigned)std::max<int64_t>(1, std::min<int64_t>((total + 255) / 256, 4096)), 256, 0, stream>>>(
        rows, cols, n_active, cuts, ctas, mark_long ? 1 : 0, slices);
    return cudaGetLastError();
}

cudaError_t launch_group_window(const GroupWindowParams& Q, bool cluster, int64_t most_rows, int64_t most_groups,
                                cudaStream_t stream) {
#elif defined(CCDB_COX_LONG)
cudaError_t launch_group_window_long(const GroupWindowParams& Q, bool cluster, int64_t most_rows, int64_t most_groups,
                                     cudaStream_t stream) {
#else
cudaError_t launch_group_window_traced(const GroupWindowParams& Q, bool cluster, int64_t most_rows, int64_t most_groups,
                                       cudaStream_t stream) {
#endif
    const int C = Q.ctas;
    if (C < 1 || C > (cluster ? kWindowCluster : kGroupWindowCtas)) return cudaErrorInvalidValue;
    int64_t limits[3];
    cudaError_t e = smem_limits(limits);
    if (e != cudaSuccess) return e;
    const int64_t smem = limits[cluster ? 1 + (Q.cox != 0) : 0];
    const int64_t vals = Q.any_vals ? kStagedVals : 0, groups = group_bytes(Q.cox != 0, most_groups);
    int where = kGlobal;
    int64_t state = 0;
    if (kStagedRows + even(groups + row_bytes(most_rows)) + vals <= smem) {
        where = kRowsShared;
        state = even(groups + row_bytes(most_rows));
    } else if (kStagedRows + even(groups) + vals <= smem) {
        where = kGroupsShared;
        state = even(groups);
    }
    GroupWindowParams R = Q;
    R.vals_at = (int32_t)(kStagedRows + state);
    const size_t bytes = (size_t)(R.vals_at + vals);
    const Kernel fn = pick(Q.cox != 0, where, cluster, Q.P.mixed != 0, Q.any_long != 0);
    if (!fn) return cudaErrorInvalidValue;
    e = kernel_attrs(limits);
    if (e != cudaSuccess) return e;
    if (cluster) {
        cudaLaunchAttribute at[1];
        const cudaLaunchConfig_t cfg = config(C, bytes, stream, at);
        return cudaLaunchKernelEx(&cfg, fn, R);
    }
    void* args[] = {(void*)&R};
    return cudaLaunchCooperativeKernel((const void*)fn, dim3(C), dim3(kT), args, bytes, stream);
}

}  // namespace ccdb
