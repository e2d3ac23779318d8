// cox_host.cu -- host side of the Breslow Cox engine: risk-set grouping,
// per-group tables, and the per-coordinate calls on the device.
#include <algorithm>
#include <cstdio>
#include <cstdlib>
#include <cmath>
#include <cstring>
#include <type_traits>
#include <vector>

#include "cox.h"
#include "engine.h"
#include "group_window.h"

namespace ccdb {

// setPidForAccumulation (ModelSpecifics.hpp:1809-1868) on rows sorted by
// (stratum, -time, y): group id per row (N for rows dropped by a zero weight)
// and the number of groups N.  Integer work, identical to the reference.
int64_t cox_group_rows(const std::vector<int32_t>& pid0, const std::vector<double>& time,
                       const std::vector<double>& y, const double* weights,
                       std::vector<int32_t>& grp) {
    const int64_t K = (int64_t)y.size();
    const int ignore = -1;
    grp.assign(K, 0);
    for (int64_t k = 0; k < K; ++k) grp[k] = pid0[k];
    int64_t index = 0;
    while (weights != nullptr && index < K && weights[index] == 0.0) {
        grp[index] = ignore;
        index++;
    }
    if (index >= K) {  // every row dropped
        for (int64_t k = 0; k < K; ++k) grp[k] = 0;
        return 0;
    }
    int lastPid = grp[index];
    double lastTime = time[index];
    double lastEvent = y[index];
    int pid = grp[index] = 0;
    for (int64_t k = index + 1; k < K; ++k) {
        if (weights == nullptr || weights[k] != 0.0) {
            const int nextPid = grp[k];
            if (nextPid != lastPid) {
                pid++;
                lastPid = nextPid;
            } else if (!(lastEvent == 1.0 && lastTime == time[k] && lastEvent == y[k])) {
                pid++;
            }
            lastTime = time[k];
            lastEvent = y[k];
            grp[k] = pid;
        } else {
            grp[k] = ignore;
        }
    }
    const int64_t N = (int64_t)pid + 1;
    for (int64_t k = 0; k < K; ++k)
        if (grp[k] == ignore) grp[k] = (int32_t)N;
    return N;
}

CoxParams Fit::cox_params() const {
    CoxParams P{};
    P.col_ptr = m->d_col_ptr;
    P.rows = m->d_rows;
    P.val_ptr = m->d_val_ptr;
    P.vals = m->d_vals;
    P.fmt = m->d_fmt;
    P.K = K;
    P.N = cox.N;
    P.xbe = cox.xbe;
    P.w = w;
    P.y = y;
    P.grp = cox.grp;
    P.rstrat = cox.rstrat;
    P.weighted = weighted ? 1 : 0;
    P.mixed = (is_cox() && precision == CCDB_PRECISION_MIXED) ? 1 : 0;
    P.denom = cox.denom;
    P.D = cox.D;
    P.S1 = cox.S1;
    P.S2 = cox.S2;
    P.nEv = cox.nEv;
    P.gfirst = cox.gfirst;
    P.glast = cox.glast;
    P.grow = cox.grow;
    P.xjy = xjy;
    P.st = st;
    P.wait_limit_ns = wait_limit_ns;
    return P;
}

void Fit::cox_allocate() {
    // stratum index of each row, as ModelData::loadY numbers them (ModelData.cpp:96-125)
    std::vector<int32_t> rs(K);
    int32_t p = 0;
    for (int64_t k = 0; k < K; ++k) {
        if (k > 0 && stratum_h[k] != stratum_h[k - 1]) p++;
        rs[k] = p;
    }
    pid0_h = rs;
    const int64_t n_strata = K > 0 ? (int64_t)p + 1 : 0;
    // Cox: the most groups any weighting can produce; grouped models: the strata; + slot N
    const size_t G = is_cox() ? (size_t)K + 1 : (size_t)n_strata + 1;
    cox.xbe = static_cast<double2*>(ctx->alloc(sizeof(double2) * K));
    cox.grp = static_cast<int32_t*>(ctx->alloc(sizeof(int32_t) * K));
    cox.rstrat = static_cast<int32_t*>(ctx->alloc(sizeof(int32_t) * K));
    cox.denom = static_cast<double*>(ctx->alloc(sizeof(double) * G));
    cox.D = static_cast<double*>(ctx->alloc(sizeof(double) * G));
    cox.S1 = static_cast<double*>(ctx->alloc(sizeof(double) * G));
    cox.S2 = static_cast<double*>(ctx->alloc(sizeof(double) * G));
    cox.nEv = static_cast<double*>(ctx->alloc(sizeof(double) * G));
    cox.gfirst = static_cast<uint8_t*>(ctx->alloc(G));
    cox.glast = static_cast<uint8_t*>(ctx->alloc(G));
    cox.grow = static_cast<int64_t*>(ctx->alloc(sizeof(int64_t) * (G + 1)));
    const int tiles = cox_scan_tiles((int64_t)G);
    cox.tickets = static_cast<unsigned*>(ctx->alloc(2 * sizeof(unsigned)));
    cox.status = static_cast<int*>(ctx->alloc(sizeof(int) * 2 * std::max(1, tiles)));
    cox.tails = ctx->alloc(cox_tail_bytes() * 2 * std::max(1, tiles));
    cox.batch_cols = static_cast<int32_t*>(ctx->alloc(sizeof(int32_t) * kBatchMax));
    cox.batch_out = static_cast<double2*>(ctx->alloc(sizeof(double2) * kBatchMax));
    check_cuda(cudaMemsetAsync(cox.status, 0, sizeof(int) * 2 * std::max(1, tiles), stream), "status");
    check_cuda(cudaMemsetAsync(cox.S1, 0, sizeof(double) * G, stream), "S1");
    check_cuda(cudaMemsetAsync(cox.S2, 0, sizeof(double) * G, stream), "S2");
    check_cuda(cudaMemsetAsync(cox.xbe, 0, sizeof(double2) * K, stream), "xbe");
    check_cuda(cudaMemcpyAsync(cox.rstrat, rs.data(), sizeof(int32_t) * K, cudaMemcpyHostToDevice, stream),
               "rstrat");
    if (is_grouped()) {  // the group of a row is its stratum (GroupedData::getGroup)
        cox.N = n_strata;
        std::vector<int64_t> grow(n_strata + 1, K);
        for (int64_t k = K - 1; k >= 0; --k) grow[rs[k]] = k;
        grow[n_strata] = K;
        check_cuda(cudaMemcpyAsync(cox.grp, rs.data(), sizeof(int32_t) * K, cudaMemcpyHostToDevice, stream),
                   "grp");
        check_cuda(cudaMemcpyAsync(cox.grow, grow.data(), sizeof(int64_t) * (n_strata + 1),
                                   cudaMemcpyHostToDevice, stream), "grow");
        cox_grow_h = grow;
    }
    check_cuda(ctx->wait(), "cox alloc");
}

void Fit::cox_release() {
    for (void* p : {(void*)cox.xbe, (void*)cox.grp, (void*)cox.rstrat, (void*)cox.denom, (void*)cox.D,
                    (void*)cox.S1, (void*)cox.S2, (void*)cox.nEv, (void*)cox.gfirst, (void*)cox.glast,
                    (void*)cox.grow, (void*)cox.tickets, (void*)cox.status, cox.tails,
                    (void*)cox.batch_cols, (void*)cox.batch_out, cox.block_mem})
        ctx->release(p);
}

// setWeights for the Cox model (ModelSpecifics.hpp:427-484): regroup with the
// weights, N-weights = events (observationCount = y) times weight per group,
// then computeXjY (x * y * w; survival models use observationCount(y) = y).
void Fit::cox_apply_weights() {
    std::vector<double> wh(K, 1.0);
    if (weighted) wh = w_h;
    if (is_grouped()) {
        // setWeights (ModelSpecifics.hpp:427-484): nEv per stratum = y * w
        // (observationCount = y); computeXjY: x * y * w; fixed terms for CPR.
        const int64_t N = cox.N;
        std::vector<double> nev(N + 1, 0.0);
        for (int64_t k = 0; k < K; ++k) nev[pid0_h[k]] += y_h[k] * wh[k];
        check_cuda(cudaMemcpyAsync(w, wh.data(), sizeof(double) * K, cudaMemcpyHostToDevice, stream), "w");
        check_cuda(cudaMemcpyAsync(cox.nEv, nev.data(), sizeof(double) * (N + 1), cudaMemcpyHostToDevice,
                                   stream), "nev");
        check_cuda(launch_xjy(m->d_col_ptr, m->d_rows, m->d_val_ptr, m->d_vals, m->d_fmt, y,
                              weighted ? w : nullptr, K, J, xjy, stream), "xjy");
        ++launches;
        ll_fixed = 0.0;
        if (model == M_CPR) {  // ConditionalPoissonRegression::logLikeFixedTermsContrib (ModelSpecifics.h:722-727)
            for (int64_t i = 0; i < K; ++i) {
                double t = 0.0;
                for (int c = 2; c <= (int)y_h[i]; c++) t -= std::log((double)c);
                ll_fixed += weighted ? t * wh[i] : t;
            }
        }
        check_cuda(ctx->wait(), "grouped weights");
        valid_weights = true;
        suff_known = false;
        return;
    }
    std::vector<int32_t> grp;
    const int64_t N = cox_group_rows(pid0_h, time_h, y_h, weighted ? w_h.data() : nullptr, grp);
    cox.N = N;
    std::vector<double> nev(N + 1, 0.0);
    for (int64_t k = 0; k < K; ++k) nev[grp[k]] += y_h[k] * wh[k];
    std::vector<uint8_t> gf(N + 1, 0), gl(N + 1, 0);
    std::vector<int64_t> grow(N + 2, K);
    std::vector<int32_t> gstrat(N + 1, -1);
    for (int64_t k = K - 1; k >= 0; --k)
        if (grp[k] < N) {
            grow[grp[k]] = k;
            gstrat[grp[k]] = pid0_h[k];
        }
    for (int64_t g = N - 1; g >= 0; --g)
        if (grow[g] == K) grow[g] = grow[g + 1];
    for (int64_t g = 0; g < N; ++g) {
        gf[g] = (g == 0 || gstrat[g] != gstrat[g - 1]) ? 1 : 0;
        gl[g] = (g == N - 1 || gstrat[g] != gstrat[g + 1]) ? 1 : 0;
    }
    grow[N] = K;
    ++cox.grouping;
    check_cuda(cudaMemcpyAsync(w, wh.data(), sizeof(double) * K, cudaMemcpyHostToDevice, stream), "w");
    check_cuda(cudaMemcpyAsync(cox.grp, grp.data(), sizeof(int32_t) * K, cudaMemcpyHostToDevice, stream), "grp");
    check_cuda(cudaMemcpyAsync(cox.nEv, nev.data(), sizeof(double) * (N + 1), cudaMemcpyHostToDevice, stream), "nev");
    check_cuda(cudaMemcpyAsync(cox.gfirst, gf.data(), N + 1, cudaMemcpyHostToDevice, stream), "gfirst");
    check_cuda(cudaMemcpyAsync(cox.glast, gl.data(), N + 1, cudaMemcpyHostToDevice, stream), "glast");
    check_cuda(cudaMemcpyAsync(cox.grow, grow.data(), sizeof(int64_t) * (N + 1), cudaMemcpyHostToDevice, stream),
               "grow");
    check_cuda(cudaMemsetAsync(cox.S1 + N, 0, sizeof(double), stream), "S1N");
    check_cuda(cudaMemsetAsync(cox.S2 + N, 0, sizeof(double), stream), "S2N");
    // slot N gathers the rows a zero weight drops; like the reference's denomPid[N]
    // it holds 0, which the MM bound reads (0 * e / 0 for such a row, as there)
    check_cuda(cudaMemsetAsync(cox.denom + N, 0, sizeof(double), stream), "denomN");
    check_cuda(cudaMemsetAsync(cox.D + N, 0, sizeof(double), stream), "DN");
    check_cuda(launch_xjy(m->d_col_ptr, m->d_rows, m->d_val_ptr, m->d_vals, m->d_fmt, y,
                          weighted ? w : nullptr, K, J, xjy, stream),
               "xjy");
    ++launches;
    ll_fixed = 0.0;
    check_cuda(ctx->wait(), "cox weights");
    cox_groups_h.row_group = std::move(grp);
    cox_groups_h.stratum = std::move(gstrat);
    cox_groups_h.first_row = std::move(grow);
    cox_groups_h.events = std::move(nev);
    valid_weights = true;
    suff_known = false;
}

// Blocks: runs of groups up to one with events, or to their stratum's end.  D
// counts only where there are events, and S1 and S2 change only there, so the
// windowed sweep keeps one denominator, one D and one pair of suffix sums per block.
// Built when a sweep needs them: a predictive log-likelihood regroups twice and
// sweeps never (300,000 rows: 5.6 ms, 8.1 with the blocks).  One allocation and one
// copy: ten of the one and six of the other had cost a fit of 100 rows 50 us.
void Fit::ensure_cox_blocks() {
    if (cox.blocks == cox.grouping) return;
    const auto& g = cox_groups_h;
    const int64_t N = cox.N;
    auto begins = [&](int64_t i) { return i == 0 || g.stratum[i] != g.stratum[i - 1]; };
    std::vector<int32_t> bgrp, group_block(N + 1);
    std::vector<int32_t> bstrat;
    for (int64_t i = 0; i < N; ++i) {
        if (begins(i) || g.events[i - 1] != 0.0) {
            bgrp.push_back((int32_t)i);
            bstrat.push_back(g.stratum[i]);
        }
        group_block[i] = (int32_t)bgrp.size() - 1;
    }
    const int64_t NB = (int64_t)bgrp.size();
    bgrp.push_back((int32_t)N);
    group_block[N] = (int32_t)NB;  // the rows that a zero weight drops
    Parts p;
    const size_t at_row = p.add(sizeof(int64_t) * (NB + 1)), at_nev = p.add(sizeof(double) * (NB + 1)),
                 at_blk = p.add(sizeof(int32_t) * K), at_grp = p.add(sizeof(int32_t) * (NB + 1)), at_first = p.add(NB + 1),
                 at_last = p.add(NB + 1), host_bytes = p.bytes;
    size_t at[4];
    for (size_t& a : at) a = p.add(sizeof(double) * (NB + 1));
    std::unique_ptr<char[]> host(new char[host_bytes]);
    auto* const brow = reinterpret_cast<int64_t*>(host.get() + at_row);
    auto* const bnev = reinterpret_cast<double*>(host.get() + at_nev);
    auto* const blk = reinterpret_cast<int32_t*>(host.get() + at_blk);
    auto* const bf = reinterpret_cast<uint8_t*>(host.get() + at_first);
    auto* const bl = reinterpret_cast<uint8_t*>(host.get() + at_last);
    for (int64_t k = 0; k < K; ++k) blk[k] = group_block[g.row_group[k]];
    std::memcpy(host.get() + at_grp, bgrp.data(), sizeof(int32_t) * (NB + 1));
    brow[NB] = K;
    bnev[NB] = 0.0;
    bf[NB] = bl[NB] = 0;
    for (int64_t b = 0; b < NB; ++b) {
        const int64_t last = bgrp[b + 1] - 1;
        bnev[b] = g.events[last];
        bf[b] = begins(bgrp[b]) ? 1 : 0;
        bl[b] = (last == N - 1 || begins(last + 1)) ? 1 : 0;
        brow[b] = g.first_row[bgrp[b]];
    }
    ctx->release(cox.block_mem);
    cox.block_mem = nullptr;
    cox.blocks = -1;
    cox.block_mem = ctx->alloc(p.bytes);
    char* const d = static_cast<char*>(cox.block_mem);
    check_cuda(cudaMemcpyAsync(d, host.get(), host_bytes, cudaMemcpyHostToDevice, stream), "blocks");
    cox.brow = reinterpret_cast<int64_t*>(d + at_row);
    cox.bnev = reinterpret_cast<double*>(d + at_nev);
    cox.blk = reinterpret_cast<int32_t*>(d + at_blk);
    cox.bgrp = reinterpret_cast<int32_t*>(d + at_grp);
    cox.bfirst = reinterpret_cast<uint8_t*>(d + at_first);
    cox.blast = reinterpret_cast<uint8_t*>(d + at_last);
    cox.bden = reinterpret_cast<double*>(d + at[0]);
    cox.bD = reinterpret_cast<double*>(d + at[1]);
    cox.bS1 = reinterpret_cast<double*>(d + at[2]);
    cox.bS2 = reinterpret_cast<double*>(d + at[3]);
    cox_grow_h.assign(brow, brow + NB + 1);
    cox_bstrat_h = std::move(bstrat);
    cox.NB = NB;
    cox.blocks = cox.grouping;
}

void Fit::cox_scans() {
    if (!is_cox()) return;
    ++cox.epoch;
    CoxParams P = cox_params();
    check_cuda(launch_cox_scans(P, cox.tickets, cox.status, cox.tails, cox.epoch, stream), "cox scans");
    launches += 2;
}

// computeRemainingStatistics (ModelSpecifics.hpp:1588-1617) + the accumulated scans.
// `rows_done`: the rows' exp(xBeta) belongs to their xBeta, as a sweep leaves it.
void Fit::cox_remaining(bool rows_done) {
    const double* const fresh = xb_pending ? xb_tmp : nullptr;  // xBeta computed into xb_tmp
    xb_pending = false;
    CoxParams P = cox_params();
    if (!rows_done || fresh) {
        check_cuda(launch_cox_exp(P, fresh, stream), "exp");
        ++launches;
    }
    if (is_cox()) check_cuda(launch_cox_denominators(P, stream), "cox remaining");
    else check_cuda(launch_grouped_denominators(P, stream), "grouped remaining");
    ++launches;
    cox_scans();
    suff_known = true;
}

void Fit::cox_objective_terms(double* out4) {
    const int nb = ctx->n_sm;
    CoxParams P = cox_params();
    if (is_cox()) check_cuda(launch_cox_objective(P, red, nb, stream), "cox objective");
    else check_cuda(launch_grouped_objective(P, red, nb, stream), "grouped objective");
    ++launches;
    std::vector<double2> parts(2 * nb);
    check_cuda(cudaMemcpyAsync(parts.data(), red, sizeof(double2) * 2 * nb, cudaMemcpyDeviceToHost, stream),
               "objective copy");
    check_cuda(ctx->wait(), "objective sync");
    double t[4] = {0, 0, 0, 0};
    for (int c = 0; c < nb; ++c) {
        t[0] += parts[2 * c].x;
        t[1] += parts[2 * c].y;
        t[2] += parts[2 * c + 1].x;
    }
    // log prior on the host (JointPrior.h:121-128)
    for (int j = 0; j < J; ++j) t[3] += log_prior_host(beta_h[j], ptype_h[j], pvar_h[j]);
    for (int i = 0; i < 4; ++i) out4[i] = t[i];
}

void Fit::cox_gh_batch(const int32_t* cols, int n, double2* out) {
    // one column: its index and its result in the fit's pinned words, no copies
    double2* const slot = n == 1 ? ctx->result(result_slot) : nullptr;
    int32_t* const which = slot ? reinterpret_cast<int32_t*>(slot + 1) : cox.batch_cols;
    if (slot) *which = cols[0];
    else check_cuda(cudaMemcpyAsync(which, cols, sizeof(int32_t) * n, cudaMemcpyHostToDevice, stream), "batch cols");
    double2* const to = slot ? slot : cox.batch_out;
    CoxParams P = cox_params();
    if (is_cox()) check_cuda(launch_cox_gh(P, which, n, to, stream), "cox gh");
    else check_cuda(launch_grouped_gh(P, which, n, to, stream), "grouped gh");
    ++launches;
    if (!slot) check_cuda(cudaMemcpyAsync(out, to, sizeof(double2) * n, cudaMemcpyDeviceToHost, stream), "gh copy");
    check_cuda(ctx->wait(), "gh sync");
    if (slot) *out = *slot;
}

void Fit::cox_update(int j, double delta) {
    CoxParams P = cox_params();
    if (is_cox()) check_cuda(launch_cox_update(P, j, delta, stream), "cox update");
    else check_cuda(launch_grouped_update(P, j, delta, stream), "grouped update");
    ++launches;
    cox_scans();
}

// The plan of the group models' windowed sweep on `ctas` CTAs: whole groups, in
// equal numbers, and what each CTA's strata share with its neighbours'.
void Fit::ensure_group_window(int ctas, bool cluster) {
    if (window && window->ctas == ctas && window->cluster == cluster && window->grouping == cox.grouping &&
        window->fixed == fixed)
        return;
    release_window();
    window.reset(new DevWindow());  // owned by the fit from here on, complete or not
    std::vector<WinCol> cols;
    for (int j = 0; j < J; ++j) {
        if (fixed[j]) continue;
        const uint8_t f = m->fmt[j];
        WinCol c{};
        c.cb = m->col_start[j];
        c.vb = m->val_start[j];
        c.j = j;
        c.n = (int32_t)m->entries(j);
        c.flags = ((f == F_SPARSE || f == F_INDICATOR) ? 1 : 0) | ((f == F_SPARSE || f == F_DENSE) ? 2 : 0) |
                  ((f == F_INDICATOR || f == F_INTERCEPT) ? 4 : 0);
        window->any_vals |= (c.flags & 2) != 0;
        window->any_long |= !is_cox() && c.n > kGroupLong;
        cols.push_back(c);
    }
    // Where a CTA's groups begin.  Cox: at the nearest start of a stratum, when no CTA
    // then owns a quarter more than its even share, so that no stratum spans CTAs and
    // a step needs no tail and head sums; else in even shares.  (The line weighs balance
    // alone.  With fewer blocks a CTA than worker threads, 512, the longer share costs the
    // scans nothing, and the two exchanges, 1,300 to 1,800 clocks each, are paid for it.)
    std::vector<GroupCut> cuts(ctas + 1);
    const int64_t N = is_cox() ? cox.NB : cox.N;
    std::vector<int64_t> first_group(ctas + 1);
    for (int r = 0; r <= ctas; ++r) first_group[r] = N * r / ctas;
    if (is_cox() && ctas > 1) {
        std::vector<int64_t> starts, aligned(first_group);
        for (int64_t g = 0; g < N; ++g)
            if (g == 0 || cox_bstrat_h[g] != cox_bstrat_h[g - 1]) starts.push_back(g);
        starts.push_back(N);
        int64_t most = 0;
        for (int r = 1; r < ctas; ++r) {
            const auto above = std::lower_bound(starts.begin(), starts.end(), first_group[r]);
            const auto below = above == starts.begin() ? above : above - 1;
            aligned[r] = *above - first_group[r] < first_group[r] - *below ? *above : *below;
        }
        bool each = true;
        for (int r = 0; r < ctas; ++r) {
            most = std::max(most, aligned[r + 1] - aligned[r]);
            each &= aligned[r + 1] > aligned[r];
        }
        if (each && most * ctas * 4 <= N * 5) first_group = aligned;
    }
    for (int r = 0; r <= ctas; ++r) {
        GroupCut& c = cuts[r];
        const int64_t g0 = first_group[r], g1 = r < ctas ? first_group[r + 1] : N;
        c.g0 = (int32_t)g0;
        c.row0 = (int32_t)(r == 0 ? 0 : r == ctas ? K : cox_grow_h[g0]);
        c.lo = c.hi = r;
        if (is_cox() && r < ctas && g1 > g0) {
            c.first = cox_bstrat_h[g0];
            c.last = cox_bstrat_h[g1 - 1];
            c.flags = ((g0 > 0 && cox_bstrat_h[g0 - 1] == c.first) ? 1 : 0) | (c.first == c.last ? 2 : 0);
        } else {
            c.first = c.last = -1;
        }
    }
    int32_t row = 1;
    for (int r = 0; r < ctas; ++r) {
        GroupCut& c = cuts[r];
        window->most_rows = std::max<int64_t>(window->most_rows, cuts[r + 1].row0 - c.row0);
        window->most_groups = std::max<int64_t>(window->most_groups, cuts[r + 1].g0 - c.g0);
        window->meet |= (c.flags & 1) != 0;
        window->chain = std::max(window->chain, r > 0 && c.flags == 3 ? ++row : (row = 1));
        if (c.flags & 1) {
            c.lo = r - 1;
            while (c.lo > 0 && cuts[c.lo].flags == 3) --c.lo;
        }
        if (r + 1 < ctas && (cuts[r + 1].flags & 1)) {
            c.hi = r + 1;
            while (c.hi + 1 < ctas && (cuts[c.hi].flags & 2) && (cuts[c.hi + 1].flags & 1)) ++c.hi;
        }
    }
    // Cox: by a column's even share of the fullest CTA's rows (which columns are marked
    // long, their true slices say)
    for (const WinCol& c : cols) window->any_long |= is_cox() && c.n * window->most_rows > kGroupLong * K;
    const size_t n = cols.size();
    const size_t col_bytes = sizeof(WinCol) * n, cut_bytes = sizeof(GroupCut) * cuts.size(), grid = cluster ? 0 : 2 * ctas;
    Parts p;
    const size_t at_cols = p.add(col_bytes), at_cuts = p.add(cut_bytes), at_slices = p.add(sizeof(WinSlice) * n * ctas),
                 at_scal = p.add(sizeof(WinScal) * n), at_bh = p.add(sizeof(double2) * n),
                 at_part = p.add(sizeof(double2) * kWindow * 3 * grid), at_tails = p.add(sizeof(double) * grid),
                 at_heads = p.add(sizeof(double2) * grid);
    place_window(p.bytes, {at_cols, col_bytes, cols.data()}, {at_cuts, cut_bytes, cuts.data()});
    char* const d = static_cast<char*>(window->mem);
    window->cols = reinterpret_cast<WinCol*>(d + at_cols);
    window->cuts = reinterpret_cast<GroupCut*>(d + at_cuts);
    window->slices = reinterpret_cast<WinSlice*>(d + at_slices);
    window->scal = reinterpret_cast<WinScal*>(d + at_scal);
    window->bh = reinterpret_cast<double2*>(d + at_bh);
    if (!cluster) {
        window->part = reinterpret_cast<double2*>(d + at_part);
        window->tails = reinterpret_cast<double*>(d + at_tails);
        window->heads = reinterpret_cast<double2*>(d + at_heads);
    }
    check_cuda(launch_window_slices(m->d_rows, window->cols, (int32_t)n, window->cuts, ctas, window->any_long, window->slices,
                                    stream),
               "sweep plan");
    ++launches;
    window->n_active = (int32_t)n;
    window->fixed = fixed;
    window->grouping = cox.grouping;
    window->cluster = cluster;
    window->ctas = ctas;
}

// findMode (CyclicCoordinateDescent.cpp:909-1216) of the Cox and grouped models
// in one launch (group_window.cu).  The bounds are set by the caller.
void Fit::find_mode_group_window(const ccdb_mode_args& a, int* flag, int* iters, double* obj, float* ms) {
    if (std::find(fixed.begin(), fixed.end(), uint8_t(0)) == fixed.end()) {
        // an empty cycle: the first check sees conv = 0
        *obj = objective(a.convergence_type);
        *flag = (*obj != *obj) ? R_ILLCONDITIONED
                : (a.tolerance > 0 ? R_SUCCESS : (a.max_iterations == 1 ? R_MAX_ITERATIONS : R_SUCCESS));
        *iters = 1;
        *ms = 0.f;
        return;
    }
    if (is_cox()) ensure_cox_blocks();
    GroupWindowLimits& lim = ctx->group_window;
    if (lim.cluster < 0) check_cuda(group_window_limits(&lim), "cluster occupancy");
    bool any_vals = false;
    for (int j = 0; j < J; ++j) any_vals |= !fixed[j] && (m->fmt[j] == F_SPARSE || m->fmt[j] == F_DENSE);
    // The cluster form, on the largest cluster of the context's share, when the groups
    // fit its CTAs' shared memory and a CTA's slice of a column is not over about 128
    // entries; else the grid form, on 64 CTAs or as many as the groups need: more of
    // them lengthen every exchange.  CCDB_SWEEP_GRID_LEVELS asks for the grid form,
    // CCDB_SWEEP_LEVELS for the cluster form.  Milliseconds per fit on a cluster of 4,
    // 8, 16 and a grid of 32, 64, 148: conditional logistic, 4,000 sets, 512 entries a
    // column: 4.60 3.27 2.82 3.13 3.41 4.74; 20,000 sets, 2,601 entries: 26.8 14.3 4.78
    // 4.22 3.84 4.14; Cox, 20,000 rows, 199 entries: 2.75 2.94 2.52 4.47 4.73 6.35;
    // 200,000 rows, 2,001 entries: 17.7 11.0 7.62 6.68 6.55 7.84.  The line of 128 lies
    // above where the forms cross.  200,000 rows, cluster of 16 and grid of 64, Cox: mean
    // 800 7.13 and 7.58, 1,200 7.88 and 7.75, 2,000 9.98 and 8.76; conditional logistic:
    // 200 1.00 and 1.37, 400 0.95 and 0.98, 800 1.58 and 1.21, 2,000 4.47 and 2.45.
    const int64_t N = is_cox() ? cox.NB : cox.N;
    int64_t total = 0, active = 0;
    for (int j = 0; j < J; ++j)
        if (!fixed[j]) {
            total += m->entries(j);
            ++active;
        }
    int n_cta = ctx->n_sm;
    if (ctx->max_ctas > 0) n_cta = std::min(n_cta, ctx->max_ctas);
    int c = lim.cluster;
    while (c > 1 && (c > n_cta || c > N)) c /= 2;
    const int64_t smem_grid = lim.smem[0], smem_cluster = lim.smem[is_cox() ? 2 : 1];
    const bool use_cluster = c >= 1 && a.strategy != CCDB_SWEEP_GRID_LEVELS &&
                             (a.strategy == CCDB_SWEEP_LEVELS || n_cta <= lim.cluster + lim.cluster / 4 ||
                              (group_window_fits(is_cox(), N, c, any_vals, smem_cluster) && total / active <= 128 * c));
    if (use_cluster) {
        n_cta = c;
    } else {
        const int most = (int)std::max<int64_t>(1, std::min<int64_t>({n_cta, N, kGroupWindowCtas}));
        n_cta = std::min(64, most);
        while (n_cta < most && !group_window_fits(is_cox(), N, n_cta, any_vals, smem_grid)) ++n_cta;
    }
    ensure_group_window(n_cta, use_cluster);
    if (!beta_dirty_host) upload_beta();
    DevStatus zero{};
    zero.flag = R_FAIL;
    check_cuda(cudaMemcpyAsync(st, &zero, sizeof(zero), cudaMemcpyHostToDevice, stream), "status");
    check_cuda(cudaMemsetAsync(grid_bar, 0, sizeof(unsigned), stream), "barrier");
    GroupWindowParams Q{};
    Q.P = cox_params();
    Q.cox = is_cox() ? 1 : 0;
    if (is_cox()) {
        check_cuda(launch_cox_blocks(Q.P, cox.bgrp, cox.NB, cox.bden, cox.bD, cox.bS1, cox.bS2, stream), "blocks");
        ++launches;
        Q.P.N = cox.NB;
        Q.P.grp = cox.blk;
        Q.P.denom = cox.bden;
        Q.P.D = cox.bD;
        Q.P.S1 = cox.bS1;
        Q.P.S2 = cox.bS2;
        Q.P.nEv = cox.bnev;
        Q.P.gfirst = cox.bfirst;
        Q.P.glast = cox.blast;
        Q.P.grow = cox.brow;
    }
    Q.n_active = window->n_active;
    Q.cols = window->cols;
    Q.slices = window->slices;
    Q.scal = window->scal;
    Q.bh = window->bh;
    Q.cuts = window->cuts;
    Q.beta = beta;
    Q.hdelta = hdelta;
    Q.ptype = ptype;
    Q.pvar = pvar;
    Q.J = J;
    Q.conv = a.convergence_type;
    Q.max_iter = a.max_iterations;
    Q.tol = a.tolerance;
    Q.ctas = window->ctas;
    Q.ll_fixed = ll_fixed;
    Q.any_vals = window->any_vals ? 1 : 0;
    Q.any_long = window->any_long ? 1 : 0;
    Q.meet = window->meet ? 1 : 0;
    Q.chain = window->chain;
    Q.st = st;
    Q.part = window->part;
    Q.tails = window->tails;
    Q.heads = window->heads;
    Q.red = red;
    Q.grid_bar = grid_bar;
    Q.wait_limit_ns = wait_limit_ns;
    RoundTrace trace(ctx);
    Q.trace = trace.d;
    check_cuda(cudaEventRecord(ctx->fev[0], stream), "event");
    const auto launch = trace.d                         ? launch_group_window_traced
                        : is_cox() && window->any_long ? launch_group_window_long
                                                       : launch_group_window;
    check_cuda(launch(Q, use_cluster, window->most_rows, window->most_groups, stream), "group sweep launch");
    ++launches;
    check_cuda(cudaEventRecord(ctx->fev[1], stream), "event");
    if (is_cox()) cox_remaining(true);  // the groups' own denominators and sums, for the calls that follow
    check_cuda(ctx->wait(), "group sweep");  // the sweep is done before a copy is queued behind it
    DevStatus out{};
    check_cuda(cudaMemcpyAsync(&out, st, sizeof(out), cudaMemcpyDeviceToHost, stream), "status");
    check_cuda(ctx->wait(), "group sweep");
    check_cuda(cudaEventElapsedTime(ms, ctx->fev[0], ctx->fev[1]), "elapsed");
    trace.write();
    if (out.error != E_NONE)
        throw Error(CCDB_ERR_TIMEOUT, "device wait timed out (code " + std::to_string(out.error) + " at " +
                                          std::to_string(out.error_where) + ")");
    nz_steps += (int64_t)out.nonzero_steps;
    *flag = out.flag;
    *iters = out.iterations;
    *obj = out.objective;
    beta_dirty_host = true;
}

}  // namespace ccdb
