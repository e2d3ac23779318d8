// api.cu -- the C ABI of libccdb.so (include/ccdb.h) and the host runtime
// behind it: device memory under a per-context HBM budget, matrix upload,
// per-fit lazy state (the flags of CyclicCoordinateDescent::checkAllLazyFlags,
// CyclicCoordinateDescent.cpp:388-406), schedule caching, and the mode-finding
// driver (CyclicCoordinateDescent::update, .cpp:586-615).
#include <algorithm>
#include <chrono>
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <memory>
#include <mutex>
#include <stdexcept>
#include <string>
#include <system_error>
#include <thread>
#include <vector>

#include <cuda_runtime.h>

#include "../../include/ccdb.h"
#include "batch.h"
#include "batch_window.h"
#include "csr_device.h"
#include "csr_host.h"
#include "engine.h"

namespace ccdb {

thread_local std::string g_last_error;

void check_cuda(cudaError_t e, const char* what) {
    if (e != cudaSuccess)
        throw Error(CCDB_ERR_CUDA, std::string(what) + ": " + cudaGetErrorString(e));
}

void* Context::alloc(size_t bytes) {
    if (bytes == 0) bytes = 16;
    bytes = (bytes + 255) / 256 * 256;
    {
        std::lock_guard<std::mutex> g(mu);
        if (budget && in_use + bytes > budget)
            throw Error(CCDB_ERR_BUDGET, "device allocation of " + std::to_string(bytes) +
                                             " bytes exceeds the HBM budget");
        in_use += bytes;
    }
    // stream-ordered from the context's own pool: allocation and release are
    // ordered with the context's own work and never wait on another context's
    // stream (the device's shared pool may reuse a block another stream freed by
    // making this stream wait for that one), so fits of other contexts keep
    // running through them
    void* p = nullptr;
    cudaError_t e = cudaMallocFromPoolAsync(&p, bytes, pool, stream);
    if (e != cudaSuccess) {
        std::lock_guard<std::mutex> g(mu);
        in_use -= bytes;
        check_cuda(e, "cudaMallocFromPoolAsync");
    }
    std::lock_guard<std::mutex> g(mu);
    sizes[p] = bytes;
    return p;
}

void Context::release(void* p) {
    if (!p) return;
    cudaFreeAsync(p, stream);
    std::lock_guard<std::mutex> g(mu);
    auto it = sizes.find(p);
    if (it != sizes.end()) {
        in_use -= it->second;
        sizes.erase(it);
    }
}

void Context::make_results() {
    if (cudaHostAlloc(reinterpret_cast<void**>(&results), 2 * sizeof(double2) * kResults, cudaHostAllocMapped) != cudaSuccess) {
        cudaGetLastError();
        results = nullptr;  // fits copy their results back instead
        return;
    }
    for (int i = kResults - 1; i >= 0; --i) free_results.push_back(i);
}

int Context::take_result() {
    std::lock_guard<std::mutex> g(mu);
    if (free_results.empty()) return -1;
    const int slot = free_results.back();
    free_results.pop_back();
    return slot;
}

void Context::give_result(int slot) {
    if (slot < 0) return;
    std::lock_guard<std::mutex> g(mu);
    free_results.push_back(slot);
}

cudaError_t Context::wait() {
    if (!blocking_wait) return cudaStreamSynchronize(stream);
    cudaError_t e = cudaEventRecord(ev_wait, stream);
    return e == cudaSuccess ? cudaEventSynchronize(ev_wait) : e;
}

template <typename T>
T* upload(Context* c, const T* h, size_t n, cudaStream_t s) {
    T* d = static_cast<T*>(c->alloc(sizeof(T) * (n ? n : 1)));
    if (n && h) check_cuda(cudaMemcpyAsync(d, h, sizeof(T) * n, cudaMemcpyHostToDevice, s), "upload");
    return d;
}

int64_t Matrix::entries(int j) const {
    if (fmt[j] == F_DENSE || fmt[j] == F_INTERCEPT) return K;
    return col_start[j + 1] - col_start[j];
}

int64_t Matrix::total_entries() const {
    int64_t total = 0;
    for (int j = 0; j < J; ++j) total += entries(j);
    return total;
}

Matrix::~Matrix() {
    for (void* p : {(void*)d_col_ptr, (void*)d_rows, (void*)d_val_ptr, (void*)d_vals, (void*)d_fmt,
                    (void*)d_row_ptr, (void*)d_csr_col, (void*)d_csr_val})
        ctx->release(p);
}

// Row-major copy for computeXBeta: per row, entries in increasing column order
// (dense-like columns included), built once, on the device from the uploaded
// columns (csr_device.cu); a matrix with a row longer than kCsrDeviceMaxRow
// entries is built on the host threads instead (csr_host.cpp, the same layout).
void Matrix::ensure_csr(cudaStream_t s) {
    if (d_row_ptr) return;
    const int64_t total = total_entries();
    CsrDeviceArgs a{K, J, d_col_ptr, d_rows, d_val_ptr, d_vals, d_fmt, val_start.back() > 0};
    auto* counts = static_cast<int32_t*>(ctx->alloc(sizeof(int32_t) * (size_t)std::max<int64_t>(K, 1)));
    auto* cursor = static_cast<int64_t*>(ctx->alloc(sizeof(int64_t) * (size_t)std::max<int64_t>(K, 1)));
    auto* tiles = static_cast<int64_t*>(ctx->alloc(sizeof(int64_t) * (size_t)std::max<int64_t>(csr_device_tiles(K), 1)));
    auto* d_max = static_cast<int32_t*>(ctx->alloc(sizeof(int32_t)));
    d_row_ptr = static_cast<int64_t*>(ctx->alloc(sizeof(int64_t) * (size_t)(K + 1)));
    int32_t longest = 0;
    check_cuda(csr_device_count(a, counts, tiles, d_row_ptr, cursor, d_max, s), "row counts");
    check_cuda(cudaMemcpyAsync(&longest, d_max, sizeof(int32_t), cudaMemcpyDeviceToHost, s), "longest row");
    check_cuda(ctx->wait(), "row counts");
    if (longest <= kCsrDeviceMaxRow) {
        d_csr_col = static_cast<int32_t*>(ctx->alloc(sizeof(int32_t) * (size_t)std::max<int64_t>(total, 1)));
        d_csr_val = static_cast<double*>(ctx->alloc(sizeof(double) * (size_t)std::max<int64_t>(total, 1)));
        check_cuda(csr_device_fill(a, d_row_ptr, cursor, d_csr_col, d_csr_val, s), "row-major fill");
    } else {
        ctx->release(d_row_ptr);
        const HostCsr h = build_csr(K, J, col_start.data(), rows_h.data(), val_start.data(), vals_h.data(),
                                    fmt.data(), (int)std::max(1u, std::thread::hardware_concurrency()));
        d_row_ptr = upload(ctx, h.row_ptr.data(), h.row_ptr.size(), s);
        d_csr_col = upload(ctx, h.col.data(), h.col.size(), s);
        d_csr_val = upload(ctx, h.val.data(), h.val.size(), s);
    }
    ctx->release(counts);
    ctx->release(cursor);
    ctx->release(tiles);
    ctx->release(d_max);
    check_cuda(ctx->wait(), "row-major copy");
}

// ------------------------------------------------------------------ Fit

Fit::~Fit() {
    for (void* p : {(void*)row, (void*)y, (void*)beta, (void*)hdelta, (void*)xjy, (void*)ptype,
                    (void*)pvar, (void*)st, (void*)grid_bar, (void*)red, (void*)xb_tmp, (void*)w,
                    (void*)gh_parts, (void*)gh_out, (void*)d_batch_cols, (void*)d_batch_out})
        ctx->release(p);
    ctx->give_result(result_slot);
    release_schedule();
    release_window();
    release_batch_window();
    if (group_engine()) cox_release();
}

void Fit::release_schedule() {
    if (!sched) return;
    for (void* p : {(void*)sched->segs, (void*)sched->cta_seg, (void*)sched->tasks,
                    (void*)sched->level_need, (void*)sched->level_done, (void*)sched->col_arrive,
                    (void*)sched->partials})
        ctx->release(p);
    sched.reset();
}

IndepParams Fit::params() const {
    IndepParams P{};
    P.col_ptr = m->d_col_ptr;
    P.rows = m->d_rows;
    P.val_ptr = m->d_val_ptr;
    P.vals = m->d_vals;
    P.fmt = m->d_fmt;
    P.K = K;
    P.J = J;
    P.model = model;
    P.row = row;
    P.y = y;
    P.beta = beta;
    P.hdelta = hdelta;
    P.xjy = xjy;
    P.ptype = ptype;
    P.pvar = pvar;
    P.red = red;
    P.grid_bar = grid_bar;
    P.st = st;
    P.ll_fixed = ll_fixed;
    P.wait_limit_ns = wait_limit_ns;
    if (sched) {
        P.segs = sched->segs;
        P.cta_seg = sched->cta_seg;
        P.tasks = sched->tasks;
        P.n_levels = sched->host.n_levels;
        P.level_done = sched->level_done;
        P.level_need = sched->level_need;
        P.col_arrive = sched->col_arrive;
        P.partials = sched->partials;
    }
    return P;
}

// ModelSpecifics::setWeights + computeFixedTermsInLogLikelihood + computeXjY
// (ModelSpecifics.hpp:427-484, 570-587, 486-524).  Independent rows: the
// N-weights equal the row weights (observationCount = 1).
void Fit::apply_weights() {
    if (group_engine()) {
        cox_apply_weights();
        return;
    }
    std::vector<double> wh(K, 1.0);
    if (weighted) wh = w_h;
    check_cuda(cudaMemcpyAsync(w, wh.data(), sizeof(double) * K, cudaMemcpyHostToDevice, stream),
               "weights");
    check_cuda(launch_xjy(m->d_col_ptr, m->d_rows, m->d_val_ptr, m->d_vals, m->d_fmt, y,
                          weighted ? w : nullptr, K, J, xjy, stream),
               "xjy");
    ++launches;
    ll_fixed = 0.0;
    if (model == M_POISSON) {
        // PoissonRegression::logLikeFixedTermsContrib (ModelSpecifics.h:1596-1601) sums
        // -log(c) for c = 2..y in order; the running table reproduces each sum exactly.
        std::vector<double> table(1, 0.0);
        for (int64_t i = 0; i < K; ++i) {
            const int yi = (int)y_h[i];
            while ((int)table.size() <= yi) {
                const int c = (int)table.size();
                table.push_back(c >= 2 ? table.back() + -std::log((double)c) : 0.0);
            }
            const double t = yi >= 2 ? table[yi] : 0.0;
            ll_fixed += weighted ? t * wh[i] : t;
        }
    }
    check_cuda(ctx->wait(), "weights sync");
    valid_weights = true;
    suff_known = false;
}

// CyclicCoordinateDescent::computeXBeta (.cpp:1452-1470).
void Fit::compute_xbeta() {
    int nonzero = 0, only = -1;
    for (int j = 0; j < J; ++j)
        if (beta_h[j] != 0.0) {
            ++nonzero;
            only = j;
        }
    if (nonzero == 0) {
        check_cuda(cudaMemsetAsync(xb_tmp, 0, sizeof(double) * K, stream), "xb zero");
    } else if (nonzero == 1 && (m->fmt[only] == F_DENSE || m->fmt[only] == F_INTERCEPT)) {
        // one dense-like column (the offset of a cold start): xBeta = 0 + b*x
        const double* v = (m->fmt[only] == F_DENSE) ? m->d_vals + m->val_start[only] : nullptr;
        check_cuda(launch_xbeta_dense(v, beta_h[only], K, xb_tmp, stream), "xbeta");
        ++launches;
    } else {
        const_cast<Matrix*>(m)->ensure_csr(stream);
        check_cuda(launch_xbeta_csr(m->d_row_ptr, m->d_csr_col, m->csr_values(), beta, K, xb_tmp, stream),
                   "xbeta");
        ++launches;
    }
    xb_pending = true;
    xb_known = true;
    suff_known = false;
}

// computeRemainingStatistics (ModelSpecifics.hpp:1588-1633).
void Fit::remaining_statistics() {
    if (group_engine()) {
        cox_remaining();
        return;
    }
    const double null_denom = (model == M_LOGISTIC) ? 1.0 : 0.0;
    check_cuda(launch_remaining_stats(row, xb_pending ? xb_tmp : nullptr, w, K, null_denom, stream),
               "remaining statistics");
    ++launches;
    xb_pending = false;
    suff_known = true;
}

void Fit::check_lazy() {
    if (!xb_known) compute_xbeta();
    if (!valid_weights) apply_weights();
    if (!suff_known) remaining_statistics();
}

void Fit::upload_beta() {
    check_cuda(cudaMemcpyAsync(beta, beta_h.data(), sizeof(double) * J, cudaMemcpyHostToDevice, stream),
               "beta upload");
}

void Fit::download_beta() {
    check_cuda(cudaMemcpyAsync(beta_h.data(), beta, sizeof(double) * J, cudaMemcpyDeviceToHost, stream),
               "beta download");
    check_cuda(ctx->wait(), "beta sync");
}

void Fit::ensure_schedule() {
    if (sched && sched->fixed == fixed) return;
    release_schedule();
    int bps = 0;
    check_cuda(indep_sweep_occupancy(model, &bps), "occupancy");
    if (bps < 1) throw Error(CCDB_ERR_CUDA, "sweep kernel does not fit on an SM");
    ScheduleParams sp;
    sp.n_cta = ctx->n_sm * std::min(bps, 1);
    if (ctx->max_ctas > 0) sp.n_cta = std::min(sp.n_cta, ctx->max_ctas);
    // columns up to cta_max entries run on one CTA; longer ones split over CTAs
    sp.warps_per_cta = indep_threads() / 32;
    std::vector<int64_t> entries(J);
    for (int j = 0; j < J; ++j) entries[j] = m->entries(j);
    auto s = std::make_unique<DevSchedule>();
    s->fixed = fixed;
    s->host = build_schedule(K, J, m->col_start.data(), m->rows_h.data(), m->fmt.data(),
                             fixed.data(), nullptr, K, entries.data(), sp);
    if (s->host.max_split_per_seg > indep_max_split())
        throw Error(CCDB_ERR_UNSUPPORTED, "too many split columns on one level");
    s->segs = upload(ctx, s->host.segs.data(), s->host.segs.size(), stream);
    s->cta_seg = upload(ctx, s->host.cta_seg.data(), s->host.cta_seg.size(), stream);
    s->tasks = upload(ctx, s->host.tasks.data(), s->host.tasks.size(), stream);
    s->level_need = upload(ctx, s->host.level_need.data(), s->host.level_need.size(), stream);
    s->level_done = static_cast<unsigned*>(ctx->alloc(sizeof(unsigned) * std::max(1, s->host.n_levels)));
    s->col_arrive = static_cast<unsigned*>(ctx->alloc(sizeof(unsigned) * std::max(1, J)));
    s->partials = static_cast<double2*>(ctx->alloc(sizeof(double2) * std::max(1, s->host.n_partials)));
    check_cuda(ctx->wait(), "schedule upload");
    sched = std::move(s);
}

// Objective terms {LL num, LL den, gradient objective, log prior} of the
// current state, reduced in a fixed order.
void Fit::objective_terms(double* out4) {
    check_lazy();
    if (group_engine()) {
        cox_objective_terms(out4);
        return;
    }
    const int nb = ctx->n_sm;
    IndepParams P = params();
    check_cuda(launch_indep_objective(P, nb, stream), "objective");
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
        t[3] += parts[2 * c + 1].y;
    }
    for (int i = 0; i < 4; ++i) out4[i] = t[i];
}

double Fit::log_likelihood() {
    double t[4];
    objective_terms(t);
    return (t[0] - t[1]) + ll_fixed;
}

double Fit::objective(int conv) {
    double t[4];
    objective_terms(t);
    const double ll = (t[0] - t[1]) + ll_fixed;
    if (conv == C_GRADIENT) return t[2];
    if (conv == C_MITTAL) return ll;
    return ll + t[3];
}

void Fit::gradient_hessian(int j, double* g, double* h) {
    check_lazy();
    if (group_engine()) {
        const int32_t col = j;
        double2 r;
        cox_gh_batch(&col, 1, &r);
        *g = r.x;
        *h = r.y;
        return;
    }
    IndepParams P = params();
    int launched = 0;
    // into the fit's word of pinned memory, where it has one: no copy back
    double2* const slot = ctx->result(result_slot);
    check_cuda(launch_indep_gh(P, j, m->entries(j), gh_parts, kGhParts, slot ? slot : gh_out, &launched, stream), "gh");
    launches += launched;
    double2 r;
    if (!slot) check_cuda(cudaMemcpyAsync(&r, gh_out, sizeof(double2), cudaMemcpyDeviceToHost, stream), "gh copy");
    check_cuda(ctx->wait(), "gh sync");
    if (slot) r = *slot;
    *g = r.x;
    *h = r.y;
}

void Fit::update_xbeta(int j, double delta) {
    check_lazy();
    beta_h[j] += delta;
    if (group_engine() || m->entries(j) == 0)  // else the update's kernel writes it
        check_cuda(cudaMemcpyAsync(beta + j, &beta_h[j], sizeof(double), cudaMemcpyHostToDevice, stream),
                   "beta j");
    if (group_engine()) {
        cox_update(j, delta);
        check_cuda(ctx->wait(), "update sync");
        return;
    }
    IndepParams P = params();
    check_cuda(launch_indep_update(P, j, m->fmt[j], m->entries(j), delta, beta_h[j], stream), "update");
    launches += m->entries(j) > 0 ? 1 : 0;
    check_cuda(ctx->wait(), "update sync");
}

// findMode (CyclicCoordinateDescent.cpp:909-1216), CCD algorithm.
void Fit::find_mode_once(const ccdb_mode_args& a, double bound, int* flag, int* iters,
                         double* obj, float* ms) {
    if (!valid_weights || touched_y) {
        apply_weights();
        touched_y = false;
    }
    if (!xb_known) compute_xbeta();
    if (!suff_known) remaining_statistics();
    std::vector<double> hd(J, bound);  // resetBounds
    check_cuda(cudaMemcpyAsync(hdelta, hd.data(), sizeof(double) * J, cudaMemcpyHostToDevice, stream),
               "bounds");
    if (a.algorithm == CCDB_ALGORITHM_MM) {
        auto t0 = std::chrono::steady_clock::now();
        nz_known = false;  // the MM cycle moves every coordinate at once
        find_mode_mm(a, flag, iters, obj);
        *ms = std::chrono::duration<float, std::milli>(std::chrono::steady_clock::now() - t0).count();
        return;
    }
    if (a.per_coordinate) {
        // the reference's call pattern: one host round trip per coordinate
        double last = objective(a.convergence_type);
        int iteration = 0;
        bool done = false;
        auto t0 = std::chrono::steady_clock::now();
        while (!done) {
            for (int j = 0; j < J; ++j) {
                if (fixed[j]) continue;
                double g, h;
                gradient_hessian(j, &g, &h);
                double delta = newton_prior_delta(g, h, beta_h[j], ptype_h[j], pvar_h[j]);
                delta = apply_bounds(delta, hd[j]);
                if (delta != 0.0) {
                    update_xbeta(j, delta);
                    ++nz_steps;
                }
            }
            ++iteration;
            const double cur = objective(a.convergence_type);
            double conv;
            bool ill = false;
            if (cur != cur) {
                conv = 0.0;
                ill = true;
            } else {
                conv = std::fabs(cur - last) / (std::fabs(cur) + 1.0);
            }
            last = cur;
            if (a.tolerance > 0 && conv < a.tolerance) {
                *flag = ill ? R_ILLCONDITIONED : R_SUCCESS;
                done = true;
            } else if (iteration == a.max_iterations) {
                *flag = R_MAX_ITERATIONS;
                done = true;
            }
        }
        *iters = iteration;
        *obj = last;
        *ms = std::chrono::duration<float, std::milli>(std::chrono::steady_clock::now() - t0).count();
        check_cuda(cudaMemcpyAsync(hdelta, hd.data(), sizeof(double) * J, cudaMemcpyHostToDevice, stream),
                   "bounds");
        return;
    }
    if (group_engine() && a.strategy != CCDB_SWEEP_SPECULATIVE) {
        find_mode_group_window(a, flag, iters, obj, ms);
        return;
    }
    if (!group_engine() && a.strategy != CCDB_SWEEP_SPECULATIVE && a.strategy != CCDB_SWEEP_GRID_LEVELS) {
        find_mode_window(a, flag, iters, obj, ms);
        return;
    }
    if (group_engine() || use_speculative(a)) {
        auto t0 = std::chrono::steady_clock::now();
        find_mode_batched(a, bound, flag, iters, obj);
        *ms = std::chrono::duration<float, std::milli>(std::chrono::steady_clock::now() - t0).count();
        return;
    }
    ensure_schedule();
    if (sched->host.n_levels == 0) {
        // every coordinate is fixed: each cycle changes nothing, so the first
        // convergence check sees conv = 0 (findMode with an empty cycle)
        *obj = objective(a.convergence_type);
        *flag = (*obj != *obj) ? R_ILLCONDITIONED
                : (a.tolerance > 0 ? R_SUCCESS : (a.max_iterations == 1 ? R_MAX_ITERATIONS : R_SUCCESS));
        *iters = 1;
        *ms = 0.f;
        return;
    }
    DevStatus zero{};
    zero.flag = R_FAIL;
    check_cuda(cudaMemcpyAsync(st, &zero, sizeof(zero), cudaMemcpyHostToDevice, stream), "status");
    check_cuda(cudaMemsetAsync(sched->level_done, 0, sizeof(unsigned) * std::max(1, sched->host.n_levels), stream), "reset");
    check_cuda(cudaMemsetAsync(sched->col_arrive, 0, sizeof(unsigned) * std::max(1, J), stream), "reset");
    check_cuda(cudaMemsetAsync(grid_bar, 0, sizeof(unsigned), stream), "reset");
    IndepParams P = params();
    P.conv = a.convergence_type;
    P.tol = a.tolerance;
    P.max_iter = a.max_iterations;
    // CCDB_TRACE_FILE=<path>: dump per-segment timestamps of the first sweep
    // together with the schedule (profiling aid; off by default)
    const char* trace_path = std::getenv("CCDB_TRACE_FILE");
    unsigned long long* d_trace = nullptr;
    const size_t n_seg = sched->host.segs.size();
    if (trace_path) {
        d_trace = static_cast<unsigned long long*>(ctx->alloc(sizeof(unsigned long long) * 5 * n_seg));
        check_cuda(cudaMemsetAsync(d_trace, 0, sizeof(unsigned long long) * 5 * n_seg, stream), "trace");
        P.trace = d_trace;
        P.trace2 = d_trace + 3 * n_seg;
    }
    check_cuda(cudaEventRecord(ctx->fev[0], stream), "event");
    check_cuda(launch_indep_sweep(P, sched->host.n_cta, stream), "sweep launch");
    ++launches;
    check_cuda(cudaEventRecord(ctx->fev[1], stream), "event");
    // the host waits for the sweep before it queues the copy back: a device-to-host
    // copy queued behind a long kernel held up the copies of other contexts'
    // streams, so fits served side by side finished together with the longest one
    check_cuda(ctx->wait(), "sweep");
    DevStatus out{};
    check_cuda(cudaMemcpyAsync(&out, st, sizeof(out), cudaMemcpyDeviceToHost, stream), "status");
    check_cuda(ctx->wait(), "sweep");
    check_cuda(cudaEventElapsedTime(ms, ctx->fev[0], ctx->fev[1]), "elapsed");
    if (d_trace) {
        std::vector<unsigned long long> tr(5 * n_seg);
        check_cuda(cudaMemcpy(tr.data(), d_trace, sizeof(unsigned long long) * 5 * n_seg,
                              cudaMemcpyDeviceToHost), "trace copy");
        ctx->release(d_trace);
        if (FILE* fh = std::fopen(trace_path, "wb")) {
            const int64_t ns = (int64_t)n_seg, nt = (int64_t)sched->host.tasks.size();
            std::fwrite(&ns, sizeof(ns), 1, fh);
            std::fwrite(&nt, sizeof(nt), 1, fh);
            std::fwrite(sched->host.segs.data(), sizeof(Seg), n_seg, fh);
            std::fwrite(sched->host.cta_seg.data(), sizeof(int64_t), sched->host.cta_seg.size(), fh);
            std::fwrite(sched->host.tasks.data(), sizeof(Task), nt, fh);
            std::fwrite(tr.data(), sizeof(unsigned long long), tr.size(), fh);
            std::fclose(fh);
        }
    }
    if (out.error != E_NONE)
        throw Error(CCDB_ERR_TIMEOUT, "device wait timed out (code " + std::to_string(out.error) +
                                          " at " + std::to_string(out.error_where) + ")");
    *flag = out.flag;
    *iters = out.iterations;
    *obj = out.objective;
    nz_known = false;  // the grid-wide sweep does not count them
    beta_dirty_host = true;
}

// findMode with speculative batches: the gradients of a run of consecutive
// coordinates are computed together against the same state; walking them in
// order, every zero step leaves the state untouched, so the next coordinate's
// gradient is exactly what a sequential sweep would compute.  At the first
// nonzero step the update is applied and the batch restarts after it.  The
// visiting order and every step are those of the sequential cycle
// (CyclicCoordinateDescent.cpp:1008-1021); only the wasted speculative
// gradients cost extra.  Batches shrink after a restart and grow while steps
// stay zero.
void Fit::find_mode_batched(const ccdb_mode_args& a, double bound, int* flag, int* iters, double* obj) {
    std::vector<double> hd(J, bound);
    std::vector<int32_t> cols;
    for (int j = 0; j < J; ++j)
        if (!fixed[j]) cols.push_back(j);
    const int n_active = (int)cols.size();
    std::vector<double2> gh(kBatchMax);
    double last = objective(a.convergence_type);
    int iteration = 0;
    bool done = false;
    while (!done) {
        int pos = 0, batch = 32;
        while (pos < n_active) {
            const int nb = std::min(batch, n_active - pos);
            gh_batch(cols.data() + pos, nb, gh.data());
            int advanced = nb;
            for (int i = 0; i < nb; ++i) {
                const int j = cols[pos + i];
                double delta = newton_prior_delta(gh[i].x, gh[i].y, beta_h[j], ptype_h[j], pvar_h[j]);
                delta = apply_bounds(delta, hd[j]);
                if (delta != 0.0) {
                    beta_h[j] += delta;
                    apply_step(j, delta);
                    ++nz_steps;
                    advanced = i + 1;
                    break;
                }
            }
            pos += advanced;
            batch = (advanced == nb) ? std::min(2 * batch, (int)kBatchMax) : 32;
        }
        upload_beta();
        ++iteration;
        const double cur = objective(a.convergence_type);
        double conv;
        bool ill = false;
        if (cur != cur) {
            conv = 0.0;
            ill = true;
        } else {
            conv = std::fabs(cur - last) / (std::fabs(cur) + 1.0);
        }
        last = cur;
        if (a.tolerance > 0 && conv < a.tolerance) {
            *flag = ill ? R_ILLCONDITIONED : R_SUCCESS;
            done = true;
        } else if (iteration == a.max_iterations) {
            *flag = R_MAX_ITERATIONS;
            done = true;
        }
    }
    check_cuda(cudaMemcpyAsync(hdelta, hd.data(), sizeof(double) * J, cudaMemcpyHostToDevice, stream),
               "bounds");
    check_cuda(ctx->wait(), "batched sync");
    *iters = iteration;
    *obj = last;
}

void Fit::gh_batch(const int32_t* cols, int n, double2* out) {
    if (group_engine()) {
        cox_gh_batch(cols, n, out);
        return;
    }
    if (!d_batch_cols) {
        d_batch_cols = static_cast<int32_t*>(ctx->alloc(sizeof(int32_t) * kBatchMax));
        d_batch_out = static_cast<double2*>(ctx->alloc(sizeof(double2) * kBatchMax));
    }
    check_cuda(cudaMemcpyAsync(d_batch_cols, cols, sizeof(int32_t) * n, cudaMemcpyHostToDevice, stream),
               "batch cols");
    IndepParams P = params();
    check_cuda(launch_indep_gh_batch(P, d_batch_cols, n, d_batch_out, stream), "gh batch");
    ++launches;
    check_cuda(cudaMemcpyAsync(out, d_batch_out, sizeof(double2) * n, cudaMemcpyDeviceToHost, stream),
               "gh copy");
    check_cuda(ctx->wait(), "gh sync");
}

void Fit::apply_step(int j, double delta) {
    if (group_engine()) {
        cox_update(j, delta);
        return;
    }
    IndepParams P = params();
    check_cuda(launch_indep_update(P, j, m->fmt[j], m->entries(j), delta, beta_h[j], stream), "update");
    launches += m->entries(j) > 0 ? 1 : 0;
}

// The host-driven speculative batches (one round trip per batch of gradients
// and per nonzero step) run only when asked for; every default path of the
// independent-row models is the windowed sweep.
bool Fit::use_speculative(const ccdb_mode_args& a) const { return a.strategy == CCDB_SWEEP_SPECULATIVE; }

// CTAs of the windowed sweep: as many as leave each warp about one entry per
// lane, and enough of them for the rows.  More CTAs shorten a round's gather and
// update until a column's share of entries fits one pass of a warp; after that
// each doubling only adds messages to the exchange.  Milliseconds per L1 fit on
// 1, 2, 4, 8, 16 CTAs (300 columns of m entries, K rows): K = 1,000, m = 20:
// 0.149 0.166 0.156 0.159 0.178; K = 3,000, m = 60: 1.09 0.93 0.84 0.85 0.94;
// K = 10,000, m = 200: 5.3 4.0 3.0 2.62 2.77; K = 30,000, m = 600: 20 12 11 7.8
// 6.9; K = 100,000, m = 200: 6.6 3.7 2.3 1.51 1.35.
int Fit::window_ctas() {
    if (ctx->window_cluster < 0) {
        int c = 0;
        check_cuda(window_limits(&c, &ctx->window_smem), "cluster occupancy");
        ctx->window_cluster = c;
    }
    if (ctx->window_cluster < 1) throw Error(CCDB_ERR_CUDA, "the sweep kernel does not fit on an SM");
    int64_t total = 0, active = 0;
    for (int j = 0; j < J; ++j)
        if (!fixed[j]) {
            total += m->entries(j);
            ++active;
        }
    const int64_t mean = total / std::max<int64_t>(active, 1);
    int c = 16;
    if (K <= 1024 && mean <= 64) c = 1;
    else if (K <= 4096 && mean <= 128) c = 4;
    else if (K <= 32768 && mean <= 256) c = 8;
    c = std::min(c, ctx->window_cluster);
    while (ctx->max_ctas > 0 && c > ctx->max_ctas && c > 1) c /= 2;
    return c;
}

void Fit::release_window() {
    if (!window) return;
    ctx->release(window->mem);
    window.reset();
}

// The memory of a plan, and its two parts that the host has made.  Those of a small
// plan are at the front and go up in one copy: a call of few columns had spent 8 us
// on an allocation a part and two copies.  (A copy from pageable memory has read it
// when the call returns.)
void Fit::place_window(size_t bytes, PlanPart a, PlanPart b) {
    window->mem = ctx->alloc(bytes);
    char* const d = static_cast<char*>(window->mem);
    const size_t front = b.at + b.bytes;
    if (a.at == 0 && front <= 65536) {
        std::vector<char> host(front);
        std::memcpy(host.data(), a.host, a.bytes);
        std::memcpy(host.data() + b.at, b.host, b.bytes);
        check_cuda(cudaMemcpyAsync(d, host.data(), front, cudaMemcpyHostToDevice, stream), "sweep plan upload");
        return;
    }
    check_cuda(cudaMemcpyAsync(d + a.at, a.host, a.bytes, cudaMemcpyHostToDevice, stream), "sweep plan upload");
    check_cuda(cudaMemcpyAsync(d + b.at, b.host, b.bytes, cudaMemcpyHostToDevice, stream), "sweep plan upload");
}

void Fit::ensure_window(int ctas) {
    if (window && window->ctas == ctas && window->fixed == fixed) return;
    release_window();
    const WindowPlan plan = build_window_plan(K, J, m->col_start.data(), m->rows_h.data(), m->val_start.data(),
                                              m->fmt.data(), fixed.data(), ctas);
    window.reset(new DevWindow());  // owned by the fit from here on, complete or not
    window->ctas = 0;               // not a plan to reuse until it is complete
    const size_t n = plan.cols.size();
    for (const WinCol& c : plan.cols) window->any_vals |= (c.flags & 2) != 0;
    const bool share = !window_share_fits((K + ctas - 1) / ctas, window->any_vals, ctx->window_smem);
    const size_t col_bytes = sizeof(WinCol) * n, slice_bytes = sizeof(WinSlice) * plan.slices.size();
    Parts p;
    const size_t at_cols = p.add(col_bytes), at_slices = p.add(slice_bytes), at_scal = p.add(sizeof(WinScal) * n),
                 at_bh = p.add(sizeof(double2) * n);
    place_window(p.bytes, {at_cols, col_bytes, plan.cols.data()}, {at_slices, slice_bytes, plan.slices.data()});
    char* const d = static_cast<char*>(window->mem);
    window->cols = reinterpret_cast<WinCol*>(d + at_cols);
    window->slices = reinterpret_cast<WinSlice*>(d + at_slices);
    window->scal = reinterpret_cast<WinScal*>(d + at_scal);
    window->bh = reinterpret_cast<double2*>(d + at_bh);
    window->share = share ? xb_tmp : nullptr;  // free during a sweep: no xBeta is pending
    window->n_active = (int32_t)n;
    window->fixed = fixed;
    window->ctas = ctas;
}

int64_t Fit::batch_mean() const {
    return batch_mean_entries(J, offset_col0, [&](int j) { return m->entries(j); });
}

// The batched fits' plan: every column but an offset one, whole on one CTA.
void Fit::ensure_batch_window() {
    if (batch_window) return;
    const BatchTeam t = batch_team(batch_mean());
    std::vector<uint8_t> skip(J, 0);
    if (offset_col0) skip[0] = 1;
    const WindowPlan plan = build_window_plan(K, J, m->col_start.data(), m->rows_h.data(), m->val_start.data(),
                                              m->fmt.data(), skip.data(), 1, t.short_entries, t.long_entries);
    std::vector<int32_t> longs;
    std::unique_ptr<DevWindow> w(new DevWindow());
    for (size_t q = 0; q < plan.cols.size(); ++q) {
        const WinCol& c = plan.cols[q];
        if (c.flags & 8) longs.push_back((int32_t)q);
        w->any_vals |= (c.flags & 2) != 0;
        w->entries += c.n;
    }
    w->n_active = (int32_t)plan.cols.size();
    w->n_long = (int32_t)longs.size();
    w->team = t.warps;
    release_batch_window();
    batch_window = std::move(w);  // owned by the fit from here on
    try {
        batch_window->cols = upload(ctx, plan.cols.data(), plan.cols.size(), stream);
        batch_window->slices = upload(ctx, plan.slices.data(), plan.slices.size(), stream);
        batch_window->longs = upload(ctx, longs.data(), longs.size(), stream);
    } catch (...) {
        release_batch_window();
        throw;
    }
}

void Fit::release_batch_window() {
    if (!batch_window) return;
    for (void* p : {(void*)batch_window->cols, (void*)batch_window->slices, (void*)batch_window->longs}) ctx->release(p);
    batch_window.reset();
}

RoundTrace::RoundTrace(Context* c) : ctx(c), path(std::getenv("CCDB_TRACE_FILE")) {
    if (!path) return;
    d = static_cast<RoundStamp*>(ctx->alloc(sizeof(RoundStamp) * kTracedRounds));
    check_cuda(cudaMemsetAsync(d, 0, sizeof(RoundStamp) * kTracedRounds, ctx->stream), "trace");
}

void RoundTrace::write() {
    if (!d) return;
    std::vector<RoundStamp> s(kTracedRounds);
    check_cuda(cudaMemcpyAsync(s.data(), d, sizeof(RoundStamp) * s.size(), cudaMemcpyDeviceToHost, ctx->stream), "trace copy");
    check_cuda(ctx->wait(), "trace copy");
    if (FILE* fh = std::fopen(path, "wb")) {
        std::fwrite(s.data(), sizeof(RoundStamp), s.size(), fh);
        std::fclose(fh);
    }
}

void Fit::find_mode_window(const ccdb_mode_args& a, int* flag, int* iters, double* obj, float* ms) {
    if (std::find(fixed.begin(), fixed.end(), uint8_t(0)) == fixed.end()) {
        // every coordinate is fixed: each cycle changes nothing, so the first
        // convergence check sees conv = 0 (findMode with an empty cycle)
        *obj = objective(a.convergence_type);
        *flag = (*obj != *obj) ? R_ILLCONDITIONED
                : (a.tolerance > 0 ? R_SUCCESS : (a.max_iterations == 1 ? R_MAX_ITERATIONS : R_SUCCESS));
        *iters = 1;
        *ms = 0.f;
        return;
    }
    ensure_window(window_ctas());
    DevStatus zero{};
    zero.flag = R_FAIL;
    check_cuda(cudaMemcpyAsync(st, &zero, sizeof(zero), cudaMemcpyHostToDevice, stream), "status");
    WindowParams R{};
    R.P = params();
    R.P.conv = a.convergence_type;
    R.P.tol = a.tolerance;
    R.P.max_iter = a.max_iterations;
    R.cols = window->cols;
    R.slices = window->slices;
    R.scal = window->scal;
    R.bh = window->bh;
    R.share = window->share;
    R.n_active = window->n_active;
    R.weighted = weighted ? 1 : 0;
    R.any_vals = window->any_vals ? 1 : 0;
    R.cluster = window->ctas;
    RoundTrace trace(ctx);
    R.trace = trace.d;
    check_cuda(cudaEventRecord(ctx->fev[0], stream), "event");
    check_cuda((trace.d ? launch_window_sweep_traced : launch_window_sweep)(R, ctx->window_smem, stream), "sweep launch");
    ++launches;
    check_cuda(cudaEventRecord(ctx->fev[1], stream), "event");
    // the host waits for the sweep before it queues the copy back: a device-to-host
    // copy queued behind a long kernel held up the copies of other contexts'
    // streams, so fits served side by side finished together with the longest one
    check_cuda(ctx->wait(), "sweep");
    DevStatus out{};
    check_cuda(cudaMemcpyAsync(&out, st, sizeof(out), cudaMemcpyDeviceToHost, stream), "status");
    check_cuda(ctx->wait(), "sweep");
    check_cuda(cudaEventElapsedTime(ms, ctx->fev[0], ctx->fev[1]), "elapsed");
    trace.write();
    if (out.error != E_NONE)
        throw Error(CCDB_ERR_TIMEOUT, "device wait timed out (code " + std::to_string(out.error) +
                                          " at " + std::to_string(out.error_where) + ")");
    *flag = out.flag;
    *iters = out.iterations;
    *obj = out.objective;
    nz_steps += (int64_t)out.nonzero_steps;
    beta_dirty_host = true;
}

void Fit::find_mode(const ccdb_mode_args& a, double* beta_inout, ccdb_fit_result* res) {
    if (!a.prior_type || !a.prior_var) throw Error(CCDB_ERR_INVALID, "prior arrays are required");
    ptype_h.assign(a.prior_type, a.prior_type + J);
    pvar_h.assign(a.prior_var, a.prior_var + J);
    for (int j = 0; j < J; ++j)
        if (ptype_h[j] < 0 || ptype_h[j] > 2) throw Error(CCDB_ERR_UNSUPPORTED, "prior type");
    check_cuda(cudaMemcpyAsync(ptype, ptype_h.data(), sizeof(int32_t) * J, cudaMemcpyHostToDevice, stream), "prior");
    check_cuda(cudaMemcpyAsync(pvar, pvar_h.data(), sizeof(double) * J, cudaMemcpyHostToDevice, stream), "prior");
    if (a.convergence_type < C_GRADIENT || a.convergence_type > C_MITTAL)
        throw Error(CCDB_ERR_UNSUPPORTED, "convergence type");
    if (a.algorithm != CCDB_ALGORITHM_CCD && a.algorithm != CCDB_ALGORITHM_MM)
        throw Error(CCDB_ERR_UNSUPPORTED, "algorithm");
    if (a.algorithm == CCDB_ALGORITHM_MM && !group_engine())
        throw Error(CCDB_ERR_UNSUPPORTED,
                    model == M_POISSON ? "Not model-specific" : "the MM algorithm needs stratified data");
    if (a.fixed)  // setFixedBeta for every column; the offset stays fixed
        for (int j = 0; j < J; ++j) fixed[j] = (a.fixed[j] != 0 || (offset_col0 && j == 0)) ? 1 : 0;
    bool any_laplace = false;
    for (int j = 0; j < J; ++j) any_laplace |= (ptype_h[j] == 1);
    const bool swindle = a.use_kkt_swindle && any_laplace;
    if (beta_inout) {
        for (int j = 0; j < J; ++j) beta_h[j] = beta_inout[j];
        upload_beta();
        xb_known = false;
        suff_known = false;
    }
    int active = 0;
    for (int j = 0; j < J; ++j) active += fixed[j] ? 0 : 1;
    const int64_t launches0 = launches;
    nz_steps = 0;
    nz_known = true;
    check_cuda(cudaEventRecord(ctx->fev[2], stream), "event");
    double bound = a.initial_bound;
    int count = 0, flag = R_FAIL, sweeps_total = 0;
    double obj = 0.0, secs = 0.0;
    int64_t updates = 0;
    for (;;) {
        float ms = 0.f;
        // A swindle whose active set stays empty runs no findMode and leaves the
        // count as it was: the reference then reports its lastIterationCount from
        // the previous fit (CyclicCoordinateDescent.cpp:696-709, :1209).
        int iters = -1;
        if (swindle) kkt_swindle(a, bound, &flag, &iters, &obj, &ms);
        else find_mode_once(a, bound, &flag, &iters, &obj, &ms);
        secs += ms * 1e-3;
        if (iters >= 0) {
            last_iterations = iters;
            updates += (int64_t)iters * active;
            sweeps_total += iters;
        }
        ++count;
        if (beta_dirty_host) {
            download_beta();
            beta_dirty_host = false;
        }
        if (flag == R_ILLCONDITIONED && count < a.max_bound_count) {
            bound /= 10.0;  // resetBeta (.cpp:256-264)
            for (int j = offset_col0 ? 1 : 0; j < J; ++j) beta_h[j] = 0.0;
            upload_beta();
            compute_xbeta();
            suff_known = false;
        } else {
            break;
        }
    }
    if (beta_inout)
        for (int j = 0; j < J; ++j) beta_inout[j] = beta_h[j];
    const double ll = log_likelihood();
    check_cuda(cudaEventRecord(ctx->fev[3], stream), "event");
    check_cuda(cudaEventSynchronize(ctx->fev[3]), "event sync");
    float call_ms = 0.f;
    check_cuda(cudaEventElapsedTime(&call_ms, ctx->fev[2], ctx->fev[3]), "elapsed");
    if (res) {
        res->return_flag = flag;
        res->iterations = last_iterations;
        res->objective = obj;
        res->log_likelihood = ll;
        res->coordinate_updates = updates;
        res->device_seconds = call_ms * 1e-3;
        res->kernel_seconds = secs;
        res->kernel_launches = launches - launches0;
        res->attempts = count;
        res->sweeps_total = sweeps_total;
        res->nonzero_steps = nz_known ? nz_steps : -1;
    }
}

}  // namespace ccdb

// ====================================================================== C ABI
using namespace ccdb;

struct ccdb_context : Context {};
struct ccdb_matrix : Matrix {};
struct ccdb_fit : Fit {};

namespace {

template <typename F>
int guard(F&& f) {
    try {
        f();
        return CCDB_OK;
    } catch (const Error& e) {
        g_last_error = e.what();
        return e.code;
    } catch (const std::bad_alloc&) {
        g_last_error = "host allocation failed";
        return CCDB_ERR_INVALID;
    } catch (const std::exception& e) {
        g_last_error = e.what();
        return CCDB_ERR_INVALID;
    }
}

void require(bool ok, const char* msg) {
    if (!ok) throw Error(CCDB_ERR_INVALID, msg);
}

}  // namespace

extern "C" {

const char* ccdb_last_error(void) { return g_last_error.c_str(); }

int ccdb_context_create(int device, size_t hbm_budget_bytes, ccdb_context** out) {
    return guard([&] {
        require(out != nullptr, "out is NULL");
        int n = 0;
        check_cuda(cudaGetDeviceCount(&n), "cudaGetDeviceCount");
        require(device >= 0 && device < n, "no such CUDA device");
        check_cuda(cudaSetDevice(device), "cudaSetDevice");
        auto* c = new ccdb_context();
        c->device = device;
        c->budget = hbm_budget_bytes;
        check_cuda(cudaDeviceGetAttribute(&c->n_sm, cudaDevAttrMultiProcessorCount, device), "attr");
        int coop = 0;
        check_cuda(cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, device), "attr");
        if (!coop) {
            delete c;
            throw Error(CCDB_ERR_UNSUPPORTED, "device lacks cooperative launch");
        }
        check_cuda(cudaStreamCreateWithFlags(&c->stream, cudaStreamNonBlocking), "stream");
        cudaMemPoolProps props = {};
        props.allocType = cudaMemAllocationTypePinned;
        props.location.type = cudaMemLocationTypeDevice;
        props.location.id = device;
        check_cuda(cudaMemPoolCreate(&c->pool, &props), "memory pool");
        uint64_t keep = UINT64_MAX;  // freed blocks stay reserved for the next fit
        check_cuda(cudaMemPoolSetAttribute(c->pool, cudaMemPoolAttrReleaseThreshold, &keep), "memory pool");
        check_cuda(cudaEventCreate(&c->ev_a), "event");
        check_cuda(cudaEventCreate(&c->ev_b), "event");
        for (cudaEvent_t& e : c->fev) check_cuda(cudaEventCreate(&e), "event");
        c->make_results();
        *out = c;
    });
}

int ccdb_context_destroy(ccdb_context* ctx) {
    return guard([&] {
        if (!ctx) return;
        cudaSetDevice(ctx->device);
        cudaStreamSynchronize(ctx->stream);
        cudaEventDestroy(ctx->ev_a);
        cudaEventDestroy(ctx->ev_b);
        for (cudaEvent_t e : ctx->fev) cudaEventDestroy(e);
        if (ctx->ev_wait) cudaEventDestroy(ctx->ev_wait);
        if (ctx->results) cudaFreeHost(ctx->results);
        cudaStreamDestroy(ctx->stream);
        if (ctx->pool) cudaMemPoolDestroy(ctx->pool);
        delete ctx;
    });
}

int ccdb_context_set_blocking_wait(ccdb_context* ctx, int32_t on) {
    return guard([&] {
        require(ctx != nullptr, "NULL context");
        check_cuda(cudaSetDevice(ctx->device), "cudaSetDevice");
        check_cuda(cudaStreamSynchronize(ctx->stream), "sync");
        ctx->blocking_wait = on != 0;
        if (ctx->blocking_wait && !ctx->ev_wait)
            check_cuda(cudaEventCreateWithFlags(&ctx->ev_wait, cudaEventBlockingSync | cudaEventDisableTiming),
                       "event");
        // the context's timing events follow the setting
        for (cudaEvent_t* e : {&ctx->ev_a, &ctx->ev_b, &ctx->fev[0], &ctx->fev[1], &ctx->fev[2], &ctx->fev[3]}) {
            if (*e) check_cuda(cudaEventDestroy(*e), "event");
            check_cuda(cudaEventCreateWithFlags(e, ctx->event_flags()), "event");
        }
    });
}

int ccdb_context_sm_count(const ccdb_context* ctx, int32_t* n_sm) {
    return guard([&] {
        require(ctx && n_sm, "NULL argument");
        *n_sm = ctx->n_sm;
    });
}

int ccdb_context_set_max_ctas(ccdb_context* ctx, int32_t max_ctas) {
    return guard([&] {
        require(ctx != nullptr, "NULL context");
        require(max_ctas >= 0, "max_ctas must be >= 0");
        ctx->max_ctas = max_ctas;
    });
}

int ccdb_context_memory(const ccdb_context* ctx, size_t* bytes) {
    return guard([&] {
        require(ctx && bytes, "NULL argument");
        *bytes = ctx->in_use;
    });
}

// The CompressedDataMatrix contract every matrix is checked against before any
// device work (host only).
// The first of columns [0, n_cols) whose row ids are not ascending within
// [0, K), or n_cols: column ranges of about equal entry counts checked on
// host threads (the check is a memory-bound walk of the row ids, vectorised
// within a column), the lowest failing column kept -- the one a walk in
// column order would report.
static int32_t first_row_error(int64_t K, int32_t n_cols, const int64_t* col_start, const int32_t* rows) {
    auto bad = [&](int32_t j) {
        const int64_t b = col_start[j], e = col_start[j + 1];
        if (e <= b) return false;
        unsigned ok = (unsigned)(rows[b] >= 0) & (unsigned)((int64_t)rows[e - 1] < K);
        for (int64_t p = b + 1; p < e; ++p) ok &= (unsigned)(rows[p] > rows[p - 1]);
        return ok == 0u;
    };
    const int64_t total = n_cols > 0 ? col_start[n_cols] : 0;
    const int64_t per_thread = int64_t(1) << 21;
    const int T = (int)std::max<int64_t>(
        1, std::min<int64_t>({(int64_t)std::max(1u, std::thread::hardware_concurrency()), total / per_thread, 16}));
    if (T == 1) {
        for (int32_t j = 0; j < n_cols; ++j)
            if (bad(j)) return j;
        return n_cols;
    }
    std::vector<int32_t> lo(T + 1, n_cols), found(T, n_cols);
    lo[0] = 0;
    for (int32_t j = 0, t = 1; j < n_cols && t < T; ++j)
        if (col_start[j + 1] >= total * t / T) lo[t++] = j + 1;
    auto walk = [&](int t) {
        for (int32_t j = lo[t]; j < lo[t + 1]; ++j)
            if (bad(j)) {
                found[t] = j;
                return;
            }
    };
    std::vector<std::thread> pool;
    int started = 0;
    try {
        for (; started < T; ++started) pool.emplace_back(walk, started);
    } catch (const std::system_error&) {  // no more threads: this one walks the rest
        for (int t = started; t < T; ++t) walk(t);
    }
    for (auto& th : pool) th.join();
    return *std::min_element(found.begin(), found.end());
}

static void validate_matrix(int64_t K, int32_t J, const int64_t* col_start, const int32_t* rows,
                            const int64_t* val_start, const double* vals, const uint8_t* fmt) {
    require(col_start && val_start && fmt, "NULL argument");
    require(K > 0 && K < (int64_t(1) << 31) && J > 0, "bad dimensions");
    const int64_t nnz = col_start[J], nv = val_start[J];
    require(col_start[0] == 0 && val_start[0] == 0 && nnz >= 0 && nv >= 0, "bad offsets");
    require(nnz == 0 || rows, "rows is NULL");
    require(nv == 0 || vals, "vals is NULL");
    // offsets and formats column by column; the columns before the first bad
    // one have offsets within [0, nnz] and [0, nv], so their row ids can be read
    int32_t first_bad = J;
    const char* why = nullptr;
    for (int32_t j = 0; j < J && !why; ++j) {
        const int64_t nr = col_start[j + 1] - col_start[j], nvj = val_start[j + 1] - val_start[j];
        if (nr < 0 || nvj < 0 || col_start[j + 1] > nnz || val_start[j + 1] > nv) {
            why = "offsets must be non-decreasing";
        } else {
            switch (fmt[j]) {
            case F_DENSE: if (!(nr == 0 && nvj == K)) why = "DENSE column needs K values, no rows"; break;
            case F_INTERCEPT: if (!(nr == 0 && nvj == 0)) why = "INTERCEPT column takes no data"; break;
            case F_INDICATOR: if (nvj != 0) why = "INDICATOR column takes no values"; break;
            case F_SPARSE: if (nvj != nr) why = "SPARSE column needs one value per row"; break;
            default: why = "unknown column format";
            }
        }
        if (why) first_bad = j;
    }
    // a row-id error in an earlier column comes first, as in a walk in column order
    require(first_row_error(K, first_bad, col_start, rows) == first_bad, "row ids must be ascending and < K");
    require(why == nullptr, why ? why : "");
}

int ccdb_matrix_validate(int64_t K, int32_t J, const int64_t* col_start, const int32_t* rows,
                         const int64_t* val_start, const double* vals, const uint8_t* fmt) {
    return guard([&] { validate_matrix(K, J, col_start, rows, val_start, vals, fmt); });
}

int ccdb_matrix_create(ccdb_context* ctx, int64_t K, int32_t J, const int64_t* col_start,
                       const int32_t* rows, const int64_t* val_start, const double* vals,
                       const uint8_t* fmt, ccdb_matrix** out) {
    return guard([&] {
        require(ctx && out, "NULL argument");
        validate_matrix(K, J, col_start, rows, val_start, vals, fmt);
        check_cuda(cudaSetDevice(ctx->device), "cudaSetDevice");
        std::unique_ptr<ccdb_matrix> m(new ccdb_matrix());
        m->ctx = ctx;
        m->K = K;
        m->J = J;
        m->col_start.assign(col_start, col_start + J + 1);
        m->val_start.assign(val_start, val_start + J + 1);
        m->fmt.assign(fmt, fmt + J);
        const int64_t nnz = col_start[J], nv = val_start[J];
        m->rows_h.assign(rows, rows + nnz);
        m->vals_h.assign(vals, vals + nv);
        cudaStream_t s = ctx->stream;
        m->d_col_ptr = upload(ctx, col_start, J + 1, s);
        m->d_val_ptr = upload(ctx, val_start, J + 1, s);
        m->d_fmt = upload(ctx, fmt, J, s);
        m->d_rows = upload(ctx, rows, nnz, s);
        m->d_vals = upload(ctx, vals, nv, s);
        check_cuda(ctx->wait(), "matrix upload");
        *out = m.release();
    });
}

int ccdb_matrix_destroy(ccdb_matrix* m) {
    return guard([&] { delete m; });
}

int ccdb_matrix_row_major(ccdb_matrix* m, int64_t* row_ptr, int32_t* col, double* val) {
    return guard([&] {
        require(m && row_ptr && col && val, "NULL argument");
        check_cuda(cudaSetDevice(m->ctx->device), "cudaSetDevice");
        cudaStream_t s = m->ctx->stream;
        m->ensure_csr(s);
        int64_t total = 0;
        for (int j = 0; j < m->J; ++j) total += m->entries(j);
        check_cuda(cudaMemcpyAsync(row_ptr, m->d_row_ptr, sizeof(int64_t) * (size_t)(m->K + 1),
                                   cudaMemcpyDeviceToHost, s), "row offsets");
        if (total > 0) {
            check_cuda(cudaMemcpyAsync(col, m->d_csr_col, sizeof(int32_t) * (size_t)total, cudaMemcpyDeviceToHost, s),
                       "columns");
            check_cuda(cudaMemcpyAsync(val, m->d_csr_val, sizeof(double) * (size_t)total, cudaMemcpyDeviceToHost, s),
                       "values");
        }
        check_cuda(m->ctx->wait(), "row-major copy");
    });
}

int ccdb_fit_create(ccdb_context* ctx, const ccdb_matrix* m, const ccdb_fit_desc* d, ccdb_fit** out) {
    return guard([&] {
        require(ctx && m && d && out && d->y, "NULL argument");
        require(m->ctx == ctx, "matrix belongs to another context");
        if (d->model_type != M_LOGISTIC && d->model_type != M_POISSON && d->model_type != M_COX &&
            d->model_type != M_CLR && d->model_type != M_CPR)
            throw Error(CCDB_ERR_UNSUPPORTED, "model type not supported by this engine");
        if ((d->model_type == M_CLR || d->model_type == M_CPR) && !d->stratum)
            throw Error(CCDB_ERR_INVALID, "conditional models need stratum ids");
        if (d->model_type == M_COX && !d->time)
            throw Error(CCDB_ERR_INVALID, "Cox fits need survival times");
        if (d->precision != CCDB_PRECISION_FP64 &&
            !(d->precision == CCDB_PRECISION_MIXED &&
              (d->model_type == M_LOGISTIC || d->model_type == M_POISSON || d->model_type == M_COX)))
            throw Error(CCDB_ERR_UNSUPPORTED, "precision not supported for this model");
        check_cuda(cudaSetDevice(ctx->device), "cudaSetDevice");
        std::unique_ptr<ccdb_fit> f(new ccdb_fit());
        f->ctx = ctx;
        f->m = m;
        f->model = d->model_type;
        f->precision = d->precision;
        f->K = m->K;
        f->J = m->J;
        f->offset_col0 = d->offset_col0 != 0;
        f->stream = ctx->stream;
        f->y_h.assign(d->y, d->y + m->K);
        const int64_t K = m->K;
        const int J = m->J;
        if (d->time) f->time_h.assign(d->time, d->time + K);
        if (d->stratum) f->stratum_h.assign(d->stratum, d->stratum + K);
        else f->stratum_h.assign(K, 0);  // one stratum, as R's rep(1, n) for unstratified Cox
        const bool grp_engine = (f->model == M_COX || f->model == M_CLR || f->model == M_CPR);
        if (!grp_engine) f->row = static_cast<double2*>(ctx->alloc(sizeof(double2) * 2 * K));
        f->y = upload(ctx, d->y, K, f->stream);
        f->beta = static_cast<double*>(ctx->alloc(sizeof(double) * J));
        f->hdelta = static_cast<double*>(ctx->alloc(sizeof(double) * J));
        f->xjy = static_cast<double*>(ctx->alloc(sizeof(double) * J));
        f->ptype = static_cast<int32_t*>(ctx->alloc(sizeof(int32_t) * J));
        f->pvar = static_cast<double*>(ctx->alloc(sizeof(double) * J));
        f->st = static_cast<DevStatus*>(ctx->alloc(sizeof(DevStatus)));
        f->grid_bar = static_cast<unsigned*>(ctx->alloc(sizeof(unsigned)));
        f->red = static_cast<double2*>(ctx->alloc(sizeof(double2) * 4 * ctx->n_sm * 2));
        f->xb_tmp = static_cast<double*>(ctx->alloc(sizeof(double) * K));
        f->w = static_cast<double*>(ctx->alloc(sizeof(double) * K));
        f->gh_parts = static_cast<double2*>(ctx->alloc(sizeof(double2) * Fit::kGhParts));
        f->gh_out = static_cast<double2*>(ctx->alloc(sizeof(double2)));
        f->result_slot = ctx->take_result();
        // CyclicCoordinateDescent::init (.cpp:200-239)
        f->beta_h.assign(J, 0.0);
        f->fixed.assign(J, 0);
        f->ptype_h.assign(J, 0);
        f->pvar_h.assign(J, 1.0);
        if (f->offset_col0) {
            f->beta_h[0] = 1.0;
            f->fixed[0] = 1;
            f->xb_known = false;
        } else {
            f->xb_known = false;  // xBeta = 0: computed (zero-filled) on first use
        }
        f->upload_beta();
        if (grp_engine) f->cox_allocate();
        check_cuda(f->ctx->wait(), "fit upload");
        *out = f.release();
    });
}

int ccdb_fit_destroy(ccdb_fit* f) {
    return guard([&] { delete f; });
}

// Mixed precision of logistic and Poisson fits is implemented by the batched
// engine; their single-fit calls compute in FP64 only and refuse a mixed fit
// rather than ignore its setting.  Cox fits take it in every call.
static void require_fp64(const ccdb_fit* f) {
    if (f->precision != CCDB_PRECISION_FP64 && f->model != M_COX)
        throw Error(CCDB_ERR_UNSUPPORTED, "mixed precision serves batched fits (ccdb_batch_find_mode) only");
}

int ccdb_set_weights(ccdb_fit* f, const double* w) {
    return guard([&] {
        require(f != nullptr, "NULL fit");
        if (w) {
            f->w_h.assign(w, w + f->K);
            f->weighted = true;
        } else {
            f->w_h.clear();
            f->weighted = false;
        }
        f->valid_weights = false;
        f->suff_known = false;
    });
}

int ccdb_set_beta(ccdb_fit* f, const double* beta) {
    return guard([&] {
        require(f && beta, "NULL argument");
        f->beta_h.assign(beta, beta + f->J);
        f->upload_beta();
        f->xb_known = false;
        f->suff_known = false;
    });
}

int ccdb_compute_xbeta(ccdb_fit* f, const double* beta) {
    return guard([&] {
        require(f && beta, "NULL argument");
        require_fp64(f);
        f->beta_h.assign(beta, beta + f->J);
        f->upload_beta();
        f->compute_xbeta_transpose();  // the statistics stay stale until computeRemainingStatistics
    });
}

int ccdb_compute_gradient_hessian(ccdb_fit* f, int32_t j, double* g, double* h) {
    return guard([&] {
        require(f && g && h, "NULL argument");
        require_fp64(f);
        require(j >= 0 && j < f->J, "column out of range");
        f->gradient_hessian(j, g, h);
    });
}

int ccdb_update_xbeta(ccdb_fit* f, int32_t j, double delta) {
    return guard([&] {
        require(f != nullptr, "NULL fit");
        require_fp64(f);
        require(j >= 0 && j < f->J, "column out of range");
        f->update_xbeta(j, delta);
    });
}

int ccdb_compute_remaining_statistics(ccdb_fit* f) {
    return guard([&] {
        require(f != nullptr, "NULL fit");
        require_fp64(f);
        f->check_lazy();
        f->remaining_statistics();
        check_cuda(f->ctx->wait(), "sync");
    });
}

int ccdb_get_log_likelihood(ccdb_fit* f, double* ll) {
    return guard([&] {
        require(f && ll, "NULL argument");
        require_fp64(f);
        *ll = f->log_likelihood();
    });
}

int ccdb_get_xbeta(ccdb_fit* f, double* out) {
    return guard([&] {
        require(f && out, "NULL argument");
        require_fp64(f);
        f->check_lazy();
        f->copy_xbeta(out);
    });
}

int ccdb_get_gradient_objective(ccdb_fit* f, double* out) {
    return guard([&] {
        require(f && out, "NULL argument");
        require_fp64(f);
        double t[4];
        f->objective_terms(t);
        *out = t[2];
    });
}

int ccdb_fisher_information(ccdb_fit* f, const int32_t* indices, int32_t n, double* out) {
    return guard([&] {
        require(f != nullptr, "NULL fit");
        require(n >= 0, "negative column count");
        require(n == 0 || (indices && out), "NULL argument");
        require_fp64(f);
        for (int32_t i = 0; i < n; ++i) require(indices[i] >= 0 && indices[i] < f->J, "column out of range");
        if (f->weighted)
            throw Error(CCDB_ERR_UNSUPPORTED, "Weights are not yet implemented in Fisher Information calculations");
        f->fisher_information(indices, n, out);
    });
}

int ccdb_compute_mm_gradient_hessian(ccdb_fit* f, const uint8_t* fixed, double* gradient, double* hessian) {
    return guard([&] {
        require(f && gradient && hessian, "NULL argument");
        require_fp64(f);
        if (!f->group_engine())
            throw Error(CCDB_ERR_UNSUPPORTED, f->model == M_POISSON ? "Not model-specific"
                                                                    : "the MM algorithm needs stratified data");
        std::vector<double2> gh(f->J);
        f->mm_gradient_hessian(fixed, gh.data());
        for (int j = 0; j < f->J; ++j) {
            gradient[j] = gh[j].x;
            hessian[j] = gh[j].y;
        }
    });
}

int ccdb_get_predictive_log_likelihood(ccdb_fit* f, const double* weights, double* out) {
    return guard([&] {
        require(f && weights && out, "NULL argument");
        require_fp64(f);
        *out = f->predictive_log_likelihood(weights);
    });
}

int ccdb_get_predictive_estimates(ccdb_fit* f, const double* weights, double* y) {
    return guard([&] {
        require(f && y, "NULL argument");
        require_fp64(f);
        if (!weights) {
            f->predictive_estimates(y);
            return;
        }
        std::vector<double> p(f->K);
        f->predictive_estimates(p.data());
        for (int64_t k = 0; k < f->K; ++k)
            if (weights[k] != 0.0) y[k] = p[k];
    });
}

int ccdb_set_fixed(ccdb_fit* f, const uint8_t* fixed) {
    return guard([&] {
        require(f && fixed, "NULL argument");
        for (int j = 0; j < f->J; ++j) f->fixed[j] = (fixed[j] != 0 || (f->offset_col0 && j == 0)) ? 1 : 0;
    });
}

int ccdb_fit_set_wait_limit(ccdb_fit* f, int64_t nanoseconds) {
    return guard([&] {
        require(f != nullptr, "NULL fit");
        require(nanoseconds >= 0, "the wait limit must be >= 0");
        f->wait_limit_ns = nanoseconds ? nanoseconds : Fit::kDefaultWaitNs;
        f->xch_wait_ns = nanoseconds ? nanoseconds : Fit::kDefaultXchWaitNs;
    });
}

int ccdb_get_last_call_seconds(const ccdb_fit* f, double* seconds) {
    return guard([&] {
        require(f && seconds, "NULL argument");
        *seconds = f->last_call_seconds;
    });
}

int ccdb_get_beta(ccdb_fit* f, double* out) {
    return guard([&] {
        require(f && out, "NULL argument");
        std::copy(f->beta_h.begin(), f->beta_h.end(), out);
    });
}

int ccdb_find_mode(ccdb_fit* f, const ccdb_mode_args* args, double* beta_inout, ccdb_fit_result* res) {
    return guard([&] {
        require(f && args, "NULL argument");
        require_fp64(f);
        check_cuda(cudaSetDevice(f->ctx->device), "cudaSetDevice");
        f->find_mode(*args, beta_inout, res);
    });
}

int ccdb_fit_model(ccdb_context* ctx, int64_t K, int32_t J, const int64_t* col_start, const int32_t* rows,
                   const int64_t* val_start, const double* vals, const uint8_t* fmt,
                   const ccdb_fit_desc* desc, const double* weights, const ccdb_mode_args* args,
                   double* beta_out, ccdb_fit_result* result) {
    ccdb_matrix* m = nullptr;
    ccdb_fit* f = nullptr;
    if (!ctx) {
        g_last_error = "NULL context";
        return CCDB_ERR_INVALID;
    }
    if (cudaSetDevice(ctx->device) != cudaSuccess || cudaEventRecord(ctx->ev_a, ctx->stream) != cudaSuccess) {
        g_last_error = "cannot record on the context stream";
        return CCDB_ERR_CUDA;
    }
    int rc = ccdb_matrix_create(ctx, K, J, col_start, rows, val_start, vals, fmt, &m);
    if (rc == CCDB_OK) rc = ccdb_fit_create(ctx, m, desc, &f);
    if (rc == CCDB_OK && weights) rc = ccdb_set_weights(f, weights);
    if (rc == CCDB_OK) rc = ccdb_find_mode(f, args, nullptr, result);
    if (rc == CCDB_OK && beta_out) rc = ccdb_get_beta(f, beta_out);
    if (rc == CCDB_OK && result) {
        float ms = 0.f;
        if (cudaEventRecord(ctx->ev_b, ctx->stream) == cudaSuccess &&
            cudaEventSynchronize(ctx->ev_b) == cudaSuccess &&
            cudaEventElapsedTime(&ms, ctx->ev_a, ctx->ev_b) == cudaSuccess)
            result->device_seconds = ms * 1e-3;
    }
    std::string err = g_last_error;
    if (f) ccdb_fit_destroy(f);
    if (m) ccdb_matrix_destroy(m);
    g_last_error = err;
    return rc;
}

// Longest slice of a row-indexed column when C CTAs split the rows evenly.
static int64_t batch_max_slice(const Matrix* m, int64_t K, int C) {
    int64_t mx = 0;
    for (int j = 0; j < m->J; ++j) {
        if (m->fmt[j] != F_SPARSE && m->fmt[j] != F_INDICATOR) continue;
        const int32_t* r0 = m->rows_h.data() + m->col_start[j];
        const int32_t* r1 = m->rows_h.data() + m->col_start[j + 1];
        const int32_t* lo = r0;
        for (int r = 1; r <= C; ++r) {
            const int32_t* hi = (r == C) ? r1 : std::lower_bound(lo, r1, K * r / C);
            mx = std::max<int64_t>(mx, hi - lo);
            lo = hi;
        }
    }
    return mx;
}

// CTAs per group of the mixed engine.  The per-column critical path shrinks
// when a column's rows are split over more SMs (each gathers and updates only
// its slice), and the kernel's registers suffice without spills for the small
// stage (1024 entries per slice).  Take the smallest power of two that both
// fits every slice in the small stage and puts a CTA on every SM; at most 8.
static int batch_cluster_size(const Matrix* m, int64_t K, int n_groups, int n_sm) {
    for (int C = 1; C <= 8; C *= 2)
        if ((int64_t)n_groups * C >= n_sm && batch_max_slice(m, K, C) <= 1024) return C;
    for (int C = 1; C <= 8; C *= 2)
        if (batch_max_slice(m, K, C) <= 1024) return C;
    return 8;
}

// Whether the windowed engine serves a batch whose caller names no launch shape: it
// is the faster one, and its workspace is within the context's memory budget.
static bool batch_windowed(Context* ctx, const Fit* f, int n, int ctas, bool mixed, int spill) {
    if (!batch_prefers_window({mixed, !(spill & 2), f->K, f->batch_mean(), n, ctx->n_sm})) return false;
    const size_t J = f->J, K = f->K, state = (spill & 1 ? 8 : 0) + (spill & 2 ? (mixed ? 4 : 8) : 0);
    const size_t bytes = ctas * ((sizeof(WinScal) + sizeof(double2)) * J + state * K) + sizeof(double) * J * n +
                         (sizeof(WinCol) + sizeof(WinSlice) + sizeof(int32_t)) * J + 4096;
    std::lock_guard<std::mutex> g(ctx->mu);
    return !ctx->budget || ctx->in_use + bytes <= ctx->budget;
}

// The engine of a batch, and what its choice has found out.
struct BatchRoute {
    int32_t engine;
    bool any_vals = false;
    int ctas = 0, spill = 0;  // of the windowed engine
};

static BatchRoute batch_route(const Fit* f, const ccdb_batch_desc* b) {
    const bool mixed = f->precision == CCDB_PRECISION_MIXED;
    BatchRoute r{mixed ? CCDB_BATCH_LOCKSTEP : CCDB_BATCH_COLUMNS};
    for (int j = f->offset_col0 ? 1 : 0; j < f->J; ++j) r.any_vals |= f->m->fmt[j] == F_SPARSE || f->m->fmt[j] == F_DENSE;
    r.ctas = std::min(b->n_instances, f->ctx->n_sm);
    check_cuda(batch_window_spill(f->K, mixed, r.any_vals, &r.spill), "batch sweep");
    // a launch shape, and the trace of a column's phases, ask for the lockstep engine
    if (mixed && (b->group || b->cluster || std::getenv("CCDB_BATCH_TRACE_FILE"))) return r;
    if (batch_windowed(f->ctx, f, b->n_instances, r.ctas, mixed, r.spill)) r.engine = CCDB_BATCH_WINDOWED;
    return r;
}

int ccdb_batch_engine(ccdb_fit* f, const ccdb_batch_desc* b, int32_t* engine) {
    return guard([&] {
        require(f && b && engine && b->n_instances > 0, "NULL argument");
        if (f->model != M_LOGISTIC && f->model != M_POISSON)
            throw Error(CCDB_ERR_UNSUPPORTED, "batched fits: logistic and Poisson models");
        check_cuda(cudaSetDevice(f->ctx->device), "cudaSetDevice");
        *engine = batch_route(f, b).engine;
    });
}

int ccdb_batch_find_mode(ccdb_fit* f, const ccdb_batch_desc* b, const ccdb_mode_args* a, double* beta_out,
                         ccdb_batch_result* results, double* device_seconds) {
    return guard([&] {
        require(f && b && a && a->prior_type && b->variance && b->n_instances > 0, "NULL argument");
        if (f->model != M_LOGISTIC && f->model != M_POISSON)
            throw Error(CCDB_ERR_UNSUPPORTED, "batched fits support logistic and Poisson models");
        if (a->convergence_type < C_GRADIENT || a->convergence_type > C_MITTAL)
            throw Error(CCDB_ERR_UNSUPPORTED, "convergence type");
        Context* ctx = f->ctx;
        check_cuda(cudaSetDevice(ctx->device), "cudaSetDevice");
        const int n = b->n_instances;
        const int64_t K = f->K;
        const int J = f->J;
        const Matrix* m = f->m;
        cudaStream_t s = f->stream;
        std::vector<void*> owned;
        auto keep = [&](void* p) { owned.push_back(p); return p; };
        struct Release {
            Context* c;
            std::vector<void*>* v;
            ~Release() { for (void* p : *v) c->release(p); }
        } rel{ctx, &owned};
        BatchParams P{};
        P.col_ptr = m->d_col_ptr;
        P.rows = m->d_rows;
        P.val_ptr = m->d_val_ptr;
        P.vals = m->d_vals;
        P.fmt = m->d_fmt;
        P.K = K;
        P.J = J;
        P.model = f->model;
        P.n_inst = n;
        P.conv = a->convergence_type;
        P.max_iter = a->max_iterations;
        P.tol = a->tolerance;
        P.initial_bound = a->initial_bound;
        P.xch_wait_ns = f->xch_wait_ns;
        P.y = f->y;
        if (b->row_fold) P.row_fold = (const int32_t*)keep(upload(ctx, b->row_fold, (size_t)K, s));
        std::vector<int32_t> hold(n, -1);
        if (b->holdout) hold.assign(b->holdout, b->holdout + n);
        P.holdout = (const int32_t*)keep(upload(ctx, hold.data(), (size_t)n, s));
        P.variance = (const double*)keep(upload(ctx, b->variance, (size_t)n, s));
        P.ptype = (const int32_t*)keep(upload(ctx, a->prior_type, (size_t)J, s));
        if (f->offset_col0) {
            if (m->fmt[0] != F_DENSE) throw Error(CCDB_ERR_UNSUPPORTED, "offset column must be DENSE");
            P.offset_vals = m->d_vals + m->val_start[0];
        }
        if (f->model == M_POISSON) {  // fixed terms per instance (ModelSpecifics.h:1596-1601)
            std::vector<double> table(1, 0.0), fixed(n, 0.0);
            for (int i = 0; i < n; ++i) {
                double acc = 0.0;
                for (int64_t k = 0; k < K; ++k) {
                    const int yi = (int)f->y_h[k];
                    while ((int)table.size() <= yi) {
                        const int c = (int)table.size();
                        table.push_back(c >= 2 ? table.back() + -std::log((double)c) : 0.0);
                    }
                    const double t = yi >= 2 ? table[yi] : 0.0;
                    const double w = (b->row_fold && hold[i] >= 0 && b->row_fold[k] == hold[i]) ? 0.0 : 1.0;
                    acc += t * w;
                }
                fixed[i] = acc;
            }
            P.ll_fixed = (const double*)keep(upload(ctx, fixed.data(), (size_t)n, s));
        }
        const bool mixed = f->precision == CCDB_PRECISION_MIXED;
        // weakest priors first: they need the most sweeps, so they start in the first wave
        // (and, in mixed precision, instances of similar variance share a group)
        std::vector<int32_t> order(n);
        for (int i = 0; i < n; ++i) order[i] = i;
        std::stable_sort(order.begin(), order.end(),
                         [&](int32_t x, int32_t y) { return b->variance[x] > b->variance[y]; });
        P.order = (const int32_t*)keep(upload(ctx, order.data(), (size_t)n, s));
        P.results = (BatchResult*)keep(ctx->alloc(sizeof(BatchResult) * n));
        int G = 1, n_groups = n;
        // CCDB_BATCH_TRACE_FILE: per-column phase clocks of CTA 0 in one sweep
        // (CCDB_BATCH_TRACE_SWEEP, default 1) of the mixed lockstep engine, written as int64 [J][6]
        const char* trace_path = mixed ? std::getenv("CCDB_BATCH_TRACE_FILE") : nullptr;
        if (mixed && K > kKeyRowMask)
            throw Error(CCDB_ERR_UNSUPPORTED, "mixed batched fits: at most 16,777,215 rows");
        for (int i = 0; mixed && i < n; ++i)
            if (hold[i] >= kKeyNoFold)
                throw Error(CCDB_ERR_UNSUPPORTED, "mixed batched fits: held-out fold ids below 127");
        BatchWindowParams W{};
        const BatchRoute route = batch_route(f, b);
        const bool windowed = route.engine == CCDB_BATCH_WINDOWED;
        if (windowed) {
            f->ensure_batch_window();
            const DevWindow& w = *f->batch_window;
            W.cols = w.cols;
            W.slices = w.slices;
            W.longs = w.longs;
            W.n_active = w.n_active;
            W.n_long = w.n_long;
            W.entries = w.entries;
            W.any_vals = w.any_vals ? 1 : 0;
            W.mixed = mixed ? 1 : 0;
            W.team = w.team;
            W.ctas = route.ctas;
            const size_t cols = (size_t)W.ctas * std::max(W.n_active, 1);
            W.scal = (WinScal*)keep(ctx->alloc(sizeof(WinScal) * cols));
            W.bh = (double2*)keep(ctx->alloc(sizeof(double2) * cols));
            if (route.spill & 1) W.xbeta = (double*)keep(ctx->alloc(sizeof(double) * (size_t)K * W.ctas));
            if (route.spill & 2) W.share = (double*)keep(ctx->alloc((mixed ? 4 : 8) * (size_t)K * W.ctas));
            P.queue = (int32_t*)keep(ctx->alloc(sizeof(int32_t)));
            check_cuda(cudaMemsetAsync(P.queue, 0, sizeof(int32_t), s), "batch queue");
            W.beta_out = P.beta = (double*)keep(ctx->alloc(sizeof(double) * (size_t)J * n));
        } else if (mixed) {
            G = b->group ? b->group : batch_group_size(n, ctx->n_sm);
            if (G != 1 && G != 2 && G != 4) throw Error(CCDB_ERR_INVALID, "batch group must be 1, 2 or 4");
            n_groups = (n + G - 1) / G;
            P.group = G;
            // the lockstep engine reads each entry's fold with its row id (row | fold << 24)
            const int64_t nnz = m->col_start.back();
            int32_t* keys = (int32_t*)keep(ctx->alloc(sizeof(int32_t) * (size_t)std::max<int64_t>(nnz, 1)));
            check_cuda(launch_batch_keys(m->d_rows, nnz, P.row_fold, keys, s), "batch keys");
            P.keys = keys;
            // CTAs per group (a cluster splits each column's rows among its CTAs):
            // the caller's choice, else the tuner's
            int C = b->cluster ? b->cluster : batch_cluster_size(m, K, n_groups, ctx->n_sm);
            if (C < 1 || C > 16) throw Error(CCDB_ERR_INVALID, "batch cluster size must be 1..16");
            P.cluster = C;
            // per row-indexed column, where its rows cross the CTAs' row boundaries;
            // the stage capacity is the small variant when every slice fits it
            std::vector<int32_t> split((size_t)J * (C + 1), 0);
            int64_t max_slice = 0;
            for (int j = 0; j < J; ++j) {
                const int64_t cb = m->col_start[j], ce = m->col_start[j + 1];
                const int32_t* r0 = m->rows_h.data() + cb;
                const int32_t* r1 = m->rows_h.data() + ce;
                int32_t* sp = split.data() + (size_t)j * (C + 1);
                for (int r = 0; r <= C; ++r)
                    sp[r] = (r == C) ? (int32_t)(ce - cb) : (int32_t)(std::lower_bound(r0, r1, K * r / C) - r0);
                if (m->fmt[j] == F_SPARSE || m->fmt[j] == F_INDICATOR)
                    for (int r = 0; r < C; ++r) max_slice = std::max<int64_t>(max_slice, sp[r + 1] - sp[r]);
            }
            if (C > 1) P.split = (const int32_t*)keep(upload(ctx, split.data(), split.size(), s));
            P.stage_cap = max_slice <= 1024 ? 1024 : 3072;
            P.queue = (int32_t*)keep(ctx->alloc(sizeof(int32_t) * 2));
            P.abort = P.queue + 1;
            check_cuda(cudaMemsetAsync(P.queue, 0, sizeof(int32_t) * 2, s), "batch queue");
            P.xg = (double*)keep(ctx->alloc(sizeof(double) * (size_t)K * G * n_groups));
            P.beta_g = (double*)keep(ctx->alloc(sizeof(double) * (size_t)J * G * n_groups));
            P.hd_g = (double*)keep(ctx->alloc(sizeof(double) * (size_t)J * G * n_groups));
            P.xjy_g = (double*)keep(ctx->alloc(sizeof(double) * (size_t)J * G * n_groups));
        } else {
            P.row = (double2*)keep(ctx->alloc(sizeof(double2) * 2 * (size_t)K * n));
            P.beta = (double*)keep(ctx->alloc(sizeof(double) * (size_t)J * n));
            P.hdelta = (double*)keep(ctx->alloc(sizeof(double) * (size_t)J * n));
            P.xjy = (double*)keep(ctx->alloc(sizeof(double) * (size_t)J * n));
        }
        if (trace_path) {
            const char* sw = std::getenv("CCDB_BATCH_TRACE_SWEEP");
            P.trace_sweep = sw ? std::atoi(sw) : 1;
            P.trace = (long long*)keep(ctx->alloc(sizeof(long long) * 6 * (size_t)J));
            check_cuda(cudaMemsetAsync(P.trace, 0, sizeof(long long) * 6 * (size_t)J, s), "trace");
        }
        cudaEvent_t e0, e1;
        check_cuda(cudaEventCreate(&e0), "event");
        check_cuda(cudaEventCreate(&e1), "event");
        check_cuda(cudaEventRecord(e0, s), "event");
        W.P = P;
        if (windowed) check_cuda(launch_batch_window(W, s), "batch sweep");
        else if (mixed) check_cuda(launch_batch_mixed(P, s), "batch sweep (lockstep)");
        else check_cuda(launch_batch_sweep(P, s), "batch sweep (one column at a time)");
        check_cuda(cudaEventRecord(e1, s), "event");
        check_cuda(f->ctx->wait(), "batch sync");  // the sweep is done before a copy is queued behind it
        std::vector<BatchResult> res(n);
        check_cuda(cudaMemcpyAsync(res.data(), P.results, sizeof(BatchResult) * n, cudaMemcpyDeviceToHost, s),
                   "results");
        int32_t aborted = 0;
        if (P.abort)
            check_cuda(cudaMemcpyAsync(&aborted, P.abort, sizeof(int32_t), cudaMemcpyDeviceToHost, s), "abort word");
        std::vector<double> bg;
        if (beta_out && P.beta_g) {
            bg.resize((size_t)J * G * n_groups);
            check_cuda(cudaMemcpyAsync(bg.data(), P.beta_g, sizeof(double) * bg.size(), cudaMemcpyDeviceToHost, s),
                       "beta");
        } else if (beta_out) {
            check_cuda(cudaMemcpyAsync(beta_out, P.beta, sizeof(double) * (size_t)J * n, cudaMemcpyDeviceToHost, s),
                       "beta");
        }
        check_cuda(f->ctx->wait(), "batch sync");
        if (trace_path) {
            std::vector<long long> tr(6 * (size_t)J);
            check_cuda(cudaMemcpy(tr.data(), P.trace, sizeof(long long) * tr.size(), cudaMemcpyDeviceToHost),
                       "trace copy");
            if (FILE* fh = std::fopen(trace_path, "wb")) {
                std::fwrite(tr.data(), sizeof(long long), tr.size(), fh);
                std::fclose(fh);
            }
        }
        if (beta_out && P.beta_g)  // [group][J][G] -> [instance][J]
            for (int q = 0; q < n; ++q) {
                const int grp = q / G, gi = q % G, inst = order[q];
                for (int j = 0; j < J; ++j) beta_out[(size_t)inst * J + j] = bg[((size_t)grp * J + j) * G + gi];
            }
        float ms = 0.f;
        check_cuda(cudaEventElapsedTime(&ms, e0, e1), "elapsed");
        cudaEventDestroy(e0);
        cudaEventDestroy(e1);
        if (device_seconds) *device_seconds = ms * 1e-3;
        bool timed_out = aborted != 0;
        for (int i = 0; i < n; ++i) timed_out |= (res[i].flag == kBatchTimeoutFlag);
        if (timed_out)
            throw Error(CCDB_ERR_TIMEOUT, windowed ? "batched fits: a bounded wait for a copy ran out"
                                                   : "batched fits: a bounded wait for the other CTAs of a cluster ran out");
        if (results)
            for (int i = 0; i < n; ++i) {
                results[i].return_flag = res[i].flag;
                results[i].iterations = res[i].iterations;
                results[i].log_likelihood = res[i].loglik;
                results[i].objective = res[i].objective;
                results[i].predictive_loglik = res[i].pred_loglik;
                results[i].steps = res[i].steps;
                results[i].updates = res[i].updates;
                results[i].update_entries = res[i].update_entries;
                results[i].gradient_entries = res[i].sweep_entries;
            }
    });
}

int ccdb_sweep_levels(int64_t K, int32_t J, const int64_t* col_start, const int32_t* rows,
                      const uint8_t* fmt, const uint8_t* fixed, int32_t* level_out, int32_t* n_levels) {
    return guard([&] {
        require(col_start && fmt && level_out && n_levels && K > 0 && J > 0, "bad argument");
        std::vector<int64_t> entries(J);
        for (int j = 0; j < J; ++j)
            entries[j] = (fmt[j] == F_DENSE || fmt[j] == F_INTERCEPT) ? K : col_start[j + 1] - col_start[j];
        ScheduleParams sp;
        const Schedule s = build_schedule(K, J, col_start, rows, fmt, fixed, nullptr, K, entries.data(), sp);
        std::copy(s.level_of.begin(), s.level_of.end(), level_out);
        *n_levels = s.n_levels;
    });
}

}  // extern "C"
