// engine.h -- host-side objects behind the C ABI: a device context with an
// HBM budget, an immutable device CompressedDataMatrix, and per-fit state
// mirroring ModelSpecifics + CyclicCoordinateDescent.
#pragma once

#include <cstdint>
#include <map>
#include <memory>
#include <mutex>
#include <stdexcept>
#include <string>
#include <vector>

#include <cuda_runtime.h>

#include "../../include/ccdb.h"
#include "cox.h"
#include "group_window.h"
#include "indep.h"
#include "schedule.h"
#include "step.h"
#include "window_sweep.h"

namespace ccdb {

// A failure with its C ABI status code (CCDB_ERR_*), raised by host code and
// turned into the status at the ABI boundary.
struct Error : std::runtime_error {
    int code;
    Error(int c, const std::string& m) : std::runtime_error(m), code(c) {}
};

void check_cuda(cudaError_t e, const char* what);

struct Context {
    int device = 0;
    int n_sm = 0;
    int max_ctas = 0;  // persistent sweep grids: at most this many CTAs (0: n_sm)
    int window_cluster = -1;     // largest resident cluster of the windowed sweep (-1: not queried)
    int64_t window_smem = 0;     // its shared memory per CTA
    GroupWindowLimits group_window{-1, {0, 0, 0}};  // of the group models' sweep (cluster -1: not queried)
    size_t budget = 0;
    size_t in_use = 0;
    cudaStream_t stream = nullptr;
    cudaMemPool_t pool = nullptr;  // this context's own stream-ordered pool
    std::mutex mu;
    std::map<void*, size_t> sizes;
    cudaEvent_t ev_a = nullptr, ev_b = nullptr;  // around a one-call fit
    // timing events of this context's fits (their calls are serialised on its
    // stream): [0], [1] around the sweep launches, [2], [3] around a whole
    // findMode.  Made once: creating and destroying events per fit waited on
    // other streams' work while they ran
    cudaEvent_t fev[4] = {nullptr, nullptr, nullptr, nullptr};
    // host waits: spin (default) or sleep until the device signals (blocking_wait),
    // for processes that run many contexts' calls at once (serving slots)
    bool blocking_wait = false;
    cudaEvent_t ev_wait = nullptr;

    // pinned words that kernels write a fit's per-call results to, with room behind
    // each for the call's column; a fit holds one
    static constexpr int kResults = 1024;
    double2* results = nullptr;
    std::vector<int> free_results;
    void make_results();
    int take_result();  // -1: none left
    void give_result(int slot);
    double2* result(int slot) const { return slot < 0 ? nullptr : results + 2 * slot; }

    void* alloc(size_t bytes);
    void release(void* p);
    // wait for everything queued on the context's stream
    cudaError_t wait();
    // event flags of this context's timing events
    unsigned event_flags() const { return blocking_wait ? cudaEventBlockingSync : cudaEventDefault; }
};

struct Matrix {
    Context* ctx = nullptr;
    int64_t K = 0;
    int32_t J = 0;
    std::vector<int64_t> col_start, val_start;
    std::vector<uint8_t> fmt;
    std::vector<int32_t> rows_h;
    std::vector<double> vals_h;
    int64_t* d_col_ptr = nullptr;
    int32_t* d_rows = nullptr;
    int64_t* d_val_ptr = nullptr;
    double* d_vals = nullptr;
    uint8_t* d_fmt = nullptr;
    // row-major copy, built on first need (computeXBeta with nonzero beta)
    int64_t* d_row_ptr = nullptr;
    int32_t* d_csr_col = nullptr;
    double* d_csr_val = nullptr;

    int64_t entries(int j) const;
    int64_t total_entries() const;
    // values of the row-major copy; NULL where every one is 1
    const double* csr_values() const { return val_start.back() > 0 ? d_csr_val : nullptr; }
    void ensure_csr(cudaStream_t s);
    ~Matrix();
};

struct DevSchedule {
    std::vector<uint8_t> fixed;
    Schedule host;
    Seg* segs = nullptr;
    int64_t* cta_seg = nullptr;
    Task* tasks = nullptr;
    int32_t* level_need = nullptr;
    unsigned* level_done = nullptr;
    unsigned* col_arrive = nullptr;
    double2* partials = nullptr;
};

// Parts of one allocation, each on a boundary of 256 bytes.
struct Parts {
    size_t bytes = 0;
    size_t add(size_t n) {
        const size_t at = bytes;
        bytes += (n + 255) / 256 * 256;
        return at;
    }
};

// The plan of a windowed sweep on the device, and its per-position state.
struct DevWindow {
    std::vector<uint8_t> fixed;
    int ctas = 0;
    int32_t n_active = 0;
    bool any_vals = false;
    // batched fits: the long columns' positions, the entries of all
    int32_t n_long = 0, team = 1;
    int64_t entries = 0;
    int32_t* longs = nullptr;
    void* mem = nullptr;  // what holds all of the following
    WinCol* cols = nullptr;
    WinSlice* slices = nullptr;
    WinScal* scal = nullptr;
    double2* bh = nullptr;
    double* share = nullptr;  // K (the fit's xb_tmp), where a CTA's rows do not fit its shared memory
    // group models: the CTAs' cuts, of the grouping that was current, and the grid
    // form's exchange buffers
    bool cluster = false;
    int64_t grouping = -1;
    int64_t most_rows = 0, most_groups = 0;
    bool any_long = false;  // a column may be too long for one warp
    bool meet = false;      // a stratum spans CTAs
    int32_t chain = 1;
    GroupCut* cuts = nullptr;
    double2* part = nullptr;
    double* tails = nullptr;
    double2* heads = nullptr;
};

// CCDB_TRACE_FILE=<path>: the first rounds of a windowed sweep, written to the file
// as they are (profiling aid; off by default).
struct RoundTrace {
    Context* ctx;
    const char* path;
    RoundStamp* d = nullptr;
    explicit RoundTrace(Context* c);
    ~RoundTrace() { ctx->release(d); }
    void write();
};

// Device tables of the Breslow Cox engine (cox.cu).
struct CoxDev {
    int64_t N = 0;  // risk-set groups
    int epoch = 0;  // scan epoch (status words are never reset)
    double2* xbe = nullptr;
    int32_t* grp = nullptr;
    int32_t* rstrat = nullptr;
    double *denom = nullptr, *D = nullptr, *S1 = nullptr, *S2 = nullptr, *nEv = nullptr;
    uint8_t *gfirst = nullptr, *glast = nullptr;
    int64_t* grow = nullptr;
    unsigned* tickets = nullptr;
    int* status = nullptr;
    void* tails = nullptr;
    int32_t* batch_cols = nullptr;
    double2* batch_out = nullptr;
    int64_t grouping = 0;  // changes when the rows are regrouped
    // Cox: runs of groups that end with events or with their stratum, the grouping
    // that the windowed sweep works on (block_rows); NB of them
    int64_t NB = 0, blocks = -1;  // the grouping that they belong to
    void* block_mem = nullptr;    // what holds them all
    int32_t *blk = nullptr, *bgrp = nullptr;  // block of each row, first group of each block
    double *bden = nullptr, *bD = nullptr, *bS1 = nullptr, *bS2 = nullptr, *bnev = nullptr;
    uint8_t *bfirst = nullptr, *blast = nullptr;
    int64_t* brow = nullptr;
};

int64_t cox_group_rows(const std::vector<int32_t>& pid0, const std::vector<double>& time,
                       const std::vector<double>& y, const double* weights, std::vector<int32_t>& grp);

struct Fit {
    static constexpr int kGhParts = 1024;
    static constexpr int kBatchMax = 1024;  // columns per speculative gradient batch
    Context* ctx = nullptr;
    const Matrix* m = nullptr;
    int model = 0, precision = 0;
    int64_t K = 0;
    int32_t J = 0;
    bool offset_col0 = false;
    cudaStream_t stream = nullptr;
    // bounds on device-side waits (ccdb_fit_set_wait_limit): the grid sweep's level,
    // column and grid waits and the windowed sweeps' exchanges; the batch engines'
    // cluster exchange and copies
    static constexpr long long kDefaultWaitNs = 20LL * 1000 * 1000 * 1000;
    static constexpr long long kDefaultXchWaitNs = 2LL * 1000 * 1000 * 1000;
    long long wait_limit_ns = kDefaultWaitNs;
    long long xch_wait_ns = kDefaultXchWaitNs;

    // device state
    double2* row = nullptr;
    double* y = nullptr;
    double* beta = nullptr;
    double* hdelta = nullptr;
    double* xjy = nullptr;
    int32_t* ptype = nullptr;
    double* pvar = nullptr;
    DevStatus* st = nullptr;
    unsigned* grid_bar = nullptr;
    double2* red = nullptr;
    double* xb_tmp = nullptr;
    double* w = nullptr;
    double2* gh_parts = nullptr;
    double2* gh_out = nullptr;
    int result_slot = -1;
    int64_t launches = 0;                        // engine kernels launched so far
    double last_call_seconds = 0.0;              // device time of the last fisher_information passes
    int last_iterations = 0;                     // getIterationCount: the last findMode's cycles
    int64_t nz_steps = 0;                        // nonzero coordinate steps of the current find_mode
    bool nz_known = true;                        // every path of the call counted them
    std::unique_ptr<DevSchedule> sched;
    CoxDev cox;

    // host mirror and lazy flags (CyclicCoordinateDescent.h:152-166)
    std::vector<double> y_h, w_h, beta_h, pvar_h, time_h;
    std::vector<int64_t> stratum_h;
    std::vector<int32_t> pid0_h;
    std::vector<int64_t> cox_grow_h;    // first row of each stratum (grouped) or block (Cox), then K
    std::vector<int32_t> cox_bstrat_h;  // Cox: stratum of each block
    struct {  // Cox: the group of each row (N: none); stratum, first row and weighted events of each group
        std::vector<int32_t> row_group, stratum;
        std::vector<int64_t> first_row;
        std::vector<double> events;
    } cox_groups_h;
    std::vector<int32_t> ptype_h;
    std::vector<uint8_t> fixed;
    bool weighted = false;
    bool valid_weights = false, xb_known = false, suff_known = false, touched_y = true;
    bool xb_pending = false, beta_dirty_host = false;
    double ll_fixed = 0.0;

    ~Fit();
    IndepParams params() const;
    void release_schedule();
    // the schedule of the grid-wide level sweep (one CTA per SM, levels ordered by
    // global counters)
    void ensure_schedule();
    void apply_weights();
    void compute_xbeta();
    void compute_xbeta_transpose();  // the MM cycle's product (ModelSpecifics::computeXBeta(beta))
    void remaining_statistics();
    void check_lazy();
    void upload_beta();
    void download_beta();
    void objective_terms(double* out4);
    double log_likelihood();
    double objective(int conv);
    void gradient_hessian(int j, double* g, double* h);
    void update_xbeta(int j, double delta);
    void find_mode_once(const ccdb_mode_args& a, double bound, int* flag, int* iters, double* obj,
                        float* ms);
    void find_mode(const ccdb_mode_args& a, double* beta_inout, ccdb_fit_result* res);
    // speculative batched sweeps (models without a fused sweep kernel)
    void find_mode_batched(const ccdb_mode_args& a, double bound, int* flag, int* iters, double* obj);
    // (g, h) of several columns against the current state; nonzero step of one column
    void gh_batch(const int32_t* cols, int n, double2* out);
    void apply_step(int j, double delta);
    bool use_speculative(const ccdb_mode_args& a) const;
    // the windowed sweep (window.cu) on window_ctas() CTAs, and its plan
    int window_ctas();
    void ensure_window(int ctas);
    void release_window();
    struct PlanPart {
        size_t at, bytes;
        const void* host;
    };
    void place_window(size_t bytes, PlanPart a, PlanPart b);
    int64_t batch_mean() const;  // entries of the columns that a batch steps (batch_route.h)
    void ensure_batch_window();
    void release_batch_window();
    void find_mode_window(const ccdb_mode_args& a, int* flag, int* iters, double* obj, float* ms);
    std::unique_ptr<DevWindow> window;
    std::unique_ptr<DevWindow> batch_window;
    int32_t* d_batch_cols = nullptr;  // independent-row models
    double2* d_batch_out = nullptr;
    bool is_cox() const { return model == M_COX; }
    bool is_grouped() const { return model == M_CLR || model == M_CPR; }
    // models served by the group engine (cox.cu) rather than the fused sweep
    bool group_engine() const { return is_cox() || is_grouped(); }
    // Cox engine (cox_host.cu)
    CoxParams cox_params() const;
    void cox_allocate();
    void cox_release();
    void cox_apply_weights();
    void cox_scans();
    void cox_remaining(bool rows_done = false);
    void cox_objective_terms(double* out4);
    void cox_gh_batch(const int32_t* cols, int n, double2* out);
    void cox_update(int j, double delta);
    // one findMode of the group engine in one launch (group_window.cu), and its plan
    void ensure_group_window(int ctas, bool cluster);
    void ensure_cox_blocks();
    void find_mode_group_window(const ccdb_mode_args& a, int* flag, int* iters, double* obj, float* ms);
    // mode-finding variants (modes_host.cu): the MM cycle, the KKT swindle, and
    // the MM all-coordinate (g, h) into out[J] (fixed may be nullptr)
    void find_mode_mm(const ccdb_mode_args& a, int* flag, int* iters, double* obj);
    void kkt_swindle(const ccdb_mode_args& a, double bound, int* flag, int* iters, double* obj, float* ms);
    void mm_gradient_hessian(const uint8_t* fixed_flags, double2* out);
    // post-fit calls (postfit_host.cu)
    void fisher_information(const int32_t* idx, int n, double* out);
    double predictive_log_likelihood(const double* weights);
    double predictive_sum(const double* weights);
    void predictive_estimates(double* out);
    void copy_xbeta(double* out);
    void rows_to_host(struct PredictParams P, double* out);
};

}  // namespace ccdb
