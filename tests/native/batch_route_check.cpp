// batch_route_check.cpp -- host test of the batch engine's dispatch
// (ccd_b200/csrc/batch_route.h), run by tests/test_batch_route.py.
#include <cstdio>

#include "batch_route.h"

using namespace ccdb;

static int failures = 0;
static void check(bool ok, const char* what) {
    if (ok) return;
    std::printf("failed: %s\n", what);
    ++failures;
}

// the mean of `covariates` columns of `each` entries behind an intercept, and an
// offset before it
static int64_t mean(bool offset, int64_t K, int covariates, int64_t each) {
    const int first = offset ? 2 : 1;
    return batch_mean_entries(first + covariates, offset, [&](int j) { return j < first ? K : each; });
}

static void means() {
    check(mean(false, 50000, 300, 20) == 20, "the intercept is left out");
    check(mean(true, 50000, 300, 20) == 20, "an offset beside it too");
    check(batch_team(mean(true, 50000, 300, 20)).warps == 1, "short columns behind an offset take one warp");
    check(mean(true, 100000, 100, 20) <= kBatchWindowMean, "and the windowed engine");
    check(mean(true, 100000, 0, 0) == 100000, "an intercept alone");
    check(batch_mean_entries(3, false, [](int j) { return j == 0 ? 1000 : 900; }) == 900, "dense covariates count");
    check(batch_mean_entries(1, true, [](int) { return 7; }) == 0, "an offset alone");
}

// (fits, rows, mean) on 148 SMs where one engine was measured at least 5 % faster
static void routes() {
    struct {
        bool mixed, shared;
        int64_t K;
        int n;
        int64_t mean;
        bool window;
    } const at[] = {
        {true, true, 40000, 4, 450, true},      {true, true, 40000, 4, 560, false},
        {true, true, 40000, 60, 620, true},     {true, true, 40000, 148, 400, true},
        {true, true, 40000, 250, 620, true},    {true, true, 40000, 600, 350, true},
        {true, true, 40000, 1000, 200, true},   {true, true, 40000, 1000, 450, false},
        {true, false, 100000, 4, 300, true},    {true, false, 100000, 4, 400, false},
        {true, false, 100000, 60, 500, true},   {true, false, 100000, 80, 620, false},
        {true, false, 100000, 148, 300, true},  {true, false, 100000, 148, 400, false},
        {true, false, 100000, 200, 500, true},  {true, false, 100000, 300, 300, true},
        {true, false, 100000, 300, 500, false}, {true, false, 100000, 450, 350, false},
        {true, false, 100000, 600, 200, true},  {true, false, 100000, 600, 350, false},
        {true, false, 100000, 1000, 300, false}, {true, false, 250000, 10, 300, true},
        {true, false, 250000, 10, 400, false},  {true, false, 250000, 300, 500, false},
        {false, true, 20000, 10, 560, true},    {false, true, 20000, 300, 560, true},
        {false, false, 40000, 10, 200, true},   {false, false, 40000, 10, 560, false},
        {false, false, 40000, 200, 500, true},  {false, false, 100000, 148, 300, true},
        {false, false, 100000, 148, 500, false}, {false, false, 250000, 40, 500, false},
        {false, false, 250000, 300, 300, true}, {false, false, 250000, 300, 500, false},
        {true, true, 5000, 20, 1000, false},    {false, true, 5000, 20, 1000, false},
    };
    for (const auto& c : at) {
        char what[128];
        std::snprintf(what, sizeof what, "%s, %lld rows, %d fits, mean %lld", c.mixed ? "mixed" : "FP64", (long long)c.K, c.n,
                      (long long)c.mean);
        check(batch_prefers_window({c.mixed, c.shared, c.K, c.mean, c.n, 148}) == c.window, what);
    }
}

int main() {
    means();
    routes();
    if (!failures) std::printf("all routes as expected\n");
    return failures ? 1 : 0;
}
