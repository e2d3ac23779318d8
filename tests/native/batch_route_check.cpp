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

int main() {
    means();
    if (!failures) std::printf("all routes as expected\n");
    return failures ? 1 : 0;
}
