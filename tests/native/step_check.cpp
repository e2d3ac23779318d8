// step_check.cpp -- host test of newton_quotient_step (ccd_b200/csrc/step.h): the
// same bits as newton_prior_delta_l for every combination of ordinary, zero,
// huge, infinite and not-a-number gradients and Hessians, coefficients on both
// sides of zero, and the three priors.  Exit status 0 when all agree.
#include <cstdio>
#include <cstring>
#include <limits>
#include <random>
#include <vector>

#include "step.h"

using namespace ccdb;

int main() {
    const double inf = std::numeric_limits<double>::infinity(), nan = std::numeric_limits<double>::quiet_NaN();
    std::vector<double> v = {0.0, -0.0, 1.0, -1.0, 2.0, -2.0, 0.3, -0.3, 1e-300, -1e-300, 1e300, -1e300, inf, -inf, nan};
    std::mt19937_64 rng(5);
    std::normal_distribution<double> z;
    for (int i = 0; i < 40; ++i) v.push_back(z(rng) * (i % 4 ? 1.0 : 100.0));
    long bad = 0, n = 0;
    for (double g : v)
        for (double h : v)
            for (double b : v)
                for (int pt = 0; pt <= 2; ++pt)
                    for (double var : {0.05, 1.0, 2.0, 1e6}) {
                        if (!std::isfinite(b)) continue;
                        const double lambda = pt == 1 ? std::sqrt(2.0 / var) : 0.0;
                        const double want = newton_prior_delta_l(g, h, b, pt, var, lambda);
                        const double got = newton_quotient_step(g, h, b, pt, var, lambda, pt == 2 ? 1.0 / var : 0.0,
                                                                pt == 2 ? b / var : 0.0);
                        ++n;
                        if (!(got == want || (got != got && want != want)) && bad++ < 10)
                            std::printf("g %g h %g b %g prior %d var %g: %g, not %g\n", g, h, b, pt, var, got, want);
                    }
    if (bad) return 1;
    std::printf("%ld steps identical\n", n);
    return 0;
}
