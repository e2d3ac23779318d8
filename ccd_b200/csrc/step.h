// step.h -- the coordinate step shared by host and device code: the Newton
// step with the prior's closed form and the trust-region bound.
#pragma once

#include <cmath>

#ifdef __CUDACC__
#define CCDB_HD __host__ __device__ __forceinline__
#define CCDB_HD_COLD static __host__ __device__ __noinline__
#else
#define CCDB_HD inline
#define CCDB_HD_COLD inline
#endif

namespace ccdb {

CCDB_HD int sgn_d(double x) { return x == 0 ? 0 : (x < 0 ? -1 : 1); }

// ccdUpdateBeta's clamp + JointPrior::getDelta (CyclicCoordinateDescent.cpp:1394-1413;
// priors/CovariatePrior.h:186-188 NoPrior, :240-273 Laplace, :410-415 Normal).
// `lambda` is sqrt(2 / var) of a Laplace prior (CovariatePrior.h:282-292),
// passed in by callers that take many steps under one variance.
CCDB_HD double newton_prior_delta_l(double g, double h, double beta, int ptype, double var,
                                    double lambda) {
    if (h < 0.0) {
        g = 0.0;
        h = 0.0;
    }
    if (ptype == 1) {
        const double neg = -(g - lambda) / h;
        const double pos = -(g + lambda) / h;
        const int s = sgn_d(beta);
        double delta;
        if (s == 0) {
            if (neg < 0) delta = neg;
            else if (pos > 0) delta = pos;
            else delta = 0.0;
        } else {
            delta = (s < 0) ? neg : pos;
            if (sgn_d(beta + delta) != s) delta = -beta;
        }
        return delta;
    } else if (ptype == 2) {
        return -(g + (beta / var)) / (h + (1.0 / var));
    }
    return -(g / h);
}

CCDB_HD double newton_prior_delta(double g, double h, double beta, int ptype, double var) {
    return newton_prior_delta_l(g, h, beta, ptype, var, ptype == 1 ? sqrt(2.0 / var) : 0.0);
}

// The Laplace step where the Hessian is not positive and finite, out of the way
// of the kernels that step through millions of ordinary ones.
CCDB_HD_COLD double laplace_delta_cold(double g, double h, double beta, double lambda) {
    return newton_prior_delta_l(g, h, beta, 1, 0.0, lambda);
}

// newton_prior_delta_l as one quotient num / den whose numerator is chosen before
// the division: for a positive finite h the sign of each of the two Laplace
// quotients is its numerator's, so only the one that is taken is divided, and a
// zero step divides nothing.  inv_var = 1 / var and b_var = beta / var are read
// for a normal prior only.
CCDB_HD double newton_quotient_step(double g, double h, double beta, int ptype, double var, double lambda,
                                    double inv_var, double b_var) {
    double num, den;
    if (ptype == 1) {
        if (!(h > 0.0 && h <= 1.7976931348623157e308)) return laplace_delta_cold(g, h, beta, lambda);
        if (beta == 0.0 && !(fabs(g) > lambda)) return 0.0;
        num = (beta > 0.0 || (beta == 0.0 && g < 0.0)) ? g + lambda : g - lambda;
        den = h;
    } else {
        if (h < 0.0) g = h = 0.0;
        num = g;
        den = h;
        if (ptype == 2) {
            num += b_var;
            den += inv_var;
        }
    }
    double delta = -num / den;
    // not across zero
    if (ptype == 1 && beta != 0.0 && (beta > 0.0 ? beta + delta <= 0.0 : !(beta + delta < 0.0))) delta = -beta;
    return delta;
}

// applyBounds (CyclicCoordinateDescent.cpp:1503-1520), std::max semantics.
CCDB_HD double apply_bounds(double delta, double& hd) {
    if (delta < -hd) delta = -hd;
    else if (delta > hd) delta = hd;
    double inter = fabs(delta) * 2;
    const double half = hd / 2;
    inter = (inter < half) ? half : inter;
    inter = (inter < 1E-3) ? 1E-3 : inter;
    hd = inter;
    return delta;
}

// log-density of one coefficient (priors/CovariatePrior.h:220-224, :404-408).
CCDB_HD double log_prior_one(double x, int ptype, double var) {
    if (ptype == 1) {
        const double lambda = sqrt(2.0 / var);
        return log(0.5 * lambda) - lambda * fabs(x);
    } else if (ptype == 2) {
        return -0.5 * log(2.0 * 3.14159265358979323846 * var) - 0.5 * x * x / var;
    }
    return 0.0;
}

// host alias used by the host-side objective
inline double log_prior_host(double x, int ptype, double var) { return log_prior_one(x, ptype, var); }

}  // namespace ccdb
