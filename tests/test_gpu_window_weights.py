"""Weighted windowed sweeps where the weights just fit in shared memory beside the rest
of the rows and where they just do not (a CTA of 4,940 rows of a logistic fit, 6,176 of
a Poisson one), in odd sizes, with values staged and on several CTAs: against the oracle
at the tolerances of the other sweeps."""
import numpy as np
import pytest

from ccd_b200 import native
from ccd_b200.data import MITTAL, MODEL_LOGISTIC, MODEL_POISSON, PRIOR_LAPLACE, PRIOR_NORMAL

from .test_gpu_window import check, problem

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("model,K,ctas,values", [
    (MODEL_LOGISTIC, 301, 1, False),
    (MODEL_LOGISTIC, 4_939, 1, False),
    (MODEL_LOGISTIC, 4_940, 1, False),
    (MODEL_LOGISTIC, 4_941, 1, False),
    (MODEL_LOGISTIC, 4_120, 1, True),
    (MODEL_LOGISTIC, 9_880, 2, False),
    (MODEL_LOGISTIC, 9_883, 2, False),
    (MODEL_LOGISTIC, 1_601, 16, True),
    (MODEL_POISSON, 6_176, 1, False),
    (MODEL_POISSON, 6_177, 1, False),
    (MODEL_POISSON, 12_350, 2, True),
])
def test_weights_on_both_sides_of_shared_memory(oracle_engine, model, K, ctas, values):
    d = problem(model, K, [0, 1, 40, 300, 130, 33, 220, 7, 64] * 3 + [min(K // 2, 900)], seed=K % 97,
                prior=PRIOR_NORMAL if ctas == 2 else PRIOR_LAPLACE, values=values)
    w = np.random.default_rng(K).integers(0, 4, K).astype(np.float64)
    e = oracle_engine(d)
    e.set_weights(w)
    ctx = native.Context(0)
    try:
        ctx.set_max_ctas(ctas)
        f = native.Fit(ctx, native.Matrix(ctx, d), d)
        f.set_weights(w)
        check(f.find_mode(native.ModeFindingArguments(convergence_type=MITTAL)), e.fit(MITTAL, 1e-6))
    finally:
        ctx.close()
