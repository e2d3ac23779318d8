"""Fisher information where its launch changes form: row vectors that just fit
in shared memory and that just do not (29,056 rows; rows and groups together
for the grouped models), and more columns than a warp reads ranges of at once.
Against the oracle at the tolerance of the other post-fit calls."""
import numpy as np
import pytest

from ccd_b200 import native, synthetic
from ccd_b200.data import MODEL_CONDITIONAL_LOGISTIC, MODEL_COX, MODEL_LOGISTIC, MODEL_POISSON
from oracle import checker

from .test_gpu_postfit import FISHER_TOL

pytestmark = pytest.mark.gpu

ALL = ("sparse", "dense", "indicator")


@pytest.mark.parametrize("model,kw", [
    (MODEL_LOGISTIC, dict(K=29_056, P=9, density=0.002, formats=ALL)),
    (MODEL_LOGISTIC, dict(K=29_057, P=9, density=0.002, formats=ALL)),
    (MODEL_POISSON, dict(K=29_056, P=9, density=0.002, offset=True)),
    (MODEL_CONDITIONAL_LOGISTIC, dict(K=20_000, P=9, density=0.002, n_strata=400, formats=ALL)),
    (MODEL_CONDITIONAL_LOGISTIC, dict(K=29_000, P=9, density=0.002, n_strata=400, formats=ALL)),
    (MODEL_COX, dict(K=9_000, P=9, density=0.01, n_strata=5, formats=ALL)),
    (MODEL_COX, dict(K=29_000, P=9, density=0.01, n_strata=5, tie_days=200)),
    (MODEL_LOGISTIC, dict(K=300, P=1_030, density=0.05)),
])
def test_fisher_on_both_sides_of_a_row_vector(gpu_ctx, model, kw):
    d = synthetic.small(model, seed=31, **kw)
    f = native.Fit(gpu_ctx, native.Matrix(gpu_ctx, d), d)
    rng = np.random.Generator(np.random.PCG64(2))
    beta = rng.normal(0.0, 0.1, d.J)
    if d.offset_col0:
        beta[0] = 1.0
    f.set_beta(beta)
    e = checker.RestatementEngine(d)
    e.set_beta(beta)
    cols = np.arange(1 if d.offset_col0 else 0, d.J, dtype=np.int32)
    got, want = f.compute_fisher_information(cols), e.fisher_information(cols)
    assert np.max(np.abs(got - want)) <= FISHER_TOL * np.max(np.abs(want))
    assert np.array_equal(got, got.T)
