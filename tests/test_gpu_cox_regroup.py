"""The Cox sweep's blocks follow the grouping: weights that regroup the rows, with
and without a sweep between them, and predictive log-likelihoods, which regroup
twice, leave the next sweep what a fresh handle gives."""
import numpy as np
import pytest

from ccd_b200 import native, synthetic
from ccd_b200.data import MITTAL, MODEL_COX

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("K,P", [(60, 3), (2500, 20)])
def test_sweep_after_regrouping(gpu_ctx, K, P):
    d = synthetic.small(MODEL_COX, seed=41, K=K, P=P, n_strata=4)
    rng = np.random.default_rng(42)
    weights = [None, (rng.random(K) < 0.7).astype(float), rng.integers(0, 3, K).astype(float), None]
    args = native.ModeFindingArguments(convergence_type=MITTAL)
    m = native.Matrix(gpu_ctx, d)

    def fresh(w):
        f = native.Fit(gpu_ctx, m, d)
        f.set_weights(w)
        return f.find_mode(args, beta=np.zeros(d.J))

    f = native.Fit(gpu_ctx, m, d)
    for w in weights:
        f.set_weights(w)
        f.set_beta(np.zeros(d.J))
        f.get_predictive_log_likelihood((rng.random(K) < 0.5).astype(float))
        got, want = f.find_mode(args, beta=np.zeros(d.J)), fresh(w)
        assert np.array_equal(got.beta, want.beta)
        assert (got.return_flag, got.iterations, got.log_likelihood) == (want.return_flag, want.iterations, want.log_likelihood)
        f.get_predictive_log_likelihood((rng.random(K) < 0.5).astype(float))
