"""Terms that overflow in the windowed sweep: a weighted Poisson fit with a row of weight
zero whose second moment is infinite ends as the oracle's does, not a number times zero
included; without such a value it is the oracle's fit."""
import numpy as np
import pytest

from ccd_b200 import native, synthetic
from ccd_b200.data import MITTAL, MODEL_POISSON, SPARSE

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("value", [1.0, 1e100, 1e170])
@pytest.mark.parametrize("zero_weight", [True, False])
def test_weighted_poisson(gpu_ctx, oracle_engine, value, zero_weight):
    d = synthetic.small(MODEL_POISSON, seed=8, K=300, P=6, formats=("indicator", "sparse"), intercept=False)
    j = int(np.flatnonzero(d.fmt == SPARSE)[0])
    d.vals = d.vals.copy()
    d.vals[d.val_start[j]] = value
    w = np.random.default_rng(9).integers(1, 3, d.K).astype(np.float64)
    if zero_weight:
        w[d.rows[d.col_start[j]]] = 0.0
    e = oracle_engine(d)
    e.set_weights(w)
    want = e.fit(MITTAL, 1e-6, 25)
    f = native.Fit(gpu_ctx, native.Matrix(gpu_ctx, d), d)
    f.set_weights(w)
    r = f.find_mode(native.ModeFindingArguments(convergence_type=MITTAL, max_iterations=25), beta=np.zeros(d.J))
    assert (r.return_flag, r.iterations) == (want["flag"], want["iterations"])
    assert np.array_equal(np.isfinite(r.beta), np.isfinite(want["beta"]))
    ok = np.isfinite(want["beta"])
    if ok.any():
        assert np.max(np.abs(r.beta - want["beta"])[ok]) <= 1e-6 * max(np.max(np.abs(want["beta"][ok])), 1e-8)
