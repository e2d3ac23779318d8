"""Cox fits with an unpenalised column that is constant within every risk set: the
reference's quotients make its gradient and Hessian zero and end the fit as
ill-conditioned; so must sums whose difference is rounding only, wherever the column
stands and however the strata lie on the CTAs.  Penalised, it stays at zero and the
rest of the fit is the oracle's."""
import numpy as np
import pytest

from ccd_b200 import native
from ccd_b200.data import (DENSE, ILLCONDITIONED, INDICATOR, INTERCEPT, MITTAL, MODEL_COX, PRIOR_LAPLACE, PRIOR_NONE, SPARSE,
                           CyclopsData, build_columns, cox_sort_order)

pytestmark = pytest.mark.gpu


def _problem(K, n_strata, where, kind, prior, seed):
    rng = np.random.default_rng(seed)
    stratum = np.sort(rng.integers(0, n_strata, K)).astype(np.int64)
    time, y = rng.exponential(size=K), (rng.random(K) < 0.3).astype(np.float64)
    order = cox_sort_order(stratum, time, y)
    stratum, time, y = stratum[order], time[order], y[order]
    n = max(1, K // 20)
    cols = [(np.sort(rng.choice(K, n, replace=False)).astype(np.int32), None) for _ in range(20)]
    fmts = [INDICATOR] * 20
    at = {"first": 0, "middle": 10, "last": 20}[where]
    level = rng.uniform(0.5, 1.5, n_strata)[stratum]  # a value of its own in each stratum
    full = {INTERCEPT: (None, None), INDICATOR: (np.arange(K, dtype=np.int32), None),
            SPARSE: (np.arange(K, dtype=np.int32), level), DENSE: (None, level)}[kind]
    cols.insert(at, full)
    fmts.insert(at, kind)
    cs, rows, vs, vals, fmt = build_columns(K, cols, fmts)
    pt = np.full(21, PRIOR_LAPLACE, np.int32)
    pt[at] = prior
    return CyclopsData(model_type=MODEL_COX, y=y, col_start=cs, rows=rows, val_start=vs, vals=vals, fmt=fmt, prior_type=pt,
                       prior_var=np.full(21, 0.1), time=time, stratum=stratum), at


@pytest.mark.parametrize("kind", [INTERCEPT, INDICATOR, SPARSE, DENSE])
@pytest.mark.parametrize("where", ["first", "middle", "last"])
@pytest.mark.parametrize("K,n_strata,strategy", [(60, 3, native.SWEEP_AUTO), (2600, 1, native.SWEEP_LEVELS),
                                                 (2600, 40, native.SWEEP_GRID_LEVELS)])
def test_unpenalised(gpu_ctx, oracle_engine, K, n_strata, strategy, where, kind):
    for seed in range(3):
        d, at = _problem(K, n_strata, where, kind, PRIOR_NONE, seed)
        f = native.Fit(gpu_ctx, native.Matrix(gpu_ctx, d), d)
        r = f.find_mode(native.ModeFindingArguments(convergence_type=MITTAL, strategy=strategy), beta=np.zeros(d.J))
        assert r.return_flag == ILLCONDITIONED
        if kind in (INTERCEPT, INDICATOR):
            assert oracle_engine(d).fit(MITTAL, 1e-6)["flag"] == ILLCONDITIONED


@pytest.mark.parametrize("kind", [INTERCEPT, SPARSE])
@pytest.mark.parametrize("where", ["first", "last"])
def test_penalised(gpu_ctx, oracle_engine, where, kind):
    d, at = _problem(2600, 5, where, kind, PRIOR_LAPLACE, 7)
    want = oracle_engine(d).fit(MITTAL, 1e-6)
    r = native.Fit(gpu_ctx, native.Matrix(gpu_ctx, d), d).find_mode(native.ModeFindingArguments(convergence_type=MITTAL),
                                                                    beta=np.zeros(d.J))
    assert r.return_flag == want["flag"] == 0 and r.iterations == want["iterations"]
    assert r.beta[at] == want["beta"][at] == 0.0
    assert np.max(np.abs(r.beta - want["beta"])) <= 1e-6 * max(np.max(np.abs(want["beta"])), 1e-8)
