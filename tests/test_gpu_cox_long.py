"""Long columns of the Cox windowed sweep, which run alone on every warp while steps
move: slices around the threshold and around the warps' parts of whole passes, strata
that lie in one part, go over one end of it or over many, with weights (zeros among
them), in both forms and on one, four and sixteen CTAs, against the oracle."""
import numpy as np
import pytest

from ccd_b200 import native
from ccd_b200.data import (DENSE, GRADIENT, INDICATOR, MITTAL, MODEL_COX, PRIOR_LAPLACE, PRIOR_NORMAL, SPARSE, CyclopsData,
                           build_columns, cox_sort_order)

pytestmark = pytest.mark.gpu


def _problem(K, n_strata, days, prior, lengths, seed):
    """Columns of the given lengths (0: dense), indicators and values in turn, and
    short ones between them."""
    rng = np.random.default_rng(seed)
    cols, fmts = [], []
    xb = np.zeros(K)
    for i, n in enumerate(lengths):
        for rows_n in (n, 7):
            b = rng.normal(0.0, 0.2)
            if rows_n == 0:
                v = rng.normal(0.0, 0.5, K)
                cols.append((np.arange(K), v))
                fmts.append(DENSE)
                xb += b * v
                continue
            r = rng.choice(K, rows_n, replace=False)
            v = rng.uniform(0.2, 1.0, rows_n) if i % 2 else None
            cols.append((r, v))
            fmts.append(SPARSE if i % 2 else INDICATOR)
            xb[r] += b * (1.0 if v is None else v)
    stratum = rng.integers(0, n_strata, K).astype(np.int64)
    t, c = rng.exponential(np.exp(-xb)), rng.exponential(1.0, K)
    y = (t < c).astype(np.float64)
    time = np.floor(np.minimum(t, c) * days)
    order = cox_sort_order(stratum, time, y)
    inv = np.empty(K, np.int64)
    inv[order] = np.arange(K)
    placed = []
    for (r, v), f in zip(cols, fmts):
        o = np.argsort(inv[r])
        placed.append((None if f == DENSE else inv[r][o].astype(np.int32), None if v is None else v[o]))
    cs, rows, vs, vals, fmt = build_columns(K, placed, fmts)
    J = len(fmts)
    return CyclopsData(model_type=MODEL_COX, y=y[order], col_start=cs, rows=rows, val_start=vs, vals=vals, fmt=fmt,
                       prior_type=np.full(J, prior, np.int32), prior_var=np.full(J, 0.5 if prior == PRIOR_NORMAL else 0.02),
                       time=time[order], stratum=stratum[order])


@pytest.mark.parametrize("prior,weighted", [(PRIOR_NORMAL, False), (PRIOR_LAPLACE, False), (PRIOR_NORMAL, True)])
@pytest.mark.parametrize("K,n_strata,days", [(2600, 1, 5), (2600, 3, 1000), (2600, 20, 30), (2600, 900, 30), (12000, 5, 400),
                                             (12000, 3000, 20)])
@pytest.mark.parametrize("ctas,strategy", [(1, native.SWEEP_AUTO), (4, native.SWEEP_AUTO), (0, native.SWEEP_LEVELS),
                                           (0, native.SWEEP_GRID_LEVELS)])
def test_long_columns(oracle_engine, K, n_strata, days, prior, weighted, ctas, strategy):
    d = _problem(K, n_strata, days, prior, (512, 513, 0, 544, 1024, 1025, K // 2), seed=K + n_strata)
    e = oracle_engine(d)
    w = np.random.default_rng(3).integers(0, 3, K).astype(np.float64)
    if weighted:
        e.set_weights(w)
    want = e.fit(MITTAL, 1e-6)
    ctx = native.Context(0)
    try:
        if ctas:
            ctx.set_max_ctas(ctas)
        f = native.Fit(ctx, native.Matrix(ctx, d), d)
        if weighted:
            f.set_weights(w)
        r = f.find_mode(native.ModeFindingArguments(convergence_type=MITTAL, strategy=strategy), beta=np.zeros(d.J))
        assert r.return_flag == want["flag"] == 0
        assert r.iterations == want["iterations"]
        assert np.max(np.abs(r.beta - want["beta"])) <= 1e-6 * max(np.max(np.abs(want["beta"])), 1e-8)
        assert abs(r.log_likelihood - want["loglik"]) <= 1e-9 * abs(want["loglik"])
    finally:
        ctx.close()


@pytest.mark.parametrize("K,n_strata,days", [(2600, 3, 1000), (12000, 5, 400), (12000, 3000, 20)])
@pytest.mark.parametrize("strategy", [native.SWEEP_LEVELS, native.SWEEP_GRID_LEVELS])
def test_long_columns_in_mixed_precision(gpu_ctx, oracle_engine, K, n_strata, days, strategy):
    """As the other mixed fits: to 1e-10, coefficients within 1e-6 of their scale."""
    d = _problem(K, n_strata, days, PRIOR_NORMAL, (512, 513, 0, 1025, K // 2), seed=K + n_strata)
    want = oracle_engine(d).fit(GRADIENT, 1e-10, 2000)
    f = native.Fit(gpu_ctx, native.Matrix(gpu_ctx, d), d, native.PRECISION_MIXED)
    r = f.find_mode(native.ModeFindingArguments(convergence_type=GRADIENT, tolerance=1e-10, max_iterations=2000,
                                                strategy=strategy), beta=np.zeros(d.J))
    assert r.return_flag == want["flag"] == 0
    assert np.max(np.abs(r.beta - want["beta"])) <= 1e-6 * max(np.max(np.abs(want["beta"])), 1e-8)
