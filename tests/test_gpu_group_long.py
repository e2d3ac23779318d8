"""Long columns of the grouped models' windowed sweep, which run alone on every
warp: slices around the threshold and around the warps' parts of whole passes,
strata that lie in one part, go over one end of it or over many, in both forms and
on one, four and sixteen CTAs, against the oracle."""
import numpy as np
import pytest

from ccd_b200 import native
from ccd_b200.data import (DENSE, INDICATOR, MITTAL, MODEL_CONDITIONAL_LOGISTIC, MODEL_CONDITIONAL_POISSON, PRIOR_NORMAL,
                           SPARSE, CyclopsData, build_columns)

pytestmark = pytest.mark.gpu


def _problem(model, K, n_strata, lengths, seed):
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
                cols.append((None, v))
                fmts.append(DENSE)
                xb += b * v
                continue
            r = np.sort(rng.choice(K, rows_n, replace=False)).astype(np.int32)
            v = rng.uniform(0.2, 1.0, rows_n) if i % 2 else None
            cols.append((r, v))
            fmts.append(SPARSE if i % 2 else INDICATOR)
            xb[r] += b * (1.0 if v is None else v)
    cs, rows, vs, vals, fmt = build_columns(K, cols, fmts)
    stratum = np.sort(rng.integers(0, n_strata, K)).astype(np.int64)
    if model == MODEL_CONDITIONAL_LOGISTIC:
        score = xb + rng.gumbel(size=K)
        y = np.zeros(K)
        for s in np.unique(stratum):
            m = np.flatnonzero(stratum == s)
            y[m[np.argmax(score[m])]] = 1.0
    else:
        y = rng.poisson(np.exp(np.clip(xb, -3, 1))).astype(np.float64)
    J = len(fmts)
    return CyclopsData(model_type=model, y=y, col_start=cs, rows=rows, val_start=vs, vals=vals, fmt=fmt,
                       prior_type=np.full(J, PRIOR_NORMAL, np.int32), prior_var=np.full(J, 0.5), stratum=stratum)


@pytest.mark.parametrize("model", [MODEL_CONDITIONAL_LOGISTIC, MODEL_CONDITIONAL_POISSON])
@pytest.mark.parametrize("K,n_strata", [(2600, 1), (2600, 3), (2600, 20), (2600, 900), (12000, 5), (12000, 3000)])
@pytest.mark.parametrize("ctas,strategy", [(1, native.SWEEP_AUTO), (4, native.SWEEP_AUTO), (0, native.SWEEP_LEVELS),
                                           (0, native.SWEEP_GRID_LEVELS)])
def test_long_columns(oracle_engine, model, K, n_strata, ctas, strategy):
    d = _problem(model, K, n_strata, (512, 513, 0, 544, 1024, 1025, K // 2), seed=K + n_strata)
    want = oracle_engine(d).fit(MITTAL, 1e-6)
    ctx = native.Context(0)
    try:
        if ctas:
            ctx.set_max_ctas(ctas)
        f = native.Fit(ctx, native.Matrix(ctx, d), d)
        r = f.find_mode(native.ModeFindingArguments(convergence_type=MITTAL, strategy=strategy), beta=np.zeros(d.J))
        assert r.return_flag == want["flag"] == 0
        assert r.iterations == want["iterations"]
        assert np.max(np.abs(r.beta - want["beta"])) <= 1e-6 * max(np.max(np.abs(want["beta"])), 1e-8)
        assert abs(r.log_likelihood - want["loglik"]) <= 1e-9 * abs(want["loglik"])
    finally:
        ctx.close()
