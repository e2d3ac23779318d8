"""Per-call results of small problems around the sizes where the calls take another
way: xBeta of few rows comes back as the row words, of more as a column; the MM
gradient works a row's share out once a row, or for each of few entries."""
import numpy as np
import pytest

from ccd_b200 import native, synthetic
from ccd_b200.data import (DENSE, INDICATOR, INTERCEPT, MODEL_CONDITIONAL_LOGISTIC, MODEL_COX, MODEL_LOGISTIC,
                           MODEL_POISSON, SPARSE, build_columns)

pytestmark = pytest.mark.gpu


def _xbeta(d, beta):
    out = np.zeros(d.K)
    for j in range(d.J):
        r, v = slice(d.col_start[j], d.col_start[j + 1]), slice(d.val_start[j], d.val_start[j + 1])
        if d.fmt[j] in (DENSE, INTERCEPT):
            out += beta[j] * (d.vals[v] if d.fmt[j] == DENSE else 1.0)
        else:
            out[d.rows[r]] += beta[j] * (d.vals[v] if v.stop > v.start else 1.0)
    return out


@pytest.mark.parametrize("model", [MODEL_LOGISTIC, MODEL_POISSON, MODEL_CONDITIONAL_LOGISTIC, MODEL_COX])
@pytest.mark.parametrize("K", [1, 2, 1023, 1024, 1025, 2047, 2048, 2049])
def test_xbeta_of_every_row(gpu_ctx, model, K):
    d = synthetic.small(model, seed=K, K=K, P=6, n_strata=max(1, K // 10))
    f = native.Fit(gpu_ctx, native.Matrix(gpu_ctx, d), d)
    beta = np.random.default_rng(K).normal(0.0, 0.3, d.J)
    f.set_beta(beta)
    want = _xbeta(d, beta)
    # sums of at most seven products, in whatever order: 8 roundings of their size
    assert np.max(np.abs(f.get_xbeta() - want)) <= 8 * 2.0 ** -52 * max(1.0, np.max(np.abs(want))) * 8


@pytest.mark.parametrize("model", [MODEL_CONDITIONAL_LOGISTIC, MODEL_COX])
@pytest.mark.parametrize("entries", [40, 4095, 4096, 4097])
def test_mm_gradient_with_few_entries(gpu_ctx, model, entries):
    """Either way gives the same bits, since the share is the same word; a column more
    takes the matrix over the line."""
    K, P = 6000, 7
    rng = np.random.default_rng(entries)
    d = synthetic.small(model, seed=5, K=K, P=P, n_strata=600, formats=("indicator", "sparse"))
    sizes = np.full(P, entries // P)
    sizes[: entries - sizes.sum()] += 1
    cols, fmts = [], [int(f) for f in d.fmt[-P:]]
    for n, f in zip(sizes, fmts):
        cols.append((np.sort(rng.choice(K, n, replace=False)).astype(np.int32), rng.uniform(0.5, 1.5, n) if f == SPARSE else None))
    d.col_start, d.rows, d.val_start, d.vals, d.fmt = build_columns(K, cols, fmts)
    d.prior_type, d.prior_var = d.prior_type[-P:], d.prior_var[-P:]
    assert d.nnz == entries
    f = native.Fit(gpu_ctx, native.Matrix(gpu_ctx, d), d)
    f.set_beta(rng.normal(0.0, 0.2, P))
    g, h = f.compute_mm_gradient_and_hessian()
    # the same columns before one that fills the rows
    wide = build_columns(K, cols + [(np.arange(K, dtype=np.int32), None)], fmts + [INDICATOR])
    beta = f.get_beta()
    d.col_start, d.rows, d.val_start, d.vals, d.fmt = wide
    d.prior_type, d.prior_var = np.append(d.prior_type, 0), np.append(d.prior_var, 1.0)
    d.prior_type, d.prior_var = d.prior_type.astype(np.int32), d.prior_var.astype(np.float64)
    f2 = native.Fit(gpu_ctx, native.Matrix(gpu_ctx, d), d)
    f2.set_beta(np.append(beta, 0.0))
    g2, h2 = f2.compute_mm_gradient_and_hessian()
    assert np.array_equal(g, g2[:P]) and np.array_equal(h, h2[:P])
