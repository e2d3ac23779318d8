"""Per-call results of small problems around the sizes where the calls take another
way: xBeta of few rows comes back as the row words, of more as a column."""
import numpy as np
import pytest

from ccd_b200 import native, synthetic
from ccd_b200.data import (DENSE, INTERCEPT, MODEL_CONDITIONAL_LOGISTIC, MODEL_COX, MODEL_LOGISTIC, MODEL_POISSON)

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
