"""Cox fits with tie groups of very many rows: around the size from which a warp sums
a group's denominator, with and without dropped rows, and long columns whose rows fall
into them, against the oracle."""
import numpy as np
import pytest

from ccd_b200 import native
from ccd_b200.data import MITTAL, PRIOR_LAPLACE, PRIOR_NORMAL

from .test_gpu_cox_long import _problem

pytestmark = pytest.mark.gpu


def _tied(K, sizes, prior, seed):
    """One stratum whose first tie groups have the given numbers of rows."""
    d = _problem(K, 1, 1, prior, (K // 2, 0, 700), seed)
    time = np.repeat(np.arange(len(sizes), dtype=np.float64), sizes)
    d.time = np.concatenate([time, len(sizes) + np.arange(K - len(time)) // 7])[::-1].copy()
    return d


@pytest.mark.parametrize("sizes", [(1023, 1024, 1025), (1, 1024 + 31, 40, 2048), (5000,)])
@pytest.mark.parametrize("prior", [PRIOR_LAPLACE, PRIOR_NORMAL])
@pytest.mark.parametrize("weighted", [False, True])
def test_large_tie_groups(gpu_ctx, oracle_engine, sizes, prior, weighted):
    d = _tied(6000, sizes, prior, seed=sum(sizes))
    e = oracle_engine(d)
    f = native.Fit(gpu_ctx, native.Matrix(gpu_ctx, d), d)
    if weighted:
        w = np.random.default_rng(4).integers(0, 3, d.K).astype(np.float64)
        e.set_weights(w)
        f.set_weights(w)
    want = e.fit(MITTAL, 1e-6)
    r = f.find_mode(native.ModeFindingArguments(convergence_type=MITTAL), beta=np.zeros(d.J))
    assert r.return_flag == want["flag"] == 0
    assert r.iterations == want["iterations"]
    assert np.max(np.abs(r.beta - want["beta"])) <= 1e-6 * max(np.max(np.abs(want["beta"])), 1e-8)
    assert abs(r.log_likelihood - want["loglik"]) <= 1e-9 * abs(want["loglik"])
    assert abs(f.get_log_likelihood() - want["loglik"]) <= 1e-9 * abs(want["loglik"])
