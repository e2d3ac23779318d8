"""The windowed sweeps' waits that run out, on purpose, without faulting the GPU.

ccdb_fit_set_wait_limit reaches them too: with a bound of one nanosecond any wait
not satisfied on its first look runs out, the CTAs stop stepping, wait for what is
on its way to them and leave together, and the call returns CCDB_ERR_TIMEOUT.  The
same handle then fits the same problem correctly under the default bound."""
import numpy as np
import pytest

from ccd_b200 import native, synthetic
from ccd_b200.data import MITTAL, MODEL_CONDITIONAL_LOGISTIC, MODEL_COX, MODEL_LOGISTIC, MODEL_POISSON

pytestmark = pytest.mark.gpu


def _runs_out_then_recovers(ctx, oracle_engine, d, strategy):
    m = native.Matrix(ctx, d)
    f = native.Fit(ctx, m, d)
    args = native.ModeFindingArguments(convergence_type=MITTAL, strategy=strategy)
    start = np.zeros(d.J)
    if d.offset_col0:
        start[0] = 1.0
    for _ in range(3):
        f.set_wait_limit(1)
        with pytest.raises(native.CcdbError) as ex:
            f.find_mode(args, beta=start)
        assert ex.value.code == native.ERR_TIMEOUT
        f.set_wait_limit(0)
        want = oracle_engine(d).fit(MITTAL, 1e-6)
        r = f.find_mode(args, beta=start)
        assert r.return_flag == want["flag"] == 0
        assert r.iterations == want["iterations"]
        assert np.max(np.abs(r.beta - want["beta"])) <= 1e-6 * max(np.max(np.abs(want["beta"])), 1e-8)


@pytest.mark.parametrize("model,K,P", [(MODEL_LOGISTIC, 3000, 60), (MODEL_LOGISTIC, 40000, 40), (MODEL_POISSON, 3000, 2)])
def test_windowed_sweep(gpu_ctx, oracle_engine, model, K, P):
    """Clusters of four and sixteen CTAs; many rounds a cycle, and two or three."""
    d = synthetic.small(model, seed=90 + P, K=K, P=P, density=0.02, formats=("indicator", "sparse"))
    _runs_out_then_recovers(gpu_ctx, oracle_engine, d, native.SWEEP_AUTO)


@pytest.mark.parametrize("model,n_strata", [(MODEL_COX, 1), (MODEL_COX, 40), (MODEL_CONDITIONAL_LOGISTIC, 400)])
@pytest.mark.parametrize("strategy", [native.SWEEP_LEVELS, native.SWEEP_GRID_LEVELS])
def test_group_sweep(gpu_ctx, oracle_engine, model, n_strata, strategy):
    """Strata that span CTAs (tail and head sums are exchanged) and that do not, in
    both forms."""
    _runs_out_then_recovers(gpu_ctx, oracle_engine,
                            synthetic.small(model, seed=95, K=3000, P=20, density=0.05, n_strata=n_strata), strategy)


@pytest.mark.parametrize("precision", [native.PRECISION_FP64, native.PRECISION_MIXED])
def test_batched_windowed_sweep(gpu_ctx, precision):
    d = synthetic.small(MODEL_LOGISTIC, seed=97, K=900, P=30)
    fold = synthetic.cv_folds(d.K, n_folds=4, seed=3)
    hold, var = synthetic.cv_grid(n_folds=4, n_vars=2, lower=0.05, upper=5.0)
    f = native.Fit(gpu_ctx, native.Matrix(gpu_ctx, d), d, precision=precision)
    b_want, r_want, _ = f.batch_find_mode(var, hold, fold)
    f.set_wait_limit(1)
    with pytest.raises(native.CcdbError) as ex:
        f.batch_find_mode(var, hold, fold)
    assert ex.value.code == native.ERR_TIMEOUT
    f.set_wait_limit(0)
    b, r, _ = f.batch_find_mode(var, hold, fold)
    assert np.array_equal(b, b_want)
    assert [x["iterations"] for x in r] == [x["iterations"] for x in r_want]
    assert all(x["flag"] == 0 for x in r)
