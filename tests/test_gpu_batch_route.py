"""The engine that a batch of fits runs on, as the call that asks for it tells."""
import numpy as np
import pytest

from ccd_b200 import native, synthetic
from ccd_b200.data import MODEL_COX, MODEL_LOGISTIC

pytestmark = pytest.mark.gpu
FP64, MIXED = native.PRECISION_FP64, native.PRECISION_MIXED


def _fit(ctx, d, precision):
    return native.Fit(ctx, native.Matrix(ctx, d), d, precision=precision)


@pytest.mark.parametrize("precision,n,group,engine", [
    (FP64, 10, 0, native.BATCH_WINDOWED), (FP64, 10, 2, native.BATCH_WINDOWED), (MIXED, 10, 0, native.BATCH_WINDOWED),
    (MIXED, 10, 2, native.BATCH_LOCKSTEP)])
def test_short_columns(gpu_ctx, precision, n, group, engine):
    d = synthetic.small(MODEL_LOGISTIC, seed=3, K=3000, P=20, density=0.01, formats=("indicator", "sparse"))
    assert _fit(gpu_ctx, d, precision).batch_engine(n, group=group) == engine


@pytest.mark.parametrize("precision,engine", [(FP64, native.BATCH_COLUMNS), (MIXED, native.BATCH_LOCKSTEP)])
def test_long_columns(gpu_ctx, precision, engine):
    d = synthetic.small(MODEL_LOGISTIC, seed=3, K=3000, P=6, formats=("dense",))
    assert _fit(gpu_ctx, d, precision).batch_engine(10) == engine


@pytest.mark.parametrize("precision", [FP64, MIXED])
def test_an_offset_does_not_count(gpu_ctx, precision):
    """20 covariates of 20 entries behind an offset and an intercept of 20,000."""
    d = synthetic.poisson_offset(seed=4, K=20_000, P=20, total_nnz=400, cap=40, n_true=0)
    f = _fit(gpu_ctx, d, precision)
    assert f.batch_engine(10) == native.BATCH_WINDOWED
    b, r, _ = f.batch_find_mode(np.full(2, 0.5))
    assert b.shape == (2, d.J) and all(x["flag"] == 0 for x in r)


def test_group_models_have_no_batch(gpu_ctx):
    with pytest.raises(native.CcdbError) as ex:
        _fit(gpu_ctx, synthetic.small(MODEL_COX, seed=1), FP64).batch_engine(4)
    assert ex.value.code == native.ERR_UNSUPPORTED
