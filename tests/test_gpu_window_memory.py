"""What a windowed sweep allocates: its plan, and no array of the rows' size beside the
fit's own (a context's budget that held a fit holds its sweep)."""
import numpy as np
import pytest

from ccd_b200 import native, synthetic
from ccd_b200.data import MITTAL, MODEL_LOGISTIC, MODEL_POISSON

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("model", [MODEL_LOGISTIC, MODEL_POISSON])
def test_a_sweep_of_many_rows_needs_its_plan_only(model):
    """600,000 rows: their shares do not fit the shared memory of 16 CTAs."""
    d = synthetic.small(model, seed=6, K=600_000, P=4, density=0.0005, formats=("indicator", "sparse"))
    ctx = native.Context(0)
    try:
        f = native.Fit(ctx, native.Matrix(ctx, d), d)
        before = ctx.memory_in_use()
        args = native.ModeFindingArguments(convergence_type=MITTAL)
        r = f.find_mode(args, beta=np.zeros(d.J))
        assert ctx.memory_in_use() - before <= 64 << 10
        again = f.find_mode(args, beta=np.zeros(d.J))
        assert np.array_equal(r.beta, again.beta) and r.iterations == again.iterations
        x = f.get_xbeta()  # and the scratch that the sweep uses is the calls' again
        f.set_beta(r.beta)
        assert np.max(np.abs(f.get_xbeta() - x)) <= 1e-12
    finally:
        ctx.close()
