"""CCDB_TRACE_FILE on the default sweeps: the rounds that the file holds are those of
the fit, whose result the trace does not change."""
import numpy as np
import pytest

from ccd_b200 import native, synthetic, trace
from ccd_b200.data import MITTAL, MODEL_CONDITIONAL_LOGISTIC, MODEL_COX, MODEL_LOGISTIC, MODEL_POISSON

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("model,strategy", [(MODEL_LOGISTIC, native.SWEEP_AUTO), (MODEL_POISSON, native.SWEEP_AUTO),
                                            (MODEL_COX, native.SWEEP_LEVELS), (MODEL_COX, native.SWEEP_GRID_LEVELS),
                                            (MODEL_CONDITIONAL_LOGISTIC, native.SWEEP_AUTO)])
def test_trace_of_a_windowed_sweep(gpu_ctx, monkeypatch, tmp_path, model, strategy):
    d = synthetic.small(model, seed=71, K=800, P=20, n_strata=100 if model == MODEL_CONDITIONAL_LOGISTIC else 5)
    args = native.ModeFindingArguments(convergence_type=MITTAL, strategy=strategy)
    f = native.Fit(gpu_ctx, native.Matrix(gpu_ctx, d), d)
    want = f.find_mode(args, beta=np.zeros(d.J))
    path = tmp_path / "rounds.bin"
    monkeypatch.setenv("CCDB_TRACE_FILE", str(path))
    got = f.find_mode(args, beta=np.zeros(d.J))
    assert np.array_equal(got.beta, want.beta) and got.iterations == want.iterations
    t = np.fromfile(path, trace.ROUND)
    assert len(t) == 4096
    t = t[t["end"] != 0]
    assert len(t) < 4096, "the whole fit"
    assert t["taken"].sum() == want.iterations * d.J
    assert t["moved"].sum() == want.nonzero_steps
    assert np.all(t["steps"] > t["begin"]) and np.all(t["end"] > t["steps"]) and np.all(t["taken"] <= t["flying"])
    assert "rounds traced" in trace.summarise_rounds(str(path))
