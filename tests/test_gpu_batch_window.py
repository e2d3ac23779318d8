"""GPU parity of the windowed sweep over many fits where it can go wrong:
columns at the lengths where a team's first entries, its copied entries and a
column's class end, for both team sizes; the rows' state in and out of shared
memory; more instances than SMs.

FP64 is compared with standalone oracle fits, at the tolerances of the plain
batch tests.  Mixed precision is compared with the lockstep engine, whose own
tests hold it to the oracle: an entry's FP32 terms are the same in both, their
compensated FP64 sums differ by the order of addition, some 1e-16 of a sum of
terms, and the fits take the same number of cycles, so 1e-9 leaves room for the
amplification of an ill-conditioned column."""
import numpy as np
import pytest

from ccd_b200 import native, synthetic
from ccd_b200.data import GRADIENT, LANGE, MITTAL, MODEL_LOGISTIC, MODEL_POISSON, PRIOR_LAPLACE, PRIOR_NORMAL

from .test_gpu_window import problem

pytestmark = pytest.mark.gpu

ONE_WARP = [0, 1, 31, 32, 33, 63, 64, 65, 123, 124, 125, 127, 128, 129, 512, 513] + [20] * 20
FOUR_WARPS = [0, 1, 127, 128, 129, 255, 256, 257, 319, 320, 321, 507, 508, 509, 512, 2048, 2049] + [100] * 20
# rows: xBeta and share in shared memory, the share alone, neither
ROWS = {False: (3001, 14001, 30001), True: (3001, 18001, 50001)}


@pytest.mark.parametrize("mixed", [False, True])
@pytest.mark.parametrize("place", [0, 1, 2])
@pytest.mark.parametrize("lengths", [ONE_WARP, FOUR_WARPS], ids=["one_warp", "four_warps"])
@pytest.mark.parametrize("model,prior,conv", [(MODEL_LOGISTIC, PRIOR_LAPLACE, GRADIENT), (MODEL_LOGISTIC, PRIOR_NORMAL, LANGE),
                                              (MODEL_POISSON, PRIOR_LAPLACE, MITTAL)])
def test_windowed_batch_matches_standalone_fits(gpu_ctx, oracle_engine, model, prior, conv, lengths, place, mixed):
    K = ROWS[mixed][place]
    d = problem(model, K, lengths, seed=90 + place, prior=prior, values=conv != GRADIENT)
    fold = synthetic.cv_folds(K, n_folds=3, seed=5)
    hold, var = np.array([0, 2, -1], np.int32), np.array([1.0, 0.05, 0.3])
    f = native.Fit(gpu_ctx, native.Matrix(gpu_ctx, d), d, native.PRECISION_MIXED if mixed else native.PRECISION_FP64)
    args = native.ModeFindingArguments(convergence_type=conv)
    beta, res, _ = f.batch_find_mode(var, hold, fold, args)
    if mixed:
        b_lock, r_lock, _ = f.batch_find_mode(var, hold, fold, args, group=1, cluster=1)
        assert np.max(np.abs(beta - b_lock)) <= 1e-9 * np.max(np.abs(b_lock))
        for got, want in zip(res, r_lock):
            for key in ("flag", "iterations", "steps", "updates", "update_entries", "gradient_entries"):
                assert got[key] == want[key], key
            assert abs(got["loglik"] - want["loglik"]) <= 1e-9 * abs(want["loglik"])
            assert abs(got["pred_loglik"] - want["pred_loglik"]) <= 1e-9 * max(1.0, abs(want["pred_loglik"]))
        return
    for i in range(len(var)):
        e = oracle_engine(d.with_prior(prior, float(var[i])))
        w = (fold != hold[i]).astype(float)
        e.set_weights(w)
        want = e.fit(conv, 1e-6)
        assert res[i]["flag"] == want["flag"]
        assert res[i]["iterations"] == want["iterations"]
        assert np.max(np.abs(beta[i] - want["beta"])) <= 1e-6 * max(np.max(np.abs(want["beta"])), 1e-8)
        assert abs(res[i]["loglik"] - want["loglik"]) <= 1e-9 * abs(want["loglik"])
        pred = e.predictive_loglik(1.0 - w)
        assert abs(res[i]["pred_loglik"] - pred) <= 1e-9 * max(1.0, abs(pred))


@pytest.mark.parametrize("mixed", [False, True])
def test_more_instances_than_sms(gpu_ctx, mixed):
    """An instance from the queue's second round equals the same one alone; so
    does one that stops at its limit of cycles."""
    d = problem(MODEL_LOGISTIC, 2000, ONE_WARP, seed=7)
    fold = synthetic.cv_folds(d.K, n_folds=5, seed=1)
    hold, var = synthetic.cv_grid(n_folds=5, n_vars=64, lower=0.05, upper=1.0)
    f = native.Fit(gpu_ctx, native.Matrix(gpu_ctx, d), d, native.PRECISION_MIXED if mixed else native.PRECISION_FP64)
    for cap in (1000, 2):
        args = native.ModeFindingArguments(convergence_type=GRADIENT, max_iterations=cap)
        b_all, r_all, _ = f.batch_find_mode(var, hold, fold, args)
        for i in (0, 150, 319):
            b1, r1, _ = f.batch_find_mode(var[i:i + 1], hold[i:i + 1], fold, args)
            assert np.array_equal(b1[0], b_all[i])
            assert r1[0] == r_all[i]
