"""A column's gradient and Hessian where the call changes form: columns at the
8,192 entries that one block takes, an empty column, and fits past the
context's pinned result words; an update's coefficient reaches the device."""
import numpy as np
import pytest

from ccd_b200 import native, synthetic
from ccd_b200.data import MODEL_CONDITIONAL_LOGISTIC, MODEL_COX, MODEL_LOGISTIC, MODEL_POISSON, PRIOR_NORMAL
from oracle import checker

from .test_gpu_window import problem

pytestmark = pytest.mark.gpu


def agree(got, want):
    assert np.max(np.abs(np.array(got) - np.array(want))) <= 1e-10 * max(1.0, np.max(np.abs(want)))


@pytest.mark.parametrize("model", [MODEL_LOGISTIC, MODEL_POISSON])
def test_gradients_at_the_block_limit(gpu_ctx, model):
    d = problem(model, 20_000, [0, 1, 8191, 8192, 8193, 16_385], seed=3, prior=PRIOR_NORMAL, values=True)
    f = native.Fit(gpu_ctx, native.Matrix(gpu_ctx, d), d)
    e = checker.RestatementEngine(d)
    beta = np.linspace(-0.2, 0.3, d.J)
    f.set_beta(beta)
    e.set_beta(beta)
    for j in range(d.J):
        agree(f.compute_gradient_and_hessian(j), e.grad_hess(j))
        f.update_xbeta(j, 0.05)
        e.update_beta(j, 0.05)
        beta[j] += 0.05
    agree(f.get_xbeta(), e.xbeta())
    agree(f.compute_gradient_and_hessian(3), e.grad_hess(3))
    # the device holds the coefficients: its own row sums from them
    f.set_weights(np.ones(d.K))
    assert np.array_equal(f.get_beta(), beta)
    agree([f.get_log_likelihood()], [e.loglik()])


@pytest.mark.parametrize("model", [MODEL_LOGISTIC, MODEL_CONDITIONAL_LOGISTIC, MODEL_COX])
def test_more_fits_than_result_words(model):
    ctx = native.Context(0)
    d = synthetic.small(model, seed=5, K=200, P=4)
    m = native.Matrix(ctx, d)
    fits = [native.Fit(ctx, m, d) for _ in range(1026)]
    for j in range(d.J):
        want = fits[0].compute_gradient_and_hessian(j)
        agree(want, checker.RestatementEngine(d).grad_hess(j))
        for f in (fits[1023], fits[1024], fits[1025]):  # the last word and none
            assert f.compute_gradient_and_hessian(j) == want
    for f in fits:
        f.close()
    again = native.Fit(ctx, m, d)
    agree(again.compute_gradient_and_hessian(1), checker.RestatementEngine(d).grad_hess(1))
    again.close()
    m.close()
    ctx.close()
