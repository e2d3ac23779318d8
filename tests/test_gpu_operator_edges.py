"""A column's gradient and Hessian where the call changes form: columns at the
8,192 entries that one block takes, an empty column, and fits past the
context's pinned result words; an update's coefficient reaches the device."""
import numpy as np
import pytest

from ccd_b200 import native
from ccd_b200.data import MODEL_LOGISTIC, MODEL_POISSON, PRIOR_NORMAL
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


def test_more_fits_than_result_words():
    ctx = native.Context(0)
    d = problem(MODEL_LOGISTIC, 200, [20, 30], seed=5)
    m = native.Matrix(ctx, d)
    fits = [native.Fit(ctx, m, d) for _ in range(1026)]
    want = fits[0].compute_gradient_and_hessian(1)
    for f in (fits[1023], fits[1024], fits[1025]):
        assert f.compute_gradient_and_hessian(1) == want
    for f in fits:
        f.close()
    again = native.Fit(ctx, m, d)
    assert again.compute_gradient_and_hessian(1) == want
    again.close()
    m.close()
    ctx.close()
