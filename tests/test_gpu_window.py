"""GPU parity of the windowed sweep against the CPU oracle where it can go
wrong: fewer columns than a window and just past one, columns at the lengths
where they stop being short and start running alone, every cluster size, rows in
and out of shared memory, weights, and columns that all share rows."""
import numpy as np
import pytest

from ccd_b200 import native, synthetic
from ccd_b200.data import (DENSE, GRADIENT, INDICATOR, INTERCEPT, MITTAL, MODEL_LOGISTIC, MODEL_POISSON, PRIOR_LAPLACE,
                           PRIOR_NORMAL, SPARSE, CyclopsData, build_columns)

pytestmark = pytest.mark.gpu

BETA_TOL = 1e-6
LL_TOL = 1e-9


def check(got, want):
    assert got.return_flag == want["flag"]
    assert got.iterations == want["iterations"]
    assert np.max(np.abs(got.beta - want["beta"])) <= BETA_TOL * max(np.max(np.abs(want["beta"])), 1e-8)
    assert abs(got.log_likelihood - want["loglik"]) <= LL_TOL * abs(want["loglik"])


def problem(model, K, lengths, seed, prior=PRIOR_LAPLACE, values=False):
    """An intercept and one column of each length at random rows."""
    rng = np.random.Generator(np.random.PCG64(seed))
    cols, fmts = [(None, None)], [INTERCEPT]
    xb = np.full(K, -1.0)
    for i, n in enumerate(lengths):
        r = np.sort(rng.choice(K, size=n, replace=False)).astype(np.int32)
        v = rng.uniform(0.2, 1.5, n) if values and i % 2 else None
        cols.append((r, v))
        fmts.append(INDICATOR if v is None else SPARSE)
        xb[r] += rng.normal(0.0, 0.5) * (1.0 if v is None else v)
    if model == MODEL_LOGISTIC:
        y = (rng.random(K) < 1.0 / (1.0 + np.exp(-xb))).astype(np.float64)
    else:
        y = rng.poisson(np.exp(xb)).astype(np.float64)
    cs, rows, vs, vals, fmt = build_columns(K, cols, fmts)
    pt = np.full(len(fmts), prior, np.int32)
    pt[0] = 0
    return CyclopsData(model, y, cs, rows, vs, vals, fmt, pt, np.full(len(fmts), 0.5))


@pytest.mark.parametrize("ctas", [1, 2, 4, 8, 16])
@pytest.mark.parametrize("model,prior", [(MODEL_LOGISTIC, PRIOR_LAPLACE), (MODEL_POISSON, PRIOR_NORMAL)])
def test_column_lengths_on_every_cluster(oracle_engine, ctas, model, prior):
    """Per CTA 127..129 and 511..513 entries (the ends of short and of medium),
    empty and one-entry columns, 36 of them: two windows and a bit."""
    edge = [127, 128, 129, 511, 512, 513]
    lengths = ([0, 1, 31, 32, 33] + [n * ctas for n in edge]) * 3 + [5, 700 * ctas, 40]
    d = problem(model, 1500 * ctas + 3, lengths, seed=40 + ctas, prior=prior, values=True)
    ctx = native.Context(0)
    try:
        ctx.set_max_ctas(ctas)
        for conv in (GRADIENT, MITTAL):
            got = native.fit_model(ctx, d, native.ModeFindingArguments(convergence_type=conv))
            check(got, oracle_engine(d).fit(conv, 1e-6))
    finally:
        ctx.close()


@pytest.mark.parametrize("n_columns", [1, 2, 15, 16, 17, 31, 33, 48])
def test_column_counts_around_a_window(gpu_ctx, oracle_engine, n_columns):
    d = problem(MODEL_LOGISTIC, 2500, [60] * n_columns, seed=50 + n_columns)
    check(native.fit_model(gpu_ctx, d, native.ModeFindingArguments()), oracle_engine(d).fit(GRADIENT, 1e-6))


@pytest.mark.parametrize("ctas,K", [(1, 4000), (1, 9000), (1, 20_000), (1, 40_000), (2, 16_000), (16, 90_000), (16, 420_000)])
def test_rows_in_and_out_of_shared_memory(oracle_engine, ctas, K):
    """All of a row's state in shared memory, a pair, its share alone, nothing."""
    for model, prior in ((MODEL_LOGISTIC, PRIOR_LAPLACE), (MODEL_POISSON, PRIOR_NORMAL)):
        d = problem(model, K, [80, 900, 20] * 8, seed=60, prior=prior)
        w = np.random.default_rng(5).uniform(0.0, 2.0, K)
        w[::9] = 0.0
        ctx = native.Context(0)
        try:
            ctx.set_max_ctas(ctas)
            f = native.Fit(ctx, native.Matrix(ctx, d), d)
            for weights in (None, w):
                ref = oracle_engine(d)
                ref.set_weights(weights)
                f.set_weights(weights)
                check(f.find_mode(native.ModeFindingArguments(), beta=np.zeros(d.J)), ref.fit(GRADIENT, 1e-6))
        finally:
            ctx.close()


def test_columns_that_all_share_rows(gpu_ctx, oracle_engine):
    """Dense columns short enough for a warp: each holds the next back."""
    rng = np.random.Generator(np.random.PCG64(70))
    K, P = 300, 40
    cols, fmts = [(None, None)], [INTERCEPT]
    xb = np.zeros(K)
    for j in range(P):
        if j % 3 == 0:
            v = rng.normal(0.0, 1.0, K)
            cols.append((None, v))
            fmts.append(DENSE)
            xb += 0.3 * v * rng.normal()
        else:
            cols.append((np.sort(rng.choice(K, 30, replace=False)).astype(np.int32), None))
            fmts.append(INDICATOR)
    y = (rng.random(K) < 1.0 / (1.0 + np.exp(-xb))).astype(np.float64)
    cs, rows, vs, vals, fmt = build_columns(K, cols, fmts)
    pt = np.full(P + 1, PRIOR_LAPLACE, np.int32)
    pt[0] = 0
    d = CyclopsData(MODEL_LOGISTIC, y, cs, rows, vs, vals, fmt, pt, np.full(P + 1, 0.3))
    check(native.fit_model(gpu_ctx, d, native.ModeFindingArguments()), oracle_engine(d).fit(GRADIENT, 1e-6))


def test_a_state_carried_on(gpu_ctx, oracle_engine):
    """The row state that a sweep leaves is the one that later calls read."""
    d = synthetic.logistic_l1(seed=71, K=12_000, P=120, density=0.01)
    f = native.Fit(gpu_ctx, native.Matrix(gpu_ctx, d), d)
    r = f.find_mode(native.ModeFindingArguments(), beta=np.zeros(d.J))
    ref = oracle_engine(d)
    ref.fit(GRADIENT, 1e-6)
    for j in (0, 1, 60, 120):
        g, h = f.compute_gradient_and_hessian(j)
        rg, rh = ref.grad_hess(j)
        assert abs(g - rg) <= 1e-8 * max(1.0, abs(rh)) and abs(h - rh) <= 1e-9 * abs(rh)
    again = f.find_mode(native.ModeFindingArguments())
    assert again.iterations <= 2 and np.max(np.abs(again.beta - r.beta)) <= 1e-4
