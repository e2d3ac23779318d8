"""GPU parity of the group models' windowed sweep against the CPU oracle where it
can go wrong: slices around a warp's 32 entries, the staged 128 and a CTA's 512;
one stratum over every CTA, strata that fit CTAs, fewer groups than CTAs; every
cluster size and the grid; weights with dropped rows; mixed precision."""
import numpy as np
import pytest

from ccd_b200 import native, synthetic
from ccd_b200.data import (GRADIENT, INDICATOR, MITTAL, MODEL_CONDITIONAL_LOGISTIC, MODEL_CONDITIONAL_POISSON, MODEL_COX,
                           PRIOR_LAPLACE, PRIOR_NORMAL, SPARSE, CyclopsData, build_columns, cox_sort_order)

pytestmark = pytest.mark.gpu

BETA_TOL = 1e-6
LL_TOL = 1e-9


def check(got, want, beta_tol=BETA_TOL):
    assert got.return_flag == want["flag"]
    assert got.iterations == want["iterations"]
    assert np.max(np.abs(got.beta - want["beta"])) <= beta_tol * max(np.max(np.abs(want["beta"])), 1e-8)
    assert abs(got.log_likelihood - want["loglik"]) <= LL_TOL * abs(want["loglik"])


def problem(model, K, strata, lengths, seed, prior=PRIOR_LAPLACE, variance=0.5, tied=False):
    """One column of each length at random rows, half of them with values."""
    rng = np.random.Generator(np.random.PCG64(seed))
    stratum = np.sort(rng.integers(0, strata, K)).astype(np.int64)
    cols, fmts, xb = [], [], np.zeros(K)
    for i, n in enumerate(lengths):
        r = np.sort(rng.choice(K, size=n, replace=False)).astype(np.int32)
        v = rng.uniform(0.2, 1.2, n) if i % 2 else None
        cols.append((r, v))
        fmts.append(INDICATOR if v is None else SPARSE)
        xb[r] += rng.normal(0.0, 0.4) * (1.0 if v is None else v)
    time = None
    if model == MODEL_COX:
        T, C = rng.exponential(1.0, K) / (0.05 * np.exp(xb)), rng.exponential(1.0, K) / 0.03
        y = (T < C).astype(np.float64)
        time = np.floor(np.minimum(T, C)) if tied else np.minimum(T, C)
        order = cox_sort_order(stratum, time, y)
        inv = np.empty(K, np.int64)
        inv[order] = np.arange(K)
        moved = []
        for r, v in cols:
            at = np.argsort(inv[r])
            moved.append((inv[r][at].astype(np.int32), None if v is None else v[at]))
        cols, y, time, stratum = moved, y[order], time[order], stratum[order]
    elif model == MODEL_CONDITIONAL_LOGISTIC:
        y = np.zeros(K)
        first = np.concatenate([[True], stratum[1:] != stratum[:-1]])
        y[np.flatnonzero(first)] = 1.0
        y = rng.permutation(y) if strata == 1 else y
    else:
        y = rng.poisson(np.exp(0.3 * xb)).astype(np.float64)
    cs, rows, vs, vals, fmt = build_columns(K, cols, fmts)
    J = len(fmts)
    return CyclopsData(model, y, cs, rows, vs, vals, fmt, np.full(J, prior, np.int32), np.full(J, variance), time=time,
                       stratum=stratum)


MODELS = [MODEL_COX, MODEL_CONDITIONAL_LOGISTIC, MODEL_CONDITIONAL_POISSON]


@pytest.mark.parametrize("ctas", [1, 2, 8, 16, 148])
@pytest.mark.parametrize("model", MODELS)
def test_slice_lengths(oracle_engine, model, ctas):
    """Per CTA of the cluster 31..33, 127..129 and 511..513 entries, empty and
    one-entry columns: a window and a bit.  148: the grid form."""
    per = ctas if ctas <= 16 else 4
    lengths = [0, 1, 7] + [n * per for n in (31, 32, 33, 127, 128, 129, 511, 512, 513)] + [40, 3, 90, 250, 12, 60]
    d = problem(model, 700 * per + 11, 30, lengths, seed=80 + ctas)
    strategy = native.SWEEP_LEVELS if ctas <= 16 else native.SWEEP_GRID_LEVELS
    ctx = native.Context(0)
    try:
        ctx.set_max_ctas(ctas)
        for conv in (GRADIENT, MITTAL):
            got = native.fit_model(ctx, d, native.ModeFindingArguments(convergence_type=conv, strategy=strategy))
            check(got, oracle_engine(d).fit(conv, 1e-6))
    finally:
        ctx.close()


@pytest.mark.parametrize("strategy", [native.SWEEP_LEVELS, native.SWEEP_GRID_LEVELS])
@pytest.mark.parametrize("strata", [1, 2, 16, 700])
@pytest.mark.parametrize("tied", [False, True])
def test_cox_strata_over_the_ctas(gpu_ctx, oracle_engine, strategy, strata, tied):
    """One stratum over every CTA, one and two per CTA, many per CTA; with and
    without tied events."""
    d = problem(MODEL_COX, 3000, strata, [60, 200, 15] * 8, seed=90 + strata, tied=tied)
    check(native.fit_model(gpu_ctx, d, native.ModeFindingArguments(strategy=strategy)), oracle_engine(d).fit(GRADIENT, 1e-6))


@pytest.mark.parametrize("model", MODELS)
def test_fewer_groups_than_ctas(gpu_ctx, oracle_engine, model):
    d = problem(model, 40, 3, [8, 12, 20], seed=95, prior=PRIOR_NORMAL)
    for strategy in (native.SWEEP_LEVELS, native.SWEEP_GRID_LEVELS):
        check(native.fit_model(gpu_ctx, d, native.ModeFindingArguments(strategy=strategy)), oracle_engine(d).fit(GRADIENT, 1e-6))


@pytest.mark.parametrize("strategy", [native.SWEEP_LEVELS, native.SWEEP_GRID_LEVELS])
@pytest.mark.parametrize("model", [MODEL_COX, MODEL_CONDITIONAL_LOGISTIC])
def test_weights_that_drop_rows(gpu_ctx, oracle_engine, model, strategy):
    """Zero weights inside groups, at strata's ends and over whole strata, then
    none: the groups are cut anew."""
    d = problem(model, 2500, 25, [70, 20, 300, 33] * 4, seed=97, tied=True)
    w = np.random.default_rng(9).uniform(0.5, 2.0, d.K)
    w[::6] = 0.0
    w[d.stratum == 4] = 0.0
    f = native.Fit(gpu_ctx, native.Matrix(gpu_ctx, d), d)
    for weights in (w, None, w):
        ref = oracle_engine(d)
        ref.set_weights(weights)
        f.set_weights(weights)
        got = f.find_mode(native.ModeFindingArguments(strategy=strategy), beta=np.zeros(d.J))
        check(got, ref.fit(GRADIENT, 1e-6))


@pytest.mark.parametrize("strategy", [native.SWEEP_LEVELS, native.SWEEP_GRID_LEVELS])
def test_mixed_precision_cox(gpu_ctx, oracle_engine, strategy):
    d = problem(MODEL_COX, 4000, 9, [150, 40, 500] * 5, seed=98)
    got = native.fit_model(gpu_ctx, d, native.ModeFindingArguments(strategy=strategy), precision=native.PRECISION_MIXED)
    want = oracle_engine(d).fit(GRADIENT, 1e-6)
    assert got.return_flag == want["flag"] and got.iterations == want["iterations"]
    assert np.max(np.abs(got.beta - want["beta"])) <= 1e-6 * np.max(np.abs(want["beta"]))


@pytest.mark.parametrize("rows,ctas", [(30_000, 1), (30_000, 2), (100_000, 4), (300_000, 2)])
def test_rows_and_groups_out_of_shared_memory(oracle_engine, rows, ctas):
    d = problem(MODEL_COX, rows, 40, [200, 60] * 6, seed=99)
    ctx = native.Context(0)
    try:
        ctx.set_max_ctas(ctas)
        check(native.fit_model(ctx, d), oracle_engine(d).fit(GRADIENT, 1e-6))
    finally:
        ctx.close()


def test_a_cox_state_carried_on(gpu_ctx, oracle_engine):
    """The groups' state after a sweep is the one that later calls read."""
    d = synthetic.cox_breslow(seed=7, K=5000, n_strata=6, P=60, density=0.02, n_true=20)
    f = native.Fit(gpu_ctx, native.Matrix(gpu_ctx, d), d)
    f.find_mode(native.ModeFindingArguments(), beta=np.zeros(d.J))
    ref = oracle_engine(d)
    ref.fit(GRADIENT, 1e-6)
    for j in (0, 17, 59):
        g, h = f.compute_gradient_and_hessian(j)
        rg, rh = ref.grad_hess(j)
        assert abs(g - rg) <= 1e-8 * max(1.0, abs(rh)) and abs(h - rh) <= 1e-8 * abs(rh)
