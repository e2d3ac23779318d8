"""The calls that this engine is measured on, from the smallest to the largest.

A case is a dict of plain values.  ``listed`` names twelve of them, ``draw``
gives more of the same ranges; ``prepare`` makes what a user's program holds
before the call (problem, device matrix, fit handle), ``run`` is one pass
through the public entry points of ``ccd_b200.native``, ``work`` counts what a
pass cannot do without, and ``exact`` is the same result in plain 64-bit numpy.
"""
import math

import numpy as np

from ccd_b200 import data, native, synthetic

_CONTEXT = []


def _context():
    """One device context for the process, as a program keeps it."""
    if not _CONTEXT:
        _CONTEXT.append(native.Context(0))
    return _CONTEXT[0]


def listed():
    return [
        # The reference's solver over the per-coordinate calls (the adapter of a
        # host program): one call per coordinate, latency is all there is.
        {"name": "operator_calls", "kind": "operator", "model": "logistic", "K": 5_000, "P": 24, "density": 0.05},
        # One whole fit from host buffers, the way fitCyclopsModel ends: the small
        # L1 logistic problem of the benchmark.
        {"name": "logistic_l1", "kind": "logistic_fit", "K": 10_000, "P": 1_000, "density": 0.01},
        # A larger L1 logistic fit on a kept handle (refits over one data set).
        {"name": "logistic_l1_large", "kind": "logistic_mode", "K": 60_000, "P": 2_500, "density": 0.005},
        # Poisson regression with an offset, normal prior, columns of very uneven
        # length: a safety study's covariates on a kept handle.
        {"name": "poisson_offset", "kind": "poisson_mode", "K": 50_000, "P": 4_000, "nnz": 200},
        # A served Cox request, from host buffers.
        {"name": "cox_request", "kind": "cox_fit", "K": 20_000, "P": 400, "density": 0.01},
        # A large Cox fit on a kept handle.
        {"name": "cox_large", "kind": "cox_mode", "K": 400_000, "P": 1_000, "density": 0.002, "mixed": False},
        # A served conditional logistic request (matched sets), from host buffers.
        {"name": "conditional_logistic", "kind": "clr_fit", "sets": 4_000, "P": 500, "density": 0.01},
        # The cross-validation grid: folds x prior variances in one launch, in the
        # mixed precision that it is run with, and in 64 bits.
        {"name": "cv_grid", "kind": "cv", "K": 40_000, "P": 1_000, "density": 0.005, "folds": 10, "variances": 20,
         "mixed": True},
        {"name": "cv_grid_fp64", "kind": "cv", "K": 8_000, "P": 300, "density": 0.01, "folds": 10, "variances": 10,
         "mixed": False},
        # Standard errors after a fit: the information over every column.
        {"name": "fisher", "kind": "fisher", "model": "logistic", "K": 10_000, "P": 1_000, "density": 0.01},
        # The MM algorithm on matched sets, from host buffers.
        {"name": "mm_conditional", "kind": "mm_fit", "sets": 20_000, "P": 2_000, "density": 0.01},
        # Scoring a held-out set after a fit: its log-likelihood and every row's
        # prediction.
        {"name": "predict", "kind": "predict", "K": 500_000, "P": 1_000, "density": 0.002},
    ]


def draw(rng):
    def size(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    def part(lo, hi):
        return round(math.exp(rng.uniform(math.log(lo), math.log(hi))), 5)

    kind = rng.choice(["operator", "logistic_fit", "logistic_mode", "poisson_mode", "cox_fit", "cox_mode", "clr_fit",
                       "cv", "cv", "fisher", "mm_fit", "predict"])
    if kind == "operator":
        return {"kind": kind, "model": rng.choice(["logistic", "poisson", "clr", "cox"]), "K": size(500, 50_000),
                "P": size(8, 32), "density": part(0.01, 0.1)}
    if kind == "logistic_fit":
        return {"kind": kind, "K": size(1_000, 14_000), "P": size(100, 1_200), "density": part(0.002, 0.02)}
    if kind == "logistic_mode":
        return {"kind": kind, "K": size(15_000, 60_000), "P": size(300, 2_500), "density": part(0.002, 0.005)}
    if kind == "poisson_mode":
        return {"kind": kind, "K": size(10_000, 50_000), "P": size(500, 4_000), "nnz": rng.randint(50, 200)}
    if kind == "cox_fit":
        return {"kind": kind, "K": size(1_000, 30_000), "P": size(50, 400), "density": part(0.002, 0.02)}
    if kind == "cox_mode":
        return {"kind": kind, "K": size(100_000, 400_000), "P": size(200, 800), "density": part(0.001, 0.002),
                "mixed": rng.random() < 0.5}
    if kind == "clr_fit":
        return {"kind": kind, "sets": size(500, 6_000), "P": size(50, 500), "density": part(0.005, 0.02)}
    if kind == "cv":
        mixed = rng.random() < 0.6
        return {"kind": kind, "K": size(4_000, 40_000 if mixed else 8_000), "P": size(100, 800 if mixed else 300),
                "density": part(0.004, 0.01), "folds": rng.choice([5, 10]), "variances": rng.randint(4, 20 if mixed else 10),
                "mixed": mixed}
    if kind == "fisher":
        return {"kind": kind, "model": rng.choice(["logistic", "poisson", "clr", "cox"]), "K": size(1_000, 10_000),
                "P": size(30, 1_000), "density": part(0.005, 0.02)}
    if kind == "mm_fit":
        return {"kind": kind, "sets": size(500, 20_000), "P": size(100, 1_500), "density": part(0.004, 0.01)}
    return {"kind": kind, "K": size(20_000, 500_000), "P": size(100, 1_000), "density": part(0.001, 0.002)}


def _problem(case, seed):
    kind, seed = case["kind"], int(seed)
    model = {"logistic_fit": "logistic", "logistic_mode": "logistic", "poisson_mode": "poisson", "cox_fit": "cox",
             "cox_mode": "cox", "clr_fit": "clr", "mm_fit": "clr", "cv": "logistic",
             "predict": "logistic"}.get(kind) or case["model"]
    if kind == "operator":
        return synthetic.small(data.MODEL_NAMES[model], seed=seed, K=case["K"], P=case["P"], density=case["density"],
                               n_strata=max(2, case["K"] // 50), offset=model == "poisson")
    if model == "logistic":
        return synthetic.logistic_l1(seed=seed, K=case["K"], P=case["P"], density=case["density"],
                                     intercept=-3.0 if kind == "cv" else -2.0)
    if model == "poisson":
        nnz = case.get("nnz") or max(1, int(case["K"] * case["density"]))
        d = synthetic.poisson_offset(seed=seed, K=case["K"], P=case["P"], total_nnz=nnz * case["P"],
                                     cap=case["K"] // 20, n_true=0, intercept=-2.0)
        return _scaled_poisson(d, seed)
    if model == "clr":
        sets = case.get("sets") or max(1, int(round(case["K"] / 6.5)))
        return synthetic.conditional_logistic(seed=seed, n_sets=sets, P=case["P"], density=case["density"])
    return synthetic.cox_breslow(seed=seed, K=case["K"], n_strata=max(1, case["K"] // 1000), P=case["P"],
                                 density=case["density"], n_true=50, variance=0.1)


def _scaled_poisson(d, seed):
    """The Poisson problem with its covariates' values scaled to at most 1, as a
    normalised analysis has them, and outcomes drawn from 50 of its columns."""
    rng = _rng(seed, 4)
    d.vals = d.vals.copy()
    xb = np.full(d.K, -2.0)
    for j in range(2, d.J):
        v = d.vals[d.val_start[j]:d.val_start[j + 1]]
        if v.size:
            v /= v.max()
    for j in rng.integers(2, d.J, 50):
        v = d.vals[d.val_start[j]:d.val_start[j + 1]]
        xb[d.rows[d.col_start[j]:d.col_start[j + 1]]] += rng.normal(0.0, 0.3) * (v if v.size else 1.0)
    d.y = rng.poisson(np.exp(d.vals[:d.K] + xb)).astype(np.float64)
    return d


def _mode(case):
    if case["kind"] == "mm_fit":
        return native.ModeFindingArguments(convergence_type=data.MITTAL, algorithm=native.ALGORITHM_MM)
    if case["kind"] == "logistic_fit":
        return native.ModeFindingArguments(convergence_type=data.MITTAL)
    return native.ModeFindingArguments()


def _rng(seed, part):
    return np.random.Generator(np.random.PCG64([int(seed), part]))


def _coefficients(d, seed):
    """Coefficients as a regularised fit leaves them: a tenth of the columns, the
    intercept (and the offset's 1)."""
    rng = _rng(seed, 1)
    beta = np.where(rng.random(d.J) < 0.1, rng.normal(0.0, 0.3, d.J), 0.0)
    beta[d.fmt == data.INTERCEPT] = -1.5
    if d.offset_col0:
        beta[0] = 1.0
    return beta


def _grid(case, seed):
    hold, var = synthetic.cv_grid(case["folds"], case["variances"], lower=1e-3, upper=1.0)
    return synthetic.cv_folds(case["K"], case["folds"], seed=int(seed)), hold, var


def prepare(case, seed):
    d = _problem(case, seed)
    state = {"case": case, "d": d, "args": _mode(case)}
    kind = case["kind"]
    if kind.endswith("_fit"):
        state["context"] = _context()
        return state
    precision = native.PRECISION_MIXED if case.get("mixed") else native.PRECISION_FP64
    matrix = native.Matrix(_context(), d)
    state["fit"] = native.Fit(_context(), matrix, d, precision)
    if kind.endswith("_mode"):
        state["start"] = np.zeros(d.J)
        if d.offset_col0:
            state["start"][0] = 1.0
    elif kind == "cv":
        state["fold"], state["holdout"], state["variance"] = _grid(case, seed)
    else:
        state["beta"] = _coefficients(d, seed)
        if kind == "operator":
            state["steps"] = _rng(seed, 2).normal(0.0, 0.05, d.J)
        else:
            state["fit"].set_beta(state["beta"])
        if kind == "fisher":
            state["columns"] = np.arange(1 if d.offset_col0 else 0, d.J, dtype=np.int32)
            state["fit"].get_log_likelihood()
        if kind == "predict":
            state["weights"] = (_rng(seed, 3).random(d.K) < 0.1).astype(np.float64)
    return state


def _fitted(r):
    return {"beta": r.beta, "log_likelihood": r.log_likelihood, "iterations": int(r.iterations)}


def run(state):
    kind = state["case"]["kind"]
    if kind.endswith("_fit"):
        return _fitted(native.fit_model(state["context"], state["d"], state["args"]))
    fit = state["fit"]
    if kind.endswith("_mode"):
        fitted = _fitted(fit.find_mode(state["args"], beta=state["start"]))
        fitted["xbeta"] = fit.get_xbeta()
        return fitted
    if kind == "cv":
        beta, res, _ = fit.batch_find_mode(state["variance"], state["holdout"], state["fold"], state["args"])
        return {"beta": beta, "log_likelihood": np.array([r["loglik"] for r in res]),
                "predictive": np.array([r["pred_loglik"] for r in res]),
                "iterations": np.array([r["iterations"] for r in res], np.int64)}
    if kind == "fisher":
        return fit.compute_fisher_information(state["columns"])
    if kind == "predict":
        return {"predictive": fit.get_predictive_log_likelihood(state["weights"]),
                "estimates": fit.get_predictive_estimates()}
    fit.set_beta(state["beta"])
    gh = np.zeros((state["d"].J, 2))
    for j in range(1 if state["d"].offset_col0 else 0, state["d"].J):
        gh[j] = fit.compute_gradient_and_hessian(j)
        fit.update_xbeta(j, state["steps"][j])
    return {"gradients": gh, "log_likelihood": fit.get_log_likelihood(), "xbeta": fit.get_xbeta()}


def _shape(case):
    """Rows, columns and matrix entries."""
    K = case.get("K") or int(6.5 * case["sets"])
    P = case["P"]
    if case["kind"] == "operator":
        return K, P, K * P * (1 + 2 * case["density"]) / 3
    if "nnz" in case:
        return K, P, case["nnz"] * P
    return K, P, K * P * case["density"]


def work(case):
    """Entries (a row id, and a value where there is one), outcomes and results
    once; per entry of one pass over the columns the terms of its gradient and
    Hessian, and per row its exp or log terms."""
    K, P, entries = _shape(case)
    n = case["folds"] * case["variances"] if case["kind"] == "cv" else 1
    if case["kind"] == "fisher":
        return {"bytes": 4 * entries + 24 * K + 8 * P * P, "flops": 2 * entries * entries / max(K, 1) + 6 * K}
    if case["kind"] == "predict":
        return {"bytes": 4 * entries + 24 * K + 8 * P, "flops": 2 * entries + 30 * K}
    return {"bytes": 4 * entries + 16 * K + 8 * n * (P + 2), "flops": n * (8 * entries + 30 * K)}


# ---------------------------------------------------------------- 64-bit results

class _TooLong(Exception):
    pass


class _Model:
    """State and column sums of one problem in plain numpy; `n` weighted instances
    side by side for the cross-validation grid."""

    def __init__(self, d, beta, weights=None):
        self.d, self.K = d, d.K
        self.w = weights  # K x n for the grid
        self.cols, self.left = [], 5e6  # budget in units of about 3 microseconds
        for j in range(d.J):
            if d.fmt[j] in (data.DENSE, data.INTERCEPT):
                r = np.arange(d.K)
            else:
                r = d.rows[d.col_start[j]:d.col_start[j + 1]].astype(np.int64)
            v = d.vals[d.val_start[j]:d.val_start[j + 1]] if d.fmt[j] in (data.DENSE, data.SPARSE) else None
            self.cols.append((r, v))
        self.beta = np.array(beta, dtype=np.float64)
        if d.model_type == data.MODEL_COX:
            self.group, _, self.N = data.cox_groups(d.stratum, d.time, d.y)
        elif d.stratum is not None:
            self.group = np.concatenate([[0], np.cumsum(d.stratum[1:] != d.stratum[:-1])])
            self.N = int(self.group[-1]) + 1
        if d.stratum is not None:
            self.events = np.bincount(self.group, weights=d.y, minlength=self.N)
            first = np.concatenate([[True], d.stratum[1:] != d.stratum[:-1]])
            start = self.group[first]
            self.base = np.repeat(start, np.diff(np.concatenate([start, [self.N]])))
        wy = d.y if weights is None else d.y[:, None] * weights
        self.xjy = [self._dot(v, wy[r]) for r, v in self.cols]
        self.reset()

    @staticmethod
    def _dot(v, t):
        return t.sum(axis=0) if v is None else np.tensordot(v, t, axes=(0, 0))

    def pay(self, entries):
        self.left -= 6.0 + entries / 250.0
        if self.left < 0:
            raise _TooLong()

    def reset(self):
        shape = (self.K,) if self.w is None else (self.K, self.w.shape[1])
        self.xb = np.zeros(shape)
        for j, (r, v) in enumerate(self.cols):
            if np.any(self.beta[j] != 0.0):
                self.xb[r] += self.beta[j] if v is None else np.multiply.outer(v, self.beta[j])
        self.refresh()

    def refresh(self):
        if self.d.stratum is not None:
            self.e = np.exp(self.xb)
            self.den = np.bincount(self.group, weights=self.e, minlength=self.N)
            self.risk = self.run_sum(self.den) if self.d.model_type == data.MODEL_COX else self.den

    def run_sum(self, a):
        """Running sums within strata."""
        c = np.concatenate([[0.0], np.cumsum(a)])
        return c[1:] - c[self.base]

    def gradient(self, j):
        r, v = self.cols[j]
        m = self.d.model_type
        if len(r) == 0:
            return 0.0, 0.0
        if m in (data.MODEL_LOGISTIC, data.MODEL_POISSON):
            self.pay(4 * self.xb[0].size * len(r) if self.w is not None else len(r))
            e = np.exp(self.xb[r])
            p, q = (e / (1.0 + e), e / (1.0 + e) ** 2) if m == data.MODEL_LOGISTIC else (e, e)
            if self.w is not None:
                p, q = p * self.w[r], q * self.w[r]
            return self._dot(v, p) - self.xjy[j], self._dot(None if v is None else v * v, q)
        e = self.e[r]
        n1 = e if v is None else e * v
        n2 = n1 if v is None else n1 * v
        if m == data.MODEL_COX:
            self.pay(2 * self.N)
            a = self.run_sum(np.bincount(self.group[r], weights=n1, minlength=self.N)) / self.risk
            b = self.run_sum(np.bincount(self.group[r], weights=n2, minlength=self.N)) / self.risk
            ev = self.events
        else:
            self.pay(5 * len(r))
            s = self.group[r]
            cut = np.flatnonzero(np.concatenate([[True], s[1:] != s[:-1]]))
            u = s[cut]
            a, b, ev = np.add.reduceat(n1, cut) / self.den[u], np.add.reduceat(n2, cut) / self.den[u], self.events[u]
        return (ev * a).sum() - self.xjy[j], (ev * (b - a * a)).sum()

    def step(self, j, delta):
        r, v = self.cols[j]
        self.beta[j] = self.beta[j] + delta
        if self.w is None:
            self.xb[r] += delta if v is None else delta * v
        else:
            self.xb[r] += delta if v is None else np.multiply.outer(v, delta)
        if self.d.stratum is not None:
            e = np.exp(self.xb[r])
            if self.d.model_type == data.MODEL_COX:
                self.pay(4 * self.N)
                self.e[r] = e
                self.den = np.bincount(self.group, weights=self.e, minlength=self.N)
                self.risk = self.run_sum(self.den)
            else:
                np.add.at(self.den, self.group[r], e - self.e[r])
                self.e[r] = e

    def predictive(self, w):
        """Held-out log-likelihood of a logistic model: the events' terms
        (logPredLikeContrib, ModelSpecifics.h:1002-1009)."""
        y = self.d.y if w.ndim == 1 else self.d.y[:, None]
        return (w * y * (self.xb - np.log1p(np.exp(self.xb)))).sum(axis=0)

    def log_likelihood(self):
        d, m = self.d, self.d.model_type
        y = d.y if self.w is None else d.y[:, None]
        w = 1.0 if self.w is None else self.w
        if m == data.MODEL_LOGISTIC:
            return ((y * self.xb - np.log1p(np.exp(self.xb))) * w).sum(axis=0)
        if m == data.MODEL_POISSON:
            fixed = sum(math.lgamma(v + 1.0) for v in d.y)
            return (y * self.xb - np.exp(self.xb)).sum() - fixed
        return (d.y * self.xb).sum() - (self.events * np.log(self.risk)).sum()

    def objective(self, conv):
        if conv == data.MITTAL:
            return self.log_likelihood()
        t = self.xb * (self.d.y if self.w is None else self.d.y[:, None])
        return (t if self.w is None else t * self.w).sum(axis=0)


def _newton(g, h, beta, prior, variance):
    """The prior's closed-form Newton step (priors/CovariatePrior.h:186-273, 410-415)."""
    if h < 0.0:
        g = h = 0.0
    if prior == data.PRIOR_NORMAL:
        return -(g + beta / variance) / (h + 1.0 / variance)
    if prior == data.PRIOR_NONE:
        return -g / h
    lam = math.sqrt(2.0 / variance)
    neg, pos = -(g - lam) / h, -(g + lam) / h
    if beta == 0.0:
        return neg if neg < 0.0 else (pos if pos > 0.0 else 0.0)
    delta = neg if beta < 0.0 else pos
    return delta if (beta + delta) * beta > 0.0 else -beta


def _descend(M, args, prior, variance, n):
    """Cyclic coordinate descent to convergence (CyclicCoordinateDescent.cpp:909-1216)
    of `n` instances (n = 0: one, unweighted); stopped instances stay where they are."""
    many = max(n, 1)
    bound = np.full((M.d.J, many), args.initial_bound)
    last = np.atleast_1d(M.objective(args.convergence_type)).copy()
    live, iterations, cycle = np.ones(many, bool), np.zeros(many, np.int64), 0
    while live.any() and cycle < args.max_iterations:
        cycle += 1
        for j in range(1 if M.d.offset_col0 else 0, M.d.J):
            g, h = M.gradient(j)
            g, h, b = np.atleast_1d(g), np.atleast_1d(h), np.atleast_1d(M.beta[j])
            delta = np.zeros(many)
            for i in np.flatnonzero(live):
                var = variance[i] if n else variance[j]
                with np.errstate(divide="ignore", invalid="ignore"):
                    t = _newton(g[i], h[i], b[i], prior[j], var) if h[i] != 0.0 or prior[j] == 2 else (
                        0.0 if abs(g[i]) <= math.sqrt(2.0 / var) else math.copysign(math.inf, -g[i]))
                t = min(max(t, -bound[j, i]), bound[j, i])
                bound[j, i] = max(2.0 * abs(t), bound[j, i] / 2.0, 1e-3)
                delta[i] = t
            if delta.any():
                M.step(j, delta if n else delta[0])
        now = np.atleast_1d(M.objective(args.convergence_type))
        iterations[live] = cycle
        done = np.abs(now - last) / (np.abs(now) + 1.0) < args.tolerance
        last = np.where(live, now, last)
        live &= ~done
    return iterations


def _mm(M, args):
    """The MM cycle (CyclicCoordinateDescent.cpp:974-1001): every column from one state."""
    d, cycle = M.d, 0
    last = M.objective(args.convergence_type)
    while cycle < args.max_iterations:
        cycle += 1
        M.pay(12 * d.rows.size)
        share = (M.events[M.group] * M.e / M.den[M.group])
        for j, (r, v) in enumerate(M.cols):
            t = share[r]
            M.beta[j] += _newton(M._dot(v, t) - M.xjy[j], M._dot(None if v is None else v * v, t), M.beta[j],
                                 d.prior_type[j], d.prior_var[j])
        M.reset()
        now = M.objective(args.convergence_type)
        if abs(now - last) / (abs(now) + 1.0) < args.tolerance:
            break
        last = now
    return cycle


def _information(M, columns):
    d = M.d
    X = np.zeros((d.K, len(columns)))
    for i, j in enumerate(columns):
        r, v = M.cols[j]
        X[r, i] = 1.0 if v is None else v
    e = np.exp(M.xb)
    if d.stratum is None:
        f = e / (1.0 + e) ** 2 if d.model_type == data.MODEL_LOGISTIC else e
        return X.T @ (f[:, None] * X)
    p = e / M.den[M.group]  # each group's own denominator, as ModelSpecifics.hpp:1203-1337 has it
    C = np.zeros((M.N, len(columns)))
    np.add.at(C, M.group, p[:, None] * X)
    return X.T @ (p[:, None] * X) - C.T @ C


def exact(case, seed):
    kind, d, args = case["kind"], _problem(case, seed), _mode(case)
    try:
        if kind == "cv":
            fold, hold, var = _grid(case, seed)
            w = (fold[:, None] != hold[None, :]).astype(np.float64)
            M = _Model(d, np.zeros((d.J, len(var))), w)
            iterations = _descend(M, args, d.prior_type, var, len(var))
            return {"beta": M.beta.T.copy(), "log_likelihood": M.log_likelihood(),
                    "predictive": M.predictive(1.0 - w), "iterations": iterations}
        beta = np.zeros(d.J)
        if d.offset_col0:
            beta[0] = 1.0
        if kind.endswith(("_fit", "_mode")):
            M = _Model(d, beta)
            cycles = _mm(M, args) if kind == "mm_fit" else int(_descend(M, args, d.prior_type, d.prior_var, 0)[0])
            found = {"beta": M.beta, "log_likelihood": float(M.log_likelihood()), "iterations": cycles}
            if kind.endswith("_mode"):
                found["xbeta"] = M.xb
            return found
        M = _Model(d, _coefficients(d, seed))
        if kind == "fisher":
            return _information(M, np.arange(1 if d.offset_col0 else 0, d.J))
        if kind == "predict":
            w = (_rng(seed, 3).random(d.K) < 0.1).astype(np.float64)
            return {"predictive": float(M.predictive(w)), "estimates": 1.0 / (1.0 + np.exp(-M.xb))}
        steps, gh = _rng(seed, 2).normal(0.0, 0.05, d.J), np.zeros((d.J, 2))
        for j in range(1 if d.offset_col0 else 0, d.J):
            gh[j] = M.gradient(j)
            M.step(j, steps[j])
        return {"gradients": gh, "log_likelihood": float(M.log_likelihood()), "xbeta": M.xb}
    except _TooLong:
        return None
