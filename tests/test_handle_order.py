"""The Python handles in whatever order the collector takes them: nothing is
destroyed after the context that it lives on (no GPU: a recording library)."""
import itertools
import weakref

import pytest

from ccd_b200 import native


class _Recorder:
    def __init__(self):
        self.calls = []

    def __getattr__(self, name):
        return lambda h: self.calls.append((name, h))


@pytest.mark.parametrize("order", list(itertools.permutations(range(3))))
def test_no_handle_outlives_its_context(monkeypatch, order):
    rec = _Recorder()
    monkeypatch.setattr(native, "lib", lambda: rec)
    ctx = native.Context.__new__(native.Context)
    ctx.h, ctx._children = 1, weakref.WeakSet()  # empty, as the collector leaves it
    m = native.Matrix.__new__(native.Matrix)
    m.ctx, m.h = ctx, 2
    f = native.Fit.__new__(native.Fit)
    f.ctx, f.matrix, f.h = ctx, m, 3
    handles = [ctx, m, f]
    for i in order:
        handles[i].__del__()
    names = [name for name, _ in rec.calls]
    assert names.count("ccdb_context_destroy") == 1
    assert names[-1] == "ccdb_context_destroy"
    assert all(h.h is None for h in handles)
