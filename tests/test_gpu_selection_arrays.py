"""The array filter_select returns: its own or a view of page-locked memory, it
outlives later calls and its context, can be written to, holds no page-locked
memory when small, no more than a bound together, and comes where memory cannot
be page-locked."""
import gc

import numpy as np
import pytest

from querymode_b200 import _abi as A
from querymode_b200 import engine
from querymode_b200.engine import Context
from querymode_b200.query import FilterOp, QueryDescriptor

pytestmark = pytest.mark.gpu

N = 300_000
COLS = {"i": np.random.default_rng(1).integers(0, 100, N).astype(np.int32)}


def select(ctx, limit):
    return ctx.filter_select(COLS, QueryDescriptor(filters=[FilterOp("i", "lt", limit)]))


def want(limit):
    return np.flatnonzero(COLS["i"] < limit).astype(np.uint32)


def test_arrays_outlive_their_context():
    c = Context(0)
    kept = [(limit, select(c, limit)) for limit in (0, 1, 5, 50, 100, 50)]
    c.close()
    del c
    gc.collect()
    for limit, a in kept:
        assert a.dtype == np.uint32 and np.array_equal(a, want(limit))
        a[:1] = 7  # writable
    kept.clear()
    gc.collect()


def test_small_selections_hold_nothing(ctx):
    held = [select(ctx, 1) for _ in range(50)]
    assert ctx._lent[0] == 0 and all(a.flags.owndata for a in held)


def test_bounded(ctx, monkeypatch):
    monkeypatch.setattr(engine, "SELECT_LENT_BYTES", 3 * 4 * N)
    held = [select(ctx, 100) for _ in range(10)]
    assert ctx._lent[0] == 3 * 4 * N and [a.flags.owndata for a in held] == [False] * 3 + [True] * 7
    assert all(np.array_equal(a, want(100)) for a in held)
    del held
    gc.collect()
    assert ctx._lent[0] == 0


def test_without_page_locked_memory(ctx, monkeypatch):
    class NoPinned:
        def __init__(self, lib):
            self.lib = lib

        def qm_filter_select_result(self, *args):
            return A.QM_ERR_OOM

        def __getattr__(self, name):
            return getattr(self.lib, name)

    monkeypatch.setattr(ctx, "lib", NoPinned(ctx.lib))
    for limit in (0, 1, 50):
        assert np.array_equal(select(ctx, limit), want(limit))
    sel = np.arange(0, N, 3, dtype=np.uint32)
    q = QueryDescriptor(filters=[FilterOp("i", "lt", 50)])
    assert np.array_equal(ctx.filter_select(COLS, q, sel), sel[COLS["i"][sel] < 50])
