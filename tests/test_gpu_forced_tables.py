"""Forced block-local hash tables up to the largest that a block's shared
memory takes (8,192 slots of two words, 4,096 of five, 2,048 of eleven), scans
of pairs of tiles with every share of their rows passing (a warp's queue takes
a pair at once or tile by tile), with and without a selection vector and on
columns that are not 16-byte aligned; against the oracle."""
import numpy as np
import pytest

import oracle
from querymode_b200.query import AggregateOp, FilterOp, QueryDescriptor
from tests.helpers import assert_same

pytestmark = pytest.mark.gpu

AGGS = {2: [("count", "*")], 5: [("sum", "x"), ("max", "i"), ("count", "*")],
        11: [("sum", "x"), ("min", "x"), ("max", "x"), ("sum", "f"), ("max", "i"), ("min", "i"), ("count", "*")]}


def columns(n, keys, seed=3):
    rng = np.random.default_rng(seed)
    return {"key": rng.integers(-2**62, 2**62, keys)[rng.integers(0, keys, n)], "i": rng.integers(0, 1000, n).astype(np.int32),
            "x": rng.normal(size=n), "f": rng.random(n).astype(np.float32)}


@pytest.mark.parametrize("words,slots", [(2, 8192), (2, 16384), (5, 4096), (5, 8192), (11, 2048), (11, 1)])
@pytest.mark.parametrize("keys", [13, 6_000])
def test_largest_tables(ctx, keys, words, slots):
    cols = columns(200_003, keys)
    q = QueryDescriptor(filters=[FilterOp("i", "lt", 800)], group_by=["key"], aggregates=[AggregateOp(f, c) for f, c in AGGS[words]])
    t = ctx.table(cols)
    try:
        ctx.set_tuning(local_slots=slots)
        assert_same(t.run(q), oracle.run(cols, q), ctx_msg=f"{keys} {words} {slots}")
    finally:
        ctx.set_tuning()


@pytest.mark.parametrize("hashed", [True, False])
@pytest.mark.parametrize("share", [0, 30, 55, 75, 97, 100])
def test_pairs_of_tiles(ctx, share, hashed):
    """Enough rows for four pairs a warp (8 M), of which `share` percent pass:
    an integer filter, and one on an unaligned column, and a selection."""
    import torch
    n = 8_000_123
    rng = np.random.default_rng(share)
    key = rng.integers(0, 40, n)
    if hashed:
        key = rng.integers(-2**62, 2**62, 40)[key]
    whole = {"key": np.r_[0, key], "i": rng.integers(0, 100, n + 1).astype(np.int32), "x": rng.random(n + 1)}
    cols = {k: v[1:] for k, v in whole.items()}
    q = QueryDescriptor(filters=[FilterOp("i", "lt", share)], group_by=["key"],
                        aggregates=[AggregateOp("sum", "x"), AggregateOp("max", "i"), AggregateOp("count", "*")])
    want = oracle.run(cols, q, threads=8)
    assert_same(ctx.table(cols).run(q), want, ctx_msg="aligned")
    held = {k: torch.from_numpy(v).cuda() for k, v in whole.items()}
    torch.cuda.synchronize()
    assert_same(ctx.table({k: v[1:] for k, v in held.items()}).run(q), want, ctx_msg="unaligned")
    sel = np.flatnonzero(rng.random(n) < 0.9).astype(np.uint32)
    s = ctx.aggregate(q)
    s.push({k: v[1:] for k, v in held.items()}, selection=sel)
    assert_same(s.finish(), oracle.run({k: v[sel] for k, v in cols.items()}, q, threads=8), ctx_msg="selection")
