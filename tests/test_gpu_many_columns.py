"""Plans that run in the run-time-plan kernels (five value columns and more,
deterministic sums) over hashed keys: they read the slot's words with its key
too.  Values against the oracle, with NULLs, wide and integer columns, and a
five-column plan in time against a four-column one (three times as long while
it probed the padded slots key by key, under twice now)."""
import numpy as np
import pytest

import oracle
from querymode_b200 import _abi as A
from querymode_b200.engine import Column
from querymode_b200.query import AggregateOp, FilterOp, QueryDescriptor
from tests.helpers import assert_same

pytestmark = pytest.mark.gpu

AGGS = [("sum", "x"), ("min", "x"), ("sum", "f"), ("max", "l"), ("sum", "l"), ("sum", "n"), ("avg", "n"), ("sum", "i"), ("count", "*")]


def columns(n, groups, rng):
    key = rng.integers(-2**62, 2**62, groups)[rng.integers(0, groups, n)]
    key[:2] = -2**63  # the empty-slot sentinel
    return {"key": Column(key, rng.random(n) < 0.01), "x": rng.normal(size=n), "f": rng.random(n).astype(np.float32),
            "l": rng.integers(-2**63, 2**63, n, dtype=np.int64), "n": Column(rng.normal(size=n), rng.random(n) < 0.2),
            "i": rng.integers(-1000, 1000, n).astype(np.int32), "w": np.exp(7 * rng.normal(size=n))}


@pytest.mark.parametrize("flags", [0, A.QM_FLAG_DETERMINISTIC])
@pytest.mark.parametrize("wide", [False, True])
@pytest.mark.parametrize("groups", [7, 1_300, 50_000])
def test_values(ctx, groups, wide, flags):
    rng = np.random.default_rng(groups)
    cols = columns(400_123, groups, rng)
    aggs = AGGS + ([("sum", "w")] if wide and not flags else [])
    q = QueryDescriptor(filters=[FilterOp("i", "lt", 600)], group_by=["key"], aggregates=[AggregateOp(f, c) for f, c in aggs], flags=flags)
    want = oracle.run(cols, q, threads=8)
    t = ctx.table(cols)
    for tuning in ({}, {"dedupe": 1}, {"local_slots": -1}):
        try:
            ctx.set_tuning(**tuning)
            assert_same(t.run(q), want, ctx_msg=f"{groups} {wide} {flags} {tuning}")
        finally:
            ctx.set_tuning()
    b = ctx.batch([t, t], [q, q])
    try:
        for mode in (1, 0):
            b.set_mode(mode)
            assert_same(b.run()[1], want, ctx_msg=f"batch {mode}")
    finally:
        b.close()


def test_time(ctx):
    import torch
    n, g = 20_000_000, torch.Generator(device="cuda")
    g.manual_seed(1)
    cols = {"key": torch.randint(-2**62, 2**62, (4_000,), generator=g, device="cuda")[torch.randint(0, 4_000, (n,), generator=g, device="cuda")],
            "f": torch.randint(0, 1000, (n,), generator=g, device="cuda", dtype=torch.int32)}
    for c in "abcde":
        cols[c] = torch.randn(n, generator=g, device="cuda", dtype=torch.float64)
    torch.cuda.synchronize()
    t = ctx.table(cols)
    ms = []
    for names in ("abcd", "abcde"):
        q = QueryDescriptor(filters=[FilterOp("f", "lt", 500)], group_by=["key"], aggregates=[AggregateOp("sum", c) for c in names])
        ms.append(min(t.run(q).stats.scan_ms for _ in range(8)))
    assert ms[1] < 2.2 * ms[0], ms
