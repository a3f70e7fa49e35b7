"""Forced deduplication over hashed keys keeps its block-local table beyond a
warp's first rows: few hot keys (the table takes every row) and many (it takes
few), against the oracle, and in time against the plan without it."""
import time

import numpy as np
import pytest

import oracle
from querymode_b200.query import AggregateOp, FilterOp, QueryDescriptor
from tests.helpers import assert_same

pytestmark = pytest.mark.gpu

Q = QueryDescriptor(filters=[FilterOp("i", "lt", 50)], group_by=["key"],
                    aggregates=[AggregateOp("sum", "x"), AggregateOp("max", "i"), AggregateOp("count", "*")])


def columns(n, keys):
    rng = np.random.default_rng(keys)
    return {"key": rng.integers(-2**62, 2**62, keys)[rng.integers(0, keys, n)], "i": rng.integers(0, 100, n).astype(np.int32),
            "x": rng.random(n)}


@pytest.mark.parametrize("slots", [0, 64])
@pytest.mark.parametrize("keys", [16, 60_000])
def test_results(ctx, keys, slots):
    cols = columns(12_000_017, keys)  # more than 32 drains a warp
    want = oracle.run(cols, Q, threads=8)
    t = ctx.table(cols)
    try:
        ctx.set_tuning(dedupe=1, local_slots=slots)
        assert_same(t.run(Q), want, ctx_msg=f"{keys} {slots}")
    finally:
        ctx.set_tuning()


def test_time(ctx):
    t = ctx.table(columns(20_000_000, 16))
    ms = []
    try:
        for dedupe in (0, 1):
            ctx.set_tuning(dedupe=dedupe)
            best = 1e9
            for _ in range(6):
                t0 = time.perf_counter()
                t.run(Q)
                best = min(best, time.perf_counter() - t0)
            ms.append(best)
    finally:
        ctx.set_tuning()
    assert ms[1] < 3 * ms[0], ms
