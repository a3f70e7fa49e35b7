"""Float SUM / AVG of pushed batches (no column statistics: doubles in the
block-local table, the lanes of a slot summed first): one group, groups around
the copies of a slot, hashed and NULL keys, NULL / NaN / infinite and
cancelling cells, several columns, no GROUP BY; against the oracle.  And one
group costs no more than a few hundred: without the summing it took ten times
as long."""
import time

import numpy as np
import pytest

import oracle
from querymode_b200.engine import Column
from querymode_b200.query import AggregateOp, FilterOp, QueryDescriptor
from tests.helpers import assert_same

pytestmark = pytest.mark.gpu

AGGS = {"one": [("sum", "x"), ("count", "*")], "null": [("sum", "n"), ("avg", "n"), ("count", "n")],
        "four": [("sum", "x"), ("avg", "f"), ("sum", "odd"), ("sum", "i"), ("min", "x")],
        "five": [("sum", "x"), ("sum", "f"), ("sum", "n"), ("sum", "odd"), ("max", "i")]}


@pytest.mark.parametrize("aggs", AGGS)
@pytest.mark.parametrize("kind,groups", [("none", 1), ("dense", 1), ("dense", 3), ("dense", 700), ("hashed", 2), ("hashed", 33), ("hashed", 40_000)])
def test_sums(ctx, kind, groups, aggs):
    n = 120_011
    rng = np.random.default_rng(groups)
    idx = rng.integers(0, groups, n)
    key = rng.integers(-2**62, 2**62, groups)[idx] if kind == "hashed" else idx.astype(np.int64)
    odd = rng.normal(size=n)
    odd[idx == 0] = np.where(rng.random(int((idx == 0).sum())) < 1e-3, np.nan, odd[idx == 0])
    odd[np.flatnonzero(idx == groups - 1)[:1]] = np.inf
    x = rng.normal(size=n) * 10.0 ** rng.integers(-12, 12, n)
    x[::2] = -x[1::2][:len(x[::2])] if n % 2 == 0 else np.r_[-x[1::2], 0.0]
    cols = {"key": Column(key, rng.random(n) < 0.01), "x": x, "f": rng.random(n).astype(np.float32), "odd": odd,
            "n": Column(rng.normal(size=n), rng.random(n) < 0.2), "i": rng.integers(-1000, 1000, n).astype(np.int32)}
    q = QueryDescriptor(filters=[FilterOp("i", "lt", 700)], group_by=None if kind == "none" else ["key"],
                        aggregates=[AggregateOp(f, c) for f, c in AGGS[aggs]])
    want = oracle.run(cols, q)
    s = ctx.aggregate(q)
    s.push(cols)
    assert_same(s.finish(), want, ctx_msg=f"{kind} {groups} {aggs}")
    t = ctx.table(cols)
    s = ctx.aggregate(q)
    s.push_table(t)
    s.push_table(t)
    twice = {k: Column(np.r_[c.values, c.values], np.r_[c.nulls, c.nulls]) if isinstance(c, Column) else np.r_[c, c] for k, c in cols.items()}
    assert_same(s.finish(), oracle.run(twice, q), ctx_msg=f"twice {kind} {groups} {aggs}")


def push_times(ctx, keys):
    """Seconds of a push of SUM and COUNT(*) by each of `keys`."""
    import torch
    g = torch.Generator(device="cuda")
    g.manual_seed(1)
    x = torch.randn(len(keys[0]), generator=g, device="cuda", dtype=torch.float64)
    q = QueryDescriptor(group_by=["key"], aggregates=[AggregateOp("sum", "x"), AggregateOp("count", "*")])
    out = []
    for key in keys:
        torch.cuda.synchronize()
        t = ctx.table({"key": key, "x": x})
        best = 1e9
        for _ in range(6):
            s = ctx.aggregate(q)
            t0 = time.perf_counter()
            s.push_table(t)
            best = min(best, time.perf_counter() - t0)
            s.close()
        out.append(best)
    return out


def test_one_group_costs_no_more(ctx):
    import torch
    many = torch.randint(0, 500, (20_000_000,), device="cuda")
    ms = push_times(ctx, [many, torch.zeros_like(many)])
    assert ms[1] < 3 * ms[0], ms


def test_keys_in_a_row_cost_no_more(ctx):
    """Sixteen keys that follow one another against sixteen random ones: twice
    as long while they met on one bank of shared memory."""
    import torch
    idx = torch.randint(0, 16, (50_000_000,), device="cuda")
    ms = push_times(ctx, [torch.randint(-2**62, 2**62, (16,), device="cuda")[idx], idx])
    assert ms[1] < 1.5 * ms[0], ms
