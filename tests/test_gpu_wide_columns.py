"""Float columns whose cells differ so much in size that many have bits below
the block-local integers' units: they are kept as doubles, by sampled cells of
the column (from one in 256 on).  Shares of such cells around the line, NULL
and non-finite ones among them, one group to more than a million (windows),
dense, hashed and no keys, batches and the partitioned aggregation; against
the oracle.  And a total of such a column takes no more than a few times one of
like-sized cells: without it, a hundred times."""
import time

import numpy as np
import pytest

import oracle
from querymode_b200.engine import Column
from querymode_b200.query import AggregateOp, FilterOp, QueryDescriptor
from tests.helpers import assert_same

pytestmark = pytest.mark.gpu

AGGS = [AggregateOp("sum", "w"), AggregateOp("min", "w"), AggregateOp("sum", "x"), AggregateOp("count", "*")]


def cells(kind, n, rng):
    if kind == "outlier":
        return np.r_[rng.normal(size=n - 1), 1e15]
    if kind == "lognormal":
        return np.exp(6 * rng.normal(size=n))
    if kind == "tiny":
        return np.r_[1e10, rng.random(n - 1) * 1e-25]
    if kind == "odd":
        w = np.exp(8 * rng.normal(size=n))
        w[rng.random(n) < 1e-3] = np.nan
        w[n // 2], w[n // 3] = np.inf, -0.0
        return w
    return np.where(rng.random(n) < kind, 1e-30 * (1 + rng.random(n)), 1 + rng.random(n))  # a share of small cells


@pytest.mark.parametrize("kind", ["outlier", "lognormal", "tiny", "odd", 1 / 1024, 1 / 256, 1 / 64])
@pytest.mark.parametrize("keys,groups", [("none", 1), ("dense", 1), ("dense", 5), ("dense", 3000), ("dense", 30_000), ("hashed", 5), ("hashed", 30_000)])
def test_sums(ctx, keys, groups, kind):
    n = 150_013
    rng = np.random.default_rng(groups)
    idx = rng.integers(0, groups, n)
    key = rng.integers(-2**62, 2**62, groups)[idx] if keys == "hashed" else idx
    w = cells(kind, n, rng)
    cols = {"key": key, "w": Column(w, rng.random(n) < 0.1) if kind == "odd" else w, "x": rng.random(n), "i": rng.integers(0, 100, n).astype(np.int32)}
    q = QueryDescriptor(filters=[FilterOp("i", "lt", 80)], group_by=None if keys == "none" else ["key"], aggregates=AGGS)
    want = oracle.run(cols, q)
    t = ctx.table(cols)
    assert_same(t.run(q), want, ctx_msg=f"{keys} {groups} {kind}")
    b = ctx.batch([t, t], [q, q])
    try:
        for mode in (1, 0):
            b.set_mode(mode)
            for r in b.run():
                assert_same(r, want, ctx_msg=f"batch {mode}")
    finally:
        b.close()


@pytest.mark.parametrize("partitioned", [0, 1])
@pytest.mark.parametrize("slots", [300_000, 1_300_001])
def test_large_tables(ctx, slots, partitioned):
    n = 12_000_013
    rng = np.random.default_rng(slots)
    cols = {"key": rng.integers(0, slots, n).astype(np.int64), "w": np.exp(6 * rng.normal(size=n))}
    cols["key"][rng.random(n) < 0.3] = 7
    q = QueryDescriptor(group_by=["key"], aggregates=[AggregateOp("sum", "w"), AggregateOp("count", "*")])
    t = ctx.table(cols)
    try:
        ctx.set_tuning(partitioned=partitioned)
        got = t.run(q)
    finally:
        ctx.set_tuning()
    want = oracle.run_full(cols, q)
    for c in ("key", "count_*"):
        assert np.array_equal(got.column(c).values, want.column(c).values)
    # the reference adds the hot key's 3.6M cells one after another and is itself off by more than 1e-12
    xhi, xlo, absum = want.diag["sum_w"]
    assert (np.abs(got.column("sum_w").values - (xhi + xlo)) <= 1e-12 * absum).all()


def test_a_total_costs_no_more(ctx):
    import torch
    g = torch.Generator(device="cuda")
    g.manual_seed(1)
    x = torch.randn(20_000_000, generator=g, device="cuda", dtype=torch.float64)
    ms = []
    for v in (x, torch.exp(6 * x)):
        torch.cuda.synchronize()
        t = ctx.table({"v": v})
        q = QueryDescriptor(aggregates=[AggregateOp("sum", "v")])
        best = 1e9
        for _ in range(6):
            t0 = time.perf_counter()
            t.run(q)
            best = min(best, time.perf_counter() - t0)
        ms.append(best)
    assert ms[1] < 8 * ms[0], ms
