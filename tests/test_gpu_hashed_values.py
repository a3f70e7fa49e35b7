"""Hashed keys with NULL cells, 128-bit integer sums and float columns of a
wide range: the slot's words beside its key are read with it there too.  Key
types, packed and NULL keys, the empty-slot sentinel as a key, table sizes on
both sides of the block-local table, against the oracle; and an int64 SUM in
time against a float one (1.6 times as long while its probe read the key
alone, 1.2 with the words beside it)."""
import numpy as np
import pytest

import oracle
from querymode_b200.engine import Column
from querymode_b200.query import AggregateOp, FilterOp, QueryDescriptor
from tests.helpers import assert_same

pytestmark = pytest.mark.gpu

AGGS = {"null": [("sum", "n"), ("count", "n"), ("min", "n"), ("count", "*")], "int64": [("sum", "l"), ("max", "l")],
        "wide": [("sum", "w"), ("max", "w")], "all": [("sum", "l"), ("sum", "n"), ("sum", "w"), ("min", "l"), ("count", "*")]}


@pytest.mark.parametrize("aggs", AGGS)
@pytest.mark.parametrize("kind", ["int64", "int32", "null", "packed"])
@pytest.mark.parametrize("groups", [1_300, 50_000])
def test_values(ctx, groups, kind, aggs):
    n = 400_123
    rng = np.random.default_rng(groups)
    idx = rng.integers(0, groups, n)
    key = rng.integers(-2**62, 2**62, groups)[idx]
    key[idx == 5] = -2**63
    cols = {"n": Column(rng.normal(size=n), rng.random(n) < 0.2), "l": rng.integers(-2**63, 2**63, n, dtype=np.int64),
            "w": np.exp(7 * rng.normal(size=n)), "i": rng.integers(0, 100, n).astype(np.int32)}
    by = ["key"]
    if kind == "packed":
        cols["key"], cols["b"] = rng.integers(-2**31, 2**31, groups)[idx].astype(np.int32), (idx % 7).astype(np.int32)
        by = ["key", "b"]
    elif kind == "int32":
        cols["key"] = rng.integers(-2**31, 2**31, groups)[idx].astype(np.int32)
    else:
        cols["key"] = Column(key, rng.random(n) < 0.01) if kind == "null" else key
    q = QueryDescriptor(filters=[FilterOp("i", "lt", 60)], group_by=by, aggregates=[AggregateOp(f, c) for f, c in AGGS[aggs]])
    want = oracle.run(cols, q, threads=8)
    t = ctx.table(cols)
    assert_same(t.run(q), want, ctx_msg=f"{groups} {kind} {aggs}")
    assert_same(ctx.batch([t, t], [q, q]).run()[1], want, ctx_msg="batch")


def test_time(ctx):
    import torch
    n, g = 20_000_000, torch.Generator(device="cuda")
    g.manual_seed(1)
    key = torch.randint(-2**62, 2**62, (9_000,), generator=g, device="cuda")[torch.randint(0, 9_000, (n,), generator=g, device="cuda")]
    t = {"key": key, "l": torch.randint(-2**60, 2**60, (n,), generator=g, device="cuda"),
         "x": torch.randn(n, generator=g, device="cuda", dtype=torch.float64), "i": torch.randint(0, 100, (n,), generator=g, device="cuda", dtype=torch.int32)}
    torch.cuda.synchronize()
    table = ctx.table(t)
    ms = []
    for c in ("x", "l"):
        q = QueryDescriptor(filters=[FilterOp("i", "lt", 50)], group_by=["key"], aggregates=[AggregateOp("sum", c), AggregateOp("count", "*")])
        ms.append(min(table.run(q).stats.scan_ms for _ in range(10)))
    assert ms[1] < 1.45 * ms[0], ms
