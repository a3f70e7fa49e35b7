"""Block-local accumulators kept as 32-bit limbs, against the oracle: carries
across limbs, integers at the ends of their types, float columns of a wide
dynamic range (cells below the block-local units, groups of only tiny cells,
NaN / Infinity), few slots (copies per lane) and slot counts around the edges
of the copy rule, dense, hashed, NULL and absent keys.  Float SUM / AVG within
helpers.REL_TOL (1e-12) of the oracle; everything else bit for bit."""
import numpy as np
import pytest

import oracle
from querymode_b200 import _abi as A
from querymode_b200.engine import Column
from querymode_b200.query import AggregateOp, FilterOp, QueryDescriptor
from tests.helpers import assert_same

pytestmark = pytest.mark.gpu


def columns(n, groups, seed, hashed):
    rng = np.random.default_rng(seed)
    idx = rng.integers(0, groups, n)
    key = (rng.integers(-2**62, 2**62, groups)[idx] if hashed else idx - groups // 2).astype(np.int64)
    wide = rng.normal(size=n) * 10.0 ** rng.integers(-30, 10, n)
    wide[idx == 0] = rng.random(int((idx == 0).sum())) * 1e-25  # a group of tiny cells only
    odd = rng.normal(size=n)
    odd[rng.random(n) < 1e-3] = np.nan
    odd[idx == groups - 1] = np.inf
    i32 = rng.integers(-2**31, 2**31, n).astype(np.int32)
    i64 = rng.integers(-2**63, 2**63, n, dtype=np.int64)
    i64[rng.random(n) < 0.1] = -1
    return {"key": key, "wide": wide, "odd": odd, "f": rng.random(n).astype(np.float32), "i32": i32, "i64": i64,
            "neg": -rng.integers(1, 3, n).astype(np.int32), "price": Column(rng.random(n) * 1000, rng.random(n) < 0.1)}


QUERIES = {
    "sum": [AggregateOp("sum", "f"), AggregateOp("count", "*")],
    "sums": [AggregateOp("sum", "wide"), AggregateOp("avg", "f")],
    "mixed": [AggregateOp("sum", "wide"), AggregateOp("min", "wide"), AggregateOp("max", "wide"), AggregateOp("sum", "i32"),
              AggregateOp("sum", "neg"), AggregateOp("count", "*")],
    "all": [AggregateOp("sum", "odd"), AggregateOp("min", "odd"), AggregateOp("sum", "i64"), AggregateOp("avg", "i64"),
            AggregateOp("sum", "price"), AggregateOp("count", "price"), AggregateOp("max", "i32")],
}


@pytest.mark.parametrize("aggs", QUERIES)
@pytest.mark.parametrize("groups,hashed", [(1, False), (2, False), (17, False), (33, False), (700, False), (2000, False),
                                           (3, True), (200, True), (5000, True)])
def test_local_words(ctx, groups, hashed, aggs):
    cols = columns(150_001, groups, groups + 10 * hashed, hashed)
    q = QueryDescriptor(filters=[FilterOp("f", "lt", 0.7)], group_by=["key"], aggregates=QUERIES[aggs])
    want = oracle.run(cols, q)
    assert_same(ctx.table(cols).run(q), want, ctx_msg=f"{groups} {hashed} {aggs}")
    s = ctx.aggregate(q)  # no statistics: sums compensated add by add
    s.push(cols)
    assert_same(s.finish(), want, ctx_msg=f"stream {groups} {hashed} {aggs}")


@pytest.mark.parametrize("aggs", QUERIES)
@pytest.mark.parametrize("n", [1, 31, 257, 150_001])
def test_no_group_by(ctx, n, aggs):
    cols = columns(n, 4, n, False)
    q = QueryDescriptor(filters=[FilterOp("f", "gte", 0.0)], aggregates=QUERIES[aggs])
    assert_same(ctx.table(cols).run(q), oracle.run(cols, q), ctx_msg=f"{n} {aggs}")


def test_null_keys_deterministic_and_forced_launch_shapes(ctx):
    cols = columns(150_001, 40, 5, False)
    cols["key"] = Column(cols["key"], np.random.default_rng(6).random(150_001) < 0.05)
    # (a deterministic sum is exact to a unit of the column's largest cell, so not to 1e-12 of a group of tiny cells)
    for flags, aggs in ((0, "mixed"), (A.QM_FLAG_DETERMINISTIC, "all")):
        q = QueryDescriptor(group_by=["key"], aggregates=QUERIES[aggs], flags=flags)
        want = oracle.run(cols, q)
        t = ctx.table(cols)
        try:
            for tuning in ({}, {"dedupe": 1}, {"local_slots": -1}, {"local_slots": 64}, {"partitioned": 1}):
                ctx.set_tuning(**tuning)
                assert_same(t.run(q), want, ctx_msg=f"{flags} {tuning}")
        finally:
            ctx.set_tuning()
