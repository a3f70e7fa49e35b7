"""Queries whose result one block finishes, and tables of few rows scanned in
short tiles: row counts around a tile, a block and the rows-per-lane rule,
slot counts around the one-block limit, hashed / dense / NULL keys, no GROUP BY,
nothing selected, all-NULL outputs; against the oracle (helpers.assert_same)."""
import numpy as np
import pytest

import oracle
from querymode_b200 import _abi as A
from querymode_b200.engine import Column
from querymode_b200.query import AggregateOp, FilterOp, QueryDescriptor
from tests.helpers import assert_same

pytestmark = pytest.mark.gpu

AGGS = [AggregateOp("sum", "x"), AggregateOp("min", "x"), AggregateOp("count", "x"), AggregateOp("avg", "i"),
        AggregateOp("sum", "l"), AggregateOp("count", "*")]


def columns(n, groups, kind, seed):
    rng = np.random.default_rng(seed)
    idx = rng.integers(0, groups, n)
    key = idx.astype(np.int64)
    if kind == "hashed":
        key = rng.integers(-2**62, 2**62, groups)[idx]
        key[idx == 0] = -2**63  # the empty-slot sentinel
    x = Column(rng.normal(size=n), (rng.random(n) < 0.1) | (idx == 1))
    return {"key": Column(key, rng.random(n) < 0.05) if kind == "nullable" else key, "x": x,
            "i": rng.integers(-100, 100, n).astype(np.int32), "l": rng.integers(-2**63, 2**63, n, dtype=np.int64),
            "b": rng.integers(0, 5, n).astype(np.int32)}


def check(ctx, cols, q, msg):
    want = oracle.run(cols, q)
    t = ctx.table(cols)
    for _ in range(2):
        got = t.run(q)
        assert_same(got, want, ctx_msg=msg)
    return got


@pytest.mark.parametrize("kind", ["dense", "nullable", "hashed", "none"])
@pytest.mark.parametrize("n", [1, 31, 32, 33, 511, 513, 10_007, 151_552, 151_553, 303_105, 606_209])
def test_row_counts(ctx, n, kind):
    cols = columns(n, 13, kind, n)
    q = QueryDescriptor(filters=[FilterOp("i", "lt", 60)], filter_groups=[[FilterOp("x", "gt", -0.5)], [FilterOp("b", "eq", 2)]],
                        group_by=None if kind == "none" else ["key"], aggregates=AGGS)
    check(ctx, cols, q, f"{n} {kind}")


@pytest.mark.parametrize("kind", ["dense", "nullable", "hashed"])
@pytest.mark.parametrize("groups", [1, 2, 480, 1022, 1023, 1024, 1025, 2049])
def test_slot_counts(ctx, groups, kind):
    cols = columns(30_000, groups, kind, groups)
    check(ctx, cols, QueryDescriptor(group_by=["key"], aggregates=AGGS), f"{groups} {kind}")


@pytest.mark.parametrize("kind", ["dense", "hashed", "none"])
def test_nothing_selected_and_two_keys(ctx, kind):
    cols = columns(5_000, 9, kind, 3)
    by = None if kind == "none" else ["key"]
    check(ctx, cols, QueryDescriptor(filters=[FilterOp("i", "gt", 98), FilterOp("b", "eq", 7)], group_by=by, aggregates=AGGS), kind)
    if kind == "dense":
        got = check(ctx, cols, QueryDescriptor(group_by=["key", "b"], aggregates=AGGS, flags=A.QM_FLAG_DETERMINISTIC), kind)
        assert got.stats.rows_selected == 5_000 and got.stats.groups == got.n_rows
