"""Direct tables of more than a million groups whose rows (12 million or more)
outnumber their slots are aggregated window by window in shared memory.  The
shapes below take that route: no, one and two value columns, NULL cells and
keys, both key types and packed keys, a filter, a last window and a last tile
that are not full, and rows that crowd into one window (several chunks merged
into the table).  Keys, first-seen order, COUNT, integer SUM and MIN / MAX
equal the oracle's bit for bit, float SUM / AVG within 1e-12
(tests/helpers.py)."""
import numpy as np
import pytest

import oracle
from querymode_b200.engine import Column
from querymode_b200.query import AggregateOp, FilterOp, QueryDescriptor
from tests.helpers import assert_same

pytestmark = pytest.mark.gpu

SLOTS = 1_300_001
ROWS = 12_000_013


def keys(rng, dtype, base=0, slots=SLOTS, n=ROWS):
    k = rng.integers(0, slots, n) + base
    k[0], k[-1] = base, base + slots - 1  # the whole range
    return k.astype(dtype)


def aggs(*specs):
    return [AggregateOp(f, c) for f, c in specs]


COUNT = (("count", "*"),)
SUM = (("sum", "v"), ("count", "*"))
ONE = (("sum", "v"), ("min", "v"), ("max", "v"), ("avg", "v"), ("count", "*"))
TWO = (("sum", "v"), ("count", "v"), ("sum", "w"), ("max", "w"), ("count", "*"))


@pytest.mark.parametrize("spec,dtype,nulls", [
    (COUNT, np.int32, False), (SUM, np.int64, False), (SUM, np.int32, True), (ONE, np.int64, True),
    (TWO, np.int32, False), (TWO, np.int64, True)], ids=["count", "sum", "sum-null", "one-null", "two", "two-null"])
def test_values_and_keys(ctx, spec, dtype, nulls):
    rng = np.random.default_rng(11)
    null = (lambda p: rng.random(ROWS) < p) if nulls else (lambda p: None)
    key = Column(keys(rng, dtype, -7), null(0.01))
    v = rng.normal(size=ROWS) * 1e3
    v[rng.random(ROWS) < 0.001] = -0.0
    cols = {"key": key, "v": Column(v, null(0.03)), "w": Column(rng.integers(-1000, 1000, ROWS).astype(np.int32), null(0.02))}
    q = QueryDescriptor(group_by=["key"], aggregates=aggs(*spec))
    assert_same(ctx.table(cols).run(q), oracle.run_full(cols, q))


@pytest.mark.parametrize("n", [8_192 * 1_600, 8_192 * 1_600 + 1])
def test_filtered_and_ragged(ctx, n):
    """A filter of scattered rows and one that leaves out whole zones."""
    rng = np.random.default_rng(n)
    cols = {"key": keys(rng, np.int64, 1 << 40, n=n), "v": np.exp(rng.normal(size=n)), "f": rng.integers(0, 1000, n).astype(np.int32),
            "t": np.arange(n, dtype=np.int64)}
    q = QueryDescriptor(filters=[FilterOp("f", "lt", 998), FilterOp("t", "gte", 400_000)], group_by=["key"], aggregates=aggs(*SUM))
    assert_same(ctx.table(cols).run(q), oracle.run_full(cols, q))


def test_non_finite_cells(ctx):
    rng = np.random.default_rng(5)
    v = rng.normal(size=ROWS)
    v[rng.integers(0, ROWS, 300)] = np.inf
    v[rng.integers(0, ROWS, 300)] = -np.inf
    v[rng.integers(0, ROWS, 300)] = np.nan
    cols = {"key": keys(rng, np.int32), "v": v}
    q = QueryDescriptor(group_by=["key"], aggregates=aggs(*ONE))
    assert_same(ctx.table(cols).run(q), oracle.run_full(cols, q))


def test_crowded_window(ctx):
    """Half the rows on 50 keys of one window: its list is aggregated in
    several chunks."""
    rng = np.random.default_rng(6)
    key = keys(rng, np.int64)
    hot = rng.random(ROWS) < 0.5
    key[hot] = 700_000 + rng.integers(0, 50, int(hot.sum()))
    key[0], key[-1] = 0, SLOTS - 1
    cols = {"key": key, "v": rng.normal(size=ROWS) * 1e3, "w": rng.integers(-1000, 1000, ROWS).astype(np.int32)}
    for spec in (SUM, TWO):
        q = QueryDescriptor(group_by=["key"], aggregates=aggs(*spec))
        assert_same(ctx.table(cols).run(q), oracle.run_full(cols, q))


def test_packed_keys(ctx):
    rng = np.random.default_rng(7)
    a, b = rng.integers(0, 1100, ROWS).astype(np.int32), rng.integers(-3, 1197, ROWS).astype(np.int64)
    cols = {"a": Column(a, rng.random(ROWS) < 0.01), "b": b, "v": rng.normal(size=ROWS)}
    q = QueryDescriptor(group_by=["a", "b"], aggregates=aggs(*SUM))
    assert_same(ctx.table(cols).run(q), oracle.run_full(cols, q))
