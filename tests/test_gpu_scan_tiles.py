"""The scan over pairs of tiles (a pruned zone of the table keeps it to them at
any size) and over short tiles, with every kind of filter term: integer ranges
and their complements, float comparisons, NULLs passing or not, OR groups, a
rare first term and a common one, rows ending inside a tile; against the oracle."""
import numpy as np
import pytest

import oracle
from querymode_b200 import _abi as A
from querymode_b200.engine import Column
from querymode_b200.query import AggregateOp, FilterOp, QueryDescriptor
from tests.helpers import assert_same

pytestmark = pytest.mark.gpu

F = FilterOp
TERMS = {
    "range": [F("i", "between", [-20, 70])],
    "outside": [F("i", "not_between", [-20, 70]), F("l", "neq", 5)],
    "rare": [F("flag", "eq", 1), F("x", "gt", 0.0)],
    "floats": [F("x", "lt", 1.0), F("f", "neq", 0.5), F("x", "not_between", [-0.1, 0.1])],
    "nulls": [F("n", "is_not_null"), F("n", "lte", 40)],
    "is null": [F("n", "is_null")],
}
GROUPS = {"none": None, "or": [[F("i", "gt", 80), F("x", "lt", 0.0)], [F("n", "eq", 7)], [F("f", "gte", 0.9)]]}


def columns(n):
    rng = np.random.default_rng(n)
    return {"ts": np.sort(rng.integers(0, 1 << 40, n)).astype(np.int64), "i": rng.integers(-100, 100, n).astype(np.int32),
            "l": rng.integers(0, 10, n).astype(np.int64), "flag": (rng.random(n) < 0.01).astype(np.int32),
            "x": rng.normal(size=n), "f": rng.random(n).astype(np.float32),
            "n": Column(rng.integers(0, 50, n).astype(np.int32), rng.random(n) < 0.3),
            "key": rng.integers(0, 3_000, n).astype(np.int64)}


@pytest.fixture(scope="module")
def tables(ctx):
    made = {}

    def get(n):
        if n not in made:
            cols = columns(n)
            made[n] = (cols, ctx.table(cols))
        return made[n]
    return get


@pytest.mark.parametrize("groups", GROUPS)
@pytest.mark.parametrize("terms", TERMS)
@pytest.mark.parametrize("n,pruned", [(400_123, True), (262_657, True), (400_123, False)])
def test_terms(tables, n, pruned, terms, groups):
    cols, t = tables(n)
    # the sorted column leaves out the table's last quarter: its zones are not scanned
    window = [F("ts", "lt", int(cols["ts"][3 * n // 4]))] if pruned else []
    for flags in (0, A.QM_FLAG_WASM_SCAN_SEMANTICS):
        q = QueryDescriptor(filters=window + TERMS[terms], filter_groups=GROUPS[groups], group_by=["key"], flags=flags,
                            aggregates=[AggregateOp("sum", "x"), AggregateOp("min", "x"), AggregateOp("max", "i"), AggregateOp("count", "*")])
        assert_same(t.run(q), oracle.run(cols, q, threads=8), ctx_msg=f"{n} {pruned} {terms} {groups} {flags}")


@pytest.mark.parametrize("aggs", [[AggregateOp("sum", "x"), AggregateOp("count", "*")],
                                  [AggregateOp("min", "x"), AggregateOp("max", "l"), AggregateOp("max", "x"), AggregateOp("sum", "i")],
                                  [AggregateOp("avg", "n"), AggregateOp("min", "n"), AggregateOp("sum", "l")]])
@pytest.mark.parametrize("groups", [1_200, 90_000, 400_000])
def test_hash_slots_with_words_beside_the_key(ctx, groups, aggs):
    rng = np.random.default_rng(groups)
    n = 400_123
    cols = columns(n)
    cols["key"] = rng.integers(-2**62, 2**62, groups)[rng.integers(0, groups, n)]
    cols["key"][:3] = -2**63  # the empty-slot sentinel
    cols["x"][rng.random(n) < 0.01] = np.nan
    cols["x"][rng.random(n) < 0.01] = -0.0
    cols["key"] = Column(cols["key"], rng.random(n) < 0.001)
    q = QueryDescriptor(filters=[F("i", "lt", 90)], group_by=["key"], aggregates=aggs)
    want = oracle.run(cols, q, threads=8)
    t = ctx.table(cols)
    assert_same(t.run(q), want, ctx_msg=f"{groups}")
    assert_same(ctx.batch([t, t], [q, q]).run()[1], want, ctx_msg=f"batch {groups}")
