"""Records of the window route: sized by the rows a filter selects, for every
row when the remembered bound no longer holds (the filter's column was
rewritten), and the route itself taken or not (by its launches) around its
smallest table."""
import numpy as np
import pytest

import oracle
from querymode_b200.engine import Context
from querymode_b200.query import AggregateOp, FilterOp, QueryDescriptor
from tests.helpers import assert_same

pytestmark = pytest.mark.gpu

N, SLOTS = 26_000_003, 1_300_001
Q = QueryDescriptor(filters=[FilterOp("f", "lt", 500)], group_by=["key"], aggregates=[AggregateOp("sum", "v"), AggregateOp("count", "*")])


def columns(n=N, slots=SLOTS):
    rng = np.random.default_rng(4)
    key = rng.integers(0, slots, n)
    key[0], key[-1] = 0, slots - 1
    return {"key": key, "v": rng.random(n), "f": rng.integers(0, 1000, n).astype(np.int32)}


def test_records_of_the_selected_rows():
    import torch
    c = Context(0)
    try:
        held = {k: torch.from_numpy(v).cuda() for k, v in columns().items()}
        torch.cuda.synchronize()
        t = c.table(held)
        c.trim()
        t.run(Q)
        assert N * 16 * 0.4 < c.trim() < N * 16 * 0.6  # 16 bytes a record, half of the rows
    finally:
        c.close()


def test_more_rows_than_the_bound(ctx):
    import torch
    cols = columns()
    held = {k: torch.from_numpy(v).cuda() for k, v in cols.items()}
    torch.cuda.synchronize()
    t = ctx.table(held)
    first = t.run(Q)
    assert_same(first, oracle.run_full(cols, Q))
    cols["f"] = (cols["f"] // 3).astype(np.int32)  # every row passes
    held["f"].copy_(torch.from_numpy(cols["f"]))
    torch.cuda.synchronize()
    got = t.run(Q)
    assert_same(got, oracle.run_full(cols, Q))
    # run again with its direct table, not a hashed one
    assert got.stats.retries == 1 and got.stats.table_capacity == first.stats.table_capacity


@pytest.mark.parametrize("n,slots,taken", [(12_000_000, 1_300_001, True), (11_999_999, 1_300_001, False),
                                           (12_000_000, 900_001, False), (12_000_000, 12_000_001, False)])
def test_route(ctx, n, slots, taken):
    """The windows are four launches; without them (no block-local table) one
    scan, or a pass of it per 64 MB of the table."""
    cols = {k: v for k, v in columns(n, slots).items() if k != "f"}
    q = QueryDescriptor(group_by=["key"], aggregates=Q.aggregates)
    t = ctx.table(cols)
    launches = t.run(q).stats.launches
    try:
        ctx.set_tuning(local_slots=-1)
        plain = t.run(q).stats.launches
    finally:
        ctx.set_tuning()
    passes = 1 if slots * 5 * 8 <= 64 << 20 or n < slots else -(-((slots + 1) * 5 * 8) // (64 << 20))
    assert launches - plain == (4 - passes if taken else 0)
