"""Borrowed device columns that their owner rewrites between queries: a query
rests on no statistic that an earlier query, which did not need it, left
behind.  Sum, then rewrite, then filter (zone maps); filter, then rewrite, then
GROUP BY (key range); in both orders, against the oracle on the values as they
are."""
import numpy as np
import pytest

import oracle
from querymode_b200.query import AggregateOp, FilterOp, QueryDescriptor
from tests.helpers import assert_same

pytestmark = pytest.mark.gpu

N = 300_001  # five zones


@pytest.mark.parametrize("dtype,first", [(np.float64, "sum"), (np.float32, "sum"), (np.int64, "key"), (np.int32, "key")])
def test_filter_after_rewrite(ctx, dtype, first):
    import torch
    rng = np.random.default_rng(8)
    k, v = rng.integers(0, 9, N).astype(np.int64), np.sort(rng.integers(0, 1000, N)).astype(dtype)
    dv = torch.from_numpy(v.copy()).cuda()
    t = ctx.table({"k": torch.from_numpy(k).cuda(), "v": dv})
    q1 = QueryDescriptor(group_by=["k" if first == "sum" else "v"], aggregates=[AggregateOp("sum", "v"), AggregateOp("count", "*")])
    assert_same(t.run(q1), oracle.run({"k": k, "v": v}, q1))
    v = v[::-1].copy()  # the zones of the old values exclude the rows that pass now
    dv.copy_(torch.from_numpy(v))
    torch.cuda.synchronize()
    q2 = QueryDescriptor(filters=[FilterOp("v", "gte", 900)], group_by=["k"], aggregates=[AggregateOp("count", "*")])
    assert_same(t.run(q2), oracle.run({"k": k, "v": v}, q2))


@pytest.mark.parametrize("dtype", [np.int64, np.int32])
def test_group_by_after_rewrite(ctx, dtype):
    import torch
    rng = np.random.default_rng(9)
    v = rng.integers(0, 50, N).astype(dtype)
    dv = torch.from_numpy(v.copy()).cuda()
    t = ctx.table({"v": dv})
    q1 = QueryDescriptor(filters=[FilterOp("v", "lt", 40)], aggregates=[AggregateOp("count", "*")])
    assert_same(t.run(q1), oracle.run({"v": v}, q1))
    v = (v + 1000).astype(dtype)
    dv.copy_(torch.from_numpy(v))
    torch.cuda.synchronize()
    q2 = QueryDescriptor(group_by=["v"], aggregates=[AggregateOp("count", "*")])
    g = t.run(q2)
    assert_same(g, oracle.run({"v": v}, q2))
    assert g.stats.retries == 0  # planned from the range of the values as they are
