"""ORDER BY ... LIMIT k at the edges of the parallel top k (rows the bound is
taken from: 16,384; list: 262,144; sorted in shared memory: 8,192; largest k:
1,024), against the reference's heap restated (oracle/post.py): the same rows
in the same order, ties, NULL and NaN included."""
import numpy as np
import pytest

from oracle.post import topk_order
from querymode_b200.engine import Column
from querymode_b200.query import AggregateOp, QueryDescriptor

pytestmark = pytest.mark.gpu


def values(kind, n):
    rng = np.random.default_rng(n)
    v = rng.permutation(n).astype(np.float64)  # all different
    nulls = np.zeros(n, bool)
    if kind == "ties":
        v = np.floor(v / max(1, n // 50))
    elif kind == "tie at the edge":
        v[rng.choice(n, n // 2, replace=False)] = 3.0
    elif kind == "rising":
        v = np.sort(v)
    elif kind == "falling":
        v = -np.sort(v)
    elif kind == "few values":
        nulls[rng.choice(n, n - min(n, 40), replace=False)] = True
    elif kind == "nan":
        v[rng.random(n) < 0.3] = np.nan
        v[rng.random(n) < 0.01] = np.inf
    return v, nulls


@pytest.mark.parametrize("kind", ["different", "ties", "tie at the edge", "rising", "falling", "few values", "nan"])
@pytest.mark.parametrize("n,limit,offset", [(1, 5, 0), (50, 50, 0), (5_000, 100, 3), (16_384, 10, 0), (16_385, 1, 0),
                                            (40_000, 1_024, 0), (40_000, 1_024, 1), (300_000, 100, 0)])
def test_topk_edges(ctx, n, limit, offset, kind):
    v, nulls = values(kind, n)
    cols = {"k": np.arange(n, dtype=np.int64) * 7, "v": Column(v, nulls)}
    vals = [None if nulls[i] else float(v[i]) for i in range(n)]
    t = ctx.table(cols)
    for desc in (True, False):
        q = QueryDescriptor(group_by=["k"], aggregates=[AggregateOp("sum", "v", "m")], sort_column="m", sort_desc=desc,
                            limit=limit, offset=offset)
        want = cols["k"][topk_order(vals, desc, limit, offset)]
        assert np.array_equal(t.run(q).column("k").values, want), f"desc={desc}"
