"""Column statistics (chunks of 8,192 rows, 16-byte loads): row counts around a
chunk and a zone, columns borrowed at unaligned addresses, NaN / Infinity and
extreme integers, through queries whose plans rest on them (dense key ranges,
zone pruning, split sums); against the oracle."""
import numpy as np
import pytest

import oracle
from querymode_b200.query import AggregateOp, FilterOp, QueryDescriptor
from tests.helpers import assert_same

pytestmark = pytest.mark.gpu


def columns(n):
    rng = np.random.default_rng(n)
    x = rng.normal(size=n) * 1e3
    x[rng.random(n) < 0.01] = np.nan
    if n > 9_000:
        x[8_192] = np.inf
    i = rng.integers(-50, 50, n).astype(np.int32)
    i[-1] = 2**31 - 1
    return {"key": (np.arange(n) // 70 - 3).astype(np.int64), "i": i, "x": x, "f": (rng.random(n) - 0.5).astype(np.float32),
            "ts": np.sort(rng.integers(-2**62, 2**62, n)).astype(np.int64)}


@pytest.mark.parametrize("shift", [0, 1])
@pytest.mark.parametrize("n", [1, 8_191, 8_192, 8_193, 65_536, 65_537, 300_001])
def test_plans_from_statistics(ctx, n, shift):
    import torch
    whole = columns(n + shift)
    cols = {k: v[shift:] for k, v in whole.items()}
    held = {k: torch.from_numpy(v).cuda() for k, v in whole.items()}
    torch.cuda.synchronize()
    t = ctx.table({k: v[shift:] for k, v in held.items()})  # shift: not 16-byte aligned
    lo, hi = int(cols["ts"][n // 4]), int(cols["ts"][n // 2])
    for filters in ([], [FilterOp("ts", "gte", lo), FilterOp("ts", "lt", hi)], [FilterOp("x", "gt", 4e3)],
                    [FilterOp("f", "lte", 0.25), FilterOp("i", "lt", 40)]):
        q = QueryDescriptor(filters=filters, group_by=["key"], aggregates=[AggregateOp("sum", "x"), AggregateOp("sum", "f"),
                                                                           AggregateOp("max", "i"), AggregateOp("count", "*")])
        assert_same(t.run(q), oracle.run(cols, q), ctx_msg=f"{n} {shift} {filters}")
