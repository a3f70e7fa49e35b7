"""Page ingest that fails after some columns are already crossing the host link
or being decoded: the error is reported, no later ingest or table is affected,
and the scratch is whole again."""
import numpy as np
import pytest

from querymode_b200 import _abi as A
from querymode_b200.engine import Page, PageTable
from tests.page_util import encode_column

pytestmark = pytest.mark.gpu

N, PAGE = 300_000, 10_000


def column(rng, pinned):
    v = rng.integers(-2**62, 2**62, N, dtype=np.int64)
    buf = v
    if pinned:
        import torch
        buf = torch.from_numpy(v).pin_memory().numpy()
    offs = np.arange(0, N, PAGE, dtype=np.int64) * 8
    return v, PageTable(buf.view(np.uint8), offs, np.full(len(offs), PAGE * 8), np.full(len(offs), PAGE))


@pytest.mark.parametrize("pinned", [True, False])
@pytest.mark.parametrize("at", [1, 2, 3])
@pytest.mark.parametrize("bad", ["rows", "type", "parquet", "name"])
def test_failure_part_way(ctx, bad, at, pinned):
    rng = np.random.default_rng(at)
    cols = [column(rng, pinned) for _ in range(4)]
    good = [(f"c{i}", A.QM_I64, pt) for i, (_, pt) in enumerate(cols)]
    before = ctx.table_from_pages(good)
    broken = {"rows": ("x", A.QM_I64, encode_column(cols[0][0][:N - 1], None, PAGE)), "type": ("x", A.QM_I64, cols[0][1], 99),
              "parquet": ("x", A.QM_I64, [Page(b"\x00" * 40, 5, 0, None, True)]), "name": ("c0", A.QM_I64, cols[0][1])}[bad]
    for _ in range(3):
        with pytest.raises(A.QmError) as e:
            ctx.table_from_pages(good[:at] + [broken] + good[at:])
        assert e.value.status in (A.QM_ERR_INVALID, A.QM_ERR_UNSUPPORTED)
        after = ctx.table_from_pages(good)
        for t in (before, after):
            for i, (v, _) in enumerate(cols):
                got, nulls = t.read_column(f"c{i}")
                assert np.array_equal(got, v) and not nulls.any()
        after.close()
