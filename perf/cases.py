"""The work that programs built on this library spend their time in, as measurable cases.

Every case is one call (or one begin / push / finish sequence) through the public entry points
of `querymode_b200.engine`: filter -> GROUP BY over tables resident in HBM, from a dashboard tile
of ten thousand rows to 200 million rows, the batched launch, streamed host batches, page ingest
and the filter-only selection.  Schemas, sizes and distributions are those of
`querymode_b200.datagen` and `bench.py`, made on the GPU from a seed.

    listed()             the cases
    draw(rng)            one more case of the same ranges
    prepare(case, seed)  inputs, tables and lowered queries a program holds before the call
    run(state)           one pass; the whole result, column by column
    work(case)           bytes and operations the pass cannot do without
    exact(case, seed)    the result in 64 bits by plain torch / numpy
"""
import math
import random

import numpy as np
import torch

from querymode_b200 import _abi as A
from querymode_b200.engine import Column, Context, PageTable
from querymode_b200.query import AggregateOp, CQuery, FilterOp, QueryDescriptor

YEAR_START_MS = 1_704_067_200_000  # 2024-01-01T00:00:00Z
DAY_MS = 86_400_000
PAGE_ROWS = 10_000  # rows of a scan page, as the files the reference benchmarks hold them

_context = None


def _ctx():
    """The program's context: one per process, kept for all its tables."""
    global _context
    if _context is None:
        _context = Context(0)
    return _context


def listed():
    return [
        # a dashboard tile: two small integer keys over a table of a few pages; launches and host work
        {"name": "rollup_10k", "kind": "rollup", "rows": 10_007},
        # the interactive roll-up of an in-memory table
        {"name": "orders_1m", "kind": "orders", "rows": 1_000_000},
        # the same over a fact table: few groups, many rows
        {"name": "orders_200m", "kind": "orders", "rows": 200_000_000},
        # the headline scan: a month of a year of events, per user
        {"name": "events_100m", "kind": "events", "rows": 100_000_000, "keys": 65_536, "days": 30},
        # a rare flag over wide keys: a million groups out of a long scan
        {"name": "wide_200m_filtered", "kind": "wide", "rows": 200_000_000, "keys": 1 << 24, "filtered": True},
        # a full roll-up of wide keys: 16.7M groups, a result of hundreds of megabytes
        {"name": "wide_200m_all", "kind": "wide", "rows": 200_000_000, "keys": 1 << 24, "filtered": False},
        # totals of nullable columns under an OR filter, no GROUP BY, an odd number of rows
        {"name": "totals_5m_nulls", "kind": "totals", "rows": 5_000_011},
        # the largest groups of hashed 64-bit keys: aggregate, ORDER BY, LIMIT
        {"name": "top_20m", "kind": "keyed", "rows": 20_000_003, "card": 500_000, "key64": True, "percent": 60, "limit": 100, "exact_sum": False},
        # sixteen tables' queries of mixed size in one batched launch
        {"name": "batch_16", "kind": "batch", "queries": 16, "rows_hi": 8_000_000, "card_hi": 200_000, "shapes": 3},
        # the operator interface: host batches pushed one after another, then the result
        {"name": "stream_1m", "kind": "stream", "rows": 1_000_003, "batch_rows": 65_536, "card": 1_000, "nulls": False},
        # a scan's pages from page-locked host memory (plain, nullable, narrow, Parquet dictionary), then a query
        {"name": "pages_10m", "kind": "pages", "rows": 10_000_000, "regions": 16, "pinned": True},
        # the filter-only operator: a selection vector back to the host
        {"name": "select_30m", "kind": "select", "rows": 30_000_001, "days": 30},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _card(rng, lo, hi, selected):
    """Keys of a column, each met four times or more by the selected rows."""
    return _log(rng, lo, max(lo + 1, min(hi, selected / 4)))


def draw(rng):
    kind = rng.choice(["rollup", "orders", "events", "wide", "totals", "keyed", "batch", "stream", "pages", "select"])
    if kind == "rollup":
        return {"kind": kind, "rows": _log(rng, 1_000, 200_000)}
    if kind == "orders":
        return {"kind": kind, "rows": _log(rng, 100_000, 200_000_000)}
    if kind == "events":
        rows, days = _log(rng, 100_000, 100_000_000), rng.randint(1, 365)
        return {"kind": kind, "rows": rows, "keys": _card(rng, 256, 65_536, rows * days / 365 * 0.9), "days": days}
    if kind == "wide":
        return {"kind": kind, "rows": _log(rng, 1_000_000, 200_000_000), "keys": _log(rng, 1 << 16, 1 << 24), "filtered": rng.random() < 0.5}
    if kind == "totals":
        return {"kind": kind, "rows": _log(rng, 10_000, 5_000_011)}
    if kind == "keyed":
        rows, percent = _log(rng, 10_000, 50_000_000), rng.randint(1, 90)
        return {"kind": kind, "rows": rows, "card": _card(rng, 4, 1_000_000, rows * percent / 100), "key64": rng.random() < 0.5,
                "percent": percent, "limit": rng.choice([0, 0, 10, 100]), "exact_sum": rng.random() < 0.25}
    if kind == "batch":
        return {"kind": kind, "queries": rng.randint(2, 16), "rows_hi": _log(rng, 100_000, 8_000_000), "card_hi": _log(rng, 1_000, 200_000),
                "shapes": rng.randint(0, 1 << 30)}
    if kind == "stream":
        rows = _log(rng, 10_000, 2_000_000)
        return {"kind": kind, "rows": rows, "batch_rows": _log(rng, 4_096, 262_144), "card": _card(rng, 4, 100_000, rows / 2), "nulls": rng.random() < 0.5}
    if kind == "pages":
        return {"kind": kind, "rows": _log(rng, 100_000, 10_000_000), "regions": rng.choice([3, 16, 100, 1_000]), "pinned": rng.random() < 0.5}
    return {"kind": kind, "rows": _log(rng, 10_000, 30_000_001), "days": rng.randint(1, 60)}


# ---- inputs ------------------------------------------------------------------------------------


def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    return g


def _int(g, lo, hi, n, dtype):
    return torch.randint(lo, hi, (n,), generator=g, device="cuda", dtype=dtype)


def _uniform(g, n):
    return torch.rand(n, generator=g, device="cuda", dtype=torch.float64)


def _normal(g, n):
    return torch.randn(n, generator=g, device="cuda", dtype=torch.float64)


def _rows(g, n, count):
    """`count` different rows of n."""
    return torch.randperm(n, generator=g, device="cuda")[:count]


def _zipf(g, n, keys):
    """Keys with P(k) ~ (k + 1)^-1.1 under a random permutation of the key values."""
    w = torch.arange(1, keys + 1, device="cuda", dtype=torch.float64) ** -1.1
    cdf = torch.cumsum(w, 0)
    cdf /= cdf[-1].clone()
    perm = torch.randperm(keys, generator=g, device="cuda")
    out = torch.empty(n, device="cuda", dtype=torch.int64)
    for i in range(0, n, 1 << 25):
        m = min(1 << 25, n - i)
        out[i:i + m] = perm[torch.searchsorted(cdf, _uniform(g, m), right=True).clamp_(max=keys - 1)]
    return out


def _keyed_columns(g, rows, card, key64):
    """`card` keys, each with at least one row that the filter keeps: a result's size is the case's, not the seed's."""
    idx, f = _int(g, 0, card, rows, torch.int64), _int(g, 0, 10_000, rows, torch.int32)
    at = _rows(g, rows, card)
    idx[at] = torch.arange(card, device="cuda")
    f[at] %= 50
    if key64:
        key = _int(g, -(1 << 62), 1 << 62, card, torch.int64)[idx]
    else:
        key = idx.to(torch.int32)
    return {"key": key, "f": f, "v": torch.exp(_normal(g, rows))}


def _batch_specs(case):
    rng = random.Random(case["shapes"])
    specs = []
    for _ in range(case["queries"]):
        rows, percent = _log(rng, 10_000, case["rows_hi"]), rng.randint(1, 90)
        specs.append({"rows": rows, "card": _card(rng, 4, case["card_hi"], rows * percent / 100), "key64": rng.random() < 0.5, "percent": percent})
    return specs


def _columns(case, seed):
    """The case's columns, on the GPU."""
    g, n, kind = _gen(seed), case["rows"], case["kind"]
    if kind == "rollup":
        return {"region": _int(g, 0, 4, n, torch.int32), "category": _int(g, 0, 3, n, torch.int32),
                "amount": _int(g, 0, 1_000, n, torch.int32), "score": _int(g, 0, 997, n, torch.int32).double() / 10.0}
    if kind == "orders":
        return {"status": _int(g, 0, 3, n, torch.int32), "region": _int(g, 0, 16, n, torch.int32), "amount": torch.exp(3.0 + _normal(g, n))}
    if kind == "events":
        c = {"key": _zipf(g, n, case["keys"]), "qty": _int(g, 1, 101, n, torch.int32), "price": _uniform(g, n) * 1000.0,
             "ts": _int(g, YEAR_START_MS, YEAR_START_MS + 365 * DAY_MS, n, torch.int64)}
        at = _rows(g, n, case["keys"])  # every key has an event in the window
        t0, t1 = _window(case["days"])
        c["key"][at] = torch.arange(case["keys"], device="cuda")
        c["ts"][at] = _int(g, t0, t1, len(at), torch.int64)
        c["qty"][at] = _int(g, 11, 101, len(at), torch.int32)
        return c
    if kind == "wide":
        # n / 100 flagged rows, half of them with a positive value; as many different keys as uniform draws give the
        # rows that are kept
        flagged = _rows(g, n, n // 100)
        kept = flagged[:n // 200] if case["filtered"] else _rows(g, n, n)
        flag = torch.zeros(n, device="cuda", dtype=torch.int32)
        flag[flagged] = 1
        val = _normal(g, n) * 1e3
        val[flagged[:n // 200]] = val[flagged[:n // 200]].abs() + 1e-9
        val[flagged[n // 200:]] = -val[flagged[n // 200:]].abs()
        distinct = int(round(_groups(case["keys"], len(kept))))
        some = torch.randperm(case["keys"], generator=g, device="cuda")[:distinct]
        key = _int(g, 0, case["keys"], n, torch.int64)
        key[kept] = some[torch.cat([torch.arange(distinct, device="cuda"), _int(g, 0, distinct, len(kept) - distinct, torch.int64)])]
        return {"key": key, "val": val, "flag": flag}
    if kind == "totals":
        return {"a": _normal(g, n).float(), "a_null": torch.rand(n, generator=g, device="cuda") < 0.02,
                "b": _int(g, -500, 500, n, torch.int32), "b_null": torch.rand(n, generator=g, device="cuda") < 0.05,
                "c": _uniform(g, n) * 1000.0}
    if kind == "keyed":
        return _keyed_columns(g, n, case["card"], case["key64"])
    if kind == "stream":
        c = _keyed_columns(g, n, case["card"], False)
        if case["nulls"]:
            c["v_null"] = (torch.rand(n, generator=g, device="cuda") < 0.01) & (c["f"] >= 50)
        return c
    if kind == "pages":
        return {"key": _int(g, 0, 4_096, n, torch.int64), "price": _uniform(g, n) * 1000.0,
                "price_null": torch.rand(n, generator=g, device="cuda") < 0.01, "qty": _int(g, 1, 101, n, torch.int16),
                "region": _int(g, 0, case["regions"], n, torch.int32)}
    c = {"ts": _int(g, YEAR_START_MS, YEAR_START_MS + 365 * DAY_MS, n, torch.int64), "qty": _int(g, 1, 101, n, torch.int32)}
    # as many rows pass as the window's share of the year says, whatever the seed: a few are moved in or out
    t0, t1 = _window(case["days"])
    passing = (c["ts"] >= t0) & (c["ts"] < t1) & (c["qty"] > 10)
    over = int(passing.sum()) - _passing(case)
    if over:
        rows = (passing if over > 0 else ~passing).nonzero().reshape(-1)
        rows = rows[_rows(g, len(rows), abs(over))]
        c["ts"][rows] = t0 - 1 if over > 0 else t0
        c["qty"][rows] = 50
    return c


def _passing(case):
    return int(case["rows"] * case["days"] / 365 * 0.9)


def _window(days):
    t0 = YEAR_START_MS + min(100, 365 - days) * DAY_MS
    return t0, t0 + days * DAY_MS


def _threshold(percent):
    return percent * 100


def _aggs(*specs):
    return [AggregateOp(fn, col) for fn, col in specs]


def _query(case):
    kind = case["kind"]
    if kind == "rollup":
        return QueryDescriptor(filters=[FilterOp("amount", "gte", 100)], group_by=["region", "category"],
                               aggregates=_aggs(("sum", "amount"), ("count", "*"), ("avg", "score")))
    if kind == "orders":
        return QueryDescriptor(filters=[FilterOp("status", "eq", 1)], group_by=["region"], aggregates=_aggs(("sum", "amount"), ("count", "*")))
    if kind == "events":
        t0, t1 = _window(case["days"])
        return QueryDescriptor(filters=[FilterOp("ts", "gte", t0), FilterOp("ts", "lt", t1), FilterOp("qty", "gt", 10)], group_by=["key"],
                               aggregates=_aggs(("sum", "price"), ("sum", "qty"), ("min", "price"), ("max", "price"), ("count", "*"), ("avg", "price")))
    if kind == "wide":
        return QueryDescriptor(filters=[FilterOp("flag", "eq", 1), FilterOp("val", "gt", 0)] if case["filtered"] else [], group_by=["key"],
                               aggregates=_aggs(("sum", "val"), ("count", "*")))
    if kind == "totals":
        return QueryDescriptor(filters=[FilterOp("c", "lt", 900.0)], filter_groups=[[FilterOp("a", "gt", 0.0)], [FilterOp("b", "between", [0, 250])]],
                               aggregates=_aggs(("sum", "a"), ("min", "a"), ("max", "a"), ("count", "a"), ("avg", "b"), ("sum", "c"), ("count", "*")))
    if kind == "keyed":
        q = QueryDescriptor(filters=[FilterOp("f", "lt", _threshold(case["percent"]))], group_by=["key"],
                            aggregates=_aggs(("sum", "v"), ("count", "*"), ("min", "v"), ("max", "v"), ("avg", "v")),
                            flags=A.QM_FLAG_DETERMINISTIC if case["exact_sum"] else 0)
        if case["limit"]:
            q.sort_column, q.sort_desc, q.limit = "sum_v", True, case["limit"]
        return q
    if kind == "batch":  # one member of the batch (case: its spec)
        raise ValueError("a batch has a query per table")
    if kind == "stream":
        return QueryDescriptor(filters=[FilterOp("f", "lt", 5_000)], group_by=["key"], aggregates=_aggs(("sum", "v"), ("count", "*"), ("max", "v")))
    if kind == "pages":
        return QueryDescriptor(filters=[FilterOp("qty", "gt", 10)], group_by=["region"],
                               aggregates=_aggs(("sum", "price"), ("count", "price"), ("avg", "qty"), ("max", "key")))
    t0, t1 = _window(case["days"])
    return QueryDescriptor(filters=[FilterOp("ts", "gte", t0), FilterOp("ts", "lt", t1), FilterOp("qty", "gt", 10)])


def _batch_query(spec):
    return QueryDescriptor(filters=[FilterOp("f", "lt", _threshold(spec["percent"]))], group_by=["key"],
                           aggregates=_aggs(("sum", "v"), ("count", "*"), ("max", "v")))


# ---- scan pages --------------------------------------------------------------------------------


def _zigzag(v):
    """A Thrift compact i32."""
    v = (v << 1) ^ (v >> 31)
    out = bytearray()
    while v >= 0x80:
        out.append((v & 0x7F) | 0x80)
        v >>= 7
    out.append(v)
    return bytes(out)


def _page_header(page_type, size, sub_delta, fields):
    """A Parquet page header: type, sizes, and the page type's own struct of i32 fields."""
    h = b"\x15" + _zigzag(page_type) + b"\x15" + _zigzag(size) + b"\x15" + _zigzag(size)
    return h + bytes([(sub_delta << 4) | 0x0C]) + b"".join(b"\x15" + _zigzag(f) for f in fields) + b"\x00\x00"


def _dictionary_chunk(codes, entries):
    """A Parquet column chunk: a dictionary page, then v2 data pages of bit-packed indices."""
    width = max(1, (entries - 1).bit_length())
    values = np.arange(entries, dtype=np.int32).tobytes()
    parts = [_page_header(2, len(values), 4, [entries, 0]) + values]
    for i in range(0, len(codes), PAGE_ROWS):
        c = codes[i:i + PAGE_ROWS]
        groups = (len(c) + 7) // 8
        padded = np.zeros(groups * 8, dtype="<u2")
        padded[:len(c)] = c
        bits = np.unpackbits(padded.view(np.uint8).reshape(-1, 2), axis=1, bitorder="little")[:, :width]
        run, head = np.packbits(bits.reshape(-1), bitorder="little").tobytes(), bytearray()
        h = (groups << 1) | 1
        while h >= 0x80:
            head.append((h & 0x7F) | 0x80)
            h >>= 7
        head.append(h)
        body = bytes([width]) + bytes(head) + run
        # num_values, num_nulls, num_rows, encoding RLE_DICTIONARY, no definition or repetition levels
        parts.append(_page_header(3, len(body), 5, [len(c), 0, len(c), 8, 0, 0]) + body)
    return np.frombuffer(b"".join(parts), dtype=np.uint8)


def _nullable_pages(values, nulls, starts, counts):
    """Pages of a validity bitmap and the non-NULL values behind it."""
    parts, lengths, null_counts = [], [], []
    for a, c in zip(starts, counts):
        m = nulls[a:a + c]
        parts += [np.packbits(~m, bitorder="little"), values[a:a + c][~m].view(np.uint8)]
        lengths.append(parts[-2].nbytes + parts[-1].nbytes)
        null_counts.append(int(m.sum()))
    return np.concatenate(parts), np.array(lengths, dtype=np.int64), np.array(null_counts)


def _page_columns(case, cols):
    c = {k: v.cpu().numpy() for k, v in cols.items()}
    n = case["rows"]
    starts = np.arange(0, n, PAGE_ROWS, dtype=np.int64)
    counts = np.minimum(PAGE_ROWS, n - starts)

    def held(buf):
        buf = np.ascontiguousarray(buf).view(np.uint8)
        return torch.from_numpy(buf.copy()).pin_memory().numpy() if case["pinned"] else buf

    price, lengths, null_counts = _nullable_pages(c["price"], c["price_null"], starts, counts)
    region = _dictionary_chunk(c["region"], case["regions"])
    return [
        ("key", A.QM_I64, PageTable(held(c["key"]), starts * 8, counts * 8, counts)),
        ("price", A.QM_F64, PageTable(held(price), np.concatenate([[0], np.cumsum(lengths)[:-1]]), lengths, counts, null_counts)),
        ("qty", A.QM_I32, PageTable(held(c["qty"]), starts * 2, counts * 2, counts), A.QM_PT_INT16),
        ("region", A.QM_I32, PageTable(held(region), np.array([0]), np.array([region.nbytes]), np.array([n]), parquet=np.array([1]))),
    ]


# ---- the calls ---------------------------------------------------------------------------------


def prepare(case, seed):
    ctx, kind = _ctx(), case["kind"]
    state = {"kind": kind, "ctx": ctx}
    if kind == "batch":
        g = _gen(seed)
        tables, queries = [], []
        for s in _batch_specs(case):
            cols = _keyed_columns(g, s["rows"], s["card"], s["key64"])
            torch.cuda.synchronize()
            tables.append(ctx.table(cols))
            queries.append(_batch_query(s))
        state["batch"] = ctx.batch(tables, queries)
        return state
    cols = _columns(case, seed)
    state["query"] = CQuery(_query(case))
    if kind == "totals":
        h = {k: v.cpu().numpy() for k, v in cols.items()}
        cols = {"a": Column(h["a"], h["a_null"]), "b": Column(h["b"], h["b_null"]), "c": h["c"]}
    if kind == "stream":
        h = {k: v.cpu().numpy() for k, v in cols.items()}
        state["query"] = _query(case)
        state["batches"] = []
        for i in range(0, case["rows"], case["batch_rows"]):
            b = {k: h[k][i:i + case["batch_rows"]] for k in ("key", "f", "v")}
            if case["nulls"]:
                b["v"] = Column(b["v"], h["v_null"][i:i + case["batch_rows"]])
            state["batches"].append(b)
        return state
    if kind == "pages":
        state["pages"] = _page_columns(case, cols)
        return state
    torch.cuda.synchronize()
    if kind == "select":
        state["columns"], state["query"] = cols, _query(case)
        return state
    state["table"] = ctx.table(cols)
    return state


def _result(r):
    """A result's columns (and NULL flags, where a column has NULLs), as the program reads them."""
    out = {}
    for c in r.columns:
        out[c.name] = c.values
        if c.nulls is not None:
            out[c.name + "_null"] = c.nulls
    return out


def run(state):
    kind = state["kind"]
    if kind == "batch":
        return [_result(r) for r in state["batch"].run()]
    if kind == "stream":
        s = state["ctx"].aggregate(state["query"])
        for b in state["batches"]:
            s.push(b)
        r = _result(s.finish())
        s.close()
        return r
    if kind == "pages":
        t = state["ctx"].table_from_pages(state["pages"])
        r = _result(t.run(state["query"]))
        t.close()
        return r
    if kind == "select":
        return state["ctx"].filter_select(state["columns"], state["query"])
    return _result(state["table"].run(state["query"]))


# ---- what a pass cannot do without ----------------------------------------------------------------


def _groups(card, selected):
    """Groups expected when `selected` rows fall on `card` equally likely keys."""
    return card * -math.expm1(-selected / card)


def work(case):
    """Each referenced column read once, the result written once; one operation per predicate term
    and row, and one per aggregate and selected row."""
    kind = case["kind"]
    if kind == "batch":
        b = f = 0.0
        for s in _batch_specs(case):
            sel = s["rows"] * s["percent"] / 100
            b += s["rows"] * ((8 if s["key64"] else 4) + 12) + _groups(s["card"], sel) * ((8 if s["key64"] else 4) + 24)
            f += s["rows"] + 3 * sel
        return {"bytes": b, "flops": f}
    n = case["rows"]
    if kind == "rollup":
        return {"bytes": n * 20 + 12 * 32, "flops": n + 3 * 0.9 * n}
    if kind == "orders":
        return {"bytes": n * 16 + 16 * 20, "flops": n + 2 * n / 3}
    if kind == "events":
        sel = n * case["days"] / 365 * 0.9
        return {"bytes": n * 28 + _groups(case["keys"], sel) * 56, "flops": 3 * n + 6 * sel}
    if kind == "wide":
        sel = n * 0.005 if case["filtered"] else n
        return {"bytes": n * (20 if case["filtered"] else 16) + _groups(case["keys"], sel) * 24, "flops": 2 * n + 2 * sel}
    if kind == "totals":
        return {"bytes": n * (16 + 0.25) + 56, "flops": 4 * n + 7 * 0.55 * n}
    if kind == "keyed":
        sel, k = n * case["percent"] / 100, 8 if case["key64"] else 4
        g = _groups(case["card"], sel)
        return {"bytes": n * (k + 12) + (min(case["limit"], g) if case["limit"] else g) * (k + 40), "flops": n + 5 * sel}
    if kind == "stream":
        return {"bytes": n * (16 + (0.125 if case["nulls"] else 0)) + case["card"] * 28, "flops": n + 1.5 * n}
    if kind == "pages":
        return {"bytes": n * (8 + 7.92 + 0.125 + 2 + max(1, (case["regions"] - 1).bit_length()) / 8) + case["regions"] * 36, "flops": n + 3.6 * n}
    return {"bytes": n * 12 + _passing(case) * 4, "flops": 3 * n}


# ---- the results in 64 bits ------------------------------------------------------------------------


def _pick(x, at):
    return x[at].cpu().numpy()


class _Grouped:
    """Aggregates per group id over the rows of a mask, groups in the order their first rows come."""

    def __init__(self, ids, n_ids, mask):
        rows = torch.arange(len(ids), device="cuda") if mask is None else mask.nonzero().reshape(-1)
        self.rows, self.ids, self.n = rows, ids[rows], n_ids
        first = torch.full((n_ids,), 1 << 62, device="cuda", dtype=torch.int64).scatter_reduce_(0, self.ids, rows, "amin")
        self.count = torch.bincount(self.ids, minlength=n_ids)
        seen = (self.count > 0).nonzero().reshape(-1)
        self.order = seen[torch.argsort(first[seen])]
        self.first = first[self.order]

    def sum(self, x, valid=None):
        v = x[self.rows].double()
        if valid is not None:
            v = torch.where(valid[self.rows], v, torch.zeros_like(v))
        return torch.zeros(self.n, device="cuda", dtype=torch.float64).index_add_(0, self.ids, v)

    def ext(self, x, how):
        start = -math.inf if how == "amax" else math.inf
        return torch.full((self.n,), start, device="cuda", dtype=torch.float64).scatter_reduce_(0, self.ids, x[self.rows].double(), how)

    def out(self, x):
        return _pick(x, self.order)


def _dense(key):
    uniq, ids = torch.unique(key, return_inverse=True)
    return ids, len(uniq)


def exact(case, seed):
    kind = case["kind"]
    if kind == "batch":
        g, out = _gen(seed), []
        for s in _batch_specs(case):
            c = _keyed_columns(g, s["rows"], s["card"], s["key64"])
            ids, n = _dense(c["key"])
            gr = _Grouped(ids, n, c["f"] < _threshold(s["percent"]))
            out.append({"key": _pick(c["key"], gr.first), "sum_v": gr.out(gr.sum(c["v"])), "count_*": gr.out(gr.count), "max_v": gr.out(gr.ext(c["v"], "amax"))})
        return out
    c = _columns(case, seed)
    if kind == "rollup":
        gr = _Grouped((c["region"] * 3 + c["category"]).long(), 12, c["amount"] >= 100)
        return {"region": _pick(c["region"], gr.first), "category": _pick(c["category"], gr.first), "sum_amount": gr.out(gr.sum(c["amount"])),
                "count_*": gr.out(gr.count), "avg_score": gr.out(gr.sum(c["score"]) / gr.count)}
    if kind == "orders":
        gr = _Grouped(c["region"].long(), 16, c["status"] == 1)
        return {"region": _pick(c["region"], gr.first), "sum_amount": gr.out(gr.sum(c["amount"])), "count_*": gr.out(gr.count)}
    if kind == "events":
        t0, t1 = _window(case["days"])
        gr = _Grouped(c["key"], case["keys"], (c["ts"] >= t0) & (c["ts"] < t1) & (c["qty"] > 10))
        total = gr.sum(c["price"])
        return {"key": _pick(c["key"], gr.first), "sum_price": gr.out(total), "sum_qty": gr.out(gr.sum(c["qty"])),
                "min_price": gr.out(gr.ext(c["price"], "amin")), "max_price": gr.out(gr.ext(c["price"], "amax")), "count_*": gr.out(gr.count),
                "avg_price": gr.out(total / gr.count)}
    if kind == "wide":
        gr = _Grouped(c["key"], case["keys"], (c["flag"] == 1) & (c["val"] > 0) if case["filtered"] else None)
        return {"key": _pick(c["key"], gr.first), "sum_val": gr.out(gr.sum(c["val"])), "count_*": gr.out(gr.count)}
    if kind == "totals":
        a, b, av, bv = c["a"].double(), c["b"].double(), ~c["a_null"], ~c["b_null"]
        m = (c["c"] < 900.0) & ((av & (a > 0)) | (bv & (b >= 0) & (b <= 250)))
        aa, bb = a[m & av], b[m & bv]
        one = lambda v: np.array([float(v)])  # noqa: E731
        return {"sum_a": one(aa.sum()), "min_a": one(aa.min()), "max_a": one(aa.max()), "count_a": np.array([len(aa)]), "avg_b": one(bb.mean()),
                "sum_c": one(c["c"][m].sum()), "count_*": np.array([int(m.sum())])}
    if kind == "keyed":
        ids, n = _dense(c["key"])
        gr = _Grouped(ids, n, c["f"] < _threshold(case["percent"]))
        total = gr.sum(c["v"])
        out = {"key": _pick(c["key"], gr.first), "sum_v": gr.out(total), "count_*": gr.out(gr.count), "min_v": gr.out(gr.ext(c["v"], "amin")),
               "max_v": gr.out(gr.ext(c["v"], "amax")), "avg_v": gr.out(total / gr.count)}
        if case["limit"]:
            top = np.argsort(-out["sum_v"], kind="stable")[:case["limit"]]
            out = {k: v[top] for k, v in out.items()}
        return out
    if kind == "stream":
        valid = ~c["v_null"] if case["nulls"] else None
        gr = _Grouped(c["key"].long(), case["card"], c["f"] < 5_000)
        held = c["v"] if valid is None else torch.where(valid, c["v"], torch.full_like(c["v"], -math.inf))
        return {"key": _pick(c["key"], gr.first), "sum_v": gr.out(gr.sum(c["v"], valid)), "count_*": gr.out(gr.count), "max_v": gr.out(gr.ext(held, "amax"))}
    if kind == "pages":
        valid = ~c["price_null"]
        gr = _Grouped(c["region"].long(), case["regions"], c["qty"] > 10)
        held = torch.bincount(gr.ids[valid[gr.rows]], minlength=gr.n)
        return {"region": _pick(c["region"], gr.first), "sum_price": gr.out(gr.sum(c["price"], valid)), "count_price": gr.out(held),
                "avg_qty": gr.out(gr.sum(c["qty"]) / gr.count), "max_key": gr.out(gr.ext(c["key"], "amax").long())}
    t0, t1 = _window(case["days"])
    return ((c["ts"] >= t0) & (c["ts"] < t1) & (c["qty"] > 10)).nonzero().reshape(-1).cpu().numpy()
