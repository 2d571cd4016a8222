"""The work that is timed when the operators are made faster: single calls of
the public operators (yallasql_b200.ops) on device-resident tables with the
benchmark's columns and distributions, over the range of sizes they are used
at - from one 4 MB batch to whole 64M-row tables.

listed()             the cases that are always timed
draw(rng)            one more case of the same ranges (rng: random.Random)
prepare(case, seed)  what a program holds before the call: tables, plans, output buffers
run(state)           one pass through the public entry points, outputs whole
work(case)           bytes and operations of one pass that nothing can avoid
exact(case, seed)    the computed outputs in 64 bits, by plain torch
"""
from __future__ import annotations

import math

import torch

from yallasql_b200 import _abi as A
from yallasql_b200 import datagen, ops
from yallasql_b200.expr import Aggregate, And, Arith, Cast, ColumnRef, Compare, Constant, between

RUN_BYTES = 4 << 20  # one out-of-core batch
CATEGORY_BYTES = len(datagen.CATEGORIES[0])


def listed() -> list[dict]:
    return [
        # one 4 MB batch of the engine's pull loop: latency and launches
        {"name": "filter_agg_batch", "kind": "filter_agg", "rows": 15_616, "nulls": False},
        # the plain WHERE + aggregate query on its 1M-row table
        {"name": "filter_agg_1m", "kind": "filter_agg", "rows": 1_000_000, "nulls": False},
        # WHERE + SELECT list over a large table of ragged length, one column with NULLs
        {"name": "filter_project_24m", "kind": "filter_project", "rows": 24_000_001, "nulls": True},
        # ORDER BY of one in-memory table by a nullable date, every column moved
        {"name": "sort_date_1m", "kind": "sort", "rows": 1_000_003, "key": "updated_at", "desc": False, "nulls": True},
        # ORDER BY of a whole table that arrived as 4 MB batches: the largest call
        {"name": "order_by_64m", "kind": "order_by", "rows": 64_000_000, "key": "key", "desc": True, "dist": "uniform"},
        # star join with the date dimension, fused with its SUM
        {"name": "star_agg_60m", "kind": "star_agg", "rows": 60_000_000},
        # fact rows joined to a customer dimension, columns of both sides materialised
        {"name": "join_2m_300k", "kind": "join", "rows": 2_000_000, "right": 300_000},
        # cross product with an inequality: no hash, every pair compared
        {"name": "cross_lt_20k", "kind": "cross", "rows": 20_000, "right": 20_000},
        # CSV text on the device into columns (ingest), ragged length
        {"name": "csv_scan_2m", "kind": "csv_scan", "rows": 1_999_993},
        # columns back into CSV text (result export)
        {"name": "csv_format_2m", "kind": "csv_format", "rows": 1_999_993},
        # GROUP BY a column of few values, five aggregates
        {"name": "group_by_32m", "kind": "group_by", "rows": 32_000_000, "groups": 11},
        # 64 independent ORDER BY tasks of uneven sizes in one batched call
        {"name": "order_tasks_64", "kind": "order_tasks", "tasks": 64, "lo": 1_000, "hi": 4_000_000},
    ]


def _log(rng, lo: int, hi: int) -> int:
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng) -> dict:
    kind = rng.choice(["filter_agg", "filter_project", "sort", "order_by", "star_agg", "join", "cross", "csv_scan",
                       "csv_format", "group_by", "order_tasks"])
    if kind == "filter_agg":
        return {"kind": kind, "rows": _log(rng, 1_000, 64_000_000), "nulls": rng.random() < 0.3}
    if kind == "filter_project":
        return {"kind": kind, "rows": _log(rng, 10_000, 32_000_000), "nulls": rng.random() < 0.5}
    if kind == "sort":
        return {"kind": kind, "rows": _log(rng, 1_000, 16_000_000),
                "key": rng.choice(["id", "price", "qty", "category", "updated_at"]), "desc": rng.random() < 0.5,
                "nulls": rng.random() < 0.5}
    if kind == "order_by":
        return {"kind": kind, "rows": _log(rng, 1_000_000, 64_000_000), "key": rng.choice(["key", "d"]),
                "desc": rng.random() < 0.5, "dist": rng.choice(["uniform", "zipf", "equal"])}
    if kind == "star_agg":
        return {"kind": kind, "rows": _log(rng, 100_000, 60_000_000)}
    if kind == "join":
        return {"kind": kind, "rows": _log(rng, 20_000, 2_000_000), "right": _log(rng, 2_000, 300_000)}
    if kind == "cross":
        return {"kind": kind, "rows": _log(rng, 500, 20_000), "right": _log(rng, 500, 20_000)}
    if kind in ("csv_scan", "csv_format"):
        return {"kind": kind, "rows": _log(rng, 10_000, 4_000_000)}
    if kind == "group_by":
        return {"kind": kind, "rows": _log(rng, 20_000, 32_000_000), "groups": _log(rng, 2, 500_000)}
    return {"kind": kind, "tasks": rng.randrange(16, 97), "lo": 1_000, "hi": _log(rng, 50_000, 3_000_000)}


# ------------------------------------------------------------------- tables
def _gen(seed: int) -> torch.Generator:
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _randint(g, lo: int, hi: int, n: int, dtype=torch.int32) -> torch.Tensor:
    return torch.randint(lo, hi, (n,), generator=g, device="cuda", dtype=dtype)


def _null_bytes(g, n: int) -> torch.Tensor:
    """One row in 50 is NULL."""
    return (torch.rand(n, generator=g, device="cuda") < 0.02).to(torch.uint8)


def _price(g, n: int) -> torch.Tensor:
    return (torch.rand(n, generator=g, device="cuda") * 999.0 + 1.0).clamp_(max=999.9999)


def _categories(g, n: int) -> torch.Tensor:
    cats = torch.from_numpy(datagen.text_slots(datagen.CATEGORIES)).cuda()
    return cats[_randint(g, 0, len(datagen.CATEGORIES), n, torch.int64)]


SALES = {"id": A.INT64, "price": A.FLOAT32, "qty": A.INT32, "discount": A.INT32, "category": A.TEXT,
         "updated_at": A.DATETIME}


def _order(n: int, seed: int) -> torch.Tensor:
    """A seed's order of rows that are otherwise the same for every seed: how
    many rows a query selects, how many groups or pairs it finds and how long
    its text is are then the case's own and not the seed's."""
    return torch.randperm(n, generator=_gen(seed), device="cuda")


def _sales(n: int, seed: int, null_column: str | None = None, own_prices: bool = True) -> dict:
    """The sales table; with own_prices the prices are the seed's."""
    g, order = _gen(n), _order(n, seed)
    t = {"price": _price(g, n), "qty": _randint(g, 1, 51, n), "discount": _randint(g, 0, 11, n),
         "category": _categories(g, n), "updated_at": _randint(g, datagen.DATE_LO, datagen.DATE_HI + 1, n, torch.int64)}
    t = {"id": torch.arange(n, dtype=torch.int64, device="cuda")} | {name: d[order] for name, d in t.items()}
    if own_prices:
        t["price"] = _price(_gen(seed + 1), n)
    nulls = _null_bytes(g, n)[order]
    return {name: ops.DeviceColumn(d, SALES[name], nulls if name == null_column else None) for name, d in t.items()}


def _zipf(g, n: int, distinct: int = 100_000, s: float = 1.1) -> torch.Tensor:
    values = torch.rand(distinct, generator=g, device="cuda") * 2e6 - 1e6
    w = torch.arange(1, distinct + 1, device="cuda", dtype=torch.float64) ** -s
    cdf = (torch.cumsum(w, 0) / w.sum()).float()
    return values[torch.searchsorted(cdf, torch.rand(n, generator=g, device="cuda")).clamp_(max=distinct - 1)]


def _order_table(n: int, seed: int, dist: str) -> ops.DeviceBatch:
    g = _gen(seed)
    if dist == "uniform":
        key = torch.rand(n, generator=g, device="cuda") * 2e6 - 1e6
    elif dist == "zipf":
        key = _zipf(g, n)
    else:
        key = torch.full((n,), 42.0, device="cuda")
    txt = torch.randint(97, 123, (n, datagen.TEXT_WIDTH), generator=g, device="cuda", dtype=torch.uint8)
    txt[:, -1] = 0
    return ops.DeviceBatch([ops.DeviceColumn(key, A.FLOAT32),
                            ops.DeviceColumn(torch.arange(n, dtype=torch.int64, device="cuda"), A.INT64),
                            ops.DeviceColumn(txt, A.TEXT),
                            ops.DeviceColumn(_randint(g, datagen.DATE_LO, datagen.DATE_HI + 1, n, torch.int64),
                                             A.DATETIME)])


ORDER_ROW_BYTES = 4 + 8 + datagen.TEXT_WIDTH + 8
SALES_ROW_BYTES = 8 + 4 + 4 + 4 + datagen.TEXT_WIDTH + 8


def _task_offsets(case: dict, seed: int | None) -> list[int]:
    """Row offsets of the tasks, their sizes log-uniform (the same for every
    seed, so that a case's size is its own)."""
    import random
    rng = random.Random(case["tasks"] * 1_000_003 + case["hi"])
    offs = [0]
    for _ in range(case["tasks"]):
        offs.append(offs[-1] + _log(rng, case["lo"], case["hi"]))
    return offs


def _empty_like(batch: ops.DeviceBatch) -> ops.DeviceBatch:
    return ops.DeviceBatch([ops.DeviceColumn.empty(c.type, c.rows, c.width if c.type == A.TEXT else None,
                                                   nulls=c.nulls is not None) for c in batch.columns])


# ------------------------------------------------------------- CSV text
def _digits(x: torch.Tensor, width: int):
    pw = 10 ** torch.arange(width - 1, -1, -1, device="cuda", dtype=torch.int64)
    x = x.to(torch.int64)
    ndig = (x[:, None] >= pw[None, :]).sum(1).clamp_(min=1)
    text = ((x[:, None] // pw[None, :]) % 10 + 48).to(torch.uint8)
    return text, torch.arange(width, device="cuda")[None, :] >= (width - ndig)[:, None]


def _padded(x: torch.Tensor, width: int) -> torch.Tensor:
    pw = 10 ** torch.arange(width - 1, -1, -1, device="cuda", dtype=torch.int64)
    return ((x.to(torch.int64)[:, None] // pw[None, :]) % 10 + 48).to(torch.uint8)


def _date_text(secs: torch.Tensor) -> torch.Tensor:
    """"YYYY-MM-DD HH:MM:SS" of epoch seconds after 1970 (UTC)."""
    days, rem = secs // 86400, secs % 86400
    z = days + 719468  # days since 0000-03-01
    era = z // 146097
    doe = z - era * 146097
    yoe = (doe - doe // 1460 + doe // 36524 - doe // 146096) // 365
    doy = doe - (365 * yoe + yoe // 4 - yoe // 100)
    mp = (5 * doy + 2) // 153
    d = doy - (153 * mp + 2) // 5 + 1
    m = torch.where(mp < 10, mp + 3, mp - 9)
    y = yoe + era * 400 + (m <= 2)

    def ch(c):
        return torch.full((secs.shape[0], 1), ord(c), dtype=torch.uint8, device="cuda")
    return torch.cat([_padded(y, 4), ch("-"), _padded(m, 2), ch("-"), _padded(d, 2), ch(" "), _padded(rem // 3600, 2),
                      ch(":"), _padded(rem % 3600 // 60, 2), ch(":"), _padded(rem % 60, 2)], dim=1)


def _csv_cents(n: int, seed: int) -> torch.Tensor:
    return _randint(_gen(seed), 100, 100_000, n, torch.int64)


def _csv_body(n: int, seed: int) -> torch.Tensor:
    """The sales table as CSV text without its header line: prices with two
    decimals, dates as written by the reference's own files."""
    cents = _csv_cents(n, seed)
    g = _gen(seed + 1)
    chunks = []
    for lo in range(0, n, 1 << 20):
        c = cents[lo:lo + (1 << 20)]
        k = c.shape[0]

        def full(t):
            return t, torch.ones(t.shape, dtype=torch.bool, device="cuda")
        dot = torch.full((k, 1), ord("."), dtype=torch.uint8, device="cuda")
        pi, pm = _digits(c // 100, 3)
        frac = torch.cat([dot, _padded(c % 100, 2)], dim=1)
        fields = [_digits(torch.arange(lo, lo + k, device="cuda"), 8),
                  (torch.cat([pi, frac], 1), torch.cat([pm, torch.ones_like(frac, dtype=torch.bool)], 1)),
                  _digits(_randint(g, 1, 51, k), 2), _digits(_randint(g, 0, 11, k), 2),
                  full(_categories(g, k)[:, :CATEGORY_BYTES]),
                  full(_date_text(_randint(g, datagen.DATE_LO, datagen.DATE_HI + 86400, k, torch.int64)))]
        text, mask = [], []
        for i, (t, m) in enumerate(fields):
            sep = ord("\n") if i + 1 == len(fields) else ord(",")
            text += [t, torch.full((k, 1), sep, dtype=torch.uint8, device="cuda")]
            mask += [m, torch.ones((k, 1), dtype=torch.bool, device="cuda")]
        chunks.append(torch.masked_select(torch.cat(text, 1), torch.cat(mask, 1)))
    return torch.cat(chunks)


CSV_TYPES = [A.INT32, A.FLOAT32, A.INT32, A.INT32, A.TEXT, A.DATETIME]
CSV_LINE_BYTES = 52  # mean line of the body above, newline included


# ------------------------------------------------------------------- queries
def _sales_predicate(price: int, qty: int, disc: int, cat: int):
    p, q, d, c = (ColumnRef(price, A.FLOAT32), ColumnRef(qty, A.INT32), ColumnRef(disc, A.INT32),
                  ColumnRef(cat, A.TEXT))
    pred = And(between(d, Constant(1, A.INT32), Constant(3, A.INT32)), Compare(A.LT, q, Constant(25, A.INT32)),
               Compare(A.NE, c, Constant(datagen.EXCLUDED_CATEGORY, A.TEXT)))
    return pred, p, d


def _sales_keep(cols: dict) -> torch.Tensor:
    excluded = torch.from_numpy(datagen.text_slots([datagen.EXCLUDED_CATEGORY])).cuda()
    d, q = cols["discount"].data, cols["qty"].data
    return (d >= 1) & (d <= 3) & (q < 25) & (cols["category"].data != excluded).any(1)


FILTER_COLUMNS = ["price", "qty", "discount", "category"]
FILTER_ROW_BYTES = 4 + 4 + 4 + datagen.TEXT_WIDTH
SELECTED = 3 / 11 * 24 / 50 * 24 / 25  # share of rows the predicate keeps


def _star_fact(n: int, seed: int) -> dict:
    g = _gen(seed)
    return {"datekey": _randint(g, 0, 2556, n), "quantity": _randint(g, 1, 51, n), "discount": _randint(g, 0, 11, n),
            "extendedprice": torch.rand(n, generator=g, device="cuda") * 104_100.0 + 900.0}


def _date_dim() -> dict:
    dk = torch.arange(2556, dtype=torch.int32, device="cuda")
    return {"datekey": dk, "year": (1992 + dk // 365).clamp_(max=1998), "month": (1 + dk % 365 * 12 // 365).int()}


def _group_table(case: dict, seed: int) -> dict:
    n, g = case["rows"], _gen(seed)
    return {"key": _randint(_gen(case["groups"]), 0, case["groups"], n)[_order(n, seed)], "price": _price(g, n), "qty": _randint(g, 1, 51, n)}


GROUP_AGGS = [(A.AGG_COUNT_STAR, 0), (A.AGG_SUM, 1), (A.AGG_AVG, 2), (A.AGG_MIN, 1), (A.AGG_MAX, 1)]


def prepare(case: dict, seed: int) -> dict:
    kind = case["kind"]
    st = {"kind": kind}
    if kind == "filter_agg":
        cols = _sales(case["rows"], seed, "price" if case["nulls"] else None)
        st["batch"] = ops.DeviceBatch([cols[c] for c in FILTER_COLUMNS])
        pred, price, disc = _sales_predicate(0, 1, 2, 3)
        aggs = [Aggregate(A.AGG_SUM, Arith(A.MUL, price, Cast(disc, A.FLOAT32))), Aggregate(A.AGG_COUNT_STAR),
                Aggregate(A.AGG_MIN, price), Aggregate(A.AGG_MAX, price)]
        st["plan"] = ops.AggPlan([c.type for c in st["batch"].columns], pred, aggs)
        st["acc"] = ops.AggState(aggs)
    elif kind == "filter_project":
        cols = _sales(case["rows"], seed, "price" if case["nulls"] else None)
        st["batch"] = ops.DeviceBatch([cols[c] for c in FILTER_COLUMNS])
        pred, price, disc = _sales_predicate(0, 1, 2, 3)
        st["plan"] = ops.ProjectPlan([c.type for c in st["batch"].columns], [c.width for c in st["batch"].columns],
                                     pred, [3, 0, Arith(A.MUL, price, Cast(disc, A.FLOAT32))])
    elif kind == "sort":
        st["batch"] = ops.DeviceBatch(list(_sales(case["rows"], seed, case["key"] if case["nulls"] else None).values()))
        st["key"], st["desc"] = list(SALES).index(case["key"]), case["desc"]
    elif kind == "order_by":
        st["batch"] = _order_table(case["rows"], seed, case["dist"])
        offs = [0]
        for c in datagen.batch_row_counts(case["rows"], ORDER_ROW_BYTES, RUN_BYTES):
            offs.append(offs[-1] + c)
        st["job"] = ops.OrderByRuns(st["batch"], 0 if case["key"] == "key" else 3, offs)
        st["out"], st["desc"] = _empty_like(st["batch"]), case["desc"]
    elif kind == "star_agg":
        fact, dim = _star_fact(case["rows"], seed), _date_dim()
        st["fact"] = ops.DeviceBatch([ops.DeviceColumn(v, A.FLOAT32 if v.is_floating_point() else A.INT32)
                                      for v in fact.values()])
        st["dim"] = ops.DeviceBatch([ops.DeviceColumn(v, A.INT32) for v in dim.values()])
        qty, disc, ext = ColumnRef(1, A.INT32), ColumnRef(2, A.INT32), ColumnRef(3, A.FLOAT32)
        aggs = [Aggregate(A.AGG_SUM, Arith(A.MUL, ext, Cast(disc, A.FLOAT32)))]
        st["plan"] = ops.JoinAggPlan([A.INT32] * 3 + [A.FLOAT32], [A.INT32] * 3,
                                     And(between(disc, Constant(1, A.INT32), Constant(3, A.INT32)),
                                         Compare(A.LT, qty, Constant(25, A.INT32))), 0,
                                     Compare(A.EQ, ColumnRef(1, A.INT32), Constant(1993, A.INT32)), 0, aggs)
        st["acc"] = ops.AggState(aggs)
    elif kind == "join":
        g, n, r = _gen(seed), case["rows"], case["right"]
        st["left"] = ops.DeviceBatch([ops.DeviceColumn(_randint(g, 0, r, n), A.INT32),
                                      ops.DeviceColumn(_price(g, n), A.FLOAT32)])
        keys = torch.randperm(r, generator=g, device="cuda", dtype=torch.int32)
        st["right"] = ops.DeviceBatch([ops.DeviceColumn(keys, A.INT32),
                                       ops.DeviceColumn(_randint(g, 0, 1 << 40, r, torch.int64), A.INT64)])
        st["cond"], st["outputs"] = [(0, 0, A.EQ)], [(0, 0), (0, 1), (1, 1)]
    elif kind == "cross":
        g, n, r = _gen(case["rows"]), case["rows"], case["right"]
        st["left"] = ops.DeviceBatch([ops.DeviceColumn(_randint(g, 0, 1_000_000, n)[_order(n, seed)], A.INT32)])
        st["right"] = ops.DeviceBatch([ops.DeviceColumn(_randint(g, 0, 1_000_000, r)[_order(r, seed + 1)], A.INT32)])
        st["cond"], st["outputs"] = [(0, 0, A.LT)], [(0, 0), (1, 0)]
    elif kind == "csv_scan":
        st["text"] = _csv_body(case["rows"], seed)
    elif kind == "csv_format":
        # a result batch as the scan leaves it: every column with null bytes
        cols = _sales(case["rows"], seed, "price", own_prices=False)
        cols["id"] = ops.DeviceColumn(cols["id"].data.int(), A.INT32)
        for c in cols.values():
            if c.nulls is None:
                c.nulls = torch.zeros(case["rows"], dtype=torch.uint8, device="cuda")
        st["batch"] = ops.DeviceBatch(list(cols.values()))
    elif kind == "group_by":
        t = _group_table(case, seed)
        st["batch"] = ops.DeviceBatch([ops.DeviceColumn(t["key"], A.INT32), ops.DeviceColumn(t["price"], A.FLOAT32),
                                       ops.DeviceColumn(t["qty"], A.INT32)])
        st["groups"] = case["groups"]
    elif kind == "order_tasks":
        offs = _task_offsets(case, seed)
        st["batch"] = ops.DeviceBatch(list(_sales(offs[-1], seed).values()))
        st["key"], st["offsets"] = list(SALES).index("price"), offs
        st["out"] = _empty_like(st["batch"])
        st["ws"] = torch.empty(ops.order_by_segments_workspace_bytes(st["batch"].columns[st["key"]], offs),
                               dtype=torch.uint8, device="cuda")
    else:
        raise ValueError(kind)
    return st


def _tensors(batch: ops.DeviceBatch) -> list:
    """Every column's values, and its null bytes where it has some."""
    out = []
    for c in batch.columns:
        out.append(c.data)
        if c.nulls is not None:
            out.append(c.nulls)
    return out


def run(st: dict):
    kind = st["kind"]
    if kind == "filter_agg":
        st["acc"].reset()
        st["plan"].run(st["batch"], st["acc"])
        return st["acc"].read()
    if kind == "filter_project":
        return _tensors(st["plan"].run(st["batch"]))
    if kind == "sort":
        return _tensors(ops.sort_batch(st["batch"], st["key"], st["desc"]))
    if kind == "order_by":
        return _tensors(st["job"].run(st["batch"], st["desc"], st["out"]))
    if kind == "star_agg":
        st["acc"].reset()
        st["plan"].run(st["fact"], st["dim"], st["acc"])
        return st["acc"].read()
    if kind in ("join", "cross"):
        return _tensors(ops.join_project(st["left"], st["right"], st["cond"], st["outputs"]))
    if kind == "csv_scan":
        return _tensors(ops.csv_scan(st["text"], CSV_TYPES, text_width=datagen.TEXT_WIDTH))
    if kind == "csv_format":
        return ops.csv_format(st["batch"])
    if kind == "group_by":
        return _tensors(ops.group_by(st["batch"], 0, GROUP_AGGS, capacity=st["groups"]))
    return _tensors(ops.order_by_segments(st["batch"], st["key"], True, st["offsets"], st["out"], workspace=st["ws"]))


def work(case: dict) -> dict:
    """Each input column read once, each output written once; operations are
    one a row and compared or computed value (pairs for the cross product)."""
    kind, n = case["kind"], case.get("rows", 0)
    if kind == "filter_agg":
        return {"bytes": n * (FILTER_ROW_BYTES + (1 if case["nulls"] else 0)), "flops": 4 * n}
    if kind == "filter_project":
        out = datagen.TEXT_WIDTH + 4 + 4 + 3
        return {"bytes": n * (FILTER_ROW_BYTES + (1 if case["nulls"] else 0)) + int(n * SELECTED * out), "flops": 4 * n}
    if kind == "sort":
        return {"bytes": 2 * n * (SALES_ROW_BYTES + (1 if case["nulls"] else 0)), "flops": n}
    if kind == "order_by":
        return {"bytes": 2 * n * ORDER_ROW_BYTES, "flops": n}
    if kind == "star_agg":
        return {"bytes": n * 16 + 2556 * 8, "flops": 4 * n}
    if kind == "join":
        return {"bytes": n * 8 + case["right"] * 12 + n * 16, "flops": n}
    if kind == "cross":
        pairs = n * case["right"]
        return {"bytes": 4 * (n + case["right"]) + pairs // 2 * 8, "flops": pairs}
    if kind == "csv_scan":
        return {"bytes": n * (CSV_LINE_BYTES + 4 + 4 + 4 + 4 + datagen.TEXT_WIDTH + 8 + len(CSV_TYPES)), "flops": n * 6}
    if kind == "csv_format":
        return {"bytes": n * (4 + 4 + 4 + 4 + datagen.TEXT_WIDTH + 8 + len(CSV_TYPES) + CSV_LINE_BYTES + 6),
                "flops": n * 6}
    if kind == "group_by":
        return {"bytes": n * 12 + case["groups"] * 41, "flops": 4 * n}
    rows = _task_offsets(case, None)[-1]
    return {"bytes": 2 * rows * SALES_ROW_BYTES, "flops": rows}


def exact(case: dict, seed: int):
    """The computed outputs in 64 bits, laid out as run returns them; None for
    values that are only moved, counted or written as text."""
    kind = case["kind"]
    if kind in ("filter_agg", "filter_project"):
        cols = _sales(case["rows"], seed, "price" if case["nulls"] else None)
        keep = _sales_keep(cols)
        p, d = cols["price"], cols["discount"].data
        if kind == "filter_agg":
            if p.nulls is not None:
                keep &= p.nulls == 0
            v = p.data[keep].double()
            if v.numel() == 0:
                return [None] * 4
            return [float((v * d[keep].double()).sum()), None, float(v.min()), float(v.max())]
        # a NULL price leaves no computed value in its place: no exact product then
        price = p.data[keep].double()
        return [None, None, price, None, None if p.nulls is not None else price * d[keep].double(), None]
    if kind == "star_agg":
        fact, dim = _star_fact(case["rows"], seed), _date_dim()
        disc = fact["discount"]
        keep = (disc >= 1) & (disc <= 3) & (fact["quantity"] < 25) & (dim["year"][fact["datekey"].long()] == 1993)
        return [float((fact["extendedprice"][keep].double() * disc[keep].double()).sum())]
    if kind == "csv_scan":
        price = _csv_cents(case["rows"], seed).double() / 100
        return [None, None, price] + [None] * 9
    if kind == "group_by":
        t = _group_table(case, seed)
        key = t["key"].long()
        count = torch.bincount(key, minlength=case["groups"])
        present = count > 0
        total = torch.bincount(key, weights=t["price"].double(), minlength=case["groups"])[present]
        mean = torch.bincount(key, weights=t["qty"].double(), minlength=case["groups"])[present] / count[present]
        return [None, None, None, None, total, None, mean, None, None, None, None, None]
    return None
