"""The key/id merge levels (yq_order_by_tiled: runs sorted, merged pairwise) over
many runs, every key kind and every output column, and the packed gather of large
tables at every record size. yq_order_by itself sorts the whole table at once, so
only a named merge tile runs the levels."""
import numpy as np
import pytest
import torch

import oracle
from yallasql_b200 import _abi as A
from yallasql_b200 import datagen, ops

pytestmark = pytest.mark.gpu

KINDS = ["f32", "f32_special", "f64_special", "i32", "i64_low", "i64_wide", "date", "bool", "bool_bytes", "equal",
         "i32_nulls", "date_nulls", "f64_nulls", "text16"]


def keys(kind, rng, n):
    """(values, type, the oracle's type, nulls)"""
    nulls = rng.random(n) < 0.15 if kind.endswith("_nulls") else None
    if kind == "f32":
        return rng.zipf(1.3, n).clip(max=500).astype(np.float32) * np.float32(-0.5), A.FLOAT32, None, nulls
    if kind == "f32_special":
        k = rng.choice(np.array([0.0, -0.0, 1.5, -np.inf, np.inf], np.float32), n)
        k.view(np.uint32)[rng.random(n) < 0.05] = 0xffc00001
        return k, A.FLOAT32, None, nulls
    if kind.startswith("f64"):
        return rng.choice(np.array([0.0, -0.0, 1e300, -1e-300, np.nan, np.inf]), n), A.FLOAT64, None, nulls
    if kind in ("i32", "i32_nulls"):
        return rng.integers(-300, 300, n).astype(np.int32), A.INT32, None, nulls
    if kind == "i64_low":  # the high word shared: one key word
        return rng.integers(0, 1 << 31, n) + (7 << 32), A.INT64, None, nulls
    if kind == "i64_wide":
        return rng.integers(-(1 << 62), 1 << 62, n) >> rng.integers(0, 50, n), A.INT64, None, nulls
    if kind.startswith("date"):
        return rng.integers(1420070400, 1640995199, n), A.DATETIME, oracle.DATETIME, nulls
    if kind.startswith("bool"):
        return rng.integers(0, 2 if kind == "bool" else 5, n).astype(np.uint8), A.BOOL, None, nulls
    if kind == "equal":
        return np.full(n, -7, np.int32), A.INT32, None, nulls
    return datagen.text_slots([f"key{x:05d}_tail" for x in rng.integers(0, 3000, n)]), A.TEXT, None, nulls


def column(v, t, nulls=None):
    return ops.DeviceColumn(torch.from_numpy(np.ascontiguousarray(v)).cuda(), t,
                            None if nulls is None else torch.from_numpy(nulls.astype(np.uint8)).cuda())


@pytest.mark.parametrize("merge_items", [4, 8, 16])
@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("desc,nulls_first", [(False, False), (True, True)])
def test_levels_over_many_runs(cuda, merge_items, kind, desc, nulls_first):
    """84 runs (seven levels), empty ones and ones of a row among them."""
    rng = np.random.default_rng(merge_items * 100 + len(kind) + desc)
    sizes = rng.integers(0, 4000, 84)
    sizes[[3, 4, 40, 83]] = 0
    sizes[[7, 8]] = 1
    n = int(sizes.sum())
    offs = [0] + list(np.cumsum(sizes).astype(int))
    k, t, ty, nulls = keys(kind, rng, n)
    payload = np.arange(n, dtype=np.int64)
    txt = datagen.text_slots([f"r{i % 97}" for i in range(n)])
    b = ops.DeviceBatch([column(k, t, nulls), column(payload, A.INT64), column(txt, A.TEXT)])
    if merge_items == 16 and kind in ("f64_nulls", "text16"):  # keys of four words
        with pytest.raises(A.YQError) as e:
            ops.order_by(b, 0, desc, offs, nulls_first=nulls_first, merge_items=merge_items)
        assert e.value.status == A.ERR_UNSUPPORTED
        return
    out = ops.order_by(b, 0, desc, offs, nulls_first=nulls_first, merge_items=merge_items)
    perm = oracle.sort_perm(k, desc=desc, nulls=nulls, nulls_first=nulls_first, type_=ty)
    np.testing.assert_array_equal(out.columns[1].data.cpu().numpy(), payload[perm])
    np.testing.assert_array_equal(out.columns[0].data.cpu().numpy().view(np.uint8), k[perm].view(np.uint8))
    np.testing.assert_array_equal(out.columns[2].data.cpu().numpy(), txt[perm])
    if nulls is not None:
        np.testing.assert_array_equal(out.columns[0].nulls.cpu().numpy().astype(bool), nulls[perm])


# columns of a record of so many 16-byte pieces, the INT32 key's 4 bytes first
RECORDS = {
    1: [(A.INT64, 8)],
    2: [(A.TEXT, 16), (A.INT64, 8)],
    3: [(A.TEXT, 16), (A.TEXT, 16), (A.BOOL, 1)],
    4: [(A.TEXT, 32), (A.TEXT, 12), (A.INT32, 4), (A.INT64, 8)],
    5: [(A.TEXT, 32), (A.TEXT, 20), (A.TEXT, 16)],
    6: [(A.TEXT, 32), (A.TEXT, 32), (A.TEXT, 16), (A.INT32, 4)],
    7: [(A.TEXT, 32), (A.TEXT, 32), (A.TEXT, 24), (A.INT64, 8), (A.BOOL, 1)],
    8: [(A.TEXT, 32), (A.TEXT, 32), (A.TEXT, 28), (A.INT64, 8), (A.INT32, 4), (A.INT32, 4), (A.BOOL, 1)],
}


@pytest.mark.parametrize("pieces", list(RECORDS))
@pytest.mark.parametrize("nullable", [False, True])
@pytest.mark.parametrize("extra", [-1, 1, 1025])
def test_packed_gather_of_every_record(cuda, pieces, nullable, extra):
    """Rows around the 64 MiB of cells from which a table is gathered through
    packed records; the least workspace always gathers column by column."""
    cell = 4 + sum(w for _, w in RECORDS[pieces]) + (1 if nullable else 0)
    n = (64 << 20) // cell + extra
    g = torch.Generator(device="cuda")
    g.manual_seed(n)
    perm = torch.randperm(n, generator=g, device="cuda")
    key = torch.empty(n, dtype=torch.int32, device="cuda")
    key[perm] = torch.arange(n, device="cuda", dtype=torch.int32)  # sorted by it, row i is perm[i]
    cols = [ops.DeviceColumn(key, A.INT32)]
    for i, (t, w) in enumerate(RECORDS[pieces]):
        d = torch.randint(0, 256, (n, w), generator=g, device="cuda", dtype=torch.uint8)
        data = d if t == A.TEXT else d.view(ops.TORCH_DTYPE[t]).flatten()
        nulls = (torch.rand(n, generator=g, device="cuda") < 0.1).to(torch.uint8) if nullable and i == 0 else None
        cols.append(ops.DeviceColumn(data, t, nulls))
    b = ops.DeviceBatch(cols)
    offs = [0, n // 3, n]
    packed = ops.order_by_batch_workspace_bytes(b, 0, offs) - ops.order_by_workspace_bytes(cols[0], offs)
    assert (packed > 0) == (extra > 0)
    if packed > 0:
        assert pieces * 16 * n <= packed <= pieces * 16 * n + 4096
    for two_level in (True, False):
        out = ops.DeviceBatch([ops.DeviceColumn.empty(c.type, n, c.width if c.type == A.TEXT else None,
                                                      nulls=c.nulls is not None) for c in cols])
        ops.OrderByRuns(b, 0, offs, two_level=two_level).run(b, False, out)
        assert torch.equal(out.columns[0].data, torch.arange(n, device="cuda", dtype=torch.int32))
        for o, c in zip(out.columns[1:], cols[1:]):
            assert torch.equal(o.data.view(torch.uint8), c.data[perm].view(torch.uint8))
            if c.nulls is not None:
                assert torch.equal(o.nulls, c.nulls[perm])
