"""GROUP BY around the number of groups whose accumulators the sort-free path has
room for: the limit follows from the call's aggregates, results on both sides of
it agree with the oracle, and a key of more values is told by its first rows."""
import ctypes as C
import json

import numpy as np
import pytest
import torch

from tests.test_yy_group_gpu import check, dcol
from yallasql_b200 import _abi as A
from yallasql_b200 import ops

pytestmark = pytest.mark.gpu

# (aggregates over columns 1: FLOAT32, 2: INT32, 3: INT64, 4: FLOAT32 with NULLs; most groups with 4- and 8-byte keys)
# a block's 220 KB less 512 slots of two key widths, by 128 threads of 4 bytes (rows) and the arrays' sizes
MIXES = {
    "count": ([(A.AGG_COUNT_STAR, 0)], 96, 96),
    "five": ([(A.AGG_COUNT_STAR, 0), (A.AGG_SUM, 1), (A.AGG_AVG, 2), (A.AGG_MIN, 1), (A.AGG_MAX, 1)], 61, 60),
    "nullable": ([(A.AGG_COUNT, 4), (A.AGG_SUM, 4), (A.AGG_MIN, 4)], 86, 84),
    "eight": ([(A.AGG_SUM, 1), (A.AGG_SUM, 2), (A.AGG_SUM, 3), (A.AGG_AVG, 4), (A.AGG_MIN, 3), (A.AGG_MAX, 3),
               (A.AGG_MIN, 1), (A.AGG_MAX, 2)], 27, 26),
}


def profiled(call):
    L = A.load()
    L.yq_profile_enable(1)
    L.yq_profile_read(None, 0, 1)
    try:
        call()
        buf = C.create_string_buffer(1 << 14)
        L.yq_profile_read(buf, len(buf), 1)
    finally:
        L.yq_profile_enable(0)
    return json.loads(buf.value.decode() or "{}")


@pytest.mark.parametrize("ktype", [A.INT32, A.INT64])
@pytest.mark.parametrize("mix", list(MIXES))
def test_around_the_accumulators_room(cuda, ktype, mix):
    aggs, limit4, limit8 = MIXES[mix]
    limit = limit4 if ktype == A.INT32 else limit8
    rows = 120_001
    dt = np.int32 if ktype == A.INT32 else np.int64
    for groups in (limit - 1, limit, limit + 1):
        rng = np.random.default_rng(groups + ktype)
        # -1 (every bit set) and the type's ends among the keys
        pool = np.unique(np.concatenate([np.array([-1, np.iinfo(dt).min, np.iinfo(dt).max], dt),
                                         rng.integers(-10_000, 10_000, 400).astype(dt) * dt(3)]))
        pool = np.concatenate([pool[[0, -1]], np.array([-1], dt), pool[1:-1][pool[1:-1] != -1]])[:groups]
        k = pool[rng.integers(0, groups, rows)]
        k[:groups] = pool
        cols = [(k, ktype, None), (rng.normal(0, 100, rows).astype(np.float32), A.FLOAT32, None),
                (rng.integers(-(1 << 31), 1 << 31, rows).astype(np.int32), A.INT32, None),
                (rng.integers(-(1 << 50), 1 << 50, rows), A.INT64, None),
                (rng.normal(0, 1, rows).astype(np.float32), A.FLOAT32, rng.random(rows) < 0.3)]
        prof = profiled(lambda: check(cols, 0, aggs))
        assert ("group_few_accumulate" in prof) == (groups <= limit), (groups, sorted(prof))


def test_search_stops_at_the_limit(cuda):
    """One value more than there is room for: the search ends within its first
    rows (a whole search of 16M keys takes several times as long)."""
    rows = 16_000_000
    aggs = MIXES["five"][0]
    g = torch.Generator(device="cuda")
    g.manual_seed(1)
    ms = {}
    for groups in (61, 62):
        b = ops.DeviceBatch([ops.DeviceColumn(torch.randint(0, groups, (rows,), generator=g, device="cuda",
                                                            dtype=torch.int32), A.INT32),
                             ops.DeviceColumn(torch.ones(rows, device="cuda"), A.FLOAT32),
                             ops.DeviceColumn(torch.ones(rows, dtype=torch.int32, device="cuda"), A.INT32)])
        for _ in range(5):
            prof = profiled(lambda: ops.group_by(b, 0, aggs, capacity=100))
            assert ("group_few_accumulate" in prof) == (groups == 61)
            ms[groups] = min(ms.get(groups, 1e9), prof["group_few_find"]["ms"])
    assert ms[62] < 0.6 * ms[61], ms
