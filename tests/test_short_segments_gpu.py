"""Segmented sorts of short segments, around the average length below which the
histogram counts with one copy of its bins, and with warps that hold no row."""
import numpy as np
import pytest
import torch

import oracle
from yallasql_b200 import _abi as A
from yallasql_b200 import datagen, ops

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", ["i32", "f32_nulls", "i64", "i64_nulls", "text12", "text28"])
@pytest.mark.parametrize("nseg,longest", [(700, 1), (900, 9), (300, 70), (40, 1020), (40, 1030), (9, 5000), (1, 511), (1, 513)])
def test_permutation_of_every_segment(cuda, kind, nseg, longest):
    rng = np.random.default_rng(nseg * 31 + longest)
    sizes = rng.integers(0, longest + 1, nseg) if nseg > 1 else np.array([longest])
    n = int(sizes.sum())
    offs = [0] + [int(x) for x in np.cumsum(sizes)]
    nulls = rng.random(n) < 0.2 if kind.endswith("nulls") else None
    if kind == "i32":
        k, t = rng.integers(-50, 50, n).astype(np.int32), A.INT32
    elif kind == "f32_nulls":
        k, t = rng.normal(0, 1e3, n).astype(np.float32), A.FLOAT32
    elif kind.startswith("i64"):
        k, t = rng.integers(-(1 << 60), 1 << 60, n), A.INT64
    else:
        k, t = datagen.text_slots([f"{x:05d}_{'x' * (int(kind[4:]) - 8)}" for x in rng.integers(0, 90_000, n)],
                                  int(kind[4:])), A.TEXT
    col = ops.DeviceColumn(torch.from_numpy(np.ascontiguousarray(k)).cuda(), t,
                           None if nulls is None else torch.from_numpy(nulls.astype(np.uint8)).cuda())
    if n == 0:
        return
    for desc in (False, True):
        want = oracle.sort_perm(k, desc=desc, nulls=nulls, segments=offs)
        for keep in (0, 1):
            ws = torch.empty(ops.sort_workspace_bytes(col, offs), dtype=torch.uint8, device="cuda")
            got = ops.sort_segments(col, offs, descending=desc, config=ops.sort_config(keep_trivial=bool(keep)),
                                    workspace=ws)
            assert np.array_equal(got.cpu().numpy().view(np.uint32), want)
