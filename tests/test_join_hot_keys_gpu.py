"""Equi-joins with a long right side whose keys repeat on both sides: runs of any
length, further conditions, left sides that fill part of a block or many, and the
time they take against the nested loop."""
import ctypes as C

import numpy as np
import pytest
import torch

from yallasql_b200 import _abi as A
from yallasql_b200 import ops

pytestmark = pytest.mark.gpu


def dev(v):
    return ops.DeviceColumn(torch.from_numpy(np.ascontiguousarray(v)).cuda(), A.INT32)


@pytest.mark.parametrize("L,R,distinct", [(1, 8193, 1), (2, 9000, 2), (31, 5000, 3), (257, 4097, 1), (591, 6000, 7),
                                          (593, 4100, 2), (3000, 4500, 40), (70_000, 5000, 4000)])
@pytest.mark.parametrize("residual", [None, A.LT, A.NE])
def test_pairs_in_order(cuda, L, R, distinct, residual):
    rng = np.random.default_rng(L * 3 + R + distinct)
    lk, rk = rng.integers(0, distinct, L).astype(np.int32), rng.integers(0, distinct, R).astype(np.int32)
    lv, rv = rng.integers(0, 50, L).astype(np.int32), rng.integers(0, 50, R).astype(np.int32)
    if residual == A.LT:
        lv[:] = np.maximum(lv, 47)  # few of a run's rows pass
    conds = [(0, 0, A.EQ)] if residual is None else [(1, 1, residual), (0, 0, A.EQ)]
    order = np.argsort(rk, kind="stable")  # a key's right rows, ascending
    starts, ends = np.searchsorted(rk[order], lk, "left"), np.searchsorted(rk[order], lk, "right")
    wl = np.repeat(np.arange(L), ends - starts)
    wr = np.concatenate([order[a:b] for a, b in zip(starts, ends)])
    if residual is not None:
        keep = lv[wl] < rv[wr] if residual == A.LT else lv[wl] != rv[wr]
        wl, wr = wl[keep], wr[keep]
    lb, rb = ops.DeviceBatch([dev(lk), dev(lv)]), ops.DeviceBatch([dev(rk), dev(rv)])
    gl, gr = ops.join_pairs(lb, rb, conds, capacity=max(1, len(wl)))
    assert np.array_equal(gl.cpu().numpy(), wl) and np.array_equal(gr.cpu().numpy(), wr)
    if len(wl) > 1:
        with pytest.raises(A.YQError) as e:  # room for a part: refused with the exact count
            ops.join_pairs(lb, rb, conds, capacity=len(wl) // 2)
        assert e.value.status == A.ERR_CAPACITY


@pytest.mark.parametrize("L,R", [(3000, 20_000), (100, 8193)])
def test_one_key_and_a_condition_takes_no_longer_than_the_nested_loop(cuda, yq, L, R):
    """Every left row meets every right row: as much to compare as in the nested
    loop, which a workspace without room for the sort selects."""
    rng = np.random.default_rng(L)
    one = lambda n: dev(np.full(n, 7, np.int32))
    lb = ops.DeviceBatch([one(L), dev(rng.integers(0, 100, L).astype(np.int32))])
    rb = ops.DeviceBatch([one(R), dev(rng.integers(100, 200, R).astype(np.int32))])
    lc, k1 = lb.c()
    rc, k2 = rb.c()
    conds = (A.JoinCond * 2)(A.JoinCond(0, 0, A.EQ), A.JoinCond(1, 1, A.GT))  # no pair passes
    out = torch.empty(2, dtype=torch.int32, device="cuda")
    n = C.c_uint64(0)
    ms = {}
    for name, size in (("sorted", int(yq.yq_join_workspace_size(L, R))), ("nested", 1 << 16)):
        ws = torch.empty(size, dtype=torch.uint8, device="cuda")
        for _ in range(4):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record()
            st = yq.yq_join_pairs(C.byref(lc), C.byref(rc), conds, 2, out.data_ptr(), out.data_ptr() + 4, 1, C.byref(n),
                                  ws.data_ptr(), ws.numel(), None)
            b.record()
            b.synchronize()
            assert (st, n.value) == (A.OK, 0)
            ms[name] = min(ms.get(name, 1e9), a.elapsed_time(b))
    assert ms["sorted"] < 1.5 * ms["nested"], ms


def test_a_row_with_millions_of_matches(cuda):
    """More pairs in a tile than its 32-bit offsets hold: three left rows, one of
    them without a match, to 1.5M right rows of two keys."""
    rows = 1_500_000
    rk = (torch.arange(rows, device="cuda", dtype=torch.int32) % 5 == 0).int()  # 1 for every fifth row
    rv = torch.arange(rows, device="cuda", dtype=torch.int32)
    lk = torch.tensor([0, 9, 0, 1], device="cuda", dtype=torch.int32)
    lb = ops.DeviceBatch([ops.DeviceColumn(lk, A.INT32), ops.DeviceColumn(lk * 100, A.INT32)])
    rb = ops.DeviceBatch([ops.DeviceColumn(rk, A.INT32), ops.DeviceColumn(rv, A.INT32)])
    zero, one = (rk == 0).nonzero().flatten().int(), (rk == 1).nonzero().flatten().int()
    wl = torch.cat([torch.full_like(zero, 0), torch.full_like(zero, 2), torch.full_like(one, 3)])
    wr = torch.cat([zero, zero, one])
    gl, gr = ops.join_pairs(lb, rb, [(0, 0, A.EQ)], capacity=len(wl))
    assert torch.equal(gl, wl) and torch.equal(gr, wr)
    out = ops.join_project(lb, rb, [(0, 0, A.EQ)], [(1, 1), (0, 1)], capacity=len(wl))
    assert torch.equal(out.columns[0].data, rv[wr.long()])
    assert torch.equal(out.columns[1].data, (lk * 100)[wl.long()])
