"""An equi-join without room for the sorted right side and its table gives the same
pairs through a form that needs a few words a tile."""
import ctypes as C

import pytest
import torch

from yallasql_b200 import _abi as A
from yallasql_b200 import ops

pytestmark = pytest.mark.gpu


def test_join_without_room_for_its_table(cuda, yq):
    """16 left rows, 20M right rows: the sorted table takes a gigabyte, the nested
    loop nothing; and a caller's workspace that only holds the nested loop."""
    rows = 20_000_000
    right = torch.arange(rows, dtype=torch.int32, device="cuda")
    left = torch.tensor([5, -1, rows - 1, rows, 7, 7, 123_456, 0] * 2, dtype=torch.int32, device="cuda")
    lb, rb = ops.DeviceBatch([ops.DeviceColumn(left, A.INT32)]), ops.DeviceBatch([ops.DeviceColumn(right, A.INT32)])
    want = [(i, int(v)) for i, v in enumerate(left.cpu().tolist()) if 0 <= v < rows]
    assert yq.yq_workspace_trim() == A.OK
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    hog = torch.empty(torch.cuda.mem_get_info()[0] - (320 << 20), dtype=torch.uint8, device="cuda")
    ol, orr = ops.join_pairs(lb, rb, [(0, 0, A.EQ)])
    assert list(zip(ol.cpu().tolist(), orr.cpu().tolist())) == want
    del hog
    torch.cuda.empty_cache()
    small = torch.empty(1 << 16, dtype=torch.uint8, device="cuda")
    outs = [torch.empty(64, dtype=torch.int32, device="cuda") for _ in range(2)]
    lc, k1 = lb.c()
    rc, k2 = rb.c()
    cond = (A.JoinCond * 1)(A.JoinCond(0, 0, A.EQ))
    n = C.c_uint64(0)
    st = yq.yq_join_pairs(C.byref(lc), C.byref(rc), cond, 1, outs[0].data_ptr(), outs[1].data_ptr(), 64, C.byref(n),
                          small.data_ptr(), small.numel(), None)
    assert st == A.OK
    got = list(zip(*[o[: n.value].cpu().tolist() for o in outs]))
    assert got == want
