"""The workspace pool at the device's limits: what it keeps goes back on request,
and is there for other allocations of the process (torch's, the engine's, the
library's own outside the pool) that find the device full."""
import pytest
import torch

from yallasql_b200 import _abi as A
from yallasql_b200 import ops
from yallasql_b200.expr import Aggregate, ColumnRef

pytestmark = pytest.mark.gpu

MB = 1 << 20


def free_bytes():
    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]


def fill_pool(yq, rows=60_000_000):
    """The pool keeps a sort's workspace (20 bytes a row); nothing else is left behind."""
    col = ops.DeviceColumn(torch.arange(rows, dtype=torch.int32, device="cuda"), A.INT32)
    perm = torch.empty(rows, dtype=torch.int32, device="cuda")
    ops.sort_indices(col, descending=True, out=perm)
    torch.cuda.synchronize()
    del col, perm
    torch.cuda.empty_cache()


def fill_device(leave):
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    hog = torch.empty(free_bytes() - leave, dtype=torch.uint8, device="cuda")
    assert free_bytes() <= leave
    return hog


@pytest.fixture
def pool_on_full_device(cuda, yq):
    """About 320 MB free, a gigabyte of idle workspaces in the pool."""
    fill_pool(yq)
    hog = fill_device(320 * MB)
    yield yq
    del hog
    torch.cuda.empty_cache()
    assert yq.yq_workspace_trim() == A.OK


def test_trim_gives_the_memory_back(cuda, yq):
    torch.cuda.empty_cache()
    assert yq.yq_workspace_trim() == A.OK
    before = free_bytes()
    fill_pool(yq)
    held = before - free_bytes()
    assert 1000 * MB < held < 3000 * MB  # a sixty-fourth of the device at most
    assert yq.yq_workspace_trim() == A.OK
    assert before - free_bytes() < 64 * MB


def test_python_allocations(pool_on_full_device):
    col = ops.DeviceColumn.empty(A.INT64, 100_000_000)
    assert col.data.numel() == 100_000_000


def test_autotuner(pool_on_full_device):
    rows = 20_000_000
    col = ops.DeviceColumn(torch.arange(rows, dtype=torch.int32, device="cuda"), A.INT32)
    best = ops.sort_autotune(col, [0, rows])
    assert best.digit_bits in (4, 6, 8)


def test_rows_dropped_by_a_csv_scan(pool_on_full_device):
    """Dropping a row of the wrong field count copies each column: 256 MB here."""
    rows = 1 << 20
    body = b"x\n" * rows + b"x,y\n"
    text = torch.frombuffer(bytearray(body), dtype=torch.uint8).cuda()
    batch = ops.csv_scan(text, [A.TEXT], text_width=256)
    assert batch.rows == rows
    assert bool((batch.columns[0].data[:, 0] == ord("x")).all())


def test_engine_csv_text(pool_on_full_device):
    from yallasql_b200.plan import Plan
    rows = 45_000_000  # 405 MB of text, 180 MB of record starts
    p = Plan()
    root = p.aggregate(p.scan_csv(b"v(N)\n" + b"12345678\n" * rows, ["v"]),
                       [Aggregate(A.AGG_COUNT_STAR), Aggregate(A.AGG_SUM, ColumnRef(0, A.INT32))])
    got = [int(c[0][0]) for c in p.execute(root)]
    assert got == [rows, rows * 12345678]
