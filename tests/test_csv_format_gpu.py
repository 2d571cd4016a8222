"""CSV writer at the limits of its one-pass form: a buffer of exactly the bound,
the longest cell of every type, and text past the 32-bit offsets."""
import ctypes as C
import json

import numpy as np
import pytest
import torch

import oracle
from yallasql_b200 import _abi as A
from yallasql_b200 import ops

pytestmark = pytest.mark.gpu

I64_MIN_DATE = b'"-292277022657-01-27 08:29:52"'  # INT64_MIN seconds, 30 bytes


def col(v, t):
    return ops.DeviceColumn(torch.from_numpy(np.ascontiguousarray(v)).cuda(), t)


def format_into(yq, batch, room, offset=0):
    """The text, and whether every byte around it stayed as it was."""
    bc, keep = batch.c()
    n = C.c_uint64(0)
    out = torch.full((room + offset + 256,), 0x7f, dtype=torch.uint8, device="cuda")
    st = yq.yq_csv_format(C.byref(bc), out.data_ptr() + offset, room, C.byref(n), None, 0, None)
    torch.cuda.synchronize()
    host = out.cpu().numpy()
    used = int(n.value) if st == A.OK else 0
    clean = bool((host[:offset] == 0x7f).all() and (host[offset + used:] == 0x7f).all())
    return st, int(n.value), host[offset:offset + used].tobytes(), clean


@pytest.mark.parametrize("rows", [1, 128, 129, 5000])
def test_buffer_of_exactly_the_bound(cuda, yq, rows):
    i64 = np.iinfo(np.int64)
    date = col(np.full(rows, i64.min), A.DATETIME)
    wide = ops.DeviceBatch([date, col(np.full(rows, i64.min), A.INT64),
                            col(np.full(rows, np.iinfo(np.int32).min, np.int32), A.INT32),
                            col(np.full((rows, 20), ord("x"), np.uint8), A.TEXT)])
    line = I64_MIN_DATE + b",-9223372036854775808,-2147483648,\"" + b"x" * 20 + b"\"\n"
    for batch, want in ((ops.DeviceBatch([date]), (I64_MIN_DATE + b"\n") * rows), (wide, line * rows)):
        bc, keep = batch.c()
        bound = int(yq.yq_csv_format_bound(C.byref(bc)))
        assert bound == len(want)  # every cell here is its type's longest
        for offset in (0, 3):
            st, n, text, clean = format_into(yq, batch, bound, offset)
            assert (st, n, clean) == (A.OK, bound, True) and text == want
        st, n, _, clean = format_into(yq, batch, bound - 1)
        assert (st, n, clean) == (A.ERR_CAPACITY, bound, True)
        assert ops.csv_format(batch).cpu().numpy().tobytes() == want


def test_extreme_numbers_within_the_bound(cuda, yq):
    f = np.array([np.finfo(np.float32).max, -np.finfo(np.float32).max, np.inf, -np.inf, np.nan, -0.0], np.float32)
    d = np.array([np.iinfo(np.int64).max, 0, -1, 1 << 32, (1 << 32) - 1, -(1 << 40)], np.int64)
    i = np.array([np.iinfo(np.int64).min, np.iinfo(np.int64).max, 0, -1, 10, 1 << 32], np.int64)
    nulls = np.array([0, 0, 1, 0, 1, 0], np.uint8)
    batch = ops.DeviceBatch([col(f, A.FLOAT32), ops.DeviceColumn(col(i, A.INT64).data, A.INT64,
                                                                 torch.from_numpy(nulls).cuda())])
    want = oracle.csv_format([(A.FLOAT32, 4, f, None), (A.INT64, 8, i, nulls)], len(f))
    bc, keep = batch.c()
    st, n, text, clean = format_into(yq, batch, int(yq.yq_csv_format_bound(C.byref(bc))))
    assert (st, clean) == (A.OK, True) and text == want
    dates = ops.DeviceBatch([col(d, A.DATETIME)])
    bc, keep = dates.c()
    st, n, text, clean = format_into(yq, dates, int(yq.yq_csv_format_bound(C.byref(bc))))
    assert (st, clean) == (A.OK, True)
    assert text.split(b"\n")[:5] == [b'"292277026596-12-04 15:30:07"', b'"1970-01-01 00:00:00"', b'"1969-12-31 23:59:59"',
                                     b'"2106-02-07 06:28:16"', b'"2106-02-07 06:28:15"']


def test_text_past_32_bit_offsets(cuda, yq):
    """140M dates: accepted by 29 bytes a date, 4.06 GB; their text is counted
    when it stays below 4 GiB and refused when thirty bytes a date pass it."""
    rows = 140_000_000
    data = torch.full((rows,), 86_400, dtype=torch.int64, device="cuda")
    batch = ops.DeviceBatch([ops.DeviceColumn(data, A.DATETIME)])
    bc, keep = batch.c()
    assert int(yq.yq_csv_format_bound(C.byref(bc))) >= 1 << 32
    n = C.c_uint64(0)
    assert yq.yq_csv_format(C.byref(bc), None, 0, C.byref(n), None, 0, None) == A.ERR_CAPACITY
    assert n.value == rows * 22
    data.fill_(np.iinfo(np.int64).min)
    assert yq.yq_csv_format(C.byref(bc), None, 0, C.byref(n), None, 0, None) == A.ERR_UNSUPPORTED
    more = ops.DeviceBatch([ops.DeviceColumn(torch.empty(143_165_577, dtype=torch.int64, device="cuda"), A.DATETIME)])
    bc, keep = more.c()  # 30 bytes a line with a date's 29: refused by its size
    assert yq.yq_csv_format(C.byref(bc), None, 0, C.byref(n), None, 0, None) == A.ERR_UNSUPPORTED


def test_result_is_the_texts_own_size(cuda):
    """The tensor holds the text and nothing else, and no more than the text is
    allocated for it on the way; another stream, no rows, a failed allocation."""
    rows = 300_000  # 7 bytes a line; the longest such line has 48 and 12
    batch = ops.DeviceBatch([col(np.full(rows, 7, np.float32), A.FLOAT32), col(np.arange(rows, dtype=np.int32) % 10, A.INT32)])
    want = b"".join(b"7.0000,%d\n" % (i % 10) for i in range(rows))
    torch.cuda.synchronize()
    torch.cuda.reset_peak_memory_stats()
    before = torch.cuda.memory_allocated()
    text = ops.csv_format(batch)
    assert torch.cuda.max_memory_allocated() - before <= len(want) + 4096
    assert text.untyped_storage().nbytes() == text.numel() == len(want)
    assert text.cpu().numpy().tobytes() == want
    side = torch.cuda.Stream()
    assert ops.csv_format(batch, stream=side).cpu().numpy().tobytes() == want
    assert ops.write_csv(["a", "b"], batch, stream=side) == b"a,b\n" + want
    none = ops.csv_format(ops.DeviceBatch([ops.DeviceColumn(torch.empty(0, device="cuda"), A.FLOAT32)]))
    assert none.numel() == 0 and none.is_cuda


def test_failed_allocation_of_the_text(cuda, monkeypatch):
    batch = ops.DeviceBatch([col(np.arange(1000, dtype=np.int32), A.INT32)])
    want = ops.csv_format(batch).cpu()

    def no_memory(*a, **k):
        raise torch.cuda.OutOfMemoryError("no room")
    with monkeypatch.context() as m:
        m.setattr(ops.torch, "empty", no_memory)
        with pytest.raises(torch.cuda.OutOfMemoryError, match="no room"):
            ops.csv_format(batch)
    assert torch.equal(ops.csv_format(batch).cpu(), want)


def test_profiled_bytes_hold_the_text(cuda, yq):
    """The write kernel's profiled bytes are the cells in and the text out, also
    where the text's length is read after the launch."""
    rows = 1000
    batch = ops.DeviceBatch([col(np.full(rows, 123456, np.int32), A.INT32)])
    bc, keep = batch.c()
    bound = int(yq.yq_csv_format_bound(C.byref(bc)))
    for room in (bound, rows * 7):  # one pass; the length first
        yq.yq_profile_enable(1)
        yq.yq_profile_read(None, 0, 1)
        st, n, text, _ = format_into(yq, batch, room)
        buf = C.create_string_buffer(1 << 14)
        yq.yq_profile_read(buf, len(buf), 1)
        yq.yq_profile_enable(0)
        assert (st, n) == (A.OK, rows * 7)
        got = json.loads(buf.value.decode())["csv_format_write"]
        assert got["launches"] == 1 and got["units"] == rows * 4 + rows * 7
