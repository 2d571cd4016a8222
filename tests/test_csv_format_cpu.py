"""The CSV writer's bound: the longest text of every cell type, formatted by the
writer's own code compiled for the host, against max_cell (from which buffers
for the one-pass writer are sized)."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
INT32, FLOAT32, DATETIME, TEXT, INT64 = 0, 1, 2, 3, 4


@pytest.fixture(scope="module")
def shim(tmp_path_factory):
    out = str(tmp_path_factory.mktemp("csvformat") / "libcsvformat.so")
    subprocess.check_call(["g++", "-std=c++17", "-O2", "-shared", "-fPIC", "-o", out,
                           os.path.join(HERE, "csv_format_shim.cpp")])
    return C.CDLL(out)


def cells(L, type_, values, nulls=None):
    values = np.ascontiguousarray(values)
    width = values.shape[1] if type_ == TEXT else values.itemsize
    out = []
    for r in range(len(values)):
        buf = C.create_string_buffer(1024)
        n = L.hs_format_cell(C.c_void_p(values.ctypes.data), None if nulls is None else C.c_void_p(nulls.ctypes.data),
                             type_, width, C.c_uint64(r), buf)
        assert n >= 0, "counted and written lengths differ"
        out.append(buf.raw[:n].decode("latin-1"))
    return out


def test_longest_cells(shim):
    i32, i64, f32 = np.iinfo(np.int32), np.iinfo(np.int64), np.finfo(np.float32)
    rng = np.random.default_rng(7)
    dates = np.concatenate([np.array([i64.min, i64.min + 1, i64.max, 0, -1, -(1 << 62), -3_155_760_000_000_000_000],
                                     np.int64),
                            rng.integers(i64.min, i64.max, 20_000, dtype=np.int64)])
    floats = np.concatenate([np.array([f32.max, -f32.max, np.inf, -np.inf, np.nan, -0.0, f32.tiny], np.float32),
                             rng.integers(0, 1 << 32, 20_000, dtype=np.uint64).astype(np.uint32).view(np.float32)])
    values = {INT32: np.array([i32.min, i32.max, 0], np.int32), INT64: np.array([i64.min, i64.max, 0], np.int64),
              FLOAT32: floats, DATETIME: dates}
    longest = {t: max(cells(shim, t, v), key=len) for t, v in values.items()}
    assert longest[INT32] == str(i32.min) and longest[INT64] == str(i64.min)
    assert longest[DATETIME] == '"-292277022657-01-27 08:29:52"'  # INT64_MIN seconds: a sign and twelve digits
    for t, text in longest.items():
        assert len(text) <= shim.hs_max_cell(t, values[t].itemsize), (t, text)
    for width in (1, 4, 16, 255, 256):
        full = np.full((1, width), ord("x"), np.uint8)
        assert len(cells(shim, TEXT, full)[0]) == width + 2 == shim.hs_max_cell(TEXT, width)
    one_null = np.ones(1, np.uint8)
    for t, v in values.items():
        assert cells(shim, t, v[:1], one_null) == ['""'] and shim.hs_max_cell(t, v.itemsize) >= 2
    assert shim.hs_max_cell(5, 1) == -1  # no text form


def test_year_beyond_eleven_digits(shim):
    """The first second of the year -99,999,999,999 and the one before it (year
    -100,000,000,000): the text grows from 29 bytes to 30 there."""
    y = -99_999_999_999 - 1  # January belongs to the year that began in March before: its day 306
    era = y // 400
    yoe = y - era * 400
    days = era * 146097 + yoe * 365 + yoe // 4 - yoe // 100 + 306 - 719468
    secs = days * 86400
    texts = cells(shim, DATETIME, np.array([secs, secs - 1], np.int64))
    assert texts == ['"-99999999999-01-01 00:00:00"', '"-100000000000-12-31 23:59:59"']
    assert len(texts[1]) == shim.hs_max_cell(DATETIME, 8)
