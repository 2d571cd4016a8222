"""Inequality joins that write other columns than the condition's own: every cell
width and null bytes of both sides, runs that start and end anywhere, room for a
part of the pairs, against a plain comparison of every pair."""
import ctypes as C

import numpy as np
import pytest
import torch

from yallasql_b200 import _abi as A
from yallasql_b200 import ops

pytestmark = pytest.mark.gpu

WIDTHS = [("flag", A.BOOL, 1), ("i32", A.INT32, 4), ("i64", A.INT64, 8), ("t12", A.TEXT, 12), ("t16", A.TEXT, 16),
          ("t20", A.TEXT, 20), ("t64", A.TEXT, 64)]


def side(rng, n, nullable):
    """The condition's column, then one of every width (as bytes and on the device)."""
    key = rng.integers(0, 1000, n).astype(np.int32)
    cols, host = [ops.DeviceColumn(torch.from_numpy(key).cuda(), A.INT32)], [(key.view(np.uint8).reshape(n, 4), None)]
    for _, t, w in WIDTHS:
        b = rng.integers(0, 256, (n, w), dtype=np.uint8)
        if t == A.BOOL:
            b &= 1
        nulls = (rng.random(n) < 0.2).astype(np.uint8) if nullable else None
        d = torch.from_numpy(b).cuda()
        data = d if t == A.TEXT else d.view(ops.TORCH_DTYPE[t]).flatten()
        cols.append(ops.DeviceColumn(data, t, None if nulls is None else torch.from_numpy(nulls).cuda()))
        host.append((b, nulls))
    return key, ops.DeviceBatch(cols), host


@pytest.mark.parametrize("cmp", [A.LT, A.NE])
@pytest.mark.parametrize("nullable", [False, True])
@pytest.mark.parametrize("L,R", [(1, 1), (3, 127), (17, 129), (5, 1000), (33, 4097), (1000, 33)])
def test_every_width(cuda, cmp, nullable, L, R):
    rng = np.random.default_rng(L * 7 + R + cmp)
    lk, lb, lh = side(rng, L, nullable)
    rk, rb, rh = side(rng, R, nullable)
    hit = lk[:, None] < rk[None, :] if cmp == A.LT else lk[:, None] != rk[None, :]
    wl, wr = np.nonzero(hit)  # left row major, right rows ascending
    alternate = [(i % 2, 1 + i) for i in range(len(WIDTHS))] + [(0, 0)]
    for outputs in (alternate, [(1 - s, c) for s, c in alternate]):
        got = ops.join_project(lb, rb, [(0, 0, cmp)], outputs)
        for (s, c), o in zip(outputs, got.columns):
            b, nulls = (rh if s else lh)[c]
            rows = wr if s else wl
            assert np.array_equal(o.data.view(torch.uint8).cpu().numpy().reshape(b[rows].shape), b[rows]), (s, c)
            if nulls is not None:
                assert np.array_equal(o.nulls.cpu().numpy(), nulls[rows]), (s, c)


@pytest.mark.parametrize("room", [1, 130, 1000, 4000])
@pytest.mark.parametrize("first", [0, 1])
def test_room_for_a_part(cuda, yq, room, first):
    """The first pairs are written, the exact count comes back, and nothing past
    the room is touched; null bytes of an input without any are zero."""
    rng = np.random.default_rng(room)
    lk, lb, lh = side(rng, 50, False)
    rk, rb, rh = side(rng, 300, False)
    wl, wr = np.nonzero(lk[:, None] < rk[None, :])
    assert len(wl) > 4000
    outputs = [((first + i) % 2, 1 + i) for i in range(len(WIDTHS))]
    guard = 64
    outs = []
    for s, c in outputs:
        _, t, w = WIDTHS[c - 1]
        raw = torch.full(((room + guard) * w,), 0x5a, dtype=torch.uint8, device="cuda")
        outs.append((raw, torch.full((room + guard,), 0x5a, dtype=torch.uint8, device="cuda"), t, w))
    oc = (A.Column * len(outs))(*[A.Column(r.data_ptr(), n.data_ptr(), t, w) for r, n, t, w in outs])
    oj = (A.JoinOutput * len(outputs))(*[A.JoinOutput(s, c) for s, c in outputs])
    cond = (A.JoinCond * 1)(A.JoinCond(0, 0, A.LT))
    lc, k1 = lb.c()
    rc, k2 = rb.c()
    n = C.c_uint64(0)
    st = yq.yq_join_project(C.byref(lc), C.byref(rc), cond, 1, oj, len(outputs), oc, room, C.byref(n), None, 0, None)
    torch.cuda.synchronize()
    assert st == A.ERR_CAPACITY and n.value == len(wl)
    for (s, c), (raw, nul, t, w) in zip(outputs, outs):
        b = (rh if s else lh)[c][0]
        rows = (wr if s else wl)[:room]
        host = raw.cpu().numpy().reshape(-1, w)
        assert np.array_equal(host[:room], b[rows]) and (host[room:] == 0x5a).all(), (s, c)
        nb = nul.cpu().numpy()
        assert not nb[:room].any() and (nb[room:] == 0x5a).all()


@pytest.mark.parametrize("kind", [A.INT32, A.FLOAT32, A.INT64, A.FLOAT64])
@pytest.mark.parametrize("L,R", [(1, 1), (255, 40), (257, 41), (5000, 5), (150_001, 3), (40_000, 33), (200_003, 40), (499_999, 41), (500_000, 72),
                                 (500_001, 73)])
def test_few_right_rows(cuda, kind, L, R):
    """Right sides around the 40 rows (72 from 500,000 left rows on) up to which
    every right row is a candidate of every left row (NaN meets nothing but under
    <>, -0.0 equals 0.0)."""
    rng = np.random.default_rng(L + R + kind)
    dt = {A.INT32: np.int32, A.FLOAT32: np.float32, A.INT64: np.int64, A.FLOAT64: np.float64}[kind]
    x, y = rng.integers(-40, 40, L).astype(dt), rng.integers(-40, 40, R).astype(dt)
    if L * R > 10_000_000:  # few pairs
        x[:] = 39
        x[::1000] = rng.integers(-40, 40, len(x[::1000]))
        y[:] = 39
        y[::9] = 38
    if kind in (A.FLOAT32, A.FLOAT64):
        x[::7], y[::5] = np.nan, -0.0
    wide = rng.integers(0, 256, (L, 20), dtype=np.uint8)
    dev = lambda v, t: ops.DeviceColumn(torch.from_numpy(np.ascontiguousarray(v)).cuda(), t)
    lb = ops.DeviceBatch([dev(x, kind), dev(wide, A.TEXT)])
    rb = ops.DeviceBatch([dev(y, kind), dev(np.arange(R, dtype=np.int64), A.INT64)])
    few = ((A.LT, np.less), (A.GT, np.greater), (A.NE, np.not_equal))
    for cmp, f in few if L * R > 10_000_000 else few + ((A.LE, np.less_equal), (A.GE, np.greater_equal)):
        wl, wr = np.nonzero(f(x[:, None], y[None, :]))
        gl, gr = ops.join_pairs(lb, rb, [(0, 0, cmp)], capacity=max(1, len(wl)))
        assert np.array_equal(gl.cpu().numpy(), wl) and np.array_equal(gr.cpu().numpy(), wr), cmp
        out = ops.join_project(lb, rb, [(0, 0, cmp)], [(0, 1), (1, 1)], capacity=max(1, len(wl)))
        assert np.array_equal(out.columns[0].data.cpu().numpy(), wide[wl]) and \
            np.array_equal(out.columns[1].data.cpu().numpy(), wr), cmp
