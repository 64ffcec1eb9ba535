"""Edges of the vector forms of the layout and elementwise kernels: widths of every alignment class, element counts around
one thread block's share (1 024 vectors), buffers whose address allows only a narrower access.  Copies are exact."""
import numpy as np
import pytest

from gpu_util import host, normal

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx(talos):
    c = talos.torch_context(0)
    yield c
    c.synchronize()


def _at(a, offset):
    """`a` on the device, `offset` floats behind a 256-byte boundary."""
    import torch
    buf = torch.full((a.size + offset + 8,), -7.0, device="cuda:0")
    buf[offset:offset + a.size] = torch.tensor(np.ascontiguousarray(a, dtype=np.float32).ravel(), device="cuda:0")
    return buf, buf.data_ptr() + 4 * offset


@pytest.mark.parametrize("shape,d0,d1", [((3, 5, 7, 4), 1, 2), ((2, 33, 31, 6), 1, 2), ((5, 3, 9, 5), 0, 2), ((4, 16, 16, 1), 1, 2), ((7, 2, 3, 8), 2, 0),
                                         ((1, 64, 8, 32), 1, 2), ((1, 65, 4, 16), 2, 1), ((2, 3, 4, 5, 8), 1, 3)])
@pytest.mark.parametrize("offset", [0, 1, 2])
def test_axis_swap(talos, ctx, shape, d0, d1, offset):
    x = normal(3, shape)
    bx, px = _at(x, offset); by, py = _at(np.zeros(x.size), offset)
    shp = np.array(shape, dtype=np.int64)
    talos.lib.talos_transpose(ctx.handle, px, py, talos.ptr(shp), len(shape), d0, d1, 0)
    got = host(by)
    assert np.array_equal(got[offset:offset + x.size].reshape(np.swapaxes(x, d0, d1).shape), np.swapaxes(x, d0, d1))
    assert np.all(got[:offset] == -7.0) and np.all(got[offset + x.size:] == -7.0)


@pytest.mark.parametrize("rows,da,db", [(1, 4, 4), (13, 8, 20), (85, 4, 8), (86, 4, 8), (37, 3, 5), (1025, 12, 4), (300, 0, 8)])
@pytest.mark.parametrize("acc", [0, 1])
def test_concat_and_split(talos, ctx, rows, da, db, acc):
    a, b = normal(4, (rows, da)), normal(5, (rows, db))
    ba, pa = _at(a, 0); bb, pb = _at(b, 0); bo, po = _at(np.zeros(rows * (da + db)), 0)
    talos.lib.talos_concat_last(ctx.handle, pa, pb, po, rows, da, db)
    both = np.concatenate([a, b], axis=1)
    assert np.array_equal(host(bo)[:both.size].reshape(both.shape), both)
    talos.lib.talos_split_last(ctx.handle, po, pa, pb, rows, da, db, acc)
    f = 2.0 if acc else 1.0                                   # x + x is exact
    assert np.array_equal(host(ba)[:a.size], f * a.ravel()) and np.array_equal(host(bb)[:b.size], f * b.ravel())
    assert np.all(host(ba)[a.size:] == -7.0) and np.all(host(bb)[b.size:] == -7.0)


@pytest.mark.parametrize("n", [1, 3, 4, 5, 2047, 2048, 2051, 4099])
@pytest.mark.parametrize("offset", [0, 1])
@pytest.mark.parametrize("op", ["add", "sub", "mul", "div"])
def test_binary_lengths(talos, ctx, n, offset, op):
    a, b = normal(6, (n,)), normal(7, (n,)); b[np.abs(b) < 0.1] = 0.5
    ba, pa = _at(a, offset); bb, pb = _at(b, offset)
    talos.lib.talos_eltwise_binary(ctx.handle, talos.EW[op], pa, pb, pa, n)        # in place, as a residual add may be
    f32 = np.float32
    ref = {"add": np.add, "sub": np.subtract, "mul": np.multiply, "div": np.divide}[op](a.astype(f32), b.astype(f32))     # one IEEE operation: exact
    got = host(ba)
    assert np.array_equal(got[offset:offset + n].astype(f32), ref)
    assert np.all(got[:offset] == -7.0) and np.all(got[offset + n:] == -7.0)


@pytest.mark.parametrize("act", ["relu", "tanh", "silu"])
@pytest.mark.parametrize("rows,width", [(1, 4), (5, 3), (129, 16), (64, 65)])
def test_linear_backward_without_bias_gradient(talos, ctx, act, rows, width, monkeypatch):
    # dZ = dY * act'(saved) as a pass of its own (no bias gradient asked for, and not the one launch that takes layers of this
    # size otherwise), in vectors and, for 15 elements, one by one; seen through an identity weight: dX = dZ
    monkeypatch.setenv("TALOS_TC_NO_SMALL", "1")
    saved, dy = normal(8, (rows, width)) * 0.7, normal(9, (rows, width))
    eye = np.eye(width)
    bs, ps = _at(saved, 0); bd, pd = _at(dy, 0); be, pe = _at(eye, 0); bx, px = _at(np.zeros(rows * width), 0)
    ctx.timeline_begin()
    talos.lib.talos_linear_bwd(ctx.handle, None, pe, ps, pd, px, None, None, rows, width, width, talos.ACTS[act], 0, 0)
    assert [name for name, _ in ctx.timeline_end()][0] == "dact_mul"
    if act == "relu":
        d = (saved > 0).astype(np.float64)
    elif act == "tanh":
        d = 1 - saved ** 2
    else:
        g = 1 / (1 + np.exp(-saved)); d = g * (1 + saved * (1 - g))
    assert np.allclose(host(bx)[:rows * width].reshape(rows, width), dy * d, rtol=1e-5, atol=1e-6)
