"""Broadcasts and column sums at the edges of the kernels that keep a column per thread: rows shorter and longer than a warp,
ragged and between words, one CTA of rows and more, both types; and the fill of segments.  Broadcasts are single
operations (exact); a column sum of at most 4099 values in fp32 1e-5, in fp64 1e-13 of the largest."""
import numpy as np
import pytest

from zigrad_b200 import opspec
from zigrad_b200.device import DeviceSlice

from .backends import GpuBackend
from .test_gpu_ops import rel_err, rng

pytestmark = pytest.mark.gpu


def past(s, n):
    return DeviceSlice(s.ptr + n * s.itemsize, s.len - n, s.dtype, 0)


@pytest.mark.parametrize("ty", [np.float32, np.float64])
@pytest.mark.parametrize("off", [0, 1])
@pytest.mark.parametrize("rows,L", [(1, 32), (9, 31), (300, 33), (5000, 36), (7, 1003), (4099, 1003), (33, 2048), (2, 100001), (3, 40), (801, 64), (70, 257),
                                    (15001, 33), (15301, 33), (20800, 96), (20801, 97), (20619, 97), (19999, 300), (20003, 301)])
def test_broadcast(gpu, rows, L, off, ty):
    g, be = rng(rows + L), GpuBackend(gpu)
    x, s = g.standard_normal(rows * L + off).astype(ty), g.standard_normal(L + off).astype(ty)
    X, S, Z = be.up(x, ty), be.up(s, ty), be.up(np.zeros(rows * L + off), ty)
    want = x[off:].reshape(rows, L)
    for a, b, w in ((past(X, off), past(S, off), want - s[off:]), (past(S, off), past(X, off), s[off:] - want)):
        gpu.dispatch(opspec.sub(a, b, past(Z, off)))
        np.testing.assert_array_equal(gpu.to_numpy(Z)[off:].reshape(rows, L), w)
    gpu.dispatch(opspec.add(past(X, off), past(S, off), past(X, off)))
    np.testing.assert_array_equal(be.down(X)[off:].reshape(rows, L), want + s[off:])


@pytest.mark.parametrize("ty", [np.float32, np.float64])
@pytest.mark.parametrize("rows,col", [(1, 5), (128, 10), (129, 127), (100, 128), (65, 129), (4099, 1003), (200, 4096), (5000, 1)])
def test_column_sums(gpu, rows, col, ty):
    g, be = rng(rows + col), GpuBackend(gpu)
    x, y = g.standard_normal((rows, col)).astype(ty), g.standard_normal(col).astype(ty)
    X, Y = be.up(x, ty), be.up(y, ty)
    gpu.dispatch(opspec.unbroadcast(X, [rows, col], Y, [col], None, 1.0, 0.5))
    assert rel_err(be.down(Y), x.astype(np.float64).sum(0) + 0.5 * y) <= (1e-5 if ty == np.float32 else 1e-13)


def test_fill_segments(gpu):
    be = GpuBackend(gpu)
    x = np.arange(70000, dtype=np.float32)
    X, want, segs = be.up(x), x.copy(), [(3, 1), (10, 0), (17, 60000), (69999, 1)] + [(61000 + 100 * i, i) for i in range(60)]
    gpu.fill_segments(X, segs, -2.5)
    for off, n in segs:
        want[off:off + n] = -2.5
    np.testing.assert_array_equal(be.down(X), want)


@pytest.mark.parametrize("ty", [np.float32, np.float64])
@pytest.mark.parametrize("rows,d", [(1, 9), (700, 13), (5, 31), (5000, 32), (300, 33), (4099, 45), (3, 288), (2, 1003)])
def test_row_maxima(gpu, rows, d, ty):
    g, be = rng(rows + d), GpuBackend(gpu)
    x = g.standard_normal((rows, d)).astype(ty)
    x[0] = -np.inf
    X, Y = be.up(x, ty), be.up(np.zeros(rows), ty)
    gpu.dispatch(opspec.max_along(X, [rows, d], Y, [rows, 1], 1))
    np.testing.assert_array_equal(be.down(Y), x.max(1))
