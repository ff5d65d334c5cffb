"""CSR propagation over many rows (several of them per warp): the same sums, bit for bit, as a warp per row, which rows of x that
are no whole 16-byte words get."""
import numpy as np
import pytest

from zigrad_b200 import opspec

from .backends import GpuBackend
from .test_gpu_ops import rng

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("epilogue", ["none", "bias_relu"])
@pytest.mark.parametrize("transpose", [False, True])
@pytest.mark.parametrize("F", [1, 7, 8, 9, 16, 17, 32])
def test_rows_by_lanes_equal_a_warp_per_row(gpu, F, transpose, epilogue):
    g = rng(F)
    be = GpuBackend(gpu)
    N = (128 if F <= 16 else 64) * gpu.sm_count() + 37
    n = g.integers(0, 20, N)
    n[:9] = [0, 8, 9, 16, 17, 64, 65, 700, 4]
    n[N - 1], n[1000:1200] = 300, 12
    rp = np.concatenate([[0], np.cumsum(n)]).astype(np.uint64)
    col = g.integers(0, N, int(rp[-1])).astype(np.uint64)
    deg, x, b = (g.random(k).astype(np.float32) + 0.1 for k in (N, N * F, F))
    got = []
    for ld in ((F + 3) // 4 * 4, (F + 3) // 4 * 4 + 1):
        X = np.zeros((N, ld), np.float32)
        X[:, :F] = x.reshape(N, F)
        rows, cols, d, bias = be.up(rp, np.uint64), be.up(col, np.uint64), be.up(deg), be.up(b)  # (down() frees them)
        X, out = be.up(X), be.up(np.full((N, ld), -7.0))
        gpu.dispatch(opspec.csr_gcn_propagate(out, X, d, rows, cols, N, F, ld, ld, transpose, epilogue, bias if epilogue != "none" else None))
        o = be.down(out).reshape(N, ld)
        assert (o[:, F:] == -7.0).all()
        got.append(o[:, :F].copy())
    assert np.array_equal(*got)
    xs, order = x.reshape(N, F), lambda r: col[int(rp[r]):int(rp[r + 1])].astype(np.int64)
    for r in (0, 1, 7, 1000, N - 1):
        w = np.zeros(F, np.float32)
        for c in order(r):
            w = w + ((xs[c] * deg[r]) * deg[c] if transpose else (deg[c] * deg[r]) * xs[c])
        w = np.maximum(w + b, 0) if epilogue != "none" else w
        assert np.abs(got[0][r] - w).max() <= 2.0 ** -23 * (len(order(r)) + 2) * max(1.0, np.abs(w).max())
