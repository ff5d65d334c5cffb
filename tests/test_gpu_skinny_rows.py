"""The transposed product with selected rows against float64: counts around the warps' stride, ragged columns, padded rows."""
import numpy as np
import pytest

from zigrad_b200 import opspec
from zigrad_b200.abi import SINGLE

from .backends import GpuBackend
from .test_gpu_ops import rel_err, rng

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N,U,C,ld", [(1, 1, 1, 1), (33, 17, 3, 4), (100, 50, 7, 8), (500, 64, 10, 12), (700, 65, 16, 16), (2708, 140, 7, 8)])
def test_rows_tn(gpu, N, U, C, ld):
    g = rng(N + U)
    be = GpuBackend(gpu)
    rows = np.sort(g.permutation(N)[:U]).astype(np.uint64)
    A, x = g.standard_normal((N, N)).astype(np.float32), np.zeros((N, ld), np.float32)
    x[rows] = g.standard_normal((U, ld))
    out = be.up(np.full((N, ld), 5.0, np.float32))
    assert gpu.rows_tn_supported(SINGLE, C) and not gpu.rows_tn_supported(SINGLE, 17)
    gpu.dispatch(opspec.rows_tn(out, ld, be.up(A), N, be.up(x), ld, be.up(rows, np.uint64), N, C))
    got = be.down(out).reshape(N, ld)
    assert rel_err(got[:, :C], A.T.astype(np.float64) @ x[:, :C]) <= 1e-5
    assert (got[:, C:] == 5.0).all()


@pytest.mark.parametrize("k", [12, 16, 124, 128, 132, 512])
@pytest.mark.parametrize("m,n", [(256, 10), (1001, 16), (255, 7)])
def test_few_columns_on_both_sides_of_the_longest_row(gpu, m, n, k):
    """Rows of 16 to 128 floats are walked by a quad of threads; shorter and longer ones take the other kernels."""
    g = rng(m + n + k)
    be = GpuBackend(gpu)
    A, B, bias = (g.standard_normal(s).astype(np.float32) for s in ((m, k), (n, k), (n,)))
    c = be.up(np.zeros((m, n), np.float32))
    gpu.dispatch(opspec.linear(be.up(A), be.up(B), c, m, n, k, False, True, k, k, n, 1.0, 0.0, "bias", be.up(bias)))
    # fp32 sums of k products in any order, or three truncated tf32 products each
    assert rel_err(be.down(c).reshape(m, n), A.astype(np.float64) @ B.T + bias) <= 1e-5
