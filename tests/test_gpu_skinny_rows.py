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
