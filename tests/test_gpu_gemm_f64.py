"""The persistent fp64 kernel, and the block kernel that takes the shortest sums, at the edges of its 64 x {64, 48, 32} tiles and 32-deep slabs, with more tiles than SMs, against
numpy's product of the same operands (1e-14 of the largest element: k = 700 sums in another order, 1e-15 seen)."""
import numpy as np
import pytest

from zigrad_b200 import opspec

from .backends import GpuBackend
from .test_gpu_ops import rel_err, rng

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ta,tb", [(False, False), (False, True), (True, False), (True, True)])
@pytest.mark.parametrize("nb,m,n,k", [(2, 641, 640, 1), (3, 640, 333, 31), (1, 1000, 1025, 33), (19, 129, 191, 64), (40, 65, 97, 130), (150, 64, 63, 700)])
def test_fp64_products(gpu, nb, m, n, k, ta, tb):
    g, be = rng(m * 7 + n * 3 + k), GpuBackend(gpu)
    A, B, C0 = (g.standard_normal(s) for s in ((nb, k, m) if ta else (nb, m, k), (1, n, k) if tb else (1, k, n), (nb, m, n)))
    a, b, c = (be.up(x, np.float64) for x in (A, B, C0))
    gpu.dispatch(opspec.bmm_acc(a, b, c, (nb, m, k), (1, k, n), (nb, m, n), ta, tb, m if ta else k, k if tb else n, n, 0.5, 2.0))
    op = lambda x, t: x.transpose(0, 2, 1) if t else x
    assert rel_err(be.down(c).reshape(nb, m, n), 0.5 * (op(A, ta) @ op(B, tb)) + 2.0 * C0) <= 1e-14


@pytest.mark.parametrize("ta,tb", [(False, False), (False, True), (True, False), (True, True)])
@pytest.mark.parametrize("k", [1, 24, 48, 49, 81])
@pytest.mark.parametrize("nb,m,n", [(45, 127, 128), (44, 128, 127), (178, 63, 64), (10, 451, 397), (5, 215, 479), (2, 302, 817)])
def test_fp64_short_sums(gpu, nb, m, n, k, ta, tb):
    g, be = rng(m * 7 + n * 3 + k), GpuBackend(gpu)
    A, B = (g.standard_normal(s) for s in ((nb, k, m) if ta else (nb, m, k), (1, n, k) if tb else (1, k, n)))
    a, b, c = be.up(A, np.float64), be.up(B, np.float64), be.up(np.full((nb, m, n), np.nan), np.float64)
    gpu.dispatch(opspec.bmm_acc(a, b, c, (nb, m, k), (1, k, n), (nb, m, n), ta, tb, m if ta else k, k if tb else n, n, 0.5, 0.0))
    op = lambda x, t: x.transpose(0, 2, 1) if t else x
    assert rel_err(be.down(c).reshape(nb, m, n), 0.5 * (op(A, ta) @ op(B, tb))) <= 1e-14


@pytest.mark.parametrize("epilogue", ["bias", "bias_relu", "relu_mask"])
@pytest.mark.parametrize("beta", [0.0, 0.5])
@pytest.mark.parametrize("nb,m,n,k", [(1, 1000, 1025, 33), (1, 1000, 1025, 48), (1, 641, 1000, 130), (1, 2049, 331, 65), (1, 6000, 40, 31)])
def test_fp64_epilogues(gpu, nb, m, n, k, beta, epilogue):
    """More than half a tile per SM, so that the persistent kernel finishes C."""
    g, be = rng(m + n + k), GpuBackend(gpu)
    A, B, C0, mask, bias = (g.standard_normal(s) for s in ((m, k), (n, k), (m, n), (m, n), n))
    bias = bias.astype(np.float32)
    c = be.up(C0, np.float64)
    gpu.dispatch(opspec.linear(be.up(A, np.float64), be.up(B, np.float64), c, m, n, k, False, True, k, k, n, 0.5, beta, epilogue,
                               be.up(bias) if epilogue != "relu_mask" else None, be.up(mask, np.float64) if epilogue == "relu_mask" else None))
    want = 0.5 * (A @ B.T) + beta * C0
    if epilogue != "relu_mask":
        want = want + bias
    if epilogue == "bias_relu":
        want = np.maximum(want, 0.0)
    if epilogue == "relu_mask":
        want = np.where(mask <= 0.0, 0.0, want)
    assert rel_err(be.down(c).reshape(m, n), want) <= 1e-14
