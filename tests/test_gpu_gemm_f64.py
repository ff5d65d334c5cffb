"""The persistent fp64 kernel at the edges of its 64 x {64, 48, 32} tiles and 32-deep slabs, with more tiles than SMs, against
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
