"""The error of three-pass fp32 products against float64, in the 2-norm, where narrower tiles take fewer K ranges than 128-wide ones
would.  Bound: what 128-wide tiles with one accumulator for all three passes give there (first figure; 64-wide tiles with it
the second).  With the small products in an accumulator of their own a range of k products is off by about 2.3e-9 k + 4e-7 (7e-9
with one)."""
import numpy as np
import pytest

from zigrad_b200 import opspec

from .backends import GpuBackend
from .test_gpu_ops import rng

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,n,k,ta,tb,bound", [(80, 1840, 2192, True, True, 2.3e-6),    # 4.3e-6
                                               (114, 1678, 3087, False, True, 3.2e-6),  # 5.8e-6
                                               (659, 367, 1094, True, True, 1.7e-6),    # 3.0e-6
                                               (96, 1880, 4048, False, True, 3.9e-6),   # 7.5e-6
                                               (494, 1150, 1037, True, True, 2.8e-6)])  # 4.0e-6
def test_error_of_clustered_products(gpu, m, n, k, ta, tb, bound):
    g, be = rng(m + n + k), GpuBackend(gpu)
    A, B, bias = (g.standard_normal(s).astype(np.float32) for s in ((k, m) if ta else (m, k), (n, k) if tb else (k, n), n))
    c = be.up(np.zeros((m, n), np.float32))
    gpu.dispatch(opspec.linear(be.up(A), be.up(B), c, m, n, k, ta, tb, m if ta else k, k if tb else n, n, 1.0, 0.0, "bias", be.up(bias)))
    want = (A.T if ta else A).astype(np.float64) @ (B.T if tb else B) + bias
    assert np.linalg.norm(be.down(c).reshape(m, n) - want) <= bound * np.linalg.norm(want)
