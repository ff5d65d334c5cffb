"""The FFMA / DFMA block kernel (small, unaligned and fp64 products) at the edges of its tiles, k slabs and
cluster splits, against a float64 product of the same operands."""
import numpy as np
import pytest

import oracle
from zigrad_b200 import opspec
from zigrad_b200.abi import BF16, DOUBLE, SINGLE

from .backends import GpuBackend
from .test_gpu_ops import rel_err, rng

pytestmark = pytest.mark.gpu

# tile edges (32, 64), slab edges (64; 32 in fp64), k ranges of 1 / 2 / 4 / 8 CTAs with and without a remainder
SHAPES = [(1, 1, 1), (1, 128, 784), (31, 33, 63), (32, 32, 64), (33, 65, 65), (64, 10, 255), (10, 37, 1000), (65, 129, 257), (700, 1001, 31)]


@pytest.mark.parametrize("ta,tb", [(False, False), (False, True), (True, False), (True, True)])
@pytest.mark.parametrize("kind", ["f32", "f64", "bf16"])
@pytest.mark.parametrize("m,n,k", SHAPES)
def test_block_gemm_edges(gpu, kind, m, n, k, ta, tb):
    g = rng(m * 7 + n * 3 + k)
    be = GpuBackend(gpu)
    nb = 2 if m * n < 20000 else 1
    ty = np.float64 if kind == "f64" else np.float32
    A, B, C0 = (g.standard_normal(s).astype(ty) for s in ((nb, k, m) if ta else (nb, m, k), (1, n, k) if tb else (1, k, n), (nb, m, n)))
    if kind == "bf16":
        A, B = (oracle.round_bf16(x.ravel()).reshape(x.shape) for x in (A, B))
        up = lambda x: be.up((x.view(np.uint32) >> 16).astype(np.uint16), np.uint16)
    else:
        up = be.up if kind == "f32" else (lambda x: be.up(x, np.float64))
    a, b, c = up(A), up(B), be.up(C0, ty)
    assert (a.dtype, c.dtype) == {"f32": (SINGLE, SINGLE), "f64": (DOUBLE, DOUBLE), "bf16": (BF16, SINGLE)}[kind]
    gpu.dispatch(opspec.linear(a, b, c, m, n, k, ta, tb, m if ta else k, k if tb else n, n, 0.5, 2.0, n_batch=(nb, 1, nb)))
    op = lambda x, t: (x.transpose(0, 2, 1) if t else x).astype(np.float64)
    want = 0.5 * (op(A, ta) @ op(B, tb)) + 2.0 * C0
    assert rel_err(be.down(c).reshape(nb, m, n), want) <= (1e-14 if kind == "f64" else 1e-5)


@pytest.mark.parametrize("m,n,k", [(1, 7, 3), (100, 50, 70), (37, 101, 515), (129, 300, 333), (1000, 1001, 77)])
def test_block_gemm_mask_and_column_sums(gpu, m, n, k):
    g = rng(m + n + k)
    be = GpuBackend(gpu)
    A, B = g.standard_normal((m, k)).astype(np.float32), g.standard_normal((k, n)).astype(np.float32)
    M, s0 = np.maximum(g.standard_normal((m, n)), 0).astype(np.float32), g.standard_normal(n).astype(np.float32)
    a, b, mk, c, s = be.up(A), be.up(B), be.up(M), be.up(np.zeros((m, n), np.float32)), be.up(s0)
    gpu.dispatch(opspec.linear(a, b, c, m, n, k, False, False, k, n, n, 1.0, 0.0, "relu_mask", None, mk, colsum=s))
    want = np.where(M > 0, A.astype(np.float64) @ B, 0.0)
    assert rel_err(be.down(c).reshape(m, n), want) <= 1e-5
    assert rel_err(be.down(s), s0 + want.sum(0)) <= 1e-5
