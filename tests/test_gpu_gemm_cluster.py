"""The tensor-core GEMM where its K ranges form clusters, where C is computed as its transpose and where operands or C are
not addressable by TMA (odd row lengths, unaligned bases), with every epilogue, against a float64 product."""
import numpy as np
import pytest

from zigrad_b200 import opspec

from .backends import GpuBackend
from .test_gpu_ops import rel_err, rng

pytestmark = pytest.mark.gpu


def run(gpu, m, n, k, ta, tb, epilogue, beta=0.0, shift=0):
    g = rng(m + 3 * n + 7 * k)
    be = GpuBackend(gpu)
    A, B = g.standard_normal((k, m) if ta else (m, k)).astype(np.float32), g.standard_normal((n, k) if tb else (k, n)).astype(np.float32)
    C0, bias, M = g.standard_normal((m, n)).astype(np.float32), g.standard_normal(n).astype(np.float32), np.maximum(g.standard_normal((m, n)), 0).astype(np.float32)

    def up(x):  # `shift` floats off the 16-byte boundary
        return be.up(np.concatenate([np.zeros(shift, np.float32), x.ravel()])).view(shift, x.size)

    a, b, c, s = up(A), up(B), up(C0), be.up(np.zeros(n, np.float32))
    kw = {"none": {}, "bias_relu": dict(bias=be.up(bias)), "relu_mask": dict(mask_src=up(M), colsum=s)}[epilogue]
    gpu.dispatch(opspec.linear(a, b, c, m, n, k, ta, tb, m if ta else k, k if tb else n, n, 0.5, beta, epilogue, **kw))
    want = 0.5 * ((A.T if ta else A).astype(np.float64) @ (B.T if tb else B)) + beta * C0
    if epilogue == "bias_relu":
        want = np.maximum(want + bias, 0)
    if epilogue == "relu_mask":
        want = np.where(M > 0, want, 0)
        assert rel_err(gpu.to_numpy(s), want.sum(0)) <= 1e-4
    assert rel_err(be.down(c).reshape(m, n), want) <= 3e-5


# clusters of 2 .. 8 with and without a ragged last range; 32-, 64- and 128-wide tiles; unaligned C (n or m odd)
@pytest.mark.parametrize("epilogue", ["none", "bias_relu", "relu_mask"])
@pytest.mark.parametrize("m,n,k", [(512, 512, 512), (1000, 301, 520), (2708, 16, 2708), (2000, 256, 1000), (130, 40, 12000), (4000, 32, 2000), (1100, 64, 900)])
def test_cluster_split(gpu, m, n, k, epilogue):
    run(gpu, m, n, k, False, True, epilogue, beta=0.0 if epilogue == "bias_relu" else 0.25)


@pytest.mark.parametrize("ta,tb", [(False, False), (False, True), (True, False), (True, True)])
@pytest.mark.parametrize("m,n,k,shift", [(1000, 501, 1001, 0), (333, 701, 333, 0), (4001, 65, 257, 0), (640, 512, 512, 1), (129, 515, 1000, 2), (2049, 1030, 70, 3)])
def test_unaligned_operands(gpu, m, n, k, shift, ta, tb):
    run(gpu, m, n, k, ta, tb, "relu_mask" if k % 2 else "none", beta=0.5, shift=shift)


@pytest.mark.parametrize("ta,tb", [(False, False), (False, True), (True, False), (True, True)])
@pytest.mark.parametrize("epilogue", ["none", "bias_relu", "relu_mask"])
@pytest.mark.parametrize("m,n,k", [(1, 4096, 1000), (33, 2001, 1001), (64, 1536, 600)])
def test_short_c_as_its_transpose(gpu, m, n, k, ta, tb, epilogue):
    run(gpu, m, n, k, ta, tb, epilogue, beta=0.5)


# C with rows longer than n: whatever path takes the product, what lies past column n is the caller's
@pytest.mark.parametrize("beta", [0.0, 0.5, 1.0])
@pytest.mark.parametrize("m,n,k,ldc,ta,tb,spoil", [
    (500, 389, 641, 392, False, True, False),    # unaligned K-major operands, K split
    (128, 781, 4096, 784, False, True, True),    # aligned operands, K split, an infinity in A
    (130, 258, 8200, 260, True, False, False),
    (384, 390, 2049, 392, True, True, False),
    (512, 512, 4096, 516, False, True, False),   # whole words: the tensor map clips them
])
def test_columns_past_n_stay(gpu, m, n, k, ldc, ta, tb, spoil, beta):
    g = rng(m + n + k)
    be = GpuBackend(gpu)
    A, B = g.standard_normal((k, m) if ta else (m, k)).astype(np.float32), g.standard_normal((n, k) if tb else (k, n)).astype(np.float32)
    C0 = g.standard_normal((m, ldc)).astype(np.float32)
    want = C0.astype(np.float64)
    want[:, :n] = 0.5 * ((A.T if ta else A).astype(np.float64) @ (B.T if tb else B)) + beta * want[:, :n]
    if spoil:
        A[0, 0] = np.inf
        want[0, :n] = np.nan
    c = be.up(C0)
    gpu.dispatch(opspec.linear(be.up(A), be.up(B), c, m, n, k, ta, tb, m if ta else k, k if tb else n, ldc, 0.5, beta))
    got = be.down(c).reshape(m, ldc)
    np.testing.assert_array_equal(got[:, n:], C0[:, n:])
    assert rel_err(got[1:, :n], want[1:, :n]) <= 3e-5


@pytest.mark.parametrize("beta", [0.0, 1.0])
@pytest.mark.parametrize("m,n,k,ldc", [(4096, 4093, 2048, 4096), (2304, 4094, 4096, 4100)])
def test_columns_past_n_stay_in_the_pair_kernel(gpu, m, n, k, ldc, beta):
    g = rng(m + n + k)
    be = GpuBackend(gpu)
    A, B = (synthetic_bf16(g, s) for s in ((m, k), (n, k)))
    C0 = g.standard_normal((m, ldc)).astype(np.float32)
    c = be.up(C0)
    a, b = gpu.from_numpy(A[0]), gpu.from_numpy(B[0])
    gpu.dispatch(opspec.linear(a, b, c, m, n, k, False, True, k, k, ldc, 1.0, beta))
    got = be.down(c).reshape(m, ldc)
    np.testing.assert_array_equal(got[:, n:], C0[:, n:])
    assert rel_err(got[:, :n], A[1] @ B[1].T + beta * C0[:, :n]) <= 1e-4
    gpu.mem_cache_free(a)
    gpu.mem_cache_free(b)


def synthetic_bf16(g, shape):
    """bf16 bit patterns and their values (truncated normals)."""
    bits = (g.standard_normal(shape).astype(np.float32).view(np.uint32) >> 16).astype(np.uint16)
    return bits, (bits.astype(np.uint32) << 16).view(np.float32)
