"""bf16 products of operands without 16-byte rows into an fp32 C: sums that round to nearest, against float64 in the 2-norm.
64-wide tiles (k < 640, or few tiles) carry what an addition rounds off: what is left is one cut of a partial sum of 32 products and
the final rounding, up to 2^-24 each: 1.2e-7 (7.4e-8 seen).  128-wide ones add up k / 64 partial sums of 64 products: 2e-7 (1.7e-7 seen
up to k = 8000).  The tensor core's own sums are 4e-7 to 4e-6 off."""
import numpy as np
import pytest

import oracle
from zigrad_b200 import opspec
from zigrad_b200.abi import BF16
from zigrad_b200.device import DeviceSlice
from zigrad_b200.mlp import MlpTrainer, kaiming_uniform

from .backends import GpuBackend
from .test_gpu_gemm_repack import between_words
from .test_gpu_ops import rng

pytestmark = pytest.mark.gpu


def operands(g, nb, m, n, k, ta, tb):
    A, B = (g.standard_normal(s).astype(np.float32) for s in ((nb, k, m) if ta else (nb, m, k), (1, n, k) if tb else (1, k, n)))
    return (oracle.round_bf16(x.ravel()).reshape(x.shape) for x in (A, B))


@pytest.mark.parametrize("ta,tb", [(False, False), (False, True), (True, False), (True, True)])
@pytest.mark.parametrize("nb,m,n,k,bound", [(1, 701, 1609, 639, 1.2e-7),  # below the line
                                            (1, 701, 1609, 640, 2e-7),    # at it
                                            (1, 701, 1609, 641, 2e-7),
                                            (1, 1895, 1341, 2310, 2e-7),  # more tiles than SMs
                                            (3, 129, 67, 1851, 1.2e-7),   # clusters, batches
                                            (1, 301, 1105, 3605, 2e-7),
                                            (1, 45, 1931, 1419, 2e-7),    # C transposed
                                            (1, 1201, 289, 187, 1.2e-7),
                                            (2, 999, 501, 97, 1.2e-7)])
def test_sums_round(gpu, nb, m, n, k, bound, ta, tb):
    g, be = rng(m + n + k), GpuBackend(gpu)
    A, B = operands(g, nb, m, n, k, ta, tb)
    a, b, c = between_words(be, A, 1, True), between_words(be, B, 3, True), be.up(np.full((nb, m, n), np.nan, np.float32))
    gpu.dispatch(opspec.linear(a, b, c, m, n, k, ta, tb, m if ta else k, k if tb else n, n, 1.0, 0.0, n_batch=(nb, 1, nb)))
    op = lambda x, t: (x.transpose(0, 2, 1) if t else x).astype(np.float64)
    want = op(A, ta) @ op(B, tb)
    assert np.linalg.norm(be.down(c).reshape(nb, m, n) - want) <= bound * np.linalg.norm(want)


@pytest.mark.parametrize("dims,B", [([320, 253, 129, 24], 700), ([64, 72, 56, 152, 36], 1992)], ids=str)
def test_weight_gradients_of_padded_activations(gpu, dims, B):
    """Rows of odd hidden widths are padded to whole words; their weight gradients add up as those of dense rows do."""
    g = rng(B)
    bits = lambda a: (oracle.round_bf16(a.ravel()).view(np.uint32) >> 16).astype(np.uint16).reshape(a.shape)
    wide = lambda u: (u.astype(np.uint32) << 16).view(np.float32)
    X = bits(g.standard_normal((B, dims[0])).astype(np.float32))
    tr = MlpTrainer(gpu, dims, B, *kaiming_uniform(dims, 3), opt="none", bf16=True, index_labels=True)
    Xd, Td = gpu.from_numpy(X.view(np.uint16)), gpu.from_numpy(g.integers(0, dims[-1], B).astype(np.uint64))
    tr.step(DeviceSlice(Xd.ptr, X.size, BF16, 0), Td)
    grads = tr.get_grads()[0]
    for l, (K, N) in enumerate(zip(dims[:-1], dims[1:])):
        if K % 8 == 0 and (N if l + 2 < len(dims) else tr.ld_out) % 8 == 0:
            continue  # whole words all along: the tensor core's own sums
        dy = tr.act_numpy(l, grad=True)
        dy = wide(bits(dy)) if l + 2 == len(dims) else dy
        a = wide(X) if l == 0 else tr.act_numpy(l - 1)
        want = dy.astype(np.float64).T @ a
        assert np.linalg.norm(grads[l] - want) <= 2e-7 * np.linalg.norm(want), l
    for s in (Xd, Td):
        gpu.mem_cache_free(s)
    tr.free()


@pytest.mark.parametrize("k", [200, 1300])
def test_infinities_and_overflow(gpu, k):
    g, be, m, n = rng(k), GpuBackend(gpu), 901, 801
    A, B = operands(g, 1, m, n, k, False, True)
    A[0, 3, 40], A[0, 5, 7], A[0, 6, k - 1] = np.inf, np.nan, -np.inf
    A[0, 9], B[0, 11] = 2.0 ** 100, 2.0 ** 27  # a sum that overflows after the first part
    a, b, c = between_words(be, A, 1, True), between_words(be, B, 3, True), be.up(np.zeros((m, n), np.float32))
    gpu.dispatch(opspec.linear(a, b, c, m, n, k, False, True, k, k, n, 1.0, 0.0))
    got = be.down(c).reshape(m, n)
    B = B[0]
    np.testing.assert_array_equal(got[3], np.where(B[:, 40] > 0, np.inf, np.where(B[:, 40] < 0, -np.inf, np.nan)).astype(np.float32))
    np.testing.assert_array_equal(got[6], np.where(B[:, k - 1] > 0, -np.inf, np.where(B[:, k - 1] < 0, np.inf, np.nan)).astype(np.float32))
    assert np.isnan(got[5]).all() and got[9, 11] == np.inf
    rest = np.delete(np.delete(got, [3, 5, 6, 9], 0), 11, 1)
    assert np.isfinite(rest).all()
