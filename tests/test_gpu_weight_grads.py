"""All weight gradients of a network in one launch, at the edges of tiles, slabs and k ranges, with padded rows and each
output left out, against float64 (sums of at most 400 products in fp32: 1e-5 of the largest element, 1e-6 seen)."""
import numpy as np
import pytest

from zigrad_b200 import opspec

from .backends import GpuBackend
from .test_gpu_ops import rel_err, rng

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows", [1, 63, 64, 65, 200, 256, 400])
@pytest.mark.parametrize("dims", [(7, 1), (784, 128, 64, 10), (4, 128, 128, 2), (33, 31, 65, 3, 32)], ids=str)
@pytest.mark.parametrize("update", ["none", "both", "only"])
def test_weight_grads(gpu, dims, rows, update):
    g, be = rng(rows + len(dims)), GpuBackend(gpu)
    pad = 3
    f = lambda *s: g.standard_normal(s).astype(np.float32)
    items, want = [], []
    for k, n in zip(dims[:-1], dims[1:]):
        dy, x, W, b = f(rows, n + pad), f(rows, k + pad), f(n, k), f(n)
        dW, db = dy[:, :n].astype(np.float64).T @ x[:, :k], dy[:, :n].astype(np.float64).sum(0)
        keep, step = update != "only", update != "none"
        items.append((be.up(dy), be.up(x), be.up(f(n, k)) if keep else None, be.up(f(n)) if keep else None, be.up(W) if step else None,
                      be.up(b) if step else None, n, k, n + pad, k + pad))
        want.append((dW, db, W - 0.25 * dW, b - 0.25 * db))
    assert gpu.weight_grads_supported(items[0][0].dtype, items, rows)
    gpu.dispatch(opspec.weight_grads(items, rows, 0.25))
    for it, w in zip(items, want):
        for got, x in zip(it[2:6], w):
            if got is not None:
                assert rel_err(gpu.to_numpy(got).reshape(x.shape), x) <= 1e-5
    be.check_guards()


def test_weight_grads_leaves_large_products_to_the_tensor_cores(gpu):
    be = GpuBackend(gpu)
    s = be.up(np.zeros(4, np.float32))
    assert not gpu.weight_grads_supported(s.dtype, [(s, s, s, s, None, None, 512, 4096, 512, 4096)], 1024)


@pytest.mark.parametrize("rows", [400, 1000])
@pytest.mark.parametrize("dims", [(784, 48, 10), (146, 29, 200, 106), (256, 128, 16)], ids=str)
def test_error_of_the_sums(gpu, dims, rows):
    """Sums of 16 products that are added up, in the 2-norm: under two roundings of 2^-24 (9.6e-8 to 1.04e-7 seen; 1.11e-7 to
    1.56e-7 in one chain)."""
    g, be = rng(rows), GpuBackend(gpu)
    f = lambda *s: g.standard_normal(s).astype(np.float32)
    ops = [(f(rows, n), f(rows, k), n, k) for k, n in zip(dims[:-1], dims[1:])]
    items = [(be.up(dy), be.up(x), be.up(np.zeros((n, k))), None, None, None, n, k, n, k) for dy, x, n, k in ops]
    if not gpu.weight_grads_supported(items[0][0].dtype, items, rows):
        pytest.skip("left to the tensor cores")
    gpu.dispatch(opspec.weight_grads(items, rows))
    for it, (dy, x, n, k) in zip(items, ops):
        want = dy.astype(np.float64).T @ x
        err = np.linalg.norm(gpu.to_numpy(it[2]).reshape(n, k) - want) / np.linalg.norm(want)
        assert err <= 1.08e-7
