"""Tensor-core products of operands without 16-byte rows (odd leading dimensions, bases between words, batches), whose operands
are copied into the work space first, against a float64 product of the same operands.  bf16 inputs are exact in fp32 and
the sums of k products are fp32: 2e-5 of the largest element (5e-6 seen); fp32 inputs in three TF32 passes: 5e-5, as for
aligned ones."""
import numpy as np
import pytest

import oracle
from zigrad_b200 import opspec
from zigrad_b200.device import DeviceSlice

from .backends import GpuBackend
from .test_gpu_ops import rel_err, rng

pytestmark = pytest.mark.gpu


def between_words(be, a, off, bf16):
    """The array on the device, `off` elements past a 16-byte boundary."""
    pad = np.zeros(off, np.float32)
    x = np.concatenate([pad, a.ravel()])
    s = be.up((x.view(np.uint32) >> 16).astype(np.uint16), np.uint16) if bf16 else be.up(x)
    return DeviceSlice(s.ptr + off * s.itemsize, a.size, s.dtype, 0)


@pytest.mark.parametrize("ta,tb", [(False, False), (False, True), (True, False), (True, True)])
@pytest.mark.parametrize("bf16,nb,m,n,k,off", [(True, 1, 300, 301, 501, 0), (True, 3, 129, 257, 263, 1), (True, 2, 2049, 513, 130, 7), (True, 1, 1000, 7, 2049, 3),
                                              (False, 1, 1023, 1001, 1001, 0), (False, 2, 701, 1024, 1003, 3)])
def test_operands_without_word_rows(gpu, bf16, nb, m, n, k, off, ta, tb):
    g, be = rng(m + n + k), GpuBackend(gpu)
    A, B = (g.standard_normal(s).astype(np.float32) for s in ((nb, k, m) if ta else (nb, m, k), (1, n, k) if tb else (1, k, n)))
    if bf16:
        A, B = (oracle.round_bf16(x.ravel()).reshape(x.shape) for x in (A, B))
    C0, bias = g.standard_normal((nb, m, n)).astype(np.float32), g.standard_normal(n).astype(np.float32)
    a, b = between_words(be, A, off, bf16), between_words(be, B, off, bf16)
    c = be.up(C0)
    gpu.dispatch(opspec.linear(a, b, c, m, n, k, ta, tb, m if ta else k, k if tb else n, n, 0.5, 2.0, "bias", be.up(bias), n_batch=(nb, 1, nb)))
    op = lambda x, t: (x.transpose(0, 2, 1) if t else x).astype(np.float64)
    want = 0.5 * (op(A, ta) @ op(B, tb)) + 2.0 * C0 + bias
    assert rel_err(be.down(c).reshape(nb, m, n), want) <= (2e-5 if bf16 else 5e-5)
