"""The masked softmax cross-entropy op against mem_take, softmax_ce and scatter_add issued separately (repeated rows included)."""
import numpy as np
import pytest

from zigrad_b200 import opspec
from zigrad_b200.abi import SINGLE

from .backends import GpuBackend
from .test_gpu_ops import rel_err, rng

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("index", [False, True])
@pytest.mark.parametrize("N,M,C,ld", [(5, 1, 1, 4), (300, 140, 7, 8), (900, 33, 33, 36), (5000, 2500, 40, 40), (64, 64, 1024, 1024)])
def test_masked_ce_equals_the_separate_ops(gpu, N, M, C, ld, index):
    g = rng(N + M + C)
    be = GpuBackend(gpu)
    logits, mask, lab = g.standard_normal((N, ld)).astype(np.float32), g.integers(0, N, M), g.integers(0, C, M)
    offs = (mask[:, None] * ld + np.arange(ld)[None, :]).astype(np.uint64)
    x, o, m1, dm = be.up(logits), be.up(offs, np.uint64), be.up(np.zeros((M, ld))), be.up(np.zeros((M, ld)))
    T = be.up(lab.astype(np.uint64), np.uint64) if index else be.up(np.eye(C, dtype=np.float32)[lab])
    d1, d2, l1, l2, b1, b2 = (be.up(np.zeros(k)) for k in (N * ld, N * ld, 1, 1, C, C))
    gpu.mem_take(x, o, m1)
    gpu.dispatch(opspec.softmax_ce(m1, T, M, C, l1, dm, float(M), accumulate=False, ld=ld, bias_grad=b1))
    gpu.dispatch(opspec.scatter_add(dm, o, d1))
    assert gpu.masked_softmax_ce_supported(SINGLE, M, C) and not gpu.masked_softmax_ce_supported(SINGLE, M, 1025)
    gpu.dispatch(opspec.masked_softmax_ce(x, o, T, M, C, ld, l2, d2, float(M), b2))
    w, l, b, wb = gpu.to_numpy(d1), gpu.to_numpy(l1), gpu.to_numpy(b1), gpu.to_numpy(b2)
    assert rel_err(gpu.to_numpy(l2), l) <= 1e-5 or abs(l[0]) < 1e-6
    assert np.abs(wb - b).max() <= 1e-5 * max(1.0, np.abs(b).max())
    assert np.abs(be.down(d2) - w).max() <= 1e-6
