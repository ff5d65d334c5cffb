"""Softmax cross-entropy on few rows (a row per warp) against float64, on both sides of the limits between its kernels."""
import numpy as np
import pytest

from zigrad_b200 import opspec

from .backends import GpuBackend
from .test_gpu_ops import rng

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bias", [False, True])
@pytest.mark.parametrize("index", [False, True])
@pytest.mark.parametrize("B,C", [(1, 2), (100, 10), (33, 32), (1000, 37), (65, 129), (17, 300), (40, 512), ("limit", 40), ("over", 40)])
def test_few_rows_against_float64(gpu, B, C, index, bias):
    B = {"limit": gpu.L.zg_sm_count() * 8, "over": gpu.L.zg_sm_count() * 8 + 1}.get(B, B)
    g = rng(B + C)
    be = GpuBackend(gpu)
    logits, lab = (3 * g.standard_normal((B, C))).astype(np.float32), g.integers(0, C, B)
    x = be.up(logits)
    T = be.up(lab.astype(np.uint64), np.uint64) if index else be.up(np.eye(C, dtype=np.float32)[lab])
    loss, d, db = be.up(np.zeros(1)), be.up(np.ones(B * C)), be.up(np.zeros(C))
    gpu.dispatch(opspec.softmax_ce(x, T, B, C, loss, d, float(B), accumulate=True, bias_grad=db if bias else None))
    z = logits.astype(np.float64) - logits.max(1, keepdims=True)
    p = np.exp(z) / np.exp(z).sum(1, keepdims=True)
    want = (p - np.eye(C)[lab]) / B
    assert np.abs(be.down(d).reshape(B, C) - 1 - want).max() <= 1e-6
    assert abs(be.down(loss)[0] + np.log(np.clip(p[np.arange(B), lab], 1e-7, 1 - 1e-7)).mean()) <= 1e-5
    if bias:
        assert np.abs(be.down(db) - want.sum(0)).max() <= 1e-6
