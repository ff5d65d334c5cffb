"""Softmax cross-entropy on few rows of at most 128 classes (one cluster) against fp64: edges of the lanes per row, of the CTAs
and of their trips; probabilities, accumulation, padded rows, labels past the classes."""
import numpy as np
import pytest

from zigrad_b200 import opspec

from .backends import GpuBackend
from .test_gpu_ops import rng

pytestmark = pytest.mark.gpu

WIDTHS = [(1, 1), (1, 8), (33, 7), (128, 10), (257, 9), (140, 16), (64, 17), (1000, 32), (31, 33), (257, 37), (1025, 64), (65, 65), (256, 127), (512, 128), (513, 128), (1024, 64),
          (2048, 16), (3072, 8), (3073, 8)]


@pytest.mark.parametrize("index", [False, True])
@pytest.mark.parametrize("R,C", WIDTHS)
def test_few_rows(gpu, R, C, index):
    g = rng(1000 * R + C)
    be = GpuBackend(gpu)
    ld, div = C + R % 3, float(R) if C % 2 else 64.0
    z, lab, old = g.standard_normal((R, ld)).astype(np.float32) * 3, g.integers(0, C, R), g.standard_normal((R, ld)).astype(np.float32)
    t = np.eye(C)[lab]
    if index and R > 2:
        lab[1] = C + 5  # in no class: no loss, nothing subtracted
        t[1] = 0.0
    z64 = z[:, :C].astype(np.float64)
    lp = z64 - z64.max(1, keepdims=True)
    lp -= np.log(np.exp(lp).sum(1, keepdims=True))
    p = np.exp(lp)
    loss = -(t * np.clip(lp, np.log(1e-7), np.log1p(-1.1920929e-07))).sum() / div
    dz = (p - t) / div
    x, dl, pr, ls, db = be.up(z), be.up(old), be.up(np.zeros((R, ld))), be.up(np.zeros(1)), be.up(np.zeros(C))
    T = be.up(lab.astype(np.uint64), np.uint64) if index else be.up(t.astype(np.float32))
    gpu.dispatch(opspec.softmax_ce(x, T, R, C, ls, dl, div, accumulate=True, ld=ld, bias_grad=db, probs=pr))
    # a probability: the exponential (2^-22, and 2^-24 |x - max| of the rounded product), its sum and the reciprocal
    eps = 2.0 ** -22 + 2.0 ** -24 * np.ptp(z64, axis=1).max() + 2.0 ** -22
    probs, bias, lo = (gpu.to_numpy(v) for v in (pr, db, ls))
    got = be.down(dl).reshape(R, ld)  # (frees them all)
    probs = probs.reshape(R, ld)
    assert np.abs(probs[:, :C] - p).max() <= 2 * eps
    assert np.abs(got[:, :C] - (old[:, :C] + dz)).max() <= 2 * eps / div + 2.0 ** -23 * np.abs(old).max()
    assert np.array_equal(got[:, C:], old[:, C:]) and not probs[:, C:].any()
    n = R + 16
    assert np.abs(bias - dz.sum(0)).max() <= (2 * eps * p.sum(0).max() + 2.0 ** -24 * n * (p + t).sum(0).max()) / div + 1e-9
    assert abs(lo[0] - loss) <= (2 * eps + 2.0 ** -24 * (R / 8 + 64)) * max(1.0, abs(loss)) * max(1.0, R / div)


@pytest.mark.parametrize("index", [False, True])
@pytest.mark.parametrize("R,C", [(129, 8), (65, 9), (1280, 32), (1281, 32), (200, 65), (2561, 16)])
def test_few_masked_rows(gpu, R, C, index):
    g = rng(R + C)
    be = GpuBackend(gpu)
    N, ld = R // 2, C + 1  # rows repeat
    z, mask, lab, old = g.standard_normal((N, ld)).astype(np.float32), g.integers(0, N, R), g.integers(0, C, R), g.standard_normal((N, ld)).astype(np.float32)
    lp = z[mask, :C].astype(np.float64)
    lp -= lp.max(1, keepdims=True)
    lp -= np.log(np.exp(lp).sum(1, keepdims=True))
    d = (np.exp(lp) - np.eye(C)[lab]) / R
    want = old.astype(np.float64)
    np.add.at(want[:, :C], mask, d)
    x, dl, ls, db = be.up(z), be.up(old), be.up(np.zeros(1)), be.up(np.zeros(C))
    o = be.up((mask[:, None] * ld + np.arange(ld)[None, :]).astype(np.uint64), np.uint64)
    T = be.up(lab.astype(np.uint64), np.uint64) if index else be.up(np.eye(C, dtype=np.float32)[lab])
    gpu.dispatch(opspec.masked_softmax_ce(x, o, T, R, C, ld, ls, dl, float(R), db))
    eps = 2.0 ** -21 + 2.0 ** -24 * 10
    bias, lo = gpu.to_numpy(db), gpu.to_numpy(ls)
    got, times = be.down(dl).reshape(N, ld), np.bincount(mask).max()
    assert np.abs(got - want).max() <= times * (2 * eps / R + 2.0 ** -23 * (np.abs(old).max() + times / R))
    assert np.array_equal(got[:, C:], old[:, C:])
    assert np.abs(bias - d.sum(0)).max() <= 2 * eps + 2.0 ** -24 * (R / 8 + 64)
    loss = -np.take_along_axis(lp, lab[:, None], 1).sum() / R
    assert abs(lo[0] - loss) <= (2 * eps + 2.0 ** -24 * (R / 8 + 64)) * max(1.0, loss)
