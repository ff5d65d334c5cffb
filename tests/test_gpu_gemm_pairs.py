"""Large single-pass products (256 x 256 tiles of CTA pairs) where the output path changes: ragged masked tiles in both output
types, rows of C that no tensor map describes, a tile whose second CTA has no rows, batches."""
import numpy as np
import pytest

import oracle
from zigrad_b200 import opspec

from .backends import GpuBackend
from .test_gpu_gemm import to_bf16_bits
from .test_gpu_ops import rel_err, rng

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,n,k,ldc,c16,epi,beta", [
    (2600, 1090, 520, 1096, True, "relu_mask", 0.0), (2600, 1090, 520, 1092, False, "relu_mask", 0.0), (2600, 1090, 520, 1090, False, "relu_mask", 0.0),
    (2433, 1025, 576, 1032, True, "bias_relu", 0.0), (2433, 1025, 576, 1025, False, "bias", 0.0), (2600, 1090, 2120, 1092, False, "none", 1.0),
    (2600, 1090, 2120, 1092, False, "none", 0.5), (2600, 1090, 2120, 1091, False, "none", 1.0)])
def test_output_paths_of_the_pair_kernel(gpu, m, n, k, ldc, c16, epi, beta):
    g = rng(m + n + k)
    r16 = lambda a: oracle.round_bf16(np.ascontiguousarray(a, np.float32).ravel()).reshape(a.shape)
    A, B, C0, mask = (r16(g.standard_normal(s).astype(np.float32)) for s in ((m, k), (n, k), (m, ldc), (m, ldc)))
    bias = g.standard_normal(n).astype(np.float32)
    be = GpuBackend(gpu)
    up = lambda x: be.up(to_bf16_bits(x), np.uint16) if c16 else be.up(x)
    c, cs = up(C0), be.up(np.zeros(n))
    gpu.dispatch(opspec.linear(be.up(to_bf16_bits(A), np.uint16), be.up(to_bf16_bits(B), np.uint16), c, m, n, k, False, True, k, k, ldc, 1.0, beta, epi,
                               be.up(bias) if epi.startswith("bias") else None, up(mask) if epi == "relu_mask" else None,
                               colsum=None if epi == "none" else cs))
    want = A.astype(np.float64) @ B.T.astype(np.float64) + beta * C0[:, :n] + (bias if epi.startswith("bias") else 0)
    if epi == "bias_relu":
        want = np.maximum(want, 0)
    if epi == "relu_mask":
        want[mask[:, :n] <= 0] = 0
    got = be.down(c)
    got = ((got.astype(np.uint32) << 16).view(np.float32) if c16 else got).reshape(m, ldc)
    assert rel_err(got[:, :n], want) <= (4e-3 if c16 else 1e-5)
    assert np.array_equal(got[:, n:], C0[:, n:])
    if epi != "none":
        assert rel_err(be.down(cs), want.sum(0)) <= 1e-4
