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


@pytest.mark.parametrize("beta", [0.0, 1.0])
@pytest.mark.parametrize("nb,m,n,k,ldc", [(1, 3000, 1700, 4104, 1704), (2, 1500, 1780, 2568, 1780), (1, 2817, 1793, 2600, 1796)])
def test_tiles_of_the_last_wave_as_k_ranges(gpu, nb, m, n, k, ldc, beta):
    """84 tiles of 256 x 256 for 74 pairs: ten are split in K.  With beta = 0 they are cleared and added to, the others stored,
    whatever C holds; padding columns stay (n = 1793: element by element)."""
    g, be = rng(m + n + k), GpuBackend(gpu)
    A, B = (oracle.round_bf16(g.standard_normal(s).astype(np.float32).ravel()).reshape(s) for s in ((nb, m, k), (1, n, k)))
    C0 = g.standard_normal((nb, m, ldc)).astype(np.float32)
    if beta == 0.0:
        C0[:, ::3, :n] = np.nan
    c = be.up(C0)
    gpu.dispatch(opspec.linear(be.up(to_bf16_bits(A), np.uint16), be.up(to_bf16_bits(B), np.uint16), c, m, n, k, False, True, k, k, ldc, 1.0, beta,
                               n_batch=(nb, 1, nb)))
    want = A.astype(np.float64) @ B.transpose(0, 2, 1).astype(np.float64) + (C0[:, :, :n] if beta else 0.0)
    got = be.down(c).reshape(nb, m, ldc)
    assert rel_err(got[:, :, :n], want) <= 1e-5
    assert np.array_equal(got[:, :, n:], C0[:, :, n:])
