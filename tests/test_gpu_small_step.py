"""Clipped optimizer steps over small tensors (one launch) against the oracle: lengths around the cluster sizes, clipped and not."""
import numpy as np
import pytest

from zigrad_b200 import opspec

from .backends import GpuBackend, OracleBackend
from .test_gpu_ops import rel_err, rng

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("limit", [0.5, 1e6])
@pytest.mark.parametrize("lens", [(1,), (4096, 1), (4097, 2, 3), (32768, 129), (32769, 129), (0, 500), (64,) * 13, (9000,) * 40], ids=lambda x: str(x[:3]))
def test_clipped_step(gpu, lens, limit):
    n, g = sum(lens), rng(sum(lens))
    segs, off = [], 1  # tensors start on any element
    for k in lens:
        segs.append((off, k))
        off += k
    p, gr, m = (g.standard_normal(off).astype(np.float32) for _ in range(3))
    v = g.random(off).astype(np.float32)
    be = GpuBackend(gpu)
    P, G, M, V, N = (be.up(x) for x in (p, gr, m, v, np.zeros(len(segs))))
    gpu.dispatch(opspec.adam(P, G, M, V, segs, 5, 1e-3, clip=True, max_norm=limit, norms=N))
    want = OracleBackend().adam(p, gr, m, v, segs, 5, 1e-3, clip=True, max_norm=limit)
    for got, w in zip((P, G, M, V), want):
        assert rel_err(gpu.to_numpy(got), w) <= 1e-6
    norms = [np.linalg.norm(gr[o:o + k].astype(np.float64)) for o, k in segs]
    assert np.allclose(be.down(N), norms, rtol=1e-6)
    for zero in (False, True):
        P, G, N = be.up(p), be.up(gr), be.up(np.zeros(len(segs)))
        gpu.dispatch(opspec.sgd(P, G, segs, 0.1, True, limit, 1e-6, N, zero))
        wp, wg = OracleBackend().sgd(p, gr, segs, 0.1, True, limit, 1e-6)
        assert rel_err(gpu.to_numpy(P), wp) <= 1e-6
        got = gpu.to_numpy(G)
        for o, k in segs:
            assert np.array_equal(got[o:o + k], np.zeros(k)) if zero else np.allclose(got[o:o + k], wg[o:o + k], rtol=1e-6, atol=0)
