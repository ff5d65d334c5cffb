"""CSR propagation with hub rows (taken by a whole CTA): bit-identical to adding the neighbours in edge order, at the edges of
the hub threshold, of a gathered batch and of the feature tiles."""
import numpy as np
import pytest

from zigrad_b200 import opspec

from .test_gpu_ops import rng

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("F", [1, 7, 8, 9, 16, 17, 33])
@pytest.mark.parametrize("transpose", [False, True])
def test_hub_rows_in_edge_order(gpu, F, transpose):
    g = rng(F)
    N, ld = 300, F + 3
    counts = g.integers(0, 6, N)
    for r, n in zip((3, 50, 51, 120, 299), (64, 65, 225, 449, 1000)):
        counts[r] = n
    rp = np.concatenate([[0], np.cumsum(counts)]).astype(np.uint64)
    col = g.integers(0, N, int(rp[-1])).astype(np.uint64)
    x, deg, bias = g.standard_normal((N, ld)).astype(np.float32), g.random(N).astype(np.float32), g.standard_normal(F).astype(np.float32)
    want = np.zeros((N, F), np.float32)
    for r in range(N):
        for c in col[int(rp[r]):int(rp[r + 1])].astype(int):
            want[r] += (x[c, :F] * deg[r]) * deg[c] if transpose else (deg[c] * deg[r]) * x[c, :F]
        want[r] += bias
    bufs = [gpu.from_numpy(a) for a in (np.zeros((N, F), np.float32), x, deg, rp, col, bias)]
    o, xd, dd, rd, cd, bd = bufs
    gpu.dispatch(opspec.csr_gcn_propagate(o, xd, dd, rd, cd, N, F, ld, F, transpose, "bias", bd))
    np.testing.assert_array_equal(gpu.to_numpy(o).reshape(N, F), want)
    for b in bufs:
        gpu.mem_cache_free(b)
