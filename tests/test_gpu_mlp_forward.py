"""The one-launch forward pass on one row against float64: widths around its limits, one layer and many."""
import numpy as np
import pytest

from zigrad_b200.abi import DOUBLE, SINGLE
from zigrad_b200.mlp import MlpTrainer, kaiming_uniform

from .backends import GpuBackend
from .test_gpu_ops import rel_err, rng

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims", [[784, 128, 64, 10], [1, 1], [7, 3, 129, 1], [1030, 157, 5], [33, 1100, 130], [6, 5, 4, 3, 4, 5, 6, 7, 8], [1025, 190]],
                         ids=lambda d: "-".join(map(str, d)))
def test_forward_on_one_row(gpu, dims):
    assert gpu.mlp_forward_supported(SINGLE, dims) and not gpu.mlp_forward_supported(DOUBLE, dims)
    assert not gpu.mlp_forward_supported(SINGLE, [4] * 10) and not gpu.mlp_forward_supported(SINGLE, [1000, 200, 1])
    Ws, bs = kaiming_uniform(dims, 3)
    g = rng(dims[0])
    bs = [g.standard_normal(b.shape).astype(np.float32) for b in bs]
    x = g.standard_normal((1, dims[0])).astype(np.float32)
    tr = MlpTrainer(gpu, dims, 1, Ws, bs, "none")
    X = GpuBackend(gpu).up(x)
    want = x.astype(np.float64)
    for _ in range(4):  # issued, then replayed
        tr.forward(X)
    for l, (W, b) in enumerate(zip(Ws, bs)):
        want = want @ np.asarray(W, np.float64).reshape(dims[l + 1], dims[l]).T + b
        if l + 2 < len(dims):
            want = np.maximum(want, 0)
        assert rel_err(tr.act_numpy(l), want) <= 1e-5
    tr.free()
