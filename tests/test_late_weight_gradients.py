"""Weight gradients behind the dX chain, side by side: their shares of the SMs, and the same gradients as beside the chain."""
import numpy as np
import pytest

from zigrad_b200.mlp import MlpTrainer, kaiming_uniform, late_weight_gradients

from .test_gpu_ops import rel_err, rng


@pytest.mark.parametrize("dims,batch", [([1000, 501, 301, 37], 1000), ([700, 900, 300, 100], 3000), ([512] * 6, 128), ([129, 65, 33, 17], 40000),
                                        ([784, 128, 64, 10], 8192), ([1024] * 5, 8192), ([8, 8, 8], 1), ([512, 512, 512], 2000)])
def test_shares(dims, batch):
    tiles = lambda l: -(-dims[l + 1] // 128) * -(-dims[l] // 128)
    for sms in (148, 132, 20):
        got = late_weight_gradients(sms, dims, batch)
        assert sum(got.values()) <= sms and len(got) != 1 and (not got or 0 in got)
        for l, share in got.items():
            assert share % tiles(l) == 0 and 1 <= share // tiles(l) <= max(1, -(-batch // 32) // 4)
    assert late_weight_gradients(148, [1000, 501, 301, 37], 1000) == {0: 96, 1: 48}
    assert late_weight_gradients(148, [1024] * 5, 8192) == {} == late_weight_gradients(148, [700, 900, 300, 100], 3000)


@pytest.mark.gpu
@pytest.mark.parametrize("dims,batch", [([1000, 501, 301, 37], 1000), ([512, 512, 512, 512], 2000), ([1024, 1024, 1024, 40], 1025), ([640, 641, 640, 639, 17], 700)])
def test_same_gradients(gpu, dims, batch):
    g = rng(batch)
    X, T = gpu.from_numpy(g.standard_normal((batch, dims[0])).astype(np.float32)), gpu.from_numpy(g.integers(0, dims[-1], batch).astype(np.uint64))
    got = []
    for late in (True, False):
        tr = MlpTrainer(gpu, dims, batch, *kaiming_uniform(dims, 3), opt="none", index_labels=True)
        assert tr._late
        if not late:
            tr._late = {}
        tr.step(X, T)
        got.append([gpu.to_numpy(w).copy() for w in tr.dW + tr.db])
    for a, b in zip(*got):  # the same three-pass products in other ranges of k: fp32 sums of the tensor core, 3e-5 as theirs
        assert rel_err(a, b) <= 3e-5
