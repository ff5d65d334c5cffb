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


def test_late_products_keep_a_third_of_their_k_ranges():
    """The error of a three-pass product grows with the length of its K ranges, at a third of the rate that one accumulator for
    all passes had: with a third of the ranges it is what it was."""
    g, found = rng(7), 0
    for _ in range(3000):
        dims = [int(16 * 128 ** g.random())] + [int(16 * 64 ** g.random()) for _ in range(g.integers(1, 4))] + [int(2 * 500 ** g.random())]
        batch = int(16384 ** g.random())
        for l, share in late_weight_gradients(148, dims, batch).items():
            tiles, most = -(-dims[l + 1] // 128) * -(-dims[l] // 128), -(-batch // 32) // 4
            start = sum((dims[j] + 1) * dims[j + 1] for j in range(l))

            def ranges(sms):  # as gemm.cu splits: from three SMs per tile on, in clusters of eight without whole words
                n = max(1, min(sms // tiles, most))
                return 1 if n < 3 else (n if dims[l] % 4 == 0 and start % 4 == 0 else min(n, 8))

            assert 3 * ranges(share) >= ranges(148), (dims, batch, l)
            found += 1
    assert found > 100


@pytest.mark.gpu
@pytest.mark.parametrize("dims,batch", [([1000, 501, 301, 37], 1000), ([512, 512, 512, 512], 2000), ([512, 640, 257, 40], 1025), ([640, 385, 512, 300, 17], 1025)])
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
