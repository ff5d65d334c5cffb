"""A step clears of its gradients only what it accumulates into and writes those of large weights: from whatever the buffer holds it
comes out with the gradients that a new trainer's first step has, op by op and as a kept graph."""
import numpy as np
import pytest

from zigrad_b200 import replay
from zigrad_b200.mlp import MlpTrainer, kaiming_uniform

from .test_gpu_ops import rel_err, rng

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kept", [False, True], ids=["op by op", "kept graph"])
@pytest.mark.parametrize("bf16", [False, True], ids=["fp32", "bf16"])
@pytest.mark.parametrize("dims", [[1024, 1024, 96, 40], [640, 96, 1100, 1000, 24], [1030, 1020, 17]], ids=str)  # large layers first, in the middle, with odd rows
def test_gradients_behind_other_gradients(gpu, dims, bf16, kept):
    B, g = 1024, rng(len(dims))
    Ws, bs = kaiming_uniform(dims, 3)

    def batch():
        X = g.standard_normal((B, dims[0])).astype(np.float32)
        return (gpu.from_numpy((X.view(np.uint32) >> 16).astype(np.uint16) if bf16 else X), gpu.from_numpy(g.integers(0, dims[-1], B).astype(np.uint64)))

    def trainer():
        tr = MlpTrainer(gpu, dims, B, Ws, bs, opt="none", bf16=bf16, index_labels=True)
        assert not tr.grouped and any(tr._large(l) for l in range(tr.L)) and not all(tr._large(l) for l in range(tr.L))
        return tr

    first, second = batch(), batch()
    new, tr = trainer(), trainer()
    new.step(*second)
    want = [gpu.to_numpy(w).copy() for w in new.dW + new.db]
    if not kept:
        tr._graphs.evicted = replay.GIVE_UP
    tr.step(*first)
    for i in range(5):
        gpu.mem_fill(tr.grads, float("nan") if i % 2 else 3.0)
        tr.step(*second)
        for a, w in zip(tr.dW + tr.db, want):  # (sums of up to 1024 products on the tensor cores, in K ranges that are added in any order)
            assert rel_err(gpu.to_numpy(a), w) <= 3e-5, i
    for t in (new, tr):
        t.free()
    for s in first + second:
        gpu.mem_cache_free(s)
