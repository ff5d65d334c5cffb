"""Where zero_grad happens: in stream order at each forward pass, whoever issues it -- op by op, from a graph the trainer
keeps, or from a graph of the caller's -- and never on a read or in an update.  Each sequence against a trainer that
issues every op anew."""
import numpy as np
import pytest

from zigrad_b200 import replay, synthetic
from zigrad_b200.mlp import MlpTrainer, kaiming_uniform

pytestmark = pytest.mark.gpu

DIMS, B = [48, 40, 24, 12], 32


class Pair:
    """A trainer as it is and one that keeps no graphs, with two batches."""

    def __init__(self, gpu, dims=DIMS, **kw):
        Ws, bs = kaiming_uniform(dims, 5)
        self.gpu = gpu
        self.data = [tuple(gpu.from_numpy(a) for a in synthetic.mlp_batch(B, dims[0], dims[-1], s)[:2]) for s in (1, 2)]
        self.a, self.b = (MlpTrainer(gpu, dims, B, Ws, bs, **kw) for _ in range(2))
        self.b._graphs.evicted = replay.GIVE_UP

    def backward(self, tr, k=0):
        tr.loss_and_grad(self.data[k][1])
        tr.backward(self.data[k][0])

    def check(self, what="params"):
        got, want = (self.gpu.to_numpy(getattr(tr, what)) for tr in (self.a, self.b))
        np.testing.assert_allclose(got, want, rtol=1e-4, atol=1e-6)
        return want

    def free(self):
        for tr in (self.a, self.b):
            tr.free()
        for s in (s for pair in self.data for s in pair):
            self.gpu.mem_cache_free(s)


@pytest.fixture(params=[dict(opt="sgd"), dict(opt="adam", clip=True), dict(opt="sgd", zero_grads_in_update=True)], ids=["sgd", "adam", "cleared"])
def pair(gpu, request):
    p = Pair(gpu, **request.param)
    yield p
    p.free()


def test_repeated_forward_without_an_update_in_between(gpu, pair):
    X = pair.data[0][0]
    for i in range(8):
        for tr in (pair.a, pair.b):
            tr.forward(X)
            pair.backward(tr)
            if i < 4 or i == 6:  # steps 4, 5 and 7 are skipped
                tr.update()
    pair.check("grads")
    pair.check()
