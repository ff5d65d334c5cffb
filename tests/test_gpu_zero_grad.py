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


def test_graph_of_the_caller_then_evaluation_then_update(gpu, pair):
    (X, T), other = pair.data[0], pair.data[1][0]
    pair.a.forward(other)
    gpu.capture.open()
    pair.a.forward(X)
    pair.backward(pair.a)
    gpu.capture.save()
    pair.a.forward(other)  # evaluation
    gpu.capture.run()
    pair.b.forward(X)
    pair.backward(pair.b)
    assert pair.check("grads").any()
    for tr in (pair.a, pair.b):
        tr.update()
    gpu.capture.free()
    pair.check()


def test_captured_forward_and_ops_behind_it(gpu):
    # (not with zero_grads_in_update: a graph captured while the update clears relies on the update)
    pair = Pair(gpu, opt="sgd")
    X = pair.data[0][0]
    gpu.capture.open()
    pair.a.forward(X)
    gpu.capture.save()
    for _ in range(3):
        gpu.capture.run()
        pair.backward(pair.a)
        pair.b.forward(X)
        pair.backward(pair.b)
        pair.check("grads")
        for tr in (pair.a, pair.b):
            tr.update()
    gpu.capture.free()
    pair.check()
    pair.free()


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


def test_a_slice_taken_before_shows_zeros_behind_a_forward_pass(gpu):
    pair = Pair(gpu, opt="adam")
    held, layer, X = pair.a.grads, pair.a.layer_grads(1), pair.data[0][0]
    for i in range(5):
        pair.a.forward(X)
        assert not gpu.to_numpy(held).any() and not gpu.to_numpy(layer).any(), i
        pair.backward(pair.a)
        assert gpu.to_numpy(held).any() and gpu.to_numpy(layer).any(), i
    gpu.mem_fill(held, 3.0)  # somebody else's writes are cleared as well
    pair.a.forward(X)
    assert not gpu.to_numpy(held).any()
    pair.free()


def test_graph_of_the_caller_over_a_trainer_that_never_had_gradients(gpu):
    pair = Pair(gpu, opt="none")
    X = pair.data[0][0]
    gpu.capture.open()
    pair.a.forward(X)
    gpu.capture.save()
    for _ in range(4):
        pair.a.forward(X)  # nothing to clear
    pair.backward(pair.a)
    gpu.capture.run()
    assert not gpu.to_numpy(pair.a.grads).any()
    gpu.capture.free()
    pair.free()


def test_without_fused_ops_backward_overwrites(gpu):
    """Op by op every gradient is written once per backward pass; a second one gives the same, not the sum."""
    pair = Pair(gpu, opt="sgd", fused=False)
    pair.a.forward(pair.data[0][0])
    pair.backward(pair.a)
    once = gpu.to_numpy(pair.a.grads).copy()
    pair.a.loss_and_grad(pair.data[0][1])
    pair.a.backward(pair.data[0][0])
    np.testing.assert_allclose(gpu.to_numpy(pair.a.grads), once, rtol=1e-5, atol=1e-8)
    pair.free()


@pytest.mark.parametrize("dims", [DIMS, [784, 128, 64, 10]], ids=str)
def test_step_leaves_the_gradients_it_declares_clear(gpu, dims):
    """zero_grads_in_update: behind a step every gradient is zero, so that the next forward pass need not clear them, an update
    without a backward pass moves nothing, and a loss of the caller's adds into zeros."""
    pair = Pair(gpu, dims, opt="sgd", zero_grads_in_update=True)
    (X, T), other = pair.data[0], pair.data[1][0]
    for i in range(4):  # op by op, then as a kept graph
        for tr in (pair.a, pair.b):
            tr.step(X, T)
            assert not gpu.to_numpy(tr._grads).any(), i
            tr.forward(other)
            assert not gpu.to_numpy(tr._grads).any(), i
            before = gpu.to_numpy(tr.params).copy()
            tr.update()
            np.testing.assert_array_equal(gpu.to_numpy(tr.params), before)
        pair.check()
    pair.free()
