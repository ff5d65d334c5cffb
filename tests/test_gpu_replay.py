"""Steps that a trainer replays as a graph of its own: same results as op-by-op steps, and never used for a call it was not
captured from (other buffers, other hyper-parameters, inside a caller's capture or branch)."""
import threading

import numpy as np
import pytest

from zigrad_b200 import replay, synthetic
from zigrad_b200.mlp import MlpTrainer, kaiming_uniform

pytestmark = pytest.mark.gpu


def graphs(tr):
    return sum(1 for e in tr._graphs.entries.values() if e.__class__ is tuple)


@pytest.mark.parametrize("kw", [dict(opt="sgd"), dict(opt="adam", clip=True), dict(opt="sgd", zero_grads_in_update=True), dict(opt="adam", fused=False)])
def test_repeated_steps_equal_op_by_op_steps(gpu, kw):
    dims, B = [100, 128, 64, 10], 96
    Ws, bs = kaiming_uniform(dims, 3)
    data = [gpu.from_numpy(a) for s in (1, 2) for a in synthetic.mlp_batch(B, 100, 10, s)[:2]]
    a, b = MlpTrainer(gpu, dims, B, Ws, bs, **kw), MlpTrainer(gpu, dims, B, Ws, bs, **kw)
    b._graphs.evicted = replay.GIVE_UP  # never replays
    for i in range(12):
        if i == 8:
            a.lr = b.lr = a.lr * 0.5
        for tr in (a, b):
            tr.step(data[2 * (i % 2)], data[2 * (i % 2) + 1])
        assert abs(a.read_loss() - b.read_loss()) <= 1e-5 * abs(b.read_loss()), i
    assert graphs(a) == 2 and graphs(b) == 0 and a.t == b.t
    if kw["opt"] == "adam":
        assert a.read_t() == a.t
    np.testing.assert_allclose(gpu.to_numpy(a.params), gpu.to_numpy(b.params), rtol=2e-3, atol=2e-6)
    for tr in (a, b):
        tr.free()
    for s in data:
        gpu.mem_cache_free(s)


def test_capture_branch_and_changing_buffers_stay_op_by_op(gpu):
    dims, B = [64, 32, 16], 40
    Ws, bs = kaiming_uniform(dims, 4)
    X, T = (gpu.from_numpy(a) for a in synthetic.mlp_batch(B, 64, 16, 1)[:2])
    tr = MlpTrainer(gpu, dims, B, Ws, bs, "sgd")
    for _ in range(2):
        tr.step(X, T)
    with gpu.branch(0):
        tr.step(X, T)
    gpu.join()
    gpu.capture.open()
    tr.step(X, T)
    gpu.capture.save()
    assert graphs(tr) == 0 and gpu.capture.kernel_count() > 3
    gpu.capture.run()
    gpu.capture.free()
    tr.step(X, T)
    assert graphs(tr) == 1
    others = [gpu.from_numpy(synthetic.mlp_batch(B, 64, 16, 2 + i)[0]) for i in range(replay.CAPACITY + 2)]
    for _ in range(4):
        for o in others:  # more buffers than places: each is forgotten before it comes back
            tr.step(o, T)
    assert graphs(tr) == 0 and len(tr._graphs.entries) <= replay.CAPACITY
    tr.free()
    for s in others + [X, T]:
        gpu.mem_cache_free(s)


def test_forward_alone_leaves_zeroed_gradients_behind(gpu):
    dims, B = [48, 40, 12], 24
    Ws, bs = kaiming_uniform(dims, 5)
    X, T = (gpu.from_numpy(a) for a in synthetic.mlp_batch(B, 48, 12, 1)[:2])
    tr = MlpTrainer(gpu, dims, B, Ws, bs, "adam")
    tr.step(X, T)
    assert gpu.to_numpy(tr.grads).any()
    first = gpu.to_numpy(tr.forward(X)).copy()
    assert not gpu.to_numpy(tr.grads).any()
    for _ in range(4):
        np.testing.assert_array_equal(gpu.to_numpy(tr.forward(X)), first)
    tr.loss_and_grad(T)
    tr.backward(X)
    once = gpu.to_numpy(tr.grads).copy()
    tr.backward(X)  # without a forward pass in between the weight gradients accumulate
    (gW, _), n = tr.get_grads(), tr.segments[0][1]
    np.testing.assert_allclose(gW[0].ravel(), 2 * once[:n], rtol=1e-4, atol=1e-7)
    tr.free()
    for s in (X, T):
        gpu.mem_cache_free(s)


def test_work_of_another_thread_stays_out_of_the_graph(gpu):
    """Fills, copies and synchronisation on the device's stream by a second thread while a step is captured happen there and
    then, and are not repeated by the steps that replay it."""
    dims, B = [64, 32, 16], 40
    Ws, bs = kaiming_uniform(dims, 4)
    X, T = (gpu.from_numpy(a) for a in synthetic.mlp_batch(B, 64, 16, 1)[:2])
    a, b = (MlpTrainer(gpu, dims, B, Ws, bs, "sgd") for _ in range(2))
    b._graphs.evicted = replay.GIVE_UP
    mine = gpu.from_numpy(np.zeros(1000, np.float32))
    seen, inner = [], a.loss_and_grad

    def other():
        gpu.mem_fill(mine, 7.0)
        seen.append(gpu.to_numpy(mine)[0])
        gpu.sync()

    def loss_and_grad(T):  # in the middle of the step
        th = threading.Thread(target=other)
        th.start()
        th.join()
        inner(T)

    a.loss_and_grad = loss_and_grad
    for i in range(6):
        gpu.mem_fill(mine, float(i))
        a.step(X, T)
        b.step(X, T)
    assert graphs(a) == 1 and seen == [7.0] * len(seen) and len(seen) == 3
    assert gpu.to_numpy(mine)[0] == 5.0  # what this thread put there last
    np.testing.assert_allclose(gpu.to_numpy(a.params), gpu.to_numpy(b.params), rtol=1e-4, atol=1e-6)
    for tr in (a, b):
        tr.free()
    for s in (X, T, mine):
        gpu.mem_cache_free(s)
