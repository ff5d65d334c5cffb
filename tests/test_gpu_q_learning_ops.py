"""The Q-learning head op against the separate ops it stands for, and the Adam step with
clipping, device step counter and soft target update against the oracle."""
import numpy as np
import pytest

from zigrad_b200 import opspec
from zigrad_b200.dqn import DqnTrainer
from zigrad_b200.mlp import kaiming_uniform

from .backends import GpuBackend, OracleBackend
from .test_gpu_ops import rel_err, rng

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,A", [(1, 1), (31, 2), (256, 18), (257, 5), (3000, 64), (70000, 3)])
def test_q_head_equals_the_separate_ops(gpu, B, A):
    g = rng(B + A)
    Ws, bs = kaiming_uniform([4, 8, A], 1)
    tr = DqnTrainer(gpu, [4, 8, A], B, Ws, bs, q_clip=1.5)
    qn, q = (g.standard_normal((B, A)).astype(np.float32) for _ in range(2))
    act, rew, done = g.integers(0, A, B).astype(np.uint64), g.standard_normal(B).astype(np.float32), (g.random(B) < 0.2).astype(np.float32)
    a, r, dn = (gpu.from_numpy(x) for x in (act, rew, done))
    outs = {}
    for how in ("ops", "op"):
        dqn, dq = gpu.from_numpy(qn), gpu.from_numpy(q)
        if how == "ops":
            tr._head(dqn, dq, a, r, dn)
            gpu.dispatch(opspec.unbroadcast(tr.policy.dact[-1], [B, A], tr.policy._db[-1], [A], None, 1.0, 0.0))
        else:
            for s in (tr.targets, tr.q, tr.dq, tr.policy.dact[-1], tr.policy._db[-1], tr.loss):
                gpu.mem_fill(s, 7.0)
            gpu.dispatch(opspec.q_head(dqn, dq, a, r, dn, B, A, tr.gamma, tr.q_clip, 1.0, tr.maxq, tr.targets, tr.q, tr.offsets, tr.loss, tr.dq,
                                       tr.policy.dact[-1], tr.policy._db[-1]))
        outs[how] = [gpu.to_numpy(s) for s in (dqn, dq, tr.maxq, tr.targets, tr.q, tr.offsets, tr.dq, tr.policy.dact[-1], tr.policy._db[-1], tr.loss)]
        gpu.mem_cache_free(dqn)
        gpu.mem_cache_free(dq)
    for x, y in zip(outs["ops"][:8], outs["op"][:8]):
        np.testing.assert_array_equal(x, y)
    assert rel_err(outs["op"][8], outs["ops"][8]) <= 1e-5 and rel_err(outs["op"][9], outs["ops"][9]) <= 1e-5
    tr.free()
    for s in (a, r, dn):
        gpu.mem_cache_free(s)


@pytest.mark.parametrize("clip", [False, True])
@pytest.mark.parametrize("lens", [(1,), (5, 3, 1), (16384, 7, 2049), (200001, 3), (64,) * 50], ids=lambda x: str(sum(x)))
def test_adam_step_with_counter_and_soft_target(gpu, lens, clip):
    n, g = sum(lens), rng(sum(lens))
    segs, off = [], 0
    for k in lens:
        segs.append((off, k))
        off += k
    p, gr, m, t = (g.standard_normal(n).astype(np.float32) for _ in range(4))
    v = g.random(n).astype(np.float32)
    gr[segs[-1][0]:] *= 1e-6  # the last tensor's norm stays below the limit
    be = GpuBackend(gpu)
    P, G, M, V, T, N = (be.up(x) for x in (p, gr, m, v, t, np.zeros(len(segs))))
    count = gpu.from_numpy(np.array([11], np.uint64))
    gpu.dispatch(opspec.adam(P, G, M, V, segs, 1, 1e-3, clip=clip, max_norm=0.5, norms=N, step_counter=count, soft_target=T, tau=0.25))
    want = OracleBackend().adam(p, gr, m, v, segs, 12, 1e-3, clip=clip, max_norm=0.5)
    for got, w in zip((P, G, M, V), want):
        assert rel_err(gpu.to_numpy(got), w) <= 1e-6
    assert rel_err(be.down(T), 0.25 * want[0] + 0.75 * t) <= 1e-6
    assert gpu.to_numpy(count)[0] == 11 + len(segs)
    gpu.mem_cache_free(count)


@pytest.mark.parametrize("lens,clip", [((200001, 3), False), ((200001, 3), True), ((700, 64, 5), True)])
def test_adam_counter_over_many_steps(gpu, lens, clip):
    """Every launch reads the counter that the launch before has moved on, in all of its CTAs."""
    n, g, steps = sum(lens), rng(sum(lens)), 60
    segs, off = [], 0
    for k in lens:
        segs.append((off, k))
        off += k
    p, gr = (g.standard_normal(n).astype(np.float32) for _ in range(2))
    gr *= 1e-3  # not clipped: the gradients stay
    be = GpuBackend(gpu)
    P, G, M, V, N = (be.up(x) for x in (p, gr, np.zeros(n), np.zeros(n), np.zeros(len(segs))))
    count = gpu.from_numpy(np.zeros(1, np.uint64))
    want = (p, gr, np.zeros(n, np.float32), np.zeros(n, np.float32))
    for i in range(steps):
        gpu.dispatch(opspec.adam(P, G, M, V, segs, 1, 1e-3, clip=clip, max_norm=10.0, norms=N, step_counter=count))
        want = OracleBackend().adam(*want, segs, 1 + i * len(segs), 1e-3, clip=clip, max_norm=10.0)
    assert gpu.to_numpy(count)[0] == steps * len(segs)
    for got, w in zip((P, G, M, V), want):
        assert rel_err(gpu.to_numpy(got), w) <= 1e-5
    gpu.mem_cache_free(count)


@pytest.mark.parametrize("opt", ["sgd", "none", "adam"])
def test_target_net_follows_whatever_updates_the_policy(gpu, opt):
    B, dims, g = 32, [4, 16, 16, 2], rng(3)
    tr = DqnTrainer(gpu, dims, B, *kaiming_uniform(dims, 1), tau=0.25)
    tr.policy.opt = opt
    batch = [gpu.from_numpy(x) for x in (g.standard_normal(B * 4).astype(np.float32), g.integers(0, 2, B).astype(np.uint64),
                                         g.standard_normal(B * 4).astype(np.float32), np.ones(B, np.float32), np.zeros(B, np.float32))]
    gpu.mem_fill(tr.target.params, 0.5)
    for _ in range(5):
        before = gpu.to_numpy(tr.target.params).astype(np.float64)
        tr.step(*batch)
        want = 0.25 * gpu.to_numpy(tr.policy.params) + 0.75 * before
        assert rel_err(gpu.to_numpy(tr.target.params), want) <= 1e-6
    tr.free()
    for s in batch:
        gpu.mem_cache_free(s)
