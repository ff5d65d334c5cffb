"""Measured cases: the work a user of this framework has it do.

Seven kinds of work, each through the entry points a user's program calls:

  train      MlpTrainer.step on inputs that are already on the device
  infer      MlpTrainer.forward (no loss, no gradients)
  stream     training steps fed from page-locked host memory through BatchStager
  graph_net  GcnTrainer.step, full batch: dense adjacency or edge list
  q_learn    DqnTrainer.step: two networks, Huber loss, Adam, soft update
  matmul     batched matrix product and its backward pass as the autograd issues them
  array      an element-wise / reduction layer and its backward pass, op by op

`replay`: the program captured its step into a graph once and runs the graph, as a training
loop over fixed buffers does; without it every pass issues its ops anew, as a program does
whose buffers or hyper-parameters change, or that never captures.

What comes back is what such a program reads: losses, outputs, updated parameters and
optimizer state.  Training cases return the parameters and moments rather than the gradient
buffer: plain SGD clears it in the step, Adam's first moment carries every gradient, and a
ReLU whose pre-activation rounds to the other side of zero changes a gradient's entries by far
more than arithmetic does, while an update is small against the weights.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from zigrad_b200 import abi, opspec, synthetic
from zigrad_b200.device import CudaDevice, DeviceSlice, USIZE
from zigrad_b200.dqn import DqnTrainer
from zigrad_b200.gcn import GcnTrainer
from zigrad_b200.input_pipeline import BatchStager
from zigrad_b200.mlp import MlpTrainer, kaiming_uniform

MNIST = "784-128-64-10"
WIDE = "4096-4096-4096-4096-1000"
TYPES = {"f32": abi.SINGLE, "f64": abi.DOUBLE, "bf16": abi.BF16}
SIZES = {"f32": 4, "f64": 8, "bf16": 2}


def listed():
    return [
        # the MNIST example's training step at its own batch, called once per batch from the loop
        train("mnist_b64", MNIST, 64),
        # the same network at the benchmark's batch: captured, gradients not kept past the step
        train("mnist_b8192_replay", MNIST, 8192, keep_grads=False, replay=True),
        # one GPU's share of the wide network's global batch: bf16 with fp32 master weights, Adam with clipping
        train("wide_bf16_b8192_replay", WIDE, 8192, dtype="bf16", optimizer="adam", clip=True, labels="index", replay=True),
        # a tabular network whose widths are no multiple of anything, fp32 Adam
        train("odd_widths_adam_b1000", "1000-501-301-37", 1000, optimizer="adam", clip=True, labels="index"),
        # the op sequence an autograd issues through the device interface, one call per op, ragged last batch
        train("mnist_ops_b100", MNIST, 100, fused=False),
        # one prediction at a time
        infer("infer_mnist_b1", MNIST, 1),
        # training fed from the host: copy of the next batch beside the current step
        stream("stream_mnist_b256", MNIST, 256),
        # full-batch GCN on a citation-sized graph: dense adjacency, then a larger graph as an edge list
        graph_net("gcn_dense_replay", 2708, 10556, 1433, 16, 7, 140, dense=True, replay=True),
        graph_net("gcn_edges_20k", 20011, 90000, 500, 16, 7, 1000, dense=False, replay=False),
        # the replay-buffer update of the DQN example
        q_learn("dqn_b256_replay", 4, 128, 2, 256, replay=True),
        # double precision products (numerical checks, small scientific models), ragged
        matmul("matmul_f64", "f64", 4, 500, 389, 640),
        # NDArray arithmetic around a layer, ragged rows
        array("array_f32", "f32", 4099, 1003),
    ]


def train(name, widths, batch, dtype="f32", optimizer="sgd", clip=False, labels="onehot", fused=True, keep_grads=True, replay=False):
    return {"name": name, "kind": "train", "widths": widths, "batch": batch, "dtype": dtype, "optimizer": optimizer, "clip": clip,
            "labels": labels, "fused": fused, "keep_grads": keep_grads, "replay": replay}


def infer(name, widths, batch, dtype="f32", replay=False):
    return {"name": name, "kind": "infer", "widths": widths, "batch": batch, "dtype": dtype, "replay": replay}


def stream(name, widths, batch):
    return {"name": name, "kind": "stream", "widths": widths, "batch": batch}


def graph_net(name, nodes, edges, features, hidden, classes, masked, dense, replay):
    return {"name": name, "kind": "graph_net", "nodes": nodes, "edges": edges, "features": features, "hidden": hidden,
            "classes": classes, "masked": masked, "dense": dense, "replay": replay}


def q_learn(name, observed, hidden, actions, batch, replay):
    return {"name": name, "kind": "q_learn", "observed": observed, "hidden": hidden, "actions": actions, "batch": batch, "replay": replay}


def matmul(name, dtype, batch, m, n, k):
    return {"name": name, "kind": "matmul", "dtype": dtype, "batch": batch, "m": m, "n": n, "k": k}


def array(name, dtype, rows, cols):
    return {"name": name, "kind": "array", "dtype": dtype, "rows": rows, "cols": cols}


# ------------------------------------------------------------------ drawn cases
def _log(rng, lo, hi):
    return int(round(lo * (hi / lo) ** rng.random()))


def _widths(rng, bf16):
    if rng.random() < 0.3 and not bf16:
        return MNIST
    dims = [_log(rng, 16, 2048)] + [_log(rng, 16, 1024) for _ in range(rng.randint(1, 3))] + [_log(rng, 2, 1000)]
    if rng.random() < 0.5:  # half of all networks have widths chosen for the hardware, half have what the data gave
        dims = [(d + 7) // 8 * 8 for d in dims[:-1]] + dims[-1:]
    return "-".join(map(str, dims))


def _draw(rng):
    kind = rng.choice(["train", "train", "infer", "stream", "graph_net", "q_learn", "matmul", "array"])
    if kind in ("train", "infer"):
        dtype = "bf16" if rng.random() < 0.3 else "f32"
        widths, batch = _widths(rng, dtype == "bf16"), _log(rng, 1, 16384)
        if kind == "infer":
            return infer("", widths, batch, dtype, rng.random() < 0.5)
        optimizer = rng.choice(["sgd", "adam"])
        fused = dtype == "bf16" or rng.random() < 0.75
        return train("", widths, batch, dtype, optimizer, rng.random() < 0.5, rng.choice(["onehot", "index"]), fused,
                     not (fused and optimizer == "sgd" and rng.random() < 0.5), rng.random() < 0.5)
    if kind == "stream":
        return stream("", MNIST, _log(rng, 16, 8192))
    if kind == "graph_net":
        dense = rng.random() < 0.5
        nodes = _log(rng, 200, 4000 if dense else 50000)
        return graph_net("", nodes, int(nodes * rng.uniform(2, 8)), _log(rng, 16, 1500), _log(rng, 8, 64), _log(rng, 2, 40),
                         max(8, nodes // 20), dense, rng.random() < 0.5)
    if kind == "q_learn":
        return q_learn("", _log(rng, 2, 64), _log(rng, 32, 512), _log(rng, 2, 18), _log(rng, 32, 1024), rng.random() < 0.5)
    if kind == "matmul":
        return matmul("", rng.choice(["f32", "f64", "bf16"]), _log(rng, 1, 64), _log(rng, 16, 2048), _log(rng, 16, 2048), _log(rng, 16, 2048))
    return array("", rng.choice(["f32", "f32", "f64"]), _log(rng, 1, 65536), _log(rng, 1, 8192))


def draw(rng):
    while True:
        case = _draw(rng)
        w = work(case)
        # no more than a few milliseconds on any path, and inputs that are made quickly
        most = {"f32": 20e9, "f64": 8e9, "bf16": 40e9}[case.get("dtype", "f32")]
        if w["flops"] <= most and w["bytes"] <= 4e8:
            del case["name"]
            return case


# ------------------------------------------------------------------- the programs
_dev = None


def _device() -> CudaDevice:
    global _dev
    if _dev is None:
        _dev = CudaDevice(0)
    return _dev


def _tensor(s: DeviceSlice, *shape) -> torch.Tensor:
    """The device memory of a slice as a torch tensor (no copy)."""
    kind = {abi.SINGLE: "<f4", abi.DOUBLE: "<f8", abi.BF16: "<i2", USIZE: "<i8"}[s.dtype]

    class Memory:
        __cuda_array_interface__ = {"shape": (s.len,), "typestr": kind, "data": (s.ptr, False), "version": 2}

    t = torch.as_tensor(Memory(), device="cuda")
    if s.dtype == abi.BF16:
        t = t.view(torch.bfloat16)
    return t.view(shape) if shape else t


class Program:
    """A user's program: its device memory, its step and the tensors it reads afterwards."""

    def __init__(self, seed):
        self.dev = _device()
        self.host = np.random.Generator(np.random.PCG64(seed))
        self.random = torch.Generator("cuda").manual_seed(seed)
        self.mine, self.owners, self.graph = [], [], None
        self.step, self.out = None, {}

    def alloc(self, dtype, n) -> DeviceSlice:
        s = self.dev.mem_cache_alloc(dtype, n)
        self.mine.append(s)
        return s

    def upload(self, a) -> DeviceSlice:
        s = self.dev.from_numpy(a)
        self.mine.append(s)
        return s

    def normal(self, dtype, n, scale=1.0) -> DeviceSlice:
        s = self.alloc(dtype, n)
        self.dev.sync()
        _tensor(s).normal_(0.0, scale, generator=self.random)
        torch.cuda.synchronize()
        return s

    def uniform(self, dtype, n) -> DeviceSlice:
        s = self.alloc(dtype, n)
        self.dev.sync()
        _tensor(s).uniform_(0.0, 1.0, generator=self.random)
        torch.cuda.synchronize()
        return s

    def moments(self, trainer, scale):
        """Adam's moments as a checkpoint taken during training holds them."""
        self.dev.sync()
        _tensor(trainer.m).normal_(0.0, scale, generator=self.random)
        _tensor(trainer.v).uniform_(0.5 * scale * scale, 1.5 * scale * scale, generator=self.random)
        torch.cuda.synchronize()

    def labels(self, batch, classes, kind) -> DeviceSlice:
        lab = self.host.integers(0, classes, batch)
        return self.upload(lab.astype(np.uint64) if kind == "index" else np.eye(classes, dtype=np.float32)[lab])

    def capture(self):
        """The step as a graph: one eager step first (work space grows there), then the capture."""
        step, dev = self.step, self.dev
        step()
        dev.capture.open()
        step()
        dev.capture.save()
        self.graph = dev.capture.detach()
        self.step = self.graph.run

    def close(self):
        self.dev.sync()
        if self.graph is not None:
            self.graph.free()
        for o in self.owners:
            getattr(o, "free", None) and o.free()
            getattr(o, "close", None) and o.close()
        for s in self.mine:
            self.dev.mem_cache_free(s)
        self.mine, self.owners, self.graph, self.out = [], [], None, {}

    def __del__(self):
        self.close()


def _dims(case):
    return [int(d) for d in case["widths"].split("-")]


def _mlp_out(tr, batch):
    out = {"loss": _tensor(tr.loss), "logits": _tensor(tr.act[-1], batch, tr.ld_out), "params": _tensor(tr.params)}
    if tr.opt == "adam":
        out.update(m=_tensor(tr.m), v=_tensor(tr.v))
    if tr.bf16:
        out["params_bf16"] = _tensor(tr.params_bf16)
    return out


def _train(p, case, seed):
    dims, B, bf16 = _dims(case), case["batch"], case["dtype"] == "bf16"
    Ws, bs = kaiming_uniform(dims, seed)
    tr = MlpTrainer(p.dev, dims, B, Ws, bs, case["optimizer"], lr=0.01 if case["optimizer"] == "sgd" else 1e-3, clip=case["clip"],
                    fused=case["fused"], bf16=bf16, zero_grads_in_update=not case["keep_grads"])
    p.owners.append(tr)
    if tr.opt == "adam":
        p.moments(tr, 0.3 / math.sqrt(B))
    X = p.normal(abi.BF16, B * dims[0]) if bf16 else p.uniform(abi.SINGLE, B * dims[0])
    T = p.labels(B, dims[-1], case["labels"])
    p.step = lambda: tr.step(X, T)
    p.out = _mlp_out(tr, B)


def _infer(p, case, seed):
    dims, B, bf16 = _dims(case), case["batch"], case["dtype"] == "bf16"
    Ws, bs = kaiming_uniform(dims, seed)
    tr = MlpTrainer(p.dev, dims, B, Ws, bs, "none", bf16=bf16)
    p.owners.append(tr)
    X = p.normal(abi.BF16, B * dims[0]) if bf16 else p.uniform(abi.SINGLE, B * dims[0])
    p.step = lambda: tr.forward(X)
    p.out = {"logits": _tensor(tr.act[-1], B, tr.ld_out)}


def _stream(p, case, seed):
    dims, B = _dims(case), case["batch"]
    Ws, bs = kaiming_uniform(dims, seed)
    tr = MlpTrainer(p.dev, dims, B, Ws, bs, "sgd", lr=0.01, zero_grads_in_update=True)
    stager = BatchStager(p.dev, [(B * dims[0], abi.SINGLE), (B, USIZE)], depth=2, packed=True)
    p.owners += [tr, stager]
    batches = [stager.pack([p.host.random((B, dims[0]), dtype=np.float32), p.host.integers(0, dims[-1], B).astype(np.uint64)])
               for _ in range(3)]
    stager.put(batches[0])
    count = 0

    def step():
        nonlocal count
        count += 1
        stager.put(batches[count % 3])  # the next batch travels while this one trains
        X, T = stager.get()
        tr.step(X, T)
        stager.release()

    p.step = step
    p.out = _mlp_out(tr, B)


def _edges(host, nodes, edges):
    """A directed edge list with a power-law degree profile (exponent 2.5)."""
    w = np.arange(1, nodes + 1, dtype=np.float64) ** (-1.0 / 1.5)
    host.shuffle(w)
    c = np.cumsum(w / w.sum())
    pick = lambda: np.minimum(np.searchsorted(c, host.random(edges)), nodes - 1).astype(np.uint64)
    return pick(), pick()


def _graph_net(p, case, seed):
    N, F, H, C, M = (case[k] for k in ("nodes", "features", "hidden", "classes", "masked"))
    src, tgt = _edges(p.host, N, case["edges"])
    X = (p.host.random((N, F), dtype=np.float32) < 0.013).astype(np.float32)
    (W1, W2), (b1, b2) = kaiming_uniform([F, H, C], seed)
    mask = np.sort(p.host.permutation(N)[:M]).astype(np.int64)
    if case["dense"]:
        tr = GcnTrainer(p.dev, synthetic.gcn_dense_adjacency(src, tgt, N), X, W1, b1, W2, b2, mask)
    else:
        tr = GcnTrainer(p.dev, None, X, W1, b1, W2, b2, mask, edges=(src, tgt, synthetic.gcn_degree_scale(tgt, N)))
    p.owners.append(tr)
    p.moments(tr, 0.03 / math.sqrt(M))
    T = p.labels(M, C, "onehot")
    p.step = lambda: tr.step(T)
    p.out = {"loss": _tensor(tr.loss), "embedding": _tensor(tr.a1, N, H), "logits": _tensor(tr.logits, N, -1),
             "params": _tensor(tr.params), "m": _tensor(tr.m), "v": _tensor(tr.v)}


def _q_learn(p, case, seed):
    D, A, B = case["observed"], case["actions"], case["batch"]
    dims = [D, case["hidden"], case["hidden"], A]
    tr = DqnTrainer(p.dev, dims, B, *kaiming_uniform(dims, seed))
    p.owners.append(tr)
    p.moments(tr.policy, 0.3 / math.sqrt(B))
    batch = [p.normal(abi.SINGLE, B * D), p.upload(p.host.integers(0, A, B).astype(np.uint64)), p.normal(abi.SINGLE, B * D),
             p.upload(np.ones(B, np.float32)), p.upload((p.host.random(B) < 0.05).astype(np.float32))]
    p.step = lambda: tr.step(*batch)
    p.out = {"loss": _tensor(tr.loss), "q": _tensor(tr.q), "policy": _tensor(tr.policy.params), "target": _tensor(tr.target.params),
             "m": _tensor(tr.policy.m), "v": _tensor(tr.policy.v)}


def _matmul(p, case, seed):
    t, nb, m, n, k = TYPES[case["dtype"]], case["batch"], case["m"], case["n"], case["k"]
    A, B, dC = p.normal(t, nb * m * k), p.normal(t, nb * k * n, 1 / math.sqrt(k)), p.normal(t, nb * m * n)
    C, dA = p.alloc(t, nb * m * n), p.alloc(t, nb * m * k)
    dB = p.alloc(abi.SINGLE if t == abi.BF16 else t, nb * k * n)  # a weight's gradient accumulates in fp32
    d, bmm, keep = p.dev, opspec.bmm_acc, t != abi.BF16

    def step():
        d.dispatch(bmm(A, B, C, (nb, m, k), (nb, k, n), (nb, m, n), False, False, k, n, n, 1.0, 0.0))
        if keep:  # ensure_grad(0), then accumulate
            d.mem_fill(dA, 0.0)
        d.dispatch(bmm(dC, B, dA, (nb, m, n), (nb, n, k), (nb, m, k), False, True, n, n, k, 1.0, 1.0 if keep else 0.0))
        d.mem_fill(dB, 0.0)
        d.dispatch(bmm(A, dC, dB, (nb, k, m), (nb, m, n), (nb, k, n), True, False, k, n, n, 1.0, 1.0))

    p.step = step
    p.out = {"C": _tensor(C, nb, m, n), "dA": _tensor(dA, nb, m, k), "dB": _tensor(dB, nb, k, n)}


def _array(p, case, seed):
    """y = tanh(x * gain + bias) with its row sums and row maxima, and the gradients of x, gain and bias."""
    t, R, C = TYPES[case["dtype"]], case["rows"], case["cols"]
    x, gain, bias, dy = p.normal(t, R * C), p.normal(t, C), p.normal(t, C), p.normal(t, R * C)
    y, dz, dx, tmp = (p.alloc(t, R * C) for _ in range(4))
    total, top = p.alloc(t, R), p.alloc(t, R)
    dgain, dbias = p.alloc(t, C), p.alloc(t, C)
    d, o = p.dev, opspec

    def step():
        d.dispatch(o.mul(x, gain, y))
        d.dispatch(o.add(y, bias, y))
        d.dispatch(o.tanh_fwd(y, y))
        d.dispatch(o.sum_along(y, [R, C], total, [R, 1], 1))
        d.dispatch(o.max_along(y, [R, C], top, [R, 1], 1))
        d.mem_fill(dz, 0.0)
        d.dispatch(o.tanh_bwd(dz, y, dy))
        d.dispatch(o.unbroadcast(dz, [R, C], dbias, [C], None))
        d.dispatch(o.mul(dz, x, tmp))
        d.dispatch(o.unbroadcast(tmp, [R, C], dgain, [C], None))
        d.dispatch(o.mul(dz, gain, dx))

    p.step = step
    p.out = {"y": _tensor(y, R, C), "sum": _tensor(total), "max": _tensor(top), "dx": _tensor(dx, R, C), "dgain": _tensor(dgain),
             "dbias": _tensor(dbias)}


BUILD = {"train": _train, "infer": _infer, "stream": _stream, "graph_net": _graph_net, "q_learn": _q_learn, "matmul": _matmul, "array": _array}


def prepare(case, seed):
    p = Program(seed)
    BUILD[case["kind"]](p, case, seed)
    if case.get("replay"):
        p.capture()
    p.dev.sync()
    abi.check()
    return p


def run(state):
    state.step()
    return state.out


# ---------------------------------------------------------------- work and tolerance
def work(case):
    """Operations of the products, and each input read once and each output written once."""
    kind = case["kind"]
    if kind in ("train", "infer", "stream"):
        dims, B = _dims(case), case["batch"]
        pairs = list(zip(dims[:-1], dims[1:]))
        weights = sum(a * b for a, b in pairs)
        params = weights + sum(dims[1:])
        es = SIZES[case.get("dtype", "f32")]
        io = B * (dims[0] * es + 4 * dims[-1])
        if kind == "infer":
            return {"bytes": io + es * weights + 4 * sum(dims[1:]), "flops": 2 * B * weights}
        io += B * (4 * dims[-1] if case.get("labels", "index") == "onehot" else 8)
        state = 24 if case.get("optimizer") == "adam" else 8
        return {"bytes": io + params * (state + (2 if es == 2 else 0)), "flops": 2 * B * (3 * weights - dims[0] * dims[1])}
    if kind == "graph_net":
        N, F, H, C, E, M = (case[k] for k in ("nodes", "features", "hidden", "classes", "edges", "masked"))
        params = F * H + H + H * C + C
        links, hop = (4 * N * N, 2 * N * N) if case["dense"] else (16 * E + 4 * N, 2 * E)
        return {"bytes": 4 * N * F + links + 4 * N * C + 4 * M * C + 24 * params, "flops": 4 * N * F * H + 6 * N * H * C + 2 * hop * (H + C)}
    if kind == "q_learn":
        D, H, A, B = (case[k] for k in ("observed", "hidden", "actions", "batch"))
        params = D * H + H + H * H + H + H * A + A
        weights = D * H + H * H + H * A
        return {"bytes": 8 * B * D + 16 * B + 32 * params, "flops": 2 * B * (4 * weights - D * H)}
    if kind == "matmul":
        nb, m, n, k = (case[i] for i in ("batch", "m", "n", "k"))
        es = SIZES[case["dtype"]]
        return {"bytes": nb * (es * (2 * m * k + k * n + 2 * m * n) + max(4, es) * k * n), "flops": 6 * nb * m * n * k}
    R, C, es = case["rows"], case["cols"], SIZES[case["dtype"]]
    return {"bytes": es * (4 * R * C + 4 * C + 2 * R), "flops": 9 * R * C}


def tolerance(case):
    kind, dtype = case["kind"], case.get("dtype", "f32")
    if dtype == "bf16":
        return {"rel": 1e-2, "max": 0.2}
    if dtype == "f64":
        return {"rel": 1e-13, "max": 1e-11}
    if kind == "array":
        return {"rel": 1e-5, "max": 1e-3}
    # a first moment takes a tenth of each gradient, and with it a tenth of what a ReLU on the other side of zero changes
    if kind in ("graph_net", "q_learn") or case.get("optimizer") == "adam":
        return {"rel": 1e-4, "max": 1e-2}
    # sums of up to a few thousand products in fp32
    return {"rel": 3e-5, "max": 2e-3}
