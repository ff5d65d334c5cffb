"""MLP training step on the device interface.

Restates what the reference's MNIST example does above the device boundary
(``examples/mnist/src/model.zig:17-111`` for the model,
``examples/mnist/src/main-simple.zig:61-71`` for the loop, and the autograd
backward order of ``src/graph.zig:55-85`` / ``src/ndtensor.zig:780-796,
1092-1136``) as a fixed sequence of device ops over preallocated buffers, so
that the whole step can be captured once into a CUDA graph
(``CudaDevice.capture``) and replayed.

Two op sequences produce the same tensors:

* ``fused=False`` -- the device ops the reference issues: per layer
  ``bmm_acc`` (beta 0), ``add`` (bias, in place), ``relu_fwd`` (in place); the
  loss; then per layer ``relu_inplace_bwd``, ``unbroadcast`` for the bias
  gradient, ``bmm_acc`` for dX and dW; then the optimizer.  Each gradient is written
  once per step, so where the reference fills it with zeros and accumulates
  (beta = 1) the op writes it (beta = 0), and what the dX chain does not need runs on
  the side stream: at batch 100 the fills were 8 of 27 launches of about 2.5 us each.
  A second ``backward()`` therefore gives the same gradients, as it did with the fills.
* ``fused=True``  -- one zero fill of the flat gradient buffer per forward pass (a second
  ``backward()`` behind it accumulates; ``step()`` clears only what it accumulates into and
  writes the gradients of large weights), ``linear`` ops
  with bias / ReLU / ReLU-mask epilogues, bias gradients taken from the loss
  kernel (last layer) and from the dX GEMM epilogues (hidden layers): 10 kernel
  launches + 1 memset for the three-layer model.  When the last two layers have
  the widths the ``mlp_tail`` op is built for (128 -> 64 -> at most 16 classes:
  the MNIST model), ``step()`` replaces everything between the first layer's
  forward GEMM and the weight gradients by that one op, which where it can
  (``mlp_tail_forms_dw2``) forms the classifier's weight gradient as well; with plain SGD and no
  reduction between backward and update the updates of the other two weights then ride in their
  gradient GEMMs' epilogues (``fuse_update``): 5 launches per step (forward
  GEMM, tail, two weight-gradient GEMMs, the update of the last layer and the biases).
  On few rows (``grouped``) all weight gradients, the biases' and the SGD step are one launch: 3 per step.

Parameters, gradients and optimizer state live in flat buffers in attach
order (W0, b0, W1, b1, ...), which is what a data-parallel step all-reduces
(one buffer) and what the multi-tensor optimizer kernels consume.
"""
from __future__ import annotations

import contextlib
from typing import Callable, List, Optional, Sequence

import numpy as np

from . import opspec
from .abi import BF16, SINGLE
from .device import CudaDevice, DeviceSlice
from .replay import GraphCache, numbers


def kaiming_uniform(dims: Sequence[int], seed: int):
    """Seeded U(+-sqrt(6/fan_in)) weights and zero biases (synthetic stand-in
    for the reference's initialiser, examples/mnist/src/model.zig:75-87; the
    same host arrays are uploaded to every backend under comparison)."""
    g = np.random.Generator(np.random.PCG64(seed))
    Ws, bs = [], []
    for fan_in, fan_out in zip(dims[:-1], dims[1:]):
        bound = np.sqrt(6.0 / fan_in)
        Ws.append(g.uniform(-bound, bound, (fan_out, fan_in)).astype(np.float32))
        bs.append(np.zeros(fan_out, np.float32))
    return Ws, bs


def shares_by_finish(sms: int, tiles0: int, tiles1: int, k_slabs: int, late: int = 4):
    """Shares of `sms` SMs for two split-K GEMMs that run side by side, the second behind a fork of the stream, about `late`
    k-slabs' time (3 us) after the first.  Both are grids of (output tiles x K ranges) CTAs, one CTA per SM, and a CTA's time
    goes with the 32-deep k-slabs of its range: the shares with which the later of the two ends soonest, as (SMs of the first,
    SMs of the second) or None.  At batch 8192 ranges of about the same length for both gave the second 15 SMs, and it ended
    4 us after everybody else (with the classifier's gradient out of the way as well, mlp_tail, the step went from 53.0 to
    47.2 us)."""
    best = None
    for s0 in range(1, sms // tiles0 + 1):
        s1 = (sms - tiles0 * s0) // tiles1
        if s1 < 1:
            break
        end = max(-(-k_slabs // s0), -(-k_slabs // s1) + late)
        if best is None or end <= best[0]:
            best = (end, tiles0 * s0, tiles1 * s1)
    return best and best[1:]


def late_weight_gradients(sms: int, dims: Sequence[int], batch: int):
    """{layer: SMs} of the weight gradients that run side by side behind the dX chain instead of each beside a product of it.
    A product that occupies an SM per CTA and splits its k over whatever SMs there are leaves nothing for another one: the
    chain's next product waited for the weight gradient's CTAs to leave.  Behind the chain they share the SMs, an output tile's
    K ranges as even as they come, and pay the fixed part of such a product once.

    Considered are those that go to the tensor cores (from 50 M multiply-adds) while all their 128 x 128 tiles together find an
    SM each -- larger ones fill the chip whatever the order -- and whose layers' dX products are one wave of tiles: the last of
    several leaves SMs that a weight gradient beside it fills (16 % slower without).  Not where the rows of X are no whole words: the
    first gradient then splits in clusters only (1.5 % faster on average, a third of them slower).  They go late
    where one after the other takes 1.4 times as long as together, at 6 us and 0.6 for a slab of k, and only where each keeps a
    third of the K ranges that it has by itself: the error of a product grows with the length of a range, at a third of the
    rate that one accumulator for all three passes had (gemm_tc.cuh), against which this was compared.
    650 networks of random widths, 2 to 4 layers, 300 to 15000 rows: 7 % faster on average, 3 % of them 1 % slower or more.
    Steps, us, beside -> behind: 1000-501-301-37 at 1000 rows 80.6 -> 72.8, 4000 rows 158 -> 146; 784-512-256-10 at 1000 66 -> 59;
    512-512-512-512 at 2000 106 -> 94; 1024-1024-1024-40 at 1024 125 -> 112."""
    pad, slabs = lambda n: -(-n // 32) * 32, -(-batch // 32)
    big = [l for l in range(len(dims) - 1) if dims[l + 1] > 16 and pad(dims[l + 1]) * pad(dims[l]) * batch >= 5e7]
    tiles = {l: -(-dims[l + 1] // 128) * -(-dims[l] // 128) for l in big}
    if 0 not in big or dims[0] % 4 or sum(tiles.values()) > sms:
        return {}
    time = lambda ranges: 6 + 0.6 * -(-slabs // ranges)
    ranges_alone = {l: max(1, min(sms // tiles[l], slabs // 4)) for l in big}
    alone = {l: time(ranges_alone[l]) for l in big}
    starts = [sum((dims[j] + 1) * dims[j + 1] for j in range(l)) for l in range(len(dims) - 1)]

    def used(l, ranges):  # what gemm.cu makes of it: narrower tiles of two SMs each, clusters where rows are no whole words
        return 1 if ranges < 3 else (ranges if dims[l] % 4 == 0 and starts[l] % 4 == 0 else min(ranges, 8))

    late = [0] + sorted((l for l in big if l and -(-batch // 128) * -(-dims[l] // 128) <= sms), key=lambda l: -tiles[l])
    best, found = 0.0, {}
    while len(late) > 1:  # (without the smallest, and so on: what finds too few SMs here holds up all of them)
        ranges, left = {l: 1 for l in late}, sms - sum(tiles[l] for l in late)
        while fit := [l for l in late if tiles[l] <= left and ranges[l] < slabs // 4]:
            l = min(fit, key=lambda l: (ranges[l], -tiles[l]))
            ranges[l] += 1
            left -= tiles[l]
        before, after = sum(alone[l] for l in late), time(min(ranges.values()))
        exact = all(3 * used(l, ranges[l]) >= used(l, ranges_alone[l]) for l in late)
        if exact and before >= 1.4 * after and before - after > best:
            best, found = before - after, {l: tiles[l] * ranges[l] for l in late}
        late.pop()
    return found


class MlpTrainer:
    def __init__(self, dev: CudaDevice, dims: Sequence[int], batch: int, weights, biases, opt: str = "sgd",
                 lr: float = 0.01, beta1: float = 0.9, beta2: float = 0.999, eps: float = 1e-8, clip: bool = False,
                 max_norm: float = 10.0, delta: float = 1e-6, fused: bool = True, loss_div: Optional[int] = None,
                 index_labels: bool = False, bf16: bool = False, pad_logits: bool = True, zero_grads_in_update: bool = False,
                 tail: Optional[bool] = None, fuse_update: bool = True, update_by_layer: bool = False):
        """`pad_logits`: in the fused path the rows of `act[l]` and `dact[l]`, logits and hidden layers alike, are `ld[l]`
        elements apart: dims[l + 1] rounded up to whole 16-byte words (fp32 4 elements, hidden bf16 rows 8).  False: dense rows.
        `act_numpy(l)` is the dense array either way."""
        self.dev, self.dims, self.B, self.L = dev, [int(d) for d in dims], int(batch), len(dims) - 1
        self.opt, self.lr, self.beta1, self.beta2, self.eps = opt, lr, beta1, beta2, eps
        self.clip, self.max_norm, self.delta = clip, max_norm, delta
        self.fused, self.index_labels, self.bf16 = fused, index_labels, bf16
        self.loss_div = float(loss_div if loss_div is not None else batch)
        self.t = 0  # Adam's optimizer-wide counter (advances once per tensor per step)
        if bf16 and not fused:
            raise ValueError("the bf16 path exists only as fused ops")
        # SGD only: the update kernel clears the gradients it applied, so the next step needs no
        # zero_grad launch (the gradients are then not readable after step())
        if zero_grads_in_update and not (fused and opt == "sgd"):
            raise ValueError("zero_grads_in_update needs the fused ops and SGD")
        self.zero_grads_in_update, self._grads_clear = bool(zero_grads_in_update), False
        self._bias_with_weights = False  # the loss leaves the last bias gradient to the op that forms the weights' (a grouped step)
        # the fused middle of the step (opspec.mlp_tail): on by default wherever the library has a kernel for the widths
        can_tail = (fused and not bf16 and self.L >= 3 and
                    dev.mlp_tail_supported(SINGLE, self.dims[-3], self.dims[-2], self.dims[-1]))
        if tail and not can_tail:
            raise ValueError("no mlp_tail kernel for the widths %s" % self.dims[-3:])
        self.tail = can_tail if tail is None else bool(tail)
        self._dw_shares = None
        self._late = late_weight_gradients(dev.sm_count(), self.dims, self.B) if fused and not bf16 else {}
        self.update_by_layer = bool(update_by_layer)
        # the tail path applies plain SGD from inside the backward pass (see _forward_backward_tail) unless told not to
        self.fuse_update = bool(fuse_update) and self.tail
        # flat parameter layout, attach order
        self.segments, off = [], 0
        for l in range(self.L):
            for n in (self.dims[l + 1] * self.dims[l], self.dims[l + 1]):
                self.segments.append((off, n))
                off += n
        self.n_params = off
        d = dev
        self.params = d.mem_cache_alloc(SINGLE, off)
        self._grads = d.mem_cache_alloc(SINGLE, off)
        self.norms = d.mem_cache_alloc(SINGLE, len(self.segments))
        flat = np.concatenate([np.concatenate([np.asarray(w, np.float32).ravel(), np.asarray(b, np.float32).ravel()])
                               for w, b in zip(weights, biases)])
        d.mem_transfer_htod(flat, self.params)
        d.mem_fill(self._grads, 0.0)
        self._touched = False  # a gradient has been written, or the buffer handed out
        self._graphs = GraphCache(d)  # repeated steps (replay.py)
        if opt == "adam":
            self.m, self.v = d.mem_cache_alloc(SINGLE, off), d.mem_cache_alloc(SINGLE, off)
            d.mem_fill(self.m, 0.0)
            d.mem_fill(self.v, 0.0)
            # tensor updates done so far, kept on the device so that a captured step keeps counting on replay
            self.t_dev = d.from_numpy(np.zeros(1, np.uint64))
        self.W = [self.params.view(self.segments[2 * l][0], self.segments[2 * l][1]) for l in range(self.L)]
        self.b = [self.params.view(self.segments[2 * l + 1][0], self.segments[2 * l + 1][1]) for l in range(self.L)]
        self._dW = [self._grads.view(self.segments[2 * l][0], self.segments[2 * l][1]) for l in range(self.L)]
        self._db = [self._grads.view(self.segments[2 * l + 1][0], self.segments[2 * l + 1][1]) for l in range(self.L)]
        # activations and their gradients.  bf16 mode: hidden activations and all
        # backward operands are bf16, logits / loss / parameter gradients fp32.
        act_t = BF16 if bf16 else SINGLE
        # Row stride of the logits and their gradient: padded to a multiple of 4
        # floats in the fused path so that the skinny last-layer GEMMs (n, k or m
        # = number of classes) satisfy TMA's 16-byte stride rule and run on the
        # tensor cores; the reference op sequence keeps them contiguous.
        C = self.dims[-1]
        self.ld_out = (C + 3) // 4 * 4 if (fused and pad_logits) else C
        # Rows of the hidden activations and their gradients: whole 16-byte words for the same reason, of the products that read
        # them only the weights' own rows are then left to be copied element by element (1000-501-301-37 with narrower tiles,
        # gemm.cu: 100 -> 92 us a step).
        word = (8 if bf16 else 4) if (fused and pad_logits) else 1
        self.ld = [-(-self.dims[l + 1] // word) * word if l + 1 < self.L else self.ld_out for l in range(self.L)]
        self.act = [d.mem_cache_alloc(act_t if l + 1 < self.L else SINGLE, self.B * self.ld[l]) for l in range(self.L)]
        self.dact = [d.mem_cache_alloc(act_t if l + 1 < self.L else SINGLE, self.B * self.ld[l]) for l in range(self.L)]
        if self.ld_out != C:
            d.mem_fill(self.act[-1], 0.0)
            d.mem_fill(self.dact[-1], 0.0)
        self.loss = d.mem_cache_alloc(SINGLE, 1)
        if bf16:
            self.params_bf16 = d.mem_cache_alloc(BF16, off)
            d.cast(self.params, self.params_bf16)
            self.Wb = [self.params_bf16.view(self.segments[2 * l][0], self.segments[2 * l][1]) for l in range(self.L)]
            self.dlogits_bf16 = d.mem_cache_alloc(BF16, self.B * self.ld_out)
        # Whether the weight gradients of a step go out as one op behind the dX chain (opspec.weight_grads): fused fp32 on few
        # rows, where the products one by one are launches of 2 to 4 us on forked streams.
        self.grouped = fused and not bf16 and not self.update_by_layer and d.weight_grads_supported(SINGLE, self._group_items(None, False), self.B)
        d.sync()

    # -------------------------------------------------------------- gradients
    def _zero_grad_due(self) -> bool:
        """Whether a forward pass that starts now has to clear the gradients (model.zig:57-62).  Not behind an update that
        did (zero_grads_in_update), and not while they are the zeros of construction: no backward pass has written them
        and nobody holds the buffer.  A graph of the caller's clears them all the same, since it may be run later."""
        due = not self._grads_clear and (self._touched or self.dev.capturing())
        self._grads_clear = False
        return due

    def zero_grad(self):
        """ONE fill of the flat gradient buffer."""
        self.dev.mem_fill(self._grads, 0.0)
        self._grads_clear = False

    def _large(self, l: int) -> bool:
        """Whether layer l's weight gradient has enough output tiles (64 of 128 x 128) to fill the chip without K ranges that
        are added into a cleared C.  Smaller ones are cleared with the biases, in one launch of about 2 us."""
        return self.segments[2 * l][1] >= 1 << 20

    def clear_for_backward(self):
        """The gradients that a fused backward pass(fresh=True) accumulates into: all but those of large weights."""
        large = {2 * l for l in range(self.L) if self._large(l)}
        if not large:
            return self.zero_grad()
        runs, end = [], -1  # neighbours as one segment
        for j, (off, n) in enumerate(self.segments):
            if j in large:
                continue
            if off == end:
                runs[-1][1] += n
            else:
                runs.append([off, n])
            end = off + n
        self.dev.fill_segments(self._grads, runs, 0.0)
        self._grads_clear = False

    @property
    def grads(self) -> DeviceSlice:
        self._touched = True
        return self._grads

    @property
    def dW(self) -> List[DeviceSlice]:
        self._touched = True
        return self._dW

    @property
    def db(self) -> List[DeviceSlice]:
        self._touched = True
        return self._db

    # ------------------------------------------------------------------ pieces
    def forward(self, X: DeviceSlice):
        if not self.fused:
            return self._layers(X)
        zero = self._zero_grad_due()
        self._graphs.run(("forward", X.ptr, X.dtype, zero), lambda: self._forward(X, zero), self._host_state, self._set_host_state)
        return self.act[-1]

    def _host_state(self):
        return self.t, self._grads_clear, self._touched

    def _set_host_state(self, state):
        self.t, self._grads_clear, self._touched = state

    def _forward(self, X: DeviceSlice, zero: bool):
        # The gradients are cleared here, in front of the products: the weight-gradient GEMMs accumulate with beta = 1 as
        # the reference does.
        if zero:
            self.zero_grad()
        return self._layers(X)

    def _ld_in(self, l: int) -> int:
        """Row stride of layer l's input: the caller's dense rows, or an activation's."""
        return self.dims[0] if l == 0 else self.ld[l - 1]

    def _layers(self, X: DeviceSlice):
        d, B = self.dev, self.B
        inp = X
        if self.fused and not self.bf16 and B == 1 and d.mlp_forward_supported(SINGLE, self.dims):
            d.dispatch(opspec.mlp_forward(X, self.dims, self.W, self.b, self.act))
            return self.act[-1]
        for l in range(self.L):
            K, N, ldx = self.dims[l], self.dims[l + 1], self._ld_in(l)
            last = l + 1 == self.L
            if self.fused:
                W = self.Wb[l] if self.bf16 else self.W[l]
                d.dispatch(opspec.linear(inp, W, self.act[l], B, N, K, False, True, ldx, K, self.ld[l], 1.0, 0.0,
                                         "bias" if last else "bias_relu", self.b[l]))
            else:
                d.dispatch(opspec.bmm_acc(inp, self.W[l], self.act[l], (1, B, K), (1, K, N), (1, B, N), False, True, K, K, N, 1.0, 0.0))
                d.dispatch(opspec.add(self.b[l], self.act[l], self.act[l]))
                if not last:
                    d.dispatch(opspec.relu_fwd(self.act[l], self.act[l]))
            inp = self.act[l]
        return self.act[-1]

    def loss_and_grad(self, T: DeviceSlice):
        d, B, C = self.dev, self.B, self.dims[-1]
        self._touched = True
        if self.fused:  # the bias gradient of the last layer comes out of the same pass
            d.dispatch(opspec.softmax_ce(self.act[-1], T, B, C, self.loss, self.dact[-1], self.loss_div, accumulate=False,
                                         ld=self.ld_out, bias_grad=None if self._bias_with_weights else self._db[-1]))
        else:
            d.dispatch(opspec.softmax_ce(self.act[-1], T, B, C, self.loss, self.dact[-1], self.loss_div, accumulate=False))

    def backward(self, X: DeviceSlice, last_bias_done: bool = True, on_layer_grads: Optional[Callable[[int], None]] = None,
                 update_by_layer: bool = False, fresh: bool = False):
        """Backward from dact[L-1].  `last_bias_done`: the bias gradient of the last
        layer was already produced by the loss kernel (fused path); pass False when
        dact[L-1] comes from elsewhere (e.g. the DQN's gather backward).
        `on_layer_grads(l)` (fused path) is called on the side stream right after
        layer l's weight gradient has been issued there -- dW[l] and db[l] are then
        final in stream order, so a data-parallel caller can start reducing that
        layer's slice of the gradient buffer while the backward pass goes on.
        `update_by_layer` (fused path, Adam): the optimizer step rides on the backward
        pass, a layer at a time.  Layer l's tensors are updated on a second side stream
        once its weight gradient (first side stream) and its dX product (main stream, the
        last reader of W[l]) have been issued, so the memory-bound update runs beside the
        tensor-bound GEMMs of the layers below.  Same arithmetic per element as one update
        over all tensors (zg_adam_step_part keeps every tensor's position in the step
        count); the caller must not call update() for this step.  Off by default: on the
        wide MLP the update then competes with the persistent GEMMs for memory bandwidth
        and the step got slower (2.39 ms against 2.27 ms with one update after the join).
        `fresh` (fused path): the gradients of large weights are written (beta = 0), whatever the
        buffer holds, and the others are zero already (clear_for_backward): what zeroing the
        whole buffer and accumulating gives, without the two passes over it."""
        d, B = self.dev, self.B
        self._touched = True
        if self.fused and not last_bias_done:
            if self.ld_out != self.dims[-1]:
                raise ValueError("an external output gradient needs unpadded logits (pad_logits=False)")
            d.dispatch(opspec.unbroadcast(self.dact[-1], [B, self.dims[-1]], self._db[-1], [self.dims[-1]], None, 1.0, 0.0))
        # (a caller that starts on each layer's gradients as they come gets them as they come)
        late = self._late if on_layer_grads is None and not update_by_layer else {}

        def weight_gradient(l, dy, a_in):
            K, N = self.dims[l], self.dims[l + 1]
            # (bf16: the padding of the activations' rows does not make the sums any less exact than those of dense rows)
            ragged = self.bf16 and (K % 8 != 0 or (N if l + 1 < self.L else self.ld_out) % 8 != 0)
            d.dispatch(opspec.linear(dy, a_in, self._dW[l], N, K, B, True, False, self.ld[l], self._ld_in(l), K, 1.0,
                                     0.0 if fresh and self._large(l) else 1.0, sm_budget=late.get(l, 0), rounded_sums=ragged))

        for l in range(self.L - 1, -1, -1):
            K, N = self.dims[l], self.dims[l + 1]
            a_in = X if l == 0 else self.act[l - 1]
            dy = self.dact[l]
            if self.fused:
                ldy = self.ld[l]
                if l + 1 == self.L:
                    if self.bf16:  # fp32 dlogits -> bf16 operand of the backward GEMMs
                        d.cast(dy, self.dlogits_bf16)
                        dy = self.dlogits_bf16
                # bias gradients: db[L-1] came out of the loss kernel; db[l-1] is the
                # column sum of the masked dX that this layer's dX GEMM stores
                # (added by its epilogue into the zero-filled gradient buffer)
                # The weight gradient does not feed the dX chain: it goes to the side
                # stream (a parallel branch of a captured step), forked here where dY
                # is ready, and runs next to this layer's dX GEMM.
                if l not in late:
                    with d.branch():
                        weight_gradient(l, dy, a_in)
                        if on_layer_grads is not None:
                            on_layer_grads(l)
                if l > 0:  # dX = dY . W, zeroed where the previous activation is <= 0
                    W = self.Wb[l] if self.bf16 else self.W[l]
                    d.dispatch(opspec.linear(dy, W, self.dact[l - 1], B, K, N, False, False, ldy, K, self.ld[l - 1], 1.0, 0.0,
                                             "relu_mask", None, self.act[l - 1], colsum=self._db[l - 1]))
                if update_by_layer:
                    with d.branch(1, after=(0,)):
                        self._adam_layer(l, last=(l == 0))
            else:
                if l + 1 < self.L:
                    d.dispatch(opspec.relu_inplace_bwd(self.act[l], dy))
                with d.branch():
                    d.dispatch(opspec.unbroadcast(dy, [B, N], self._db[l], [N], None, 1.0, 0.0))
                    if l > 0:
                        self._dw_op(l, dy, a_in)
                if l > 0:
                    d.dispatch(opspec.bmm_acc(dy, self.W[l], self.dact[l - 1], (1, B, N), (1, N, K), (1, B, K), False, False, N, K, K, 1.0, 0.0))
                else:
                    self._dw_op(l, dy, a_in)
        for k, l in enumerate(sorted(late, reverse=True)):
            with (d.branch(1 + k) if l > 0 else contextlib.nullcontext()):  # (not behind those beside the chain)
                weight_gradient(l, self.dact[l], X if l == 0 else self.act[l - 1])
        d.join()  # the gradients are complete before anything that follows on the main stream

    # ------------------------------------------------- few rows: one launch for all weight gradients
    def _group_items(self, X: Optional[DeviceSlice], update: bool):
        keep = not (update and self.zero_grads_in_update)  # the gradients are written unless nobody sees them past the step
        items = []
        for l in range(self.L):
            items.append((self.dact[l], X if l == 0 else self.act[l - 1], self._dW[l] if keep else None, self._db[l] if keep else None,
                          self.W[l] if update else None, self.b[l] if update else None, self.dims[l + 1], self.dims[l], self.ld[l],
                          self._ld_in(l)))
        return items

    def _weight_grads(self, X: DeviceSlice, update: bool):
        """All weight and bias gradients from dact[] (overwritten, so nothing had to be cleared), and the SGD step."""
        self.dev.dispatch(opspec.weight_grads(self._group_items(X, update), self.B, self.lr))
        if update:
            self._grads_clear = self.zero_grads_in_update

    def backward_grouped(self, X: DeviceSlice, update: bool = False):
        """backward() from dact[L-1] where `grouped`: the dX chain, then everything else in one launch."""
        d, B = self.dev, self.B
        self._touched = True
        for l in range(self.L - 1, 0, -1):
            K, N = self.dims[l], self.dims[l + 1]
            d.dispatch(opspec.linear(self.dact[l], self.W[l], self.dact[l - 1], B, K, N, False, False, self.ld[l], K, self.ld[l - 1], 1.0, 0.0,
                                     "relu_mask", None, self.act[l - 1]))
        self._weight_grads(X, update)

    def _clear_unwritten(self, update: bool):
        """The zero_grad of a grouped step: only where its gradients are not written."""
        if self._zero_grad_due() and update and self.zero_grads_in_update:
            self.zero_grad()
        self._touched = True

    def _dw_op(self, l: int, dy: DeviceSlice, a_in: DeviceSlice):
        B, K, N = self.B, self.dims[l], self.dims[l + 1]
        self.dev.dispatch(opspec.bmm_acc(dy, a_in, self._dW[l], (1, N, B), (1, B, K), (1, N, K), True, False, N, K, K, 1.0, 0.0))

    def _adam_layer(self, l: int, last: bool):
        """Adam over the two tensors of layer l: the segment list keeps every tensor (the others
        empty) so that the per-tensor step counts are those of one update over the whole model;
        the device counter is advanced by the last call of the step."""
        segs = [(off, n if j in (2 * l, 2 * l + 1) else 0) for j, (off, n) in enumerate(self.segments)]
        self.dev.dispatch(opspec.adam(self.params, self._grads, self.m, self.v, segs, self.t + 1, self.lr, self.beta1,
                                      self.beta2, self.eps, self.clip, self.max_norm, self.delta, self.norms,
                                      self.params_bf16 if self.bf16 else None, self.t_dev, advance_counter=last))
        if last:
            self.t += len(self.segments)  # host mirror (eager steps only; read_t() is the truth)

    def update(self, soft_target: Optional[DeviceSlice] = None, tau: float = 0.0):
        """`soft_target`: a target network's flat parameters, moved towards the updated ones by tau (Adam: in the same pass)."""
        d = self.dev
        if self.opt == "sgd":
            d.dispatch(opspec.sgd(self.params, self._grads, self.segments, self.lr, self.clip, self.max_norm, self.delta, self.norms,
                                  self.zero_grads_in_update))
            self._grads_clear = self.zero_grads_in_update
        elif self.opt == "adam":
            d.dispatch(opspec.adam(self.params, self._grads, self.m, self.v, self.segments, self.t + 1, self.lr, self.beta1,
                                   self.beta2, self.eps, self.clip, self.max_norm, self.delta, self.norms,
                                   self.params_bf16 if self.bf16 else None, self.t_dev, soft_target=soft_target, tau=tau))
            self.t += len(self.segments)  # host mirror (eager steps only; read_t() is the truth)
        elif self.opt != "none":
            raise ValueError(self.opt)
        if soft_target is not None and self.opt != "adam":
            d.soft_update(self.params, soft_target, tau)

    # -------------------------------------------------------------------- step
    def layer_grads(self, l: int) -> DeviceSlice:
        """The contiguous slice [dW_l ; db_l] of the flat gradient buffer."""
        off = self.segments[2 * l][0]
        self._touched = True
        return self._grads.view(off, self.segments[2 * l][1] + self.segments[2 * l + 1][1])

    def _forward_backward_tail(self, X: DeviceSlice, T: DeviceSlice, fuse_update: bool = False):
        """forward, loss and backward with the last two layers, the loss and the
        dX chain down to dact[L-3] done by one mlp_tail op.

        ``fuse_update`` (plain SGD, no all-reduce in between): the update rides on the
        backward pass instead of following it.  For layer 0 and the two tail layers nothing
        reads the weights any more once their gradient runs, so
        * with ``zero_grads_in_update`` (the gradients are not kept past the step) the
          weight-gradient GEMM accumulates straight into the weights,
          W += (-lr) * dY^T X (alpha = -lr, beta = 1, C = W): no gradient tensor, no update launch;
        * otherwise each weight gradient is followed, on its own stream, by the SGD update
          of that one tensor.
        The biases and the last layer, whose gradients the tail op has finished, are updated by a
        launch of their own (behind the last layer's product where that op does not form it); no update waits for the join of all streams.  The weights of the
        layers in between are still read by the dX products and are updated after the join."""
        d, B, L = self.dev, self.B, self.L
        grouped = self.grouped
        if grouped:
            self._clear_unwritten(fuse_update)
        elif self._zero_grad_due():
            self.zero_grad()
        self._touched = True

        in_gemm = fuse_update and self.zero_grads_in_update
        in_tail = not grouped and d.mlp_tail_forms_dw2(B)  # the classifier's weight gradient comes out of the tail op as well
        by_gemm = (0, L - 2) if in_tail else (0, L - 2, L - 1)  # layers whose update rides in their gradient's product
        nlr = -float(np.float32(self.lr))  # lr cast f64 -> f32, then negated (optim.zig:103)

        def target(l):  # (C, alpha) of layer l's weight-gradient product
            return (self.W[l], nlr) if in_gemm and l in by_gemm else (self._dW[l], 1.0)

        def update(segs):
            if in_gemm:
                segs = [sg for sg in segs if sg not in [self.segments[2 * l] for l in by_gemm]]
            if fuse_update and segs:
                d.dispatch(opspec.sgd(self.params, self._grads, segs, self.lr, False, self.max_norm, self.delta, self.norms,
                                      self.zero_grads_in_update))

        weight, bias = (lambda l: self.segments[2 * l]), (lambda l: self.segments[2 * l + 1])
        inp = X
        for l in range(L - 2):  # the layers in front of the tail
            K, N = self.dims[l], self.dims[l + 1]
            d.dispatch(opspec.linear(inp, self.W[l], self.act[l], B, N, K, False, True, self._ld_in(l), K, self.ld[l], 1.0, 0.0, "bias_relu", self.b[l]))
            inp = self.act[l]
        h1, h2, C = self.dims[L - 2], self.dims[L - 1], self.dims[L]
        d.dispatch(opspec.mlp_tail(self.act[L - 3], self.W[L - 2], self.b[L - 2], self.W[L - 1], self.b[L - 1], T, B, h1, h2, C,
                                   self.ld_out, self.loss_div, self.act[L - 2], self.act[L - 1], self.loss, self.dact[L - 1],
                                   self.dact[L - 2], self.dact[L - 3], *([None] * 3 if grouped else [self._db[L - 1], self._db[L - 2], self._db[L - 3]]),
                                   weights_ready=L - 2 >= 1, dW2=self._dW[L - 1] if in_tail else None))
        if grouped:
            for l in range(L - 3, 0, -1):
                K, N = self.dims[l], self.dims[l + 1]
                d.dispatch(opspec.linear(self.dact[l], self.W[l], self.dact[l - 1], B, K, N, False, False, self.ld[l], K, self.ld[l - 1], 1.0, 0.0,
                                         "relu_mask", None, self.act[l - 1]))
            return self._weight_grads(X, fuse_update)
        # the weight gradients of the two tail layers are independent of each other and of everything that follows:
        # one side stream each.
        # With one layer in front of the tail, its weight gradient (main stream) runs beside the two of the tail:
        # the SMs are shared out by output tiles so that the three split-K grids fit in one wave together.
        share = self._dw_sm_shares() if L == 3 else {}
        with d.branch(0):
            Cw, a = target(L - 2)
            d.dispatch(opspec.linear(self.dact[L - 2], self.act[L - 3], Cw, h2, h1, B, True, False, h2, h1, h1, a, 1.0,
                                     sm_budget=share.get(L - 2, 0)))
            update([weight(L - 2)])
        if fuse_update or not in_tail:
            with d.branch(1):
                if not in_tail:
                    Cw, a = target(L - 1)
                    d.dispatch(opspec.linear(self.dact[L - 1], self.act[L - 2], Cw, C, h2, B, True, False, self.ld_out, h2, h2, a, 1.0))
                # the tail op wrote the bias gradients of its two layers and of the layer in front of it
                update([weight(L - 1)] + [bias(l) for l in (L - 3, L - 2, L - 1)])
        for l in range(L - 3, -1, -1):
            K, N = self.dims[l], self.dims[l + 1]
            a_in = X if l == 0 else self.act[l - 1]
            if l == 0:  # nothing else is left on the main stream: the largest weight gradient runs there
                Cw, a = target(0)
                d.dispatch(opspec.linear(self.dact[l], a_in, Cw, N, K, B, True, False, self.ld[l], K, K, a, 1.0, sm_budget=share.get(0, 0)))
                update([weight(0)])
            else:
                with d.branch(0):
                    d.dispatch(opspec.linear(self.dact[l], a_in, self._dW[l], N, K, B, True, False, self.ld[l], self._ld_in(l), K, 1.0, 1.0))
                d.dispatch(opspec.linear(self.dact[l], self.W[l], self.dact[l - 1], B, K, N, False, False, self.ld[l], K, self.ld[l - 1], 1.0, 0.0,
                                         "relu_mask", None, self.act[l - 1], colsum=self._db[l - 1]))
        d.join()
        if fuse_update:
            # what did not ride on the backward pass: the weights the dX products read and the biases in front of them
            update([weight(l) for l in range(1, L - 2)] + [bias(l) for l in range(L - 3)])
            self._grads_clear = self.zero_grads_in_update

    def _dw_sm_shares(self) -> dict:
        """SMs for each tensor-core weight-gradient GEMM of a three-layer step (layers 0 and 1; the last layer's comes out of
        the tail op, or goes to a small FFMA kernel that fits beside the others)."""
        if self._dw_shares is None:
            t0, t1 = (-(-self.dims[l + 1] // 128) * -(-self.dims[l] // 128) for l in (0, 1))
            best = shares_by_finish(self.dev.sm_count(), t0, t1, -(-self.B // 32))
            self._dw_shares = {0: best[0], 1: best[1]} if best else {}
        return self._dw_shares

    def step(self, X: DeviceSlice, T: DeviceSlice, allreduce: Optional[Callable[[DeviceSlice], None]] = None):
        """forward + loss + backward [+ gradient all-reduce] + update, all
        asynchronous on the device stream.  The loss stays in ``self.loss``."""
        if allreduce is not None:
            return self._step(X, T, allreduce)
        key = (X.ptr, X.dtype, T.ptr, T.dtype, numbers(self.lr, self.beta1, self.beta2, self.eps, self.max_norm, self.delta, self.loss_div),
               self.opt, str(self.clip), self.fused, self.tail, self.fuse_update, self.update_by_layer, self.zero_grads_in_update, self._grads_clear)
        self._graphs.run(key, lambda: self._step(X, T, None), self._host_state, self._set_host_state)

    def _step(self, X: DeviceSlice, T: DeviceSlice, allreduce):
        if self.tail:
            fuse = self.fuse_update and allreduce is None and self.opt == "sgd" and not self.clip
            self._forward_backward_tail(X, T, fuse_update=fuse)
            if fuse:
                return
        else:
            by_layer = self.update_by_layer and self.fused and self.opt == "adam" and allreduce is None
            if self.grouped:
                fuse = self.opt == "sgd" and not self.clip and allreduce is None
                self._clear_unwritten(fuse)
                self._layers(X)
                # (nothing else clears what the loss would write where the gradients are not kept)
                self._bias_with_weights = True
                try:
                    self.loss_and_grad(T)
                finally:
                    self._bias_with_weights = False
                self.backward_grouped(X, fuse)
                return None if fuse else self._reduce_and_update(allreduce)
            # The whole step is issued here: of its gradients only those it accumulates into have to be cleared (a fill of
            # all of them is 35 us of the wide network's step, and the additions read the 218 MB once more)
            if self.fused and self._zero_grad_due():
                self.clear_for_backward()
            self._layers(X)
            self.loss_and_grad(T)
            self.backward(X, update_by_layer=by_layer, fresh=self.fused)
            if by_layer:
                return
        self._reduce_and_update(allreduce)

    def _reduce_and_update(self, allreduce):
        if allreduce is not None:
            fused = getattr(allreduce, "reduce_and_sgd", None)
            if fused is not None and self.opt == "sgd" and not self.clip:
                if self.zero_grads_in_update:
                    fused(self._grads, self.params, self.lr, True)  # reduction, update and zero_grad in one kernel
                    self._grads_clear = True
                else:
                    fused(self._grads, self.params, self.lr)  # reduction and update in one kernel
                return
            allreduce(self._grads)
        self.update()

    def read_loss(self) -> float:
        return float(self.dev.to_numpy(self.loss)[0])

    def read_t(self) -> int:
        """Adam's counter as the device holds it (tensor updates done so far)."""
        return int(self.dev.to_numpy(self.t_dev)[0]) if self.opt == "adam" else 0

    # ------------------------------------------------------------- inspection
    def act_numpy(self, l: int, grad: bool = False) -> np.ndarray:
        """Activation (or its gradient) of layer l as a [B, dims[l+1]] fp32 array
        (row padding of the logits stripped, bf16 widened)."""
        s = (self.dact if grad else self.act)[l]
        a = self.dev.to_numpy(s)
        if s.dtype == BF16:
            a = (a.astype(np.uint32) << 16).view(np.float32)
        return a.reshape(self.B, self.ld[l])[:, :self.dims[l + 1]].copy()

    def get_params(self):
        flat = self.dev.to_numpy(self.params)
        return self._split(flat)

    def get_grads(self):
        return self._split(self.dev.to_numpy(self.grads))

    def _split(self, flat):
        Ws, bs = [], []
        for l in range(self.L):
            o, n = self.segments[2 * l]
            Ws.append(flat[o:o + n].reshape(self.dims[l + 1], self.dims[l]).copy())
            o, n = self.segments[2 * l + 1]
            bs.append(flat[o:o + n].copy())
        return Ws, bs

    def free(self):
        d = self.dev
        d.sync()
        self._graphs.clear()
        for s in [self.params, self._grads, self.norms, self.loss] + self.act + self.dact:
            d.mem_cache_free(s)
        if self.opt == "adam":
            d.mem_cache_free(self.m)
            d.mem_cache_free(self.v)
            d.mem_cache_free(self.t_dev)
        if self.bf16:
            d.mem_cache_free(self.params_bf16)
            d.mem_cache_free(self.dlogits_bf16)
