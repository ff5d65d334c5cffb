"""Two-layer GCN training step with a dense normalised adjacency.

Restates the reference's GCN example above the device boundary
(``examples/gcn/src/model.zig:17-112`` model and layer, ``:296-353`` MaskLayer,
``examples/gcn/src/main.zig:40-95`` Adam + loop).  Each GraphConvLayer is
``h = x . W^T`` (``bmm_acc`` with ``trans_b``), a propagation step, then
``+ bias``; the reference propagates with an edge scatter
(``scatter_gcn_deg_scaled``, ``src/device/host_device.zig:1356-1370``), this
configuration uses the dense matrix that scatter equals, ``p = A_hat . h``.

Device op sequence (fused path): 4 forward GEMMs (bias / bias+ReLU epilogues),
row gather of the masked logits, softmax-CE (+ last bias gradient), row scatter,
2 transposed propagation GEMMs, dW2, dA1 (ReLU mask + bias-gradient column sums),
dW1, Adam.  Rows of X and W1 are padded to a multiple of 4 floats and the class
dimension to a multiple of 4 so that every operand meets TMA's 16-byte stride
rule; padding columns are zero and stay zero.
"""
from __future__ import annotations

from typing import Optional

import numpy as np

from . import opspec
from .abi import SINGLE
from .device import USIZE, CudaDevice, DeviceSlice
from .replay import GraphCache, numbers


def _pad4(n: int) -> int:
    return (n + 3) // 4 * 4


class GcnTrainer:
    def __init__(self, dev: CudaDevice, A_hat: Optional[np.ndarray], X: np.ndarray, W1, b1, W2, b2, mask_idx: np.ndarray,
                 lr: float = 0.01, beta1: float = 0.9, beta2: float = 0.999, eps: float = 1e-8, clip: bool = True,
                 max_norm: float = 10.0, delta: float = 1e-6, opt: str = "adam", edges=None):
        """`A_hat`: dense normalised adjacency (config 4), or None with
        `edges = (src, tgt, deg)` for the reference's own sparse propagation
        (edge list + deg^-1/2 per node): the edge scatter then runs as a CSR
        row walk without atomics (opspec.csr_gcn_propagate)."""
        d = self.dev = dev
        self.sparse = edges is not None
        self.N, self.F = X.shape
        self.H, self.C = W1.shape[0], W2.shape[0]
        self.Fp, self.Cp = _pad4(self.F), _pad4(self.C)
        self.M = len(mask_idx)
        self.opt, self.lr, self.beta1, self.beta2, self.eps = opt, lr, beta1, beta2, eps
        self.clip, self.max_norm, self.delta = clip, max_norm, delta
        self.t = 0
        N, F, H, C, Fp, Cp, M = self.N, self.F, self.H, self.C, self.Fp, self.Cp, self.M
        Xp = np.zeros((N, Fp), np.float32)
        Xp[:, :F] = X
        self.X = d.from_numpy(Xp)
        if self.sparse:
            from .synthetic import edges_to_csr
            src, tgt, deg = edges
            rp, ci = edges_to_csr(tgt, src, N)      # forward: grouped by target, neighbours = sources
            rpt, cit = edges_to_csr(src, tgt, N)    # gradient w.r.t. h: grouped by source, neighbours = targets
            # ... of which the gradient of the logits needs the edges into masked nodes only: it is zero elsewhere
            into = np.isin(tgt, mask_idx)
            rpm, cim = edges_to_csr(np.asarray(src)[into], np.asarray(tgt)[into], N)
            self.csr = tuple(d.from_numpy(a) for a in (rp, ci, rpt, cit, rpm, cim))
            self.deg = d.from_numpy(np.ascontiguousarray(deg, np.float32))
            self.A = None
        else:
            self.A = d.from_numpy(np.ascontiguousarray(A_hat, np.float32))
        self.mask_rows = d.from_numpy(np.unique(np.asarray(mask_idx, np.uint64)))
        # flat parameters in attach order: W1 [H, Fp], b1 [H], W2 [C, H], b2 [C]
        W1p = np.zeros((H, Fp), np.float32)
        W1p[:, :F] = W1
        flat = np.concatenate([W1p.ravel(), np.asarray(b1, np.float32), np.asarray(W2, np.float32).ravel(), np.asarray(b2, np.float32)])
        sizes = [H * Fp, H, C * H, C]
        self.segments, off = [], 0
        for n in sizes:
            self.segments.append((off, n))
            off += n
        self.params = d.from_numpy(flat)
        # the gradients and, behind them, the gradient of the logits: what a step clears
        at = -(-off // 64) * 64
        self.cleared = d.mem_cache_alloc(SINGLE, at + N * Cp)
        self.grads, self.dlog = self.cleared.view(0, off), self.cleared.view(at, N * Cp)
        self.m, self.v = d.mem_cache_alloc(SINGLE, off), d.mem_cache_alloc(SINGLE, off)
        self.norms = d.mem_cache_alloc(SINGLE, 4)
        self.t_dev = d.from_numpy(np.zeros(1, np.uint64))  # Adam's counter on the device (graph-replay safe)
        for s in (self.cleared, self.m, self.v):
            d.mem_fill(s, 0.0)
        v = lambda buf, i: buf.view(self.segments[i][0], self.segments[i][1])
        self.W1, self.b1, self.W2, self.b2 = (v(self.params, i) for i in range(4))
        self.dW1, self.db1, self.dW2, self.db2 = (v(self.grads, i) for i in range(4))
        alloc = lambda n: d.mem_cache_alloc(SINGLE, n)
        self.h1, self.a1, self.h2, self.logits = alloc(N * H), alloc(N * H), alloc(N * Cp), alloc(N * Cp)
        self.dh2, self.da1, self.dh1 = alloc(N * Cp), alloc(N * H), alloc(N * H)
        self.mlog, self.dm = alloc(M * Cp), alloc(M * Cp)
        for s in (self.h2, self.logits, self.dh2, self.mlog, self.dm):
            d.mem_fill(s, 0.0)
        # MaskLayer as flat offsets: row r of the mask -> Cp consecutive elements of node mask_idx[r]
        offs = (np.asarray(mask_idx, np.uint64)[:, None] * np.uint64(Cp) + np.arange(Cp, dtype=np.uint64)[None, :]).ravel()
        self.offsets = d.from_numpy(np.ascontiguousarray(offs, np.uint64))
        self.loss = alloc(1)
        self._graphs = GraphCache(d)  # repeated steps (replay.py)
        d.sync()

    def _mm(self, A, B, Cbuf, m, n, k, ta, tb, lda, ldb, ldc, beta=0.0, epilogue="none", bias=None, mask=None, colsum=None):
        self.dev.dispatch(opspec.linear(A, B, Cbuf, m, n, k, ta, tb, lda, ldb, ldc, 1.0, beta, epilogue, bias, mask, colsum=colsum))

    def _prop(self, x, out, F, ld, epilogue="none", bias=None, transpose=False):
        """out = A.x (+ bias, ReLU) -- dense GEMM with the adjacency, or the CSR walk over the edges."""
        N = self.N
        if self.sparse:
            rp, ci, rpt, cit = self.csr[:4]
            self.dev.dispatch(opspec.csr_gcn_propagate(out, x, self.deg, rpt if transpose else rp, cit if transpose else ci, N, F, ld, ld,
                                                       transpose, epilogue, bias))
        else:
            self._mm(self.A, x, out, N, F, N, transpose, False, N, ld, ld, 0.0, epilogue, bias)

    def _prop_dlogits(self):
        """dh2 = A^T . dlogits, of which only the masked nodes' rows are not zero (up to a sixth of them it pays to say so)."""
        d, N, C, Cp = self.dev, self.N, self.C, self.Cp
        if self.sparse:
            d.dispatch(opspec.csr_gcn_propagate(self.dh2, self.dlog, self.deg, self.csr[4], self.csr[5], N, C, Cp, Cp, True, "none", None))
        elif 6 * self.mask_rows.len <= N and d.rows_tn_supported(SINGLE, C):
            d.dispatch(opspec.rows_tn(self.dh2, Cp, self.A, N, self.dlog, Cp, self.mask_rows, N, C))
        else:
            self._prop(self.dlog, self.dh2, C, Cp, transpose=True)

    def step(self, T_masked: DeviceSlice):
        """T_masked: one-hot targets of the masked rows, fp32 [M, C] contiguous."""
        key = (T_masked.ptr, T_masked.dtype, numbers(self.lr, self.beta1, self.beta2, self.eps, self.max_norm, self.delta), self.opt, str(self.clip))
        self._graphs.run(key, lambda: self._step(T_masked), lambda: (self.t,), self._set_t)

    def _set_t(self, state):
        (self.t,) = state

    def _step(self, T_masked: DeviceSlice):
        d, N, F, H, C, Fp, Cp, M = self.dev, self.N, self.F, self.H, self.C, self.Fp, self.Cp, self.M
        # zero_grad (model.zig:49-54) and the zero gradient the MaskLayer backward scatters into, one fill.  Nothing in the
        # forward pass needs them, but while the fill is small the fork and the join, which keeps the loss from being launched
        # while the last propagation still runs, cost more than it does: 0.16 MB 49.5 us a step in front of the forward pass,
        # 51.3 beside it; 1.5 MB 82.5 and 82.2; 3 MB 98.5 and 96.6.
        beside = self.cleared.nbytes > 1 << 20
        if beside:
            with d.branch(1):
                d.mem_fill(self.cleared, 0.0)
        else:
            d.mem_fill(self.cleared, 0.0)
        # ---- forward
        self._mm(self.X, self.W1, self.h1, N, H, F, False, True, Fp, Fp, H)                       # h1 = X . W1^T
        self._prop(self.h1, self.a1, H, H, "bias_relu", self.b1)                                   # relu(A.h1 + b1)
        self._mm(self.a1, self.W2, self.h2, N, C, H, False, True, H, H, Cp)                       # h2 = a1 . W2^T
        self._prop(self.h2, self.logits, C, Cp, "bias", self.b2)                                   # A.h2 + b2
        # ---- mask rows, loss, gradient of the masked logits (+ db2 = its column sums)
        if beside:
            d.join()
        if d.masked_softmax_ce_supported(SINGLE, M, C):
            d.dispatch(opspec.masked_softmax_ce(self.logits, self.offsets, T_masked, M, C, Cp, self.loss, self.dlog, float(M), self.db2))
        else:
            d.mem_take(self.logits, self.offsets, self.mlog)
            d.dispatch(opspec.softmax_ce(self.mlog, T_masked, M, C, self.loss, self.dm, float(M), accumulate=False, ld=Cp,
                                         bias_grad=self.db2))
            d.dispatch(opspec.scatter_add(self.dm, self.offsets, self.dlog))                        # MaskLayer backward
        # ---- backward
        self._prop_dlogits()                                                                       # dh2 = A^T . dlogits
        with d.branch(0):  # nothing below reads dW2: beside the rest of the backward pass
            self._mm(self.dh2, self.a1, self.dW2, C, H, N, True, False, Cp, H, H, 1.0)            # dW2 += dh2^T . a1
        self._mm(self.dh2, self.W2, self.da1, N, H, C, False, False, Cp, H, H, 0.0, "relu_mask", None, self.a1,
                 colsum=self.db1)                                                                   # da1, db1
        self._prop(self.da1, self.dh1, H, H, transpose=True)                                      # dh1 = A^T . da1
        # (with the padding columns, which X holds as zeros: rows of whole 16-byte words leave through the tensor map)
        self._mm(self.dh1, self.X, self.dW1, H, Fp, N, True, False, H, Fp, Fp, 1.0)               # dW1 += dh1^T . X
        d.join()
        # ---- update
        if self.opt == "adam":
            d.dispatch(opspec.adam(self.params, self.grads, self.m, self.v, self.segments, self.t + 1, self.lr, self.beta1,
                                   self.beta2, self.eps, self.clip, self.max_norm, self.delta, self.norms, None, self.t_dev))
            self.t += 4

    def read_loss(self) -> float:
        return float(self.dev.to_numpy(self.loss)[0])

    def numpy(self, name: str) -> np.ndarray:
        """A tensor by name with the padding stripped."""
        d, N, F, H, C, Fp, Cp = self.dev, self.N, self.F, self.H, self.C, self.Fp, self.Cp
        shapes = {"W1": (H, Fp, F), "dW1": (H, Fp, F), "W2": (C, H, H), "dW2": (C, H, H), "b1": (1, H, H), "db1": (1, H, H),
                  "b2": (1, C, C), "db2": (1, C, C), "a1": (N, H, H), "da1": (N, H, H), "logits": (N, Cp, C), "dlog": (N, Cp, C)}
        r, ld, c = shapes[name]
        a = d.to_numpy(getattr(self, name)).reshape(r, ld)[:, :c]
        return a.copy() if r > 1 else a.ravel().copy()

    def free(self):
        d = self.dev
        d.sync()
        self._graphs.clear()
        extra = list(self.csr) + [self.deg] if self.sparse else [self.A]
        for s in extra + [self.mask_rows, self.X, self.params, self.cleared, self.m, self.v, self.norms, self.h1, self.a1, self.h2, self.logits,
                  self.dh2, self.da1, self.dh1, self.mlog, self.dm, self.offsets, self.loss, self.t_dev]:
            d.mem_cache_free(s)
