"""DQN update step on the device interface.

Restates ``DQNAgent.train`` + ``updateTargetNetwork`` of the reference
(``examples/dqn/src/dqn_agent.zig:111-228``; that example still targets the
library's removed Model/Layer API and loops over host memory, marked there as
"illegal in the incoming device api") as a fixed sequence of device ops:

  target net forward (no grad) -> clamp +-100 -> max over dim 1
  targets = r + gamma * max * (1 - done) -> clamp
  policy net forward -> clamp in place -> gather by action
  smooth-L1 (beta 1) -> gather backward (scatter_add) -> backward -> Adam (clip on)
  soft target update: target = (1 - tau) * target + tau * policy

Every tensor is tiny (batch 256, 4-128-128-2), so the step is launch-latency
bound; it is meant to be captured into ONE CUDA graph and replayed.
"""
from __future__ import annotations

import numpy as np

from . import opspec
from .abi import SINGLE
from .device import USIZE, CudaDevice, DeviceSlice
from .mlp import MlpTrainer
from .replay import GraphCache, numbers


class DqnTrainer:
    def __init__(self, dev: CudaDevice, dims, batch: int, weights, biases, lr: float = 1e-4, gamma: float = 0.99,
                 tau: float = 0.005, q_clip: float = 100.0):
        self.dev, self.B, self.C = dev, int(batch), int(dims[-1])
        self.gamma, self.tau, self.q_clip = gamma, tau, q_clip
        # policy net: Adam with the library's default clipping; target net: forward only
        self.policy = MlpTrainer(dev, dims, batch, weights, biases, "adam", lr=lr, clip=True, fused=True, pad_logits=False)
        self.target = MlpTrainer(dev, dims, batch, weights, biases, "none", fused=True, pad_logits=False)
        d, B = dev, self.B
        self.maxq = d.mem_cache_alloc(SINGLE, B)
        self.tmp = d.mem_cache_alloc(SINGLE, B)
        self.targets = d.mem_cache_alloc(SINGLE, B)
        self.q = d.mem_cache_alloc(SINGLE, B)
        self.dq = d.mem_cache_alloc(SINGLE, B)
        self.offsets = d.mem_cache_alloc(USIZE, B)
        self.gamma_s = d.from_numpy(np.array([gamma], np.float32))
        self.one_s = d.from_numpy(np.array([1.0], np.float32))
        self.loss = d.mem_cache_alloc(SINGLE, 1)
        self._graphs = GraphCache(d)  # repeated steps (replay.py)

    def step(self, states: DeviceSlice, actions: DeviceSlice, next_states: DeviceSlice, rewards: DeviceSlice,
             dones: DeviceSlice):
        p = self.policy
        key = (states.ptr, actions.ptr, next_states.ptr, rewards.ptr, dones.ptr,
               numbers(self.gamma, self.tau, self.q_clip, p.lr, p.beta1, p.beta2, p.eps, p.max_norm, p.delta), p.opt, str(p.clip),
               self.target._touched)
        self._graphs.run(key, lambda: self._step(states, actions, next_states, rewards, dones), self._host_state, self._set_host_state)

    def _host_state(self):
        return self.policy._host_state() + self.target._host_state()

    def _set_host_state(self, state):
        half = len(state) // 2
        self.policy._set_host_state(state[:half])
        self.target._set_host_state(state[half:])

    def _step(self, states: DeviceSlice, actions: DeviceSlice, next_states: DeviceSlice, rewards: DeviceSlice, dones: DeviceSlice):
        d, B, C = self.dev, self.B, self.C
        pol, tgt = self.policy, self.target
        grouped = pol.grouped
        # ---- both forward passes (gradients disabled in the reference for the target net): independent chains of
        # small kernels; zero_grad of the policy net rides on the side stream
        with d.branch(1):
            if tgt._touched:  # (it has no backward pass: only if somebody holds its gradients)
                tgt.zero_grad()
            qn = tgt._layers(next_states)
            if not grouped:
                pol.zero_grad()
        q_all = pol._layers(states)
        d.join()
        # ---- targets, gather by action, loss and its gradient w.r.t. all Q values, last bias gradient
        fused = d.q_head_supported(SINGLE, B, C)
        if fused:
            d.dispatch(opspec.q_head(qn, q_all, actions, rewards, dones, B, C, self.gamma, self.q_clip, 1.0, self.maxq, self.targets, self.q,
                                     self.offsets, self.loss, self.dq, pol.dact[-1], pol._db[-1]))
        else:
            self._head(qn, q_all, actions, rewards, dones)
        if grouped:
            pol.backward_grouped(states)
        else:
            pol.backward(states, last_bias_done=fused)
        # ---- Adam, and the soft update of the target parameters behind it
        pol.update(soft_target=tgt.params, tau=self.tau)

    def _head(self, qn, q_all, actions, rewards, dones):
        """opspec.q_head as separate ops (more actions than it is built for)."""
        d, B, C, qc = self.dev, self.B, self.C, self.q_clip
        d.dispatch(opspec.clamp_fwd(qn, qn, -qc, qc))
        d.dispatch(opspec.max_along(qn, [B, C], self.maxq, [B, 1], 1))
        d.dispatch(opspec.mul(self.maxq, self.gamma_s, self.tmp))          # gamma * max
        d.dispatch(opspec.sub(self.one_s, dones, self.targets))            # 1 - done
        d.dispatch(opspec.mul(self.tmp, self.targets, self.tmp))           # masked
        d.dispatch(opspec.add(rewards, self.tmp, self.targets))            # r + ...
        d.dispatch(opspec.clamp_fwd(self.targets, self.targets, -qc, qc))
        # the two zero fills the loss and the gather backward accumulate into (ensure_grad(0))
        d.mem_fill(self.dq, 0.0)
        d.mem_fill(self.policy.dact[-1], 0.0)
        d.dispatch(opspec.clamp_fwd(q_all, q_all, -qc, qc))
        d.gather_rows(q_all, actions, B, C, self.q, self.offsets)
        d.dispatch(opspec.smooth_l1(self.q, self.targets, 1.0, self.loss, self.dq))
        # gather backward: scatter into a zero gradient of all Q values
        d.dispatch(opspec.scatter_add(self.dq, self.offsets, self.policy.dact[-1]))

    def read_loss(self) -> float:
        return float(self.dev.to_numpy(self.loss)[0])

    def free(self):
        d = self.dev
        d.sync()
        self._graphs.clear()
        for s in (self.maxq, self.tmp, self.targets, self.q, self.dq, self.offsets, self.gamma_s, self.one_s, self.loss):
            d.mem_cache_free(s)
        self.policy.free()
        self.target.free()
