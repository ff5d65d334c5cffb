"""The rules by which a trainer's steps become graphs, on a stand-in for the library that records what is asked of it (no
GPU): what is issued when a capture fails or a step raises, where captures happen, and what a graph is found by."""
import ctypes as C
import threading
from fractions import Fraction

import numpy as np
import pytest
import torch

from zigrad_b200 import abi, device
from zigrad_b200.mlp import MlpTrainer, kaiming_uniform
from zigrad_b200.replay import GraphCache


class Library:
    """Calls by name, with the stream they went to; handles are numbers that are given out once."""

    def __init__(self):
        self.calls, self.error, self.fail, self.given = [], 0, set(), 0
        self.open = {}  # graph -> stream

    def _new(self):
        self.given += 64
        return self.given

    def init_stream(self):
        return abi.StreamWrapper(self._new())

    def init_cublas_handle(self, s):
        return abi.CublasWrapper(self._new())

    def init_cudnn_handle(self, s):
        return abi.CudnnWrapper(self._new())

    def init_cutensor_handle(self, s):
        return abi.CutensorWrapper(self._new())

    def init_device(self, n):
        return None

    def zg_device_available(self):
        return 1

    def zg_cache_alloc(self, cache, size, stream):
        return abi.Block(self._new() << 20, self._new())

    def zg_last_error(self):
        return self.error

    def zg_clear_error(self):
        self.error = 0

    def zg_stream_capturing(self, s):
        return int(s.ptr in self.open.values())

    def open_capture(self, s):
        self.calls.append(("open_capture", s.ptr))
        if "open" in self.fail:
            self.error = 1
            return abi.GraphWrapper(0)
        g = self._new()
        self.open[g] = s.ptr
        return abi.GraphWrapper(g)

    def save_capture(self, g, s):
        if not g.ptr:
            return
        self.calls.append(("save_capture", s.ptr))
        del self.open[g.ptr]
        if "save" in self.fail:
            self.error = 1

    def __getattr__(self, name):
        def call(*args):
            streams = [a.ptr for a in args if isinstance(a, abi.StreamWrapper)]
            self.calls.append((name, streams[0] if streams else None))
            return 0
        return call

    def names(self):
        return [n for n, _ in self.calls]


@pytest.fixture()
def dev(monkeypatch):
    lib = Library()
    monkeypatch.setattr(abi, "lib", lambda: lib)
    monkeypatch.setattr(abi, "check", lambda: None)
    return device.CudaDevice(0)


class Steps:
    """A step of one launch that counts, in the host's state too."""

    def __init__(self, dev):
        self.dev, self.t, self.ran = dev, 0, []
        self.cache = GraphCache(dev)
        self.hook = lambda: None

    def body(self):
        d = self.dev
        self.t += 1
        with d.branch(0):
            d.L.kernel(d.stream)
        self.hook()
        d.join()
        self.ran.append(d.capturing())

    def step(self, key=0):
        self.cache.run(key, self.body, lambda: (self.t,), self._set)

    def _set(self, s):
        (self.t,) = s


def test_third_call_is_captured_and_replayed(dev):
    s = Steps(dev)
    for i in range(6):
        s.step()
    assert s.ran == [False, False, True] and s.t == 6
    assert dev.L.names().count("open_capture") == 1 and dev.L.names().count("run_capture") == 4
    s.cache.clear()
    assert dev.L.names().count("free_capture") == 1


def test_capture_that_does_not_open_issues_the_step_once(dev):
    s = Steps(dev)
    s.step()
    s.step()
    dev.L.fail.add("open")
    for i in range(3, 6):
        s.step()
        assert s.ran == [False] * i and s.t == i and dev.L.error == 0
    assert "run_capture" not in dev.L.names() and "save_capture" not in dev.L.names()


def test_capture_that_cannot_be_saved_issues_the_step_instead(dev):
    s = Steps(dev)
    s.step()
    s.step()
    dev.L.fail.add("save")
    s.step()
    assert s.ran == [False, False, True, False] and s.t == 3 and dev.L.error == 0
    assert dev.L.names().count("free_capture") == 1 and "run_capture" not in dev.L.names()
    s.step()
    assert s.t == 4 and "run_capture" not in dev.L.names()


@pytest.mark.parametrize("call", [1, 2, 3])
def test_step_that_raises(dev, call):
    s = Steps(dev)

    def hook():
        if len(s.ran) + 1 == call:
            s.hook = lambda: None
            raise KeyError("from the step")

    s.hook = hook
    for _ in range(call - 1):
        s.step()
    with pytest.raises(KeyError):
        s.step()
    assert s.t == (call if call < 3 else 2)  # nothing of a captured step has run
    names = dev.L.names()
    assert names.count("open_capture") == names.count("save_capture") == names.count("free_capture") == (1 if call == 3 else 0)
    dev.join()
    for _ in range(6):
        s.step()
    assert "run_capture" in dev.L.names() and not dev.L.open
    assert s.t == (call if call < 3 else 2) + 6


def test_captures_happen_beside_the_streams_that_others_use(dev):
    s, main = Steps(dev), dev.stream.ptr
    seen, mine = [], []

    def hook():  # in the middle of the step
        th = threading.Thread(target=lambda: (seen.append(dev.stream.ptr), dev.capturing() and seen.append("capturing"), dev.L.copy(dev.stream)))
        th.start()
        th.join()
        mine.append(dev.stream.ptr)

    s.hook = hook
    for _ in range(5):
        s.step()
    assert seen == [main] * 3 and [x for n, x in dev.L.calls if n == "copy"] == [main] * 3
    assert mine[0] == main and main not in mine[1:]
    assert [x for n, x in dev.L.calls if n == "open_capture"] == [mine[2]] and mine[1] == mine[2]
    assert [x for n, x in dev.L.calls if n == "run_capture"] == [main] * 3
    kernels = [x for n, x in dev.L.calls if n == "kernel"]
    assert kernels[1] == kernels[2] != kernels[0]  # side streams of their own, too
    with dev.branch(0):
        assert dev.stream.ptr == kernels[0]
    dev.join()
    assert dev.stream.ptr == main


def test_one_thread_captures_at_a_time(dev):
    first, second = Steps(dev), Steps(dev)
    for s in (first, second):
        s.step()
        s.step()

    def hook():
        th = threading.Thread(target=second.step)
        th.start()
        th.join()

    first.hook = hook
    first.step()
    assert first.ran == [False, False, True] and second.ran == [False, False, False] and second.t == 3
    second.step()
    assert second.ran[-1] is True and dev.L.names().count("run_capture") == 2


def test_stream_chosen_by_the_user_is_everybodys(dev):
    s, other = Steps(dev), dev.L.init_stream()
    main, dev.stream = dev.stream, other
    seen = []
    th = threading.Thread(target=lambda: seen.append(dev.stream.ptr))
    th.start()
    th.join()
    for _ in range(4):
        s.step()
    assert seen == [other.ptr] and "open_capture" not in dev.L.names()
    dev.stream = main


def trainer(dev, **kw):
    dims = [12, 8, 5]
    Ws, bs = kaiming_uniform(dims, 1)
    tr = MlpTrainer(dev, dims, 4, Ws, bs, "sgd", **kw)
    X, T = dev.mem_cache_alloc(abi.SINGLE, 48), dev.mem_cache_alloc(abi.SINGLE, 20)
    return tr, lambda: tr.step(X, T)


@pytest.mark.parametrize("number", [float, np.float32, np.array, torch.tensor, Fraction], ids=lambda f: f.__name__)
def test_hyper_parameters_are_found_by_value(dev, number):
    """Whatever holds the number: it is compared as a number, also if the holder is changed in place or cannot be hashed."""
    tr, step = trainer(dev)
    runs = lambda: dev.L.names().count("run_capture")
    tr.lr = number(0.25)
    for _ in range(3):
        step()
    assert runs() == 1
    tr.lr = number(0.25)
    step()
    assert runs() == 2
    if hasattr(tr.lr, "fill_") or hasattr(tr.lr, "fill") and tr.lr.__class__ is np.ndarray:
        (tr.lr.fill_ if hasattr(tr.lr, "fill_") else tr.lr.fill)(0.5)
    else:
        tr.lr = number(0.5)
    step()
    assert runs() == 2
    step()
    step()
    assert runs() == 3
