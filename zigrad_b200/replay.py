"""Steps that repeat: the device work of a trainer's step as a graph the trainer keeps.

A training loop calls ``step`` over and over with the same few buffers.  Issued op by op, a small step costs the
host more than the device (77 us of Python and launches for 45 us of kernels at batch 64), so a step that is asked
for a third time with the same arguments is captured while it runs and replayed from then on: one launch.
What is kept is the sequence of launches, never a result.

A graph is used only for exactly the call it was captured from: the key holds every address, hyper-parameter and
option that the sequence depends on.  Calls inside a capture of the caller's own, inside a ``branch`` block, or with
side streams still forked are issued op by op as before.
"""
from __future__ import annotations

from collections import OrderedDict
from typing import Callable, Hashable

CAPACITY = 8    # graphs (or candidates) per trainer; the one used longest ago goes first
GIVE_UP = 32    # evicted graphs after which a trainer stops capturing: its buffers change too often


class GraphCache:
    def __init__(self, dev):
        self.dev = dev
        self.entries: "OrderedDict[Hashable, object]" = OrderedDict()  # key -> times seen, or (graph, state change)
        self.evicted = 0

    def run(self, key: Hashable, body: Callable[[], None], save: Callable[[], tuple], restore: Callable[[tuple], None]) -> None:
        """Issue `body()`, or replay it.  `save()` returns the host-side state `body` changes, as a tuple; `restore`
        is given the state to set after a replay, in which every int has advanced as it did when captured."""
        d = self.dev
        if d.replaying or d._forked or d.stream.ptr != d.main_stream.ptr or self.evicted >= GIVE_UP or d.L.zg_stream_capturing(d.stream):
            return body()
        key = (key, d.L.zg_get_math_mode())
        hit = self.entries.get(key)
        if hit.__class__ is tuple:
            graph, delta = hit
            d.L.run_capture(graph, d.stream)
            restore(tuple(a + b if b.__class__ is int else b for a, b in zip(save(), delta)))
            self.entries.move_to_end(key)
            return
        d.replaying = True
        try:
            if hit is None or hit < 2 or d.L.zg_last_error():
                self.entries[key] = min((hit or 0) + 1, 2)
                self.entries.move_to_end(key)
                if len(self.entries) > CAPACITY:
                    self._drop(self.entries.popitem(last=False)[1])
                return body()
            before = save()
            graph = d.L.open_capture(d.stream)
            if not graph.ptr:  # what is issued now runs now: once
                d.L.zg_clear_error()
                self.evicted = GIVE_UP
                return body()
            try:
                body()
            except BaseException:  # none of it has run: as before the call, side streams included
                d.L.save_capture(graph, d.stream)
                d.L.free_capture(graph, d.stream)
                d.L.zg_clear_error()
                d._forked = []
                restore(before)
                raise
            d.L.save_capture(graph, d.stream)
            if d.L.zg_last_error():  # something in it cannot be captured: nothing ran, so issue it after all
                d.L.zg_clear_error()
                d.L.free_capture(graph, d.stream)
                self.evicted = GIVE_UP
                restore(before)
                return body()
            self.entries[key] = (graph, tuple(b - a if b.__class__ is int else b for a, b in zip(before, save())))
            d.L.run_capture(graph, d.stream)
        finally:
            d.replaying = False

    def _drop(self, entry) -> None:
        if entry.__class__ is tuple:
            self.evicted += 1
            self.dev.sync()  # it may still be running
            self.dev.L.free_capture(entry[0], self.dev.stream)

    def clear(self) -> None:
        evicted = self.evicted
        while self.entries:
            self._drop(self.entries.popitem()[1])
        self.evicted = evicted
