"""Steps that repeat: the device work of a trainer's step as a graph the trainer keeps.

A training loop calls ``step`` over and over with the same few buffers.  Issued op by op, a small step costs the
host more than the device (77 us of Python and launches for 45 us of kernels at batch 64), so a step that is asked
for a third time with the same arguments is captured and replayed from then on: one launch.
What is kept is the sequence of launches, never a result.

A graph is used only for exactly the call it was captured from: the key holds every address, hyper-parameter and
option that the sequence depends on.  Calls inside a capture of the caller's own, inside a ``branch`` block, or with
side streams still forked are issued op by op as before.

Captures happen on streams of their own (``CudaDevice.apart``), so that what another thread issues on the device's
stream meanwhile runs there and then and does not enter the graph.  The call before the capture runs on those streams
too: it leaves them with the work space that a capture cannot allocate.
"""
from __future__ import annotations

from collections import OrderedDict
from typing import Callable, Hashable

CAPACITY = 8    # graphs (or candidates) per trainer; the one used longest ago goes first
GIVE_UP = 32    # evicted graphs after which a trainer stops capturing: its buffers change too often


def numbers(*values) -> tuple:
    """Hyper-parameters as a part of a key: by value, whatever holds them (an array or tensor may be changed in place)."""
    for v in values:
        if v.__class__ is not float:
            return tuple(map(float, values))
    return values


class GraphCache:
    def __init__(self, dev):
        self.dev = dev
        self.entries: "OrderedDict[Hashable, object]" = OrderedDict()  # key -> times seen, or (graph, state change)
        self.evicted = 0

    def run(self, key: Hashable, body: Callable[[], None], save: Callable[[], tuple], restore: Callable[[tuple], None]) -> None:
        """Issue `body()`, or replay it.  `save()` returns the host-side state `body` changes, as a tuple; `restore`
        is given the state to set after a replay, in which every int has advanced as it did when captured."""
        d = self.dev
        here = d._here
        if (here.replaying or here.stream is not None or d._stream is not d.main_stream or d._main.forked or self.evicted >= GIVE_UP
                or d.L.zg_stream_capturing(d.main_stream)):
            return body()
        key = (key, d.L.zg_get_math_mode())
        hit = self.entries.get(key)
        if hit.__class__ is tuple:
            self._launch(hit[0])
            restore(tuple(a + b if b.__class__ is int else b for a, b in zip(save(), hit[1])))
            self.entries.move_to_end(key)
            return
        here.replaying = True
        try:
            if hit is None:
                self.entries[key] = 1
                if len(self.entries) > CAPACITY:
                    self._drop(self.entries.popitem(last=False)[1])
            elif not d.L.zg_last_error():
                self.entries.move_to_end(key)
                with d.apart() as lane:
                    done = lane is not None and (self._rehearse(lane, body) if hit == 1 else self._capture(key, lane, body, save, restore))
                if done:
                    if hit == 1:
                        self.entries[key] = 2
                    else:
                        self._launch(self.entries[key][0])
                    return
            return body()
        finally:
            here.replaying = False

    def _launch(self, graph) -> None:
        d = self.dev
        with d._apart_lock:  # its nodes use the work space of the streams it was captured on
            d.L.run_capture(graph, d.main_stream)

    def _rehearse(self, lane, body) -> bool:
        d = self.dev
        d.L.zg_stream_wait(lane.stream, d.main_stream)
        try:
            body()
        finally:
            d.join()
            d.L.zg_stream_wait(d.main_stream, lane.stream)
        return True

    def _capture(self, key, lane, body, save, restore) -> bool:
        """False: there is no graph, nothing of the step has been issued, and all is as before the call."""
        d = self.dev
        before = save()
        graph = d.L.open_capture(lane.stream)
        try:
            if graph.ptr:
                body()
        except BaseException:
            d.L.save_capture(graph, lane.stream)
            self._undo(graph, lane, before, restore)
            raise
        if graph.ptr:
            d.L.save_capture(graph, lane.stream)
        if d.L.zg_last_error():  # something in it cannot be captured
            self._undo(graph, lane, before, restore)
            self.evicted = GIVE_UP
            return False
        self.entries[key] = (graph, tuple(b - a if b.__class__ is int else b for a, b in zip(before, save())))
        return True

    def _undo(self, graph, lane, before, restore) -> None:
        self.dev.L.free_capture(graph, lane.stream)
        self.dev.L.zg_clear_error()
        lane.forked = []
        restore(before)

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
