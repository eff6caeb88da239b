"""Recorded passes: a fixed sequence of kernel launches over fixed buffers, replayed with one host call."""
from __future__ import annotations

import ctypes as C

import torch

from . import _lib as L
from . import kernels as K


def capturing() -> bool:
    """True while the current stream is being captured (by a caller's own CUDA graph)."""
    return bool(L.lib().grb_is_capturing(L.stream()))


class Recording:
    """``body()`` captured on a side stream as one CUDA graph.  Everything it launches must be on the current stream (or
    on streams forked from it and joined again) and must not allocate; it does not run while it is recorded."""

    def __init__(self, body, device):
        self._exec = C.c_void_p()
        side = torch.cuda.Stream(device=device)
        n0 = K.LAUNCHES
        with torch.cuda.stream(side):
            L.check(L.lib().grb_capture_begin(L.stream()), "grb_capture_begin")
            try:
                body()
            finally:
                rc = L.lib().grb_capture_end(L.stream(), C.byref(self._exec))
        L.check(rc, "grb_capture_end")
        self.launches = K.LAUNCHES - n0
        K.LAUNCHES = n0

    def replay(self) -> None:
        L.check(L.lib().grb_graph_launch(self._exec, L.stream()), "grb_graph_launch")
        K.LAUNCHES += self.launches

    def __del__(self):
        if getattr(self, "_exec", None) and L._LIB is not None:
            L._LIB.grb_graph_destroy(self._exec)


class Recorder:
    """Recordings of the passes over one set of buffers, by key.  The first two passes of a key run as they are
    (kernels are loaded and configured then, and a program with few passes pays for no recording); the third is recorded.
    At most ``limit`` keys are kept, the oldest goes first."""

    def __init__(self, limit: int = 8):
        self.limit = limit
        self._seen: dict = {}

    def __reduce__(self):
        return Recorder, (self.limit,)       # a copy of the model has buffers of its own and records for itself

    def run(self, key, body, device) -> None:
        rec = self._seen.get(key, 0)
        if isinstance(rec, Recording):
            rec.replay()
            return
        if capturing():
            body()
            return
        if rec < 2:
            while key not in self._seen and len(self._seen) >= self.limit:
                self._seen.pop(next(iter(self._seen)))
            self._seen[key] = rec + 1
            body()
            return
        self._seen[key] = rec = Recording(body, device)
        rec.replay()
