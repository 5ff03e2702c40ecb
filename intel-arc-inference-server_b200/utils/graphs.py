"""Capture of a CUDA graph in a process that does other things meanwhile.

A dead engine's graphs and buffers may be released at any time, by the collector or by a thread that lets go of them.
In the capturing thread a release makes calls that a capture does not allow, so no thread starts a collection until the last
capture has ended.  One that runs already, or a reference dropped by another thread, releases them there: the capture takes no
notice of other threads (``thread_local``; in the default mode their calls fail and invalidate it).
"""
from __future__ import annotations

import gc
import threading
from typing import Callable

import torch

_lock = threading.Lock()
_running = 0             # captures under way, by any thread
_collects = False        # the collector was on when the first of them began


def _hold(by: int):
    global _running, _collects
    with _lock:
        if by > 0 and _running == 0:
            _collects = gc.isenabled()
            gc.disable()
        _running += by
        if _running == 0 and _collects:
            gc.enable()


def capture(enqueue: Callable[[], None]) -> "torch.cuda.CUDAGraph":
    """The launches that ``enqueue`` makes, as a graph."""
    g = torch.cuda.CUDAGraph()
    _hold(1)
    try:
        with torch.cuda.graph(g, capture_error_mode="thread_local"):
            enqueue()
    finally:
        _hold(-1)
    return g
