"""Automatic garbage collection off over a block, for any number of blocks at once."""
from __future__ import annotations

import contextlib
import gc
import threading

_lock = threading.Lock()
_open = 0        # blocks being run, over all threads
_was_on = False  # collection before the first of them


@contextlib.contextmanager
def no_collection():
    """Automatic garbage collection is off until the last such block ends (of whatever thread), then as it was before the
    first. Over a CUDA graph capture: a collection may free an older step (its launch list holds it in a reference cycle) with
    its CUDA graph, and the calls that frees it with invalidate the capture. Over a serving loop: a generation-2
    collection over the tens of thousands of request and result objects stops the host for about 30 ms, which shows up
    directly in the latency tail (the serving objects hold no reference cycles)."""
    global _open, _was_on
    with _lock:
        if _open == 0:
            _was_on = gc.isenabled()
            gc.disable()
        _open += 1
    try:
        yield
    finally:
        with _lock:
            _open -= 1
            if _open == 0 and _was_on:
                gc.enable()
