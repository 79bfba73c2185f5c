"""Garbage collection and CUDA graphs: collection off over a block, for any number of blocks at once, and graphs that are not freed
within a capture."""
from __future__ import annotations

import contextlib
import gc
import threading
import weakref

import torch

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


_parked = []  # graphs of objects that went while a capture was running


def _let_go(graph):
    # Freeing a captured graph frees its memory pool, which a capture under way does not survive.
    if torch.cuda.is_current_stream_capturing():
        _parked.append(graph)
    else:
        _parked.clear()


def free_outside_captures(owner, graph) -> None:
    """Keep `graph` until `owner` goes, and past it while the current stream is being captured: the next call, or the next
    owner to go outside a capture, frees it then. An owner in a reference cycle may go at any time, in whatever capture a
    garbage collection comes due."""
    if not torch.cuda.is_current_stream_capturing():
        _parked.clear()
    weakref.finalize(owner, _let_go, graph).atexit = False
