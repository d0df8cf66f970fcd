"""Recording work into a CUDA graph without the housekeeping of ``torch.cuda.graph``."""
from __future__ import annotations

import gc
from contextlib import contextmanager

import torch

_STREAMS = {}


@contextmanager
def capture(graph: "torch.cuda.CUDAGraph", pool=None):
    """Record what the body launches into ``graph``.  ``torch.cuda.graph`` collects garbage and empties the caching
    allocator first, which takes 50 to 100 ms next to the few milliseconds of a capture and has every later allocation
    go to the driver again; here the collector is held off instead while the capture runs (freeing a captured graph in
    the middle of one is an error)."""
    dev = torch.cuda.current_device()
    stream = _STREAMS.get(dev)
    if stream is None:
        stream = _STREAMS[dev] = torch.cuda.Stream(device=dev)
    torch.cuda.synchronize()
    held = gc.isenabled()
    gc.disable()
    try:
        with torch.cuda.stream(stream):
            graph.capture_begin(*(() if pool is None else (pool,)))
            try:
                yield
            finally:
                graph.capture_end()
    finally:
        if held:
            gc.enable()
