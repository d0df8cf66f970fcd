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
    the middle of one is an error).  Where memory is short, garbage and the allocator's cached blocks do go back: a capture's
    own pool cannot use them and nothing can be freed while it records."""
    dev = torch.cuda.current_device()
    stream = _STREAMS.get(dev)
    if stream is None:
        stream = _STREAMS[dev] = torch.cuda.Stream(device=dev)
    torch.cuda.synchronize()
    free, total = torch.cuda.mem_get_info(dev)
    # no step so far has needed more than the allocator holds; an eighth of the device for steps that are larger
    if free < max(torch.cuda.memory_reserved(dev), total // 8):
        gc.collect()
        torch.cuda.empty_cache()
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
