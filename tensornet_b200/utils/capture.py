"""Recording work into a CUDA graph without the housekeeping of ``torch.cuda.graph``."""
from __future__ import annotations

import gc
import threading
from contextlib import contextmanager

import torch

_STREAMS = {}


class _CollectorOff:
    """The garbage collector is off while any thread is inside, and then back as the first one found it."""

    def __init__(self):
        self.lock, self.inside, self.was_on = threading.Lock(), 0, False

    def __enter__(self):
        with self.lock:
            if self.inside == 0:
                self.was_on = gc.isenabled()
                gc.disable()
            self.inside += 1

    def __exit__(self, *_):
        with self.lock:
            self.inside -= 1
            if self.inside == 0 and self.was_on:
                gc.enable()


_collector_off = _CollectorOff()


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
    if pool is None:               # (the first capture of a group: the others find what it needed in their common pool)
        free, total = torch.cuda.mem_get_info(dev)
        # no step so far has needed more than the allocator holds; an eighth of the device for steps that are larger
        if free < max(torch.cuda.memory_reserved(dev), total // 8):
            gc.collect()
            torch.cuda.empty_cache()
    with _collector_off, torch.cuda.stream(stream):
        graph.capture_begin(*(() if pool is None else (pool,)))
        try:
            yield
        finally:
            graph.capture_end()
