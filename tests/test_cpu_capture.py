"""Recording into a CUDA graph: what surrounds the recording, with a stand-in for the device."""
import contextlib

import pytest
import torch

from tensornet_b200.utils import capture as C


class _Graph:
    def __init__(self, log):
        self.log = log

    def capture_begin(self, *pool):
        self.log.append("begin")

    def capture_end(self):
        self.log.append("end")


@pytest.fixture()
def device(monkeypatch):
    """``device.free / device.reserved`` in GB on a device of 180; ``device.log`` of what was called."""
    class D:
        free, reserved, log = 100, 10, []
    d = D()
    d.log = []
    monkeypatch.setattr(torch.cuda, "current_device", lambda: 0)
    monkeypatch.setattr(torch.cuda, "Stream", lambda device=None: object())
    monkeypatch.setattr(torch.cuda, "stream", lambda s: contextlib.nullcontext())
    monkeypatch.setattr(torch.cuda, "synchronize", lambda *a: None)
    monkeypatch.setattr(torch.cuda, "mem_get_info", lambda *a: (d.free << 30, 180 << 30))
    monkeypatch.setattr(torch.cuda, "memory_reserved", lambda *a: d.reserved << 30)
    monkeypatch.setattr(torch.cuda, "empty_cache", lambda: d.log.append("empty"))
    monkeypatch.setattr(C, "_STREAMS", {})
    return d


@pytest.mark.parametrize("free,reserved,gives_back", [(100, 10, False), (100, 120, True), (20, 10, True), (30, 29, False)])
def test_cached_memory_goes_back_where_memory_is_short(device, free, reserved, gives_back):
    device.free, device.reserved = free, reserved
    with C.capture(_Graph(device.log)):
        device.log.append("body")
    assert device.log == (["empty"] if gives_back else []) + ["begin", "body", "end"]


def test_two_threads_leave_the_collector_as_they_found_it(device):
    """The second capture begins inside the first and ends after it."""
    import gc

    assert gc.isenabled()
    first, second = C.capture(_Graph(device.log)), C.capture(_Graph(device.log))
    first.__enter__()
    second.__enter__()
    first.__exit__(None, None, None)
    assert not gc.isenabled()              # the second one is still recording
    second.__exit__(None, None, None)
    assert gc.isenabled()
    with pytest.raises(ValueError):
        with C.capture(_Graph(device.log)):
            raise ValueError
    assert gc.isenabled() and device.log[-1] == "end"
