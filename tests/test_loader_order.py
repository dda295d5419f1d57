"""Order of the device loader's side stream against the caller's stream."""
from __future__ import annotations

import contextlib
import types

import pytest
import torch

from ade_b200 import packed_io, synth


def test_side_stream_waits_for_the_callers_stream(monkeypatch):
    """The blocks a load writes come from the caller's stream: the side stream waits for that stream after they were allocated and
    before anything is written, and the allocator is told about the side stream for every one of them."""
    log, recorded = [], []

    class Stream:
        cuda_stream = 0

        def wait_stream(self, other):
            log.append(("wait", other))

    class Event:
        def record(self, stream):
            log.append("done")

        def synchronize(self):
            pass

    @contextlib.contextmanager
    def on(what):
        if isinstance(what, Stream):
            log.append("side")
        yield

    real_empty = torch.empty
    monkeypatch.setattr(torch, "empty", lambda *a, pin_memory=False, **k: log.append("empty") or real_empty(*a, **k))
    monkeypatch.setattr(torch.cuda, "device", on)
    monkeypatch.setattr(torch.cuda, "stream", on)
    monkeypatch.setattr(torch.cuda, "Event", Event)
    monkeypatch.setattr(torch.cuda, "current_stream", lambda d=None: ("current", d))
    monkeypatch.setattr(torch.Tensor, "record_stream", lambda t, s: recorded.append(t))
    loader = object.__new__(packed_io.DeviceDeltaLoader)
    loader.device, loader.stream, loader._turn = torch.device("cpu"), Stream(), 0
    loader._pinned, loader._staged, loader._free = [None, None], [None, None], [None, None]
    loader.lib = types.SimpleNamespace(ade_b200_pack_delta=lambda *a: log.append("pack") or 0)
    out = loader.load(synth.random_packed(16, 128, 128, 0))
    wait = log.index(("wait", ("current", loader.device)))
    assert max(i for i, e in enumerate(log) if e == "empty") < wait < log.index("side") < log.index("pack") < log.index("done")
    tensors = [t for t in out.values() if torch.is_tensor(t)] + [loader._staged[0]]
    assert all(any(t is u for u in recorded) for t in tensors)


@pytest.mark.gpu
def test_load_does_not_overwrite_what_queued_kernels_read():
    """A tensor freed on the host while a copy of it is still queued: its block goes to the loader, the copy has its old values."""
    M, N, r = 8192, 1024, 512
    packed = synth.random_packed(M, N, r, 1)
    loader = packed_io.DeviceDeltaLoader("cuda")
    warm = [loader.load(packed), loader.load(packed)]                     # both staging blocks exist
    loader.finish()
    torch.cuda.synchronize()
    del warm
    torch.cuda.empty_cache()                                              # the next blocks are cut from a segment of their own
    old = torch.full((M, r // 2), 7, dtype=torch.uint8, device="cuda")
    torch.cuda.synchronize()
    torch.cuda._sleep(200_000_000)                                        # about a tenth of a second of queued work
    ptr, kept = old.data_ptr(), old.clone()
    del old
    out = loader.load(packed)
    loader.finish()
    torch.cuda.synchronize()
    assert any(t.data_ptr() == ptr for t in out.values() if torch.is_tensor(t)), "the block was not handed on: nothing was tested"
    assert bool((kept == 7).all())
