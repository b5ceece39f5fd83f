"""Scratch of the operators: who asks for it at the same time, and what becomes of an outgrown buffer."""
import contextlib
import threading

import pytest
import torch

from mini_sglang_mlx_b200 import kernel as K


@pytest.fixture
def host_scratch(monkeypatch):
    """The operators' scratch bookkeeping over host memory: no entry to begin with, none left behind."""
    monkeypatch.setattr(K, "_workspaces", {})
    monkeypatch.setattr(K, "_retired", [])
    monkeypatch.setattr(torch.cuda, "ExternalStream", lambda *a, **k: None)
    monkeypatch.setattr(torch.cuda, "stream", lambda s: contextlib.nullcontext())
    real = torch.zeros
    monkeypatch.setattr(torch, "zeros", lambda *a, device=None, **k: real(*a, **k))


def test_a_buffer_that_was_handed_out_is_kept(host_scratch, monkeypatch):
    """Two threads ask for the same scratch and meet inside the allocation (or would, if they may): the
    native calls keep the addresses they were given, so both buffers must stay alive."""
    meet = threading.Barrier(2)
    allocate = torch.zeros

    def slow(*a, **k):
        with contextlib.suppress(threading.BrokenBarrierError):
            meet.wait(timeout=1.0)
        return allocate(*a, **k)

    monkeypatch.setattr(torch, "zeros", slow)
    got = []
    threads = [threading.Thread(target=lambda: got.append(K._workspace(100, torch.device("cuda", 0), 7, "decode")))
               for _ in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    kept = {ws.data_ptr() for ws in [*K._workspaces.values(), *K._retired]}
    assert len(got) == 2 and {ws.data_ptr() for ws in got} <= kept


def test_growth_that_finds_no_memory_leaves_the_buffer_in_use(host_scratch, monkeypatch):
    dev = torch.device("cuda", 0)
    first = K._workspace(100, dev, 7, "decode")

    def none_left(*a, **k):
        raise torch.OutOfMemoryError("no memory")

    with monkeypatch.context() as m:
        m.setattr(torch, "zeros", none_left)
        with pytest.raises(torch.OutOfMemoryError):
            K._workspace(first.numel() + 1, dev, 7, "decode")
    assert K._workspace(100, dev, 7, "decode") is first and K._retired == []
    grown = K._workspace(first.numel() + 1, dev, 7, "decode")
    assert grown.numel() == 2 * first.numel() and K._retired == [first]


def test_a_report_from_before_a_buffer_grew_is_not_lost(host_scratch, monkeypatch):
    monkeypatch.setattr(torch.cuda, "synchronize", lambda device=None: None)
    dev = torch.device("cuda", 0)
    first = K._workspace(100, dev, 7, "decode")
    first[:4].view(torch.int32).fill_(2)              # (a kernel met a slot outside the pool)
    K._workspace(first.numel() + 1, dev, 7, "decode")
    assert K.device_status() == 2
    assert K.device_status() == 0
