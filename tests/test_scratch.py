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
    monkeypatch.setattr(K, "_captured_pages", {}, raising=False)
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


def test_growth_asks_for_what_it_needs_where_a_power_of_two_finds_no_memory(host_scratch, monkeypatch):
    dev, real, limit = torch.device("cuda", 0), torch.zeros, (1 << 20) + 5000

    def small(n, *a, **k):
        if n > limit:
            raise torch.OutOfMemoryError("no memory")
        return real(n, *a, **k)

    monkeypatch.setattr(torch, "zeros", small)
    assert K._workspace((1 << 20) + 4096, dev, 7, "prefill").numel() == (1 << 20) + 4096


def test_page_memory_of_a_captured_call_stays(host_scratch, monkeypatch):
    """A graph writes there whenever it is replayed, so the memory is neither given back nor taken twice; an
    uncaptured call's is its own."""
    real = torch.empty
    monkeypatch.setattr(torch, "empty", lambda n, *, dtype, device: real(n, dtype=dtype))
    monkeypatch.setattr(K, "_stream_handle", lambda stream, device: 7)
    monkeypatch.setattr(torch.cuda, "is_current_stream_capturing", lambda: False)
    a, b = K._make_pages(5000, 0, 7), K._make_pages(5000, 0, 7)
    assert a.data_ptr() != b.data_ptr()
    monkeypatch.setattr(torch.cuda, "is_current_stream_capturing", lambda: True)
    at = [K._make_pages(n, 0, stream).data_ptr() for n, stream in ((5000, 7), (4000, 7), (9000, 7), (9000, 7), (5000, 8))]
    others = [K._make_pages(5000, 0, 9 + i).data_ptr() for i in range(8)]        # (memory given back would be handed out)
    assert at[0] == at[1] != at[2] == at[3] and len({*at, *others}) == 3 + len(others)


def test_a_report_from_before_a_buffer_grew_is_not_lost(host_scratch, monkeypatch):
    monkeypatch.setattr(torch.cuda, "synchronize", lambda device=None: None)
    dev = torch.device("cuda", 0)
    first = K._workspace(100, dev, 7, "decode")
    first[:4].view(torch.int32).fill_(2)              # (a kernel met a slot outside the pool)
    K._workspace(first.numel() + 1, dev, 7, "decode")
    assert K.device_status() == 2
    assert K.device_status() == 0


@pytest.mark.gpu
@pytest.mark.parametrize("max_splits", [1, 2, 3, 32])
@pytest.mark.parametrize("kv_lens", [[5000], [1, 0, 700, 3000, 64], [40] * 50 + [2500] * 3], ids=lambda x: f"{len(x)}x{sum(x)}")
def test_decode_with_the_least_scratch_that_a_call_takes(kv_lens, max_splits):
    """Fewer partials than the op would like: fewer shares, down to a share per sequence (max_splits 1 and
    2: no room for a partial per share and sequence).  Bytes behind the scratch stay as they were."""
    import math

    from mini_sglang_mlx_b200 import _lib
    from oracle import paged_attention_oracle as O
    from tests.helpers import assert_close_to_oracle
    from tests.test_page_granular_gpu import make_pool
    hkv, hq, d, batch = 2, 8, 128, len(kv_lens)
    kc, vc, _, _, slots = make_pool(kv_lens, 16, hkv, seed=batch, d=d)
    q = torch.randn(batch, hq, d, generator=torch.Generator().manual_seed(1)).bfloat16().cuda()
    kvp = torch.from_numpy(O.build_indptr(kv_lens)).cuda()
    lib, sc = _lib.lib(), 1 / math.sqrt(d)
    need = lib.msgl_decode_workspace_bytes(batch, hq, d, max_splits)
    ws = torch.full((need + 4096,), 255, dtype=torch.uint8, device="cuda")
    ws[:65792] = 0
    out = torch.empty_like(q)
    for _ in range(2):
        _lib.check(lib.msgl_paged_decode_attention_sized(
            q.data_ptr(), kc.data_ptr(), vc.data_ptr(), kvp.data_ptr(), slots.data_ptr(), None, out.data_ptr(),
            ws.data_ptr(), need, batch, hq, hkv, d, kc.shape[0], 0, sc, max_splits, sum(kv_lens),
            torch.cuda.current_stream().cuda_stream))
        assert_close_to_oracle(out, O.paged_decode_attention_oracle(q, kc, vc, kvp, slots, sc))
    assert int(ws[:65792].sum()) == 0 and bool((ws[need:] == 255).all())


@pytest.mark.gpu
def test_a_long_prefill_over_token_slots_keeps_no_memory_and_does_without(monkeypatch):
    """Its K/V rows are laid out as pages in memory of the call's own, given back behind it; on a device
    without room for them it gathers the rows as it goes."""
    import math

    from mini_sglang_mlx_b200 import _lib
    from oracle import paged_attention_oracle as O
    from tests.helpers import assert_close_to_oracle
    from tests.test_page_granular_gpu import make_pool
    n, hkv, hq, d = 2300, 4, 32, 128
    kc, vc, _, _, slots = make_pool([n], 16, hkv, seed=4, d=d)
    q = torch.randn(n, hq, d, generator=torch.Generator().manual_seed(4)).bfloat16().cuda()
    ends, prefix = torch.tensor([0, n], dtype=torch.int32, device="cuda"), torch.zeros(1, dtype=torch.int32, device="cuda")
    pages = _lib.lib().msgl_prefill_kv_pages_bytes(1, n, n, hq, hkv, d, n, 0)
    assert pages > 1 << 20
    monkeypatch.setattr(K, "_pages_pause", {})

    def call():
        return K.paged_prefill_attention(q, kc, vc, ends, ends, slots, prefix, 1 / math.sqrt(d), n)

    out = call()
    held = torch.cuda.memory_allocated()
    again = call()
    assert torch.cuda.memory_allocated() - held <= 2 * again.numel() + 512 and K._pages_pause == {}
    assert torch.equal(out, again)
    del again
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    room, hold = torch.empty(2 * out.numel(), dtype=torch.uint8, device="cuda"), []
    total = torch.cuda.get_device_properties(0).total_memory
    try:
        torch.cuda.set_per_process_memory_fraction((torch.cuda.memory_reserved() + (64 << 20)) / total)
        with pytest.raises(torch.OutOfMemoryError):
            for _ in range(1000):
                hold.append(torch.empty(pages - 4096, dtype=torch.uint8, device="cuda"))
        del room                               # (room for the output)
        without = call()
    finally:
        torch.cuda.set_per_process_memory_fraction(1.0)
    assert K._pages_pause == {0: K._PAGES_PAUSE}
    ref = O.paged_prefill_attention_oracle(q, kc, vc, ends, ends, slots, prefix, 1 / math.sqrt(d))
    assert_close_to_oracle(out, ref, "laid out")
    assert_close_to_oracle(without, ref, "gathered")
