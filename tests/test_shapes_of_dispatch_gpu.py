"""Shapes where the kernels' work splits and dispatch rules change: pairs of CTAs for prefill (query blocks
around one 128-row half and one 256-row pair, key ranges around a 128-key tile, heads that do and do not
divide 128), equal shares of a decode batch (share and sequence boundaries, batches above a warp's 32
sequences, more pieces than one merge holds), and a layer's store and attention as one call."""
import math

import pytest
import torch

from oracle import paged_attention_oracle as O
from tests.helpers import assert_close_to_oracle
from tests.test_page_granular_gpu import make_pool

pytestmark = pytest.mark.gpu


def _i32(x):
    return torch.tensor(x, dtype=torch.int32).cuda()


def _problem(q_lens, prefixes, hkv, hq, d, seed, dtype=torch.bfloat16):
    kv_lens = [a + b for a, b in zip(q_lens, prefixes)]
    kc, vc, pip, pidx, slots = make_pool(kv_lens, 16, hkv, seed=seed, d=d, dtype=dtype)
    g = torch.Generator().manual_seed(seed + 1)
    q = torch.randn(sum(q_lens), hq, d, generator=g).to(dtype).cuda()
    gate = torch.randn(sum(q_lens), hq, d, generator=g).to(dtype).cuda()
    return q, gate, kc, vc, pip, pidx, slots, kv_lens


@pytest.mark.parametrize("d,hkv,hq", [(128, 2, 8), (128, 1, 6), (256, 1, 8), (256, 2, 12)])
@pytest.mark.parametrize("q_lens,prefixes,cross,window", [
    ([129], [0], False, 0), ([22, 43, 65], [0, 128, 127], False, 0), ([64, 33, 1], [129, 640, 300], False, 0),
    ([85, 171], [1000, 0], False, 200), ([100, 70], [513, 15], True, 0),
    ([300, 131, 217] * 12, [0, 5, 40] * 12, False, 0)], ids=lambda x: str(x)[:40])
def test_prefill_pairs(d, hkv, hq, q_lens, prefixes, cross, window):
    """Through page ids, per-token slots and with a gate; the three agree with the oracle.  (The last: enough
    short items at head_dim 128 for the one-CTA form.)"""
    from mini_sglang_mlx_b200 import paged_prefill_attention, paged_prefill_attention_p16
    q, gate, kc, vc, pip, pidx, slots, kv_lens = _problem(q_lens, prefixes, hkv, hq, d, sum(q_lens) + hq)
    qo, kvp, pre = _i32(O.build_indptr(q_lens).tolist()), _i32(O.build_indptr(kv_lens).tolist()), _i32(prefixes)
    kw = dict(is_cross_attention=cross, sliding_window_size=window)
    sc, n = 1 / math.sqrt(d), max(q_lens)
    ref = O.paged_prefill_attention_oracle(q, kc, vc, qo, kvp, slots, pre, sc, **kw)
    paged = (q, kc, vc, qo, pip, pidx, _i32(kv_lens), pre, sc, n)
    out = paged_prefill_attention_p16(*paged, page_size=16, **kw)
    assert_close_to_oracle(out, ref, "pages")
    assert_close_to_oracle(paged_prefill_attention(q, kc, vc, qo, kvp, slots, pre, sc, n, **kw), ref, "slots")
    gated = paged_prefill_attention_p16(*paged, page_size=16, gate=gate, **kw)
    assert_close_to_oracle(gated, out.float().cpu() * torch.sigmoid(gate.float()).cpu(), "gate")


@pytest.mark.parametrize("d,hkv,hq", [(128, 8, 16), (128, 2, 32), (256, 2, 16), (256, 1, 2)])
@pytest.mark.parametrize("kv_lens", [[64], [1, 0, 63, 64, 65, 4097], [20000], [0] * 5 + [17] * 31 + [900],
                                     [7, 300, 0, 1500] * 33], ids=lambda x: f"{len(x)}x{sum(x)}")
def test_decode_shares(d, hkv, hq, kv_lens):
    """(20000 tokens of one or two KV heads: more pieces than fit the merge at once.)"""
    from mini_sglang_mlx_b200 import paged_decode_attention, paged_decode_attention_p16
    q, gate, kc, vc, pip, pidx, slots, _ = _problem([1] * len(kv_lens), [max(l - 1, 0) for l in kv_lens], hkv, hq, d, 3)
    need = [max(l, 1) for l in kv_lens]       # (an empty sequence keeps its page, unread)
    kept, at = [], 0
    for l, n in zip(kv_lens, need):
        kept.append(slots[at:at + l])
        at += n
    slots, kvp, sc = torch.cat(kept), _i32(O.build_indptr(kv_lens).tolist()), 1 / math.sqrt(d)
    splits = _i32([4] * len(kv_lens))
    ref = O.paged_decode_attention_oracle(q, kc, vc, kvp, slots, sc)
    out = paged_decode_attention_p16(q, kc, vc, pip, pidx, _i32(kv_lens), splits, sc, 4, page_size=16)
    assert_close_to_oracle(out, ref, "pages")
    assert torch.equal(paged_decode_attention(q, kc, vc, kvp, slots, splits, sc, 4), out)
    gated = paged_decode_attention_p16(q, kc, vc, pip, pidx, _i32(kv_lens), splits, sc, 4, page_size=16, gate=gate)
    assert_close_to_oracle(gated, out.float().cpu() * torch.sigmoid(gate.float()).cpu(), "gate")


@pytest.mark.parametrize("page_size", [1, 16])
@pytest.mark.parametrize("phase,batch", [("DECODE", 1), ("DECODE", 40), ("DECODE", 129), ("PREFILL", 6)])
def test_a_layer_call_equals_store_then_attention(phase, batch, page_size):
    """A pool of another class keeps the separate calls; layers run back to back, with nothing between."""
    from mini_sglang_mlx_b200.attention import AttnBackend
    from mini_sglang_mlx_b200.core import Batch, BatchPhase, Req
    from mini_sglang_mlx_b200.kvcache import MHAKVCache

    class OtherPool(MHAKVCache):
        pass

    class Cfg:
        head_dim, num_kv_heads = 128, 2

    g = torch.Generator().manual_seed(batch)
    pages = torch.randperm(batch * (640 // page_size), generator=g).int().view(batch, -1)
    table = (pages[:, :, None] * page_size + torch.arange(page_size, dtype=torch.int32)).reshape(batch, -1).cuda()
    new = 1 if phase == "DECODE" else 70
    cached = torch.randint(0, 500, (batch,), generator=g).tolist()
    reqs = [Req(table_idx=i, cached_len=c, device_len=c + new) for i, c in enumerate(cached)]
    loc = torch.cat([table[i, c:c + new] for i, c in enumerate(cached)])
    n = loc.numel()
    x = [[torch.randn(n, h, 128, generator=g).bfloat16().cuda() for h in (8, 2, 2)] for _ in range(4)]
    w = [torch.randn(128, generator=g).bfloat16().cuda() for _ in range(2)]
    got = []
    for cls in (MHAKVCache, OtherPool):
        pool = cls(2, 4, 128, table.numel(), torch.bfloat16)
        pool._buffer.copy_(torch.randn(pool._buffer.shape, generator=torch.Generator().manual_seed(9)))
        be = AttnBackend(Cfg, pool, table, page_size=page_size)
        b = Batch(reqs=reqs, phase=BatchPhase[phase], out_loc=loc)
        be.prepare_metadata(b)
        outs = []
        for i, (q, k, v) in enumerate(x):
            outs.append(be.forward(q, k, v, i, b) if i % 2 else be.forward_from_projections(
                q.clone(), k, v, i, b, q_norm_weight=w[0], k_norm_weight=w[1], rope_base=1e6)
                if cls is MHAKVCache else _separate(be, pool, q, k, v, i, b, w))
        got.append((outs, pool._buffer.clone()))
    assert all(torch.equal(a, c) for a, c in zip(got[0][0], got[1][0]))
    assert torch.equal(got[0][1], got[1][1])


@pytest.mark.parametrize("page_size", [1, 16])
@pytest.mark.parametrize("d,hkv,hq,new,cached,mask,launches", [
    (128, 2, 8, [16] * 16, 3000, dict(sliding_window_size=1024), 1),                        # draft blocks
    (128, 2, 8, [8] * 70, 1500, {}, 1),                  # verification, key ranges split, merged by the last CTA
    (128, 2, 8, [8] * 5, 6000, {}, 2), (128, 2, 8, [128], 9000, {}, 2),       # merged by a second launch
    (128, 2, 6, [64 + i % 9 for i in range(40)], 500, {}, 1),       # more sequences than a warp finds its item among
    (256, 2, 16, [600, 33, 570], 900, {}, 1), (256, 2, 12, [9] * 3, 2000, {}, None), (256, 1, 6, [130] * 33, 90, {}, 1),
    (128, 1, 32, [2300, 40], 1500, {}, {1: 2, 16: 1}),              # per-token rows laid out as pages first
], ids=lambda x: str(x)[:24])
def test_a_layer_call_equals_store_then_attention_in_every_prefill_form(d, hkv, hq, new, cached, mask, launches, page_size):
    """Attention that starts while the layer's own store still writes, in the forms of prefill, against separate calls with a
    wait for the device between them: layers back to back, again with other rows over another pool."""
    from mini_sglang_mlx_b200 import _lib
    from mini_sglang_mlx_b200.attention import AttnBackend
    from mini_sglang_mlx_b200.core import Batch, BatchPhase, Req
    from mini_sglang_mlx_b200.kernel import qk_norm_rope_store
    from mini_sglang_mlx_b200.kvcache import MHAKVCache

    class WaitingPool(MHAKVCache):
        def store_kv(self, *args, **kw):
            super().store_kv(*args, **kw)
            torch.cuda.synchronize()

    class Cfg:
        head_dim, num_kv_heads = d, hkv

    g = torch.Generator().manual_seed(len(new) + d)
    batch, most = len(new), -(-(cached + max(new)) // page_size)
    lens = torch.randint(cached // 2, cached + 1, (batch,), generator=g).tolist()
    pages = torch.randperm(batch * most, generator=g).int().view(batch, -1)
    table = (pages[:, :, None] * page_size + torch.arange(page_size, dtype=torch.int32)).reshape(batch, -1).cuda()
    loc = torch.cat([table[i, c:c + x] for i, (c, x) in enumerate(zip(lens, new))])
    if launches is not None:
        total = sum(lens) + sum(new) if page_size == 1 else sum(-(-(c + x) // 16) * 16 for c, x in zip(lens, new))
        assert _lib.lib().msgl_prefill_launch_count(
            batch, sum(new), total, hq, hkv, d, max(new), mask.get("sliding_window_size", 0), int(page_size > 1)) == (
                launches if isinstance(launches, int) else launches[page_size])
    pools = [cls(hkv, 4, d, table.numel(), torch.bfloat16) for cls in (MHAKVCache, WaitingPool)]
    w = [torch.randn(d, generator=g).bfloat16().cuda() for _ in range(2)]
    dev = torch.Generator("cuda").manual_seed(d)
    for _ in range(3):
        x = [[torch.empty(sum(new), h, d, dtype=torch.bfloat16, device="cuda").normal_(generator=dev) for h in (hq, hkv, hkv)]
             for _ in range(4)]
        rows, got = torch.empty_like(pools[0]._buffer).normal_(generator=dev), []
        for pool in pools:
            pool._buffer.copy_(rows)
            be = AttnBackend(Cfg, pool, table, page_size=page_size)
            b = Batch(reqs=[Req(table_idx=i, cached_len=c, device_len=c + n) for i, (c, n) in enumerate(zip(lens, new))],
                      phase=BatchPhase.PREFILL, out_loc=loc)
            be.prepare_metadata(b)
            outs, qs = [], [q.clone() for q, _, _ in x]
            for i, (q, (_, k, v)) in enumerate(zip(qs, x)):
                if i % 2:
                    outs.append(be.forward(q, k, v, i, b, **mask))
                elif type(pool) is MHAKVCache:
                    outs.append(be.forward_from_projections(q, k, v, i, b, q_norm_weight=w[0], k_norm_weight=w[1],
                                                            rope_base=1e6, **mask))
                else:
                    q = qk_norm_rope_store(q, k, v, *w, b.attn_metadata.positions, loc, pool.k_cache(i), pool.v_cache(i),
                                           rope_base=1e6)
                    torch.cuda.synchronize()
                    outs.append(be._attend(q, pool.k_cache(i), pool.v_cache(i), b.attn_metadata, False,
                                           mask.get("sliding_window_size", 0)))
            got.append((outs, qs, pool._buffer.clone()))
        assert all(torch.equal(a, c) for kind in (0, 1) for a, c in zip(got[0][kind], got[1][kind]))
        assert torch.equal(got[0][2], got[1][2])


def _separate(be, pool, q, k, v, i, b, w):
    from mini_sglang_mlx_b200.kernel import qk_norm_rope_store
    if i % 2:
        return be.forward(q, k, v, i, b)
    md = b.attn_metadata
    q = qk_norm_rope_store(q.clone(), k, v, w[0], w[1], md.positions, b.out_loc, pool.k_cache(i), pool.v_cache(i),
                           rope_base=1e6)
    torch.cuda.synchronize()
    return be._attend(q, pool.k_cache(i), pool.v_cache(i), md, False, 0)


@pytest.mark.parametrize("batch", [31, 32, 33])
@pytest.mark.parametrize("d,hkv,hq,q_hi,window", [(128, 2, 6, 90, 0), (256, 1, 4, 90, 0), (128, 2, 8, 12, 0), (128, 1, 8, 16, 100)])
def test_items_of_up_to_32_sequences_and_of_more(batch, d, hkv, hq, q_hi, window):
    """Up to 32 sequences one warp finds a CTA's work item, beyond that the whole CTA does: pairs and one-CTA
    tiles, key ranges split or not, sequences without queries or keys, lengths that tie."""
    from mini_sglang_mlx_b200 import paged_prefill_attention, paged_prefill_attention_p16
    q_lens = [0 if i % 7 == 3 else 1 + (i * 37) % q_hi for i in range(batch)]
    prefixes = [0 if i % 3 == 0 else (i * 211) % 700 for i in range(batch)]
    q, _, kc, vc, pip, pidx, slots, kv_lens = _problem([max(n, 1) for n in q_lens], prefixes, hkv, hq, d, batch)
    kept, at = [], 0
    for n, x in zip(q_lens, kv_lens):                # (a sequence without queries has its cached tokens only)
        kept.append(slots[at:at + x - (n == 0)])
        at += x
    kv_lens = [x - (n == 0) for n, x in zip(q_lens, kv_lens)]
    slots, q = torch.cat(kept), q[:sum(q_lens)].contiguous()
    qo, kvp, pre = _i32(O.build_indptr(q_lens).tolist()), _i32(O.build_indptr(kv_lens).tolist()), _i32(prefixes)
    sc, n = 1 / math.sqrt(d), max(q_lens)
    ref = O.paged_prefill_attention_oracle(q, kc, vc, qo, kvp, slots, pre, sc, sliding_window_size=window)
    out = paged_prefill_attention_p16(q, kc, vc, qo, pip, pidx, _i32(kv_lens), pre, sc, n, page_size=16,
                                      sliding_window_size=window)
    assert_close_to_oracle(out, ref, "pages")
    out = paged_prefill_attention(q, kc, vc, qo, kvp, slots, pre, sc, n, sliding_window_size=window)
    assert_close_to_oracle(out, ref, "slots")


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("hkv,hq,q_lens,prefixes,kw", [
    (1, 32, [2600, 37, 0, 300], [100, 500, 64, 900], {}), (4, 32, [2300], [1], {}),
    (3, 48, [17, 1800], [0, 700], dict(sliding_window_size=900)), (2, 32, [2300, 1100], [3, 0], dict(is_cross_attention=True))],
    ids=lambda x: str(x)[:30])
def test_long_prefill_over_per_token_slots(hkv, hq, q_lens, prefixes, kw, dtype):
    """Rows laid out as pages first, with room for them in the scratch: the page-granular call's bits; slots outside
    the pool are zeros and reported.  With the least scratch the attention kernel gathers them itself."""
    from mini_sglang_mlx_b200 import _lib, paged_prefill_attention, paged_prefill_attention_p16
    from mini_sglang_mlx_b200.kernel import device_status
    d, lib = 128, _lib.lib()
    need = [max(n, 1) for n in q_lens]
    q, _, kc, vc, pip, pidx, slots, kv_lens = _problem(need, prefixes, hkv, hq, d, sum(q_lens), dtype=dtype)
    kept, at = [], 0
    for n, x in zip(q_lens, kv_lens):
        kept.append(slots[at:at + x - (n == 0)])
        at += x
    kv_lens = [x - (n == 0) for n, x in zip(q_lens, kv_lens)]
    slots, q = torch.cat(kept), q[:sum(q_lens)].contiguous()
    qo, kvp, pre = _i32(O.build_indptr(q_lens).tolist()), _i32(O.build_indptr(kv_lens).tolist()), _i32(prefixes)
    sc, n, batch, tq, tkv = 1 / math.sqrt(d), max(q_lens), len(q_lens), sum(q_lens), sum(kv_lens)
    window, cross = kw.get("sliding_window_size", 0), kw.get("is_cross_attention", False)
    shape = (batch, tq, tkv, hq, hkv, d, n, window)
    assert lib.msgl_prefill_launch_count(*shape, 0) == 2          # (the rows are laid out)
    args = (qo, kvp, slots, pre, sc, n)
    device_status()
    out = paged_prefill_attention(q, kc, vc, *args, **kw)
    paged = paged_prefill_attention_p16(q, kc, vc, qo, pip, pidx, _i32(kv_lens), pre, sc, n, page_size=16, **kw)
    assert torch.equal(out, paged) and device_status() == 0
    ref = O.paged_prefill_attention_oracle(q, kc, vc, qo, kvp, slots, pre, sc, **kw)
    assert_close_to_oracle(out, ref, "laid out")
    least, full = lib.msgl_prefill_workspace_bytes(*shape), lib.msgl_prefill_workspace_bytes_full(*shape)
    assert least < full <= least + (256 << 20)
    for size in (least, full - 1, full):
        ws = torch.full((size + 4096,), 255, dtype=torch.uint8, device="cuda")
        ws[:65792] = 0
        got = torch.empty_like(q)
        _lib.check(lib.msgl_paged_prefill_attention(
            q.data_ptr(), kc.data_ptr(), vc.data_ptr(), qo.data_ptr(), kvp.data_ptr(), slots.data_ptr(), pre.data_ptr(),
            got.data_ptr(), ws.data_ptr(), size, batch, tq, tkv, hq, hkv, d, kc.shape[0], int(dtype == torch.float16), sc, n,
            int(cross), window, torch.cuda.current_stream().cuda_stream))
        assert_close_to_oracle(got, ref, str(size))
        assert torch.equal(got, out) or size < full
        assert int(ws[:65792].sum()) == 0 and bool((ws[size:] == 255).all())
    bad = slots.clone()
    bad[::5], bad[1::7] = -1, kc.shape[0] + 3
    out = paged_prefill_attention(q, kc, vc, qo, kvp, bad, pre, sc, n, **kw)
    assert device_status() == 2
    kz, vz = torch.cat([kc, torch.zeros_like(kc[:1])]), torch.cat([vc, torch.zeros_like(vc[:1])])
    zeros = torch.where((bad < 0) | (bad >= kc.shape[0]), kc.shape[0], bad)
    assert_close_to_oracle(out, O.paged_prefill_attention_oracle(q, kz, vz, qo, kvp, zeros, pre, sc, **kw), "zeros")


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("hkv,hq,q_lens,prefixes,launches", [
    (2, 8, [64], [4 * 1024 - 40], 2), (2, 8, [64] * 3, [2 * 1024 - 40] * 3, 2), (2, 12, [43, 86], [3 * 1024 - 20, 1024 - 70], 2), (1, 8, [16], [2 * 1024 - 9], 2),
    (2, 8, [300, 131, 217] * 12, [-300, 5, -217] * 6 + [0, -131, 40] * 6, 1)], ids=lambda x: str(x)[:30])
def test_sub_tiles_without_keys(hkv, hq, q_lens, prefixes, launches, dtype):
    """Key ranges cut inside the new tokens, so that the first rows of an item have no key in a piece and the last ones
    do, and sequences without any key: zero rows and empty partials are staged where the queries land."""
    from mini_sglang_mlx_b200 import _lib, paged_prefill_attention, paged_prefill_attention_p16
    d, n = 128, max(q_lens)
    kv_lens = [a + b for a, b in zip(q_lens, prefixes)]
    kc, vc, pip, pidx, slots = make_pool([max(x, 1) for x in kv_lens], 16, hkv, seed=hq, d=d, dtype=dtype)
    keep, at = [], 0
    for x in kv_lens:
        keep.append(slots[at:at + x])
        at += max(x, 1)
    slots, q = torch.cat(keep), torch.randn(sum(q_lens), hq, d, generator=torch.Generator().manual_seed(hq)).to(dtype).cuda()
    shape = (len(q_lens), sum(q_lens), sum(kv_lens), hq, hkv, d, n, 0)
    assert _lib.lib().msgl_prefill_launch_count(*shape, 0) == launches
    qo, kvp, pre = (_i32(x) for x in (O.build_indptr(q_lens).tolist(), O.build_indptr(kv_lens).tolist(),
                                      [max(x, 0) for x in prefixes]))
    sc = 1 / math.sqrt(d)
    ref = O.paged_prefill_attention_oracle(q, kc, vc, qo, kvp, slots, pre, sc)
    out = paged_prefill_attention(q, kc, vc, qo, kvp, slots, pre, sc, n)
    assert_close_to_oracle(out, ref, "slots")
    paged = paged_prefill_attention_p16(q, kc, vc, qo, pip, pidx, _i32(kv_lens), pre, sc, n, page_size=16)
    assert_close_to_oracle(paged, ref, "pages")
    for b, x in enumerate(kv_lens):
        if x == 0:
            rows = slice(sum(q_lens[:b]), sum(q_lens[:b + 1]))
            assert not out[rows].any() and not paged[rows].any()


@pytest.mark.parametrize("lens", [[(8000, 6000)] + [(3, 5 * i) for i in range(39)], [(1, 0)] * 33 + [(8000, 6000)],
                                  [(7, 9)] * 2 + [(8000, 4001)] + [(0, 0)] * 3 + [(1, 6)]], ids=lambda x: str(len(x)))
def test_rows_of_a_long_sequence_among_short_ones_are_laid_out(lens):
    """Tokens are dealt to the copying warps across sequences: more than a warp's 32 of them, ends inside a warp's eight
    tokens, sequences without keys."""
    from mini_sglang_mlx_b200 import _lib, kernel as K, paged_prefill_attention, paged_prefill_attention_p16
    from mini_sglang_mlx_b200.kernel import device_status
    q_lens, prefixes = [a for a, _ in lens], [p for _, p in lens]
    hkv, hq, d, n, kv_lens = 1, 32, 128, max(q_lens), [a + p for a, p in lens]
    assert _lib.lib().msgl_prefill_launch_count(len(lens), sum(q_lens), sum(kv_lens), hq, hkv, d, n, 0, 0) == 2
    kc, vc, pip, pidx, slots = make_pool([max(x, 1) for x in kv_lens], 16, hkv, seed=len(lens), d=d)
    slots = torch.cat([s[:x] for s, x in zip(slots.split([max(x, 1) for x in kv_lens]), kv_lens)])
    q = torch.empty(sum(q_lens), hq, d, dtype=torch.bfloat16, device="cuda").normal_(generator=torch.Generator("cuda").manual_seed(1))
    qo, kvp, pre = _i32(O.build_indptr(q_lens).tolist()), _i32(O.build_indptr(kv_lens).tolist()), _i32(prefixes)
    device_status()
    out = paged_prefill_attention(q, kc, vc, qo, kvp, slots, pre, 0.1, n)
    paged = paged_prefill_attention_p16(q, kc, vc, qo, pip, pidx, _i32(kv_lens), pre, 0.1, n, page_size=16)
    assert torch.equal(out, paged) and device_status() == 0
    made = []          # (what the memory held before is not read: NaN here)
    _lib.host.set_pages_maker(lambda size, index, stream: made.append(torch.full(
        (size,), 255, dtype=torch.uint8, device="cuda")) or made[-1])
    try:
        again = paged_prefill_attention(q, kc, vc, qo, kvp, slots, pre, 0.1, n)
    finally:
        _lib.host.set_pages_maker(K._make_pages)
    assert made and torch.equal(again, paged)
