"""Hand-overs between threads and CTAs inside a kernel: inputs on which data that comes too late, or a
value that is paired with another's tag, changes the result."""
import math

import pytest
import torch

from oracle import paged_attention_oracle as O
from tests.helpers import assert_close_to_oracle
from tests.test_page_granular_gpu import make_pool

pytestmark = pytest.mark.gpu


def _i32(x):
    return torch.tensor(x, dtype=torch.int32).cuda()


@pytest.mark.parametrize("n,keys", [(200, 256), (200, 384), (1400, 2000), (1400, 9000)])
def test_v_copied_by_the_peers_threads_is_what_the_leader_multiplies(n, keys):
    """Pairs of CTAs with per-token slots copy V with their own threads, the page-granular form by TMA: the
    same tiles in the same order, so the same bits.  The pool changes from call to call: a row that is
    read before its copy is there would be one of the call before.  (Query tokens enough that the key range
    is not split.)"""
    from mini_sglang_mlx_b200 import _lib, paged_prefill_attention, paged_prefill_attention_p16
    hkv, hq, d = 4, 8, 256
    kc, vc, pip, pidx, slots = make_pool([keys], 16, hkv, seed=keys, d=d)
    g = torch.Generator(device="cuda").manual_seed(keys)
    q = torch.empty(n, hq, d, dtype=torch.bfloat16, device="cuda").normal_(generator=g)
    assert _lib.lib().msgl_prefill_launch_count(1, n, keys, hq, hkv, d, n, 0, 1) == 1
    qo, kvp, lens, pre = _i32([0, n]), _i32([0, keys]), _i32([keys]), _i32([keys - n])
    sc = 1 / math.sqrt(d)
    for _ in range(8):
        vc.normal_(generator=g)
        a = paged_prefill_attention(q, kc, vc, qo, kvp, slots, pre, sc, n)
        b = paged_prefill_attention_p16(q, kc, vc, qo, pip, pidx, lens, pre, sc, n, page_size=16)
        assert torch.equal(a, b)
    ref = O.paged_prefill_attention_oracle(q, kc, vc, qo, kvp, slots, pre, sc)
    assert (a.float().cpu() - ref).abs().max() <= 2e-2


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("n,keys,cross", [(200, 250, False), (300, 1000, False), (300, 1024, True)])
def test_a_reference_maximum_that_grows_with_every_tile(n, keys, cross, dtype):
    """At head_dim 128 the two softmax groups of a pair pass every row's reference maximum from tile to tile,
    with the tile's number.  Scores that rise by up to 40 (base 2) a tile, fall, or stay, row by row: a maximum
    of another tile would scale the row's sum and its accumulator differently.  (A key range this short is
    not split, and few items run as pairs.)"""
    from mini_sglang_mlx_b200 import paged_prefill_attention_p16
    hkv, hq, d = 2, 8, 128
    kc, vc, pip, pidx, slots = make_pool([keys], 16, hkv, seed=keys + n, d=d, dtype=dtype)
    g = torch.Generator(device="cuda").manual_seed(n)
    # score of row i and key t, base 2: slope_i * t / 128 plus noise of size 1
    slope = torch.empty(n, hq, device="cuda").uniform_(-40, 40, generator=g)
    unit = math.sqrt(d) / 8 * math.log(2)             # one in q's first column times 8 in K's: one, base 2
    q = torch.empty(n, hq, d, device="cuda").normal_(generator=g)
    q[..., 0] = slope * unit
    kc[slots.long(), :, 0] = (torch.arange(keys, device="cuda") / 16.0).to(dtype)[:, None]
    vc.uniform_(-1, 1, generator=g)
    q = q.to(dtype)
    qo, kvp, lens, pre = _i32([0, n]), _i32([0, keys]), _i32([keys]), _i32([keys - n])
    sc = 1 / math.sqrt(d)
    out = paged_prefill_attention_p16(q, kc, vc, qo, pip, pidx, lens, pre, sc, n, page_size=16,
                                      is_cross_attention=cross)
    ref = O.paged_prefill_attention_oracle(q, kc, vc, qo, kvp, slots, pre, sc, is_cross_attention=cross)
    # |V| <= 1: probabilities and output rounded to 8 bits of mantissa, 2^-9 each; the scores (up to 320) in fp32
    assert (out.float().cpu() - ref).abs().max() <= 2 ** -8 + 1e-3


@pytest.mark.parametrize("d", [128, 256])
@pytest.mark.parametrize("bad", [False, True], ids=["pages", "pages outside the pool"])
def test_a_ring_stage_changes_between_ordinary_and_bulk_copies(d, bad):
    """Decode rings run on across sequences: the stage that held a ragged last page (ordinary copies) is filled
    by TMA next, over and over, and the pool changes from call to call.  The per-token form copies every
    row the ordinary way and runs the same shares, so it gives the same bits; rows of a page outside the
    pool are zeros in both."""
    from mini_sglang_mlx_b200 import paged_decode_attention, paged_decode_attention_p16
    from mini_sglang_mlx_b200.kernel import device_status
    hkv, hq, splits = 2, 8, 4
    kv_lens = [1 + 37 * i % 113 for i in range(300)] + [1999, 4001]
    kc, vc, pip, pidx, slots = make_pool(kv_lens, 16, hkv, seed=d, d=d)
    g = torch.Generator(device="cuda").manual_seed(d)
    if bad:                                           # every third page
        pidx[::3] += kc.shape[0]
        page = torch.repeat_interleave(torch.arange(pidx.numel()).cuda(), 16)
        own = torch.cat([torch.arange(l) + 16 * int(a) for l, a in zip(kv_lens, pip.tolist())]).cuda()
        slots[page[own] % 3 == 0] = -1
    q = torch.empty(len(kv_lens), hq, d, dtype=torch.bfloat16, device="cuda").normal_(generator=g)
    kvp, lens, n = _i32(O.build_indptr(kv_lens).tolist()), _i32(kv_lens), _i32([splits] * len(kv_lens))
    sc = 1 / math.sqrt(d)
    device_status()
    for _ in range(4):
        kc.normal_(generator=g)
        vc.normal_(generator=g)
        a = paged_decode_attention_p16(q, kc, vc, pip, pidx, lens, n, sc, splits, page_size=16)
        b = paged_decode_attention(q, kc, vc, kvp, slots, n, sc, splits)
        assert torch.equal(a, b)
    assert device_status() == (2 if bad else 0)
    if not bad:
        ref = O.paged_decode_attention_oracle(q, kc, vc, kvp, slots, sc)
        assert_close_to_oracle(a, ref, "pages")


@pytest.mark.parametrize("d,hkv,hq,limit", [(256, 2, 32, 11 * 128), (128, 2, 32, 11 * 128), (256, 1, 2, 32 * 128),
                                            (128, 8, 16, 32 * 128)])
@pytest.mark.parametrize("past", [-15, 0, 1, 5000])
@pytest.mark.parametrize("others", [0, 40])
def test_pieces_of_a_long_sequence_beside_short_ones(d, hkv, hq, limit, past, others):
    """A share is 8 groups at least: 11 or 32 pieces of one sequence, one more or less, and many."""
    from mini_sglang_mlx_b200 import paged_decode_attention, paged_decode_attention_p16
    kv_lens = [limit + past] + [1 + i % 3 for i in range(others)]
    kc, vc, pip, pidx, slots = make_pool(kv_lens, 16, hkv, seed=d + 100 + past, d=d)
    g = torch.Generator(device="cuda").manual_seed(limit)
    q = torch.empty(len(kv_lens), hq, d, dtype=torch.bfloat16, device="cuda").normal_(generator=g)
    kvp, lens, n = _i32(O.build_indptr(kv_lens).tolist()), _i32(kv_lens), _i32([1] * len(kv_lens))
    sc = 1 / math.sqrt(d)
    out = paged_decode_attention_p16(q, kc, vc, pip, pidx, lens, n, sc, 1, page_size=16)
    assert_close_to_oracle(out, O.paged_decode_attention_oracle(q, kc, vc, kvp, slots, sc))
    assert torch.equal(paged_decode_attention(q, kc, vc, kvp, slots, n, sc, 1), out)


@pytest.mark.parametrize("d,hkv,hq", [(128, 2, 2), (128, 2, 6), (256, 1, 5), (128, 1, 16), (256, 2, 8)])
@pytest.mark.parametrize("kv_lens", [[128 * k + 5 for k in (1, 2, 7, 8, 9)], [128 * 16], [128 * 17 + 1, 300], [128 * 33],
                                     [200] * 33 + [2100, 0, 2300]], ids=lambda x: f"{len(x)}x{sum(x)}")
def test_a_warp_merges_the_pieces_of_its_heads(d, hkv, hq, kv_lens):
    """A warp per query head, eight or sixteen pieces at a time, whichever CTA arrives last at the head: heads that leave
    warps without one, one to 33 pieces, two partials of a share (a sequence's end and the next one's start), and
    the counters back at zero (a second call gives the same bits)."""
    from mini_sglang_mlx_b200 import paged_decode_attention
    kc, vc, _, _, slots = make_pool([max(l, 1) for l in kv_lens], 16, hkv, seed=hq, d=d)
    slots = torch.cat([s[:l] for s, l in zip(slots.split([max(l, 1) for l in kv_lens]), kv_lens)])
    g = torch.Generator(device="cuda").manual_seed(hq)
    q, gate = (torch.empty(len(kv_lens), hq, d, dtype=torch.bfloat16, device="cuda").normal_(generator=g)
               for _ in range(2))
    kvp, n = _i32(O.build_indptr(kv_lens).tolist()), _i32([1] * len(kv_lens))
    sc = 1 / math.sqrt(d)
    ref = O.paged_decode_attention_oracle(q, kc, vc, kvp, slots, sc)
    out = paged_decode_attention(q, kc, vc, kvp, slots, n, sc, 1)
    assert_close_to_oracle(out, ref)
    assert torch.equal(paged_decode_attention(q, kc, vc, kvp, slots, n, sc, 1), out)
    gated = paged_decode_attention(q, kc, vc, kvp, slots, n, sc, 1, gate=gate)
    assert_close_to_oracle(gated, out.float().cpu() * torch.sigmoid(gate.float()).cpu(), "gate")
