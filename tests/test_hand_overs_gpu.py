"""Hand-overs between threads and CTAs inside a kernel: inputs on which data that comes too late, or a
value that is paired with another's tag, changes the result."""
import math

import pytest
import torch

from oracle import paged_attention_oracle as O
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
