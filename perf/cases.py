"""The attention work of a serving engine, as cases to time and to compare.

A case is one engine step of a slice of a model's layers: the step's index arrays are built from
the requests and the page table (``AttnBackend.prepare_metadata`` / ``build_prefill_metadata``),
then every layer hands its projections over to the attention backend, which puts the new K/V
rows into the pool and attends.  ``layer`` says how a layer does that:

* ``"projections"``: ``forward_from_projections`` (q/k RMSNorm, rotary embedding and K/V store in
  one pass, then attention), the call of a layer with q/k norms;
* ``"forward"``: ``forward`` (K/V store, then attention), the call of a layer that has rotated its
  own q and k.

Each layer has its own pool, so a step of several layers walks memory as a model does.  The
request lengths of a case come from its ``lens`` number, so that its work does not depend on the
seed; page ids, q, k, v, gates, norm weights and the pool's contents do.
"""
import math
import random
from types import SimpleNamespace

import torch

from mini_sglang_mlx_b200.attention import AttnBackend
from mini_sglang_mlx_b200.core import Batch, BatchPhase, Req
from mini_sglang_mlx_b200.kvcache import MHAKVCache

DTYPES = {"bf16": torch.bfloat16, "f16": torch.float16}

# No drawn case costs more than the largest listed ones (bytes that must move, operations).
MAX_BYTES = 9.0e9
MAX_FLOPS = 2.3e12


def _case(name=None, *, kind, layer="projections", layers=1, hq=32, hkv=8, head_dim=128, rotary=0,
          gate=False, dtype="bf16", page_size=16, batch=1, lens=1, kv_lo=0, kv_hi=0, q_lo=1, q_hi=1,
          window=0, cross=False):
    """``kind``: decode | prefill | verify.  ``kv_lo`` .. ``kv_hi``: tokens a request has cached
    before the step, ``q_lo`` .. ``q_hi``: its new tokens (decode: one).  ``rotary`` 0 = the whole
    head."""
    c = dict(kind=kind, layer=layer, layers=layers, hq=hq, hkv=hkv, head_dim=head_dim, rotary=rotary,
             gate=gate, dtype=dtype, page_size=page_size, batch=batch, lens=lens, kv_lo=kv_lo,
             kv_hi=kv_hi, q_lo=q_lo, q_hi=q_hi, window=window, cross=cross)
    return c if name is None else dict(name=name, **c)


def listed():
    return [
        # One user chatting with a small model: the smallest call there is, all latency and launches.
        _case("decode_one_request", kind="decode", layers=8, hq=16, hkv=8, kv_lo=700, kv_hi=700),
        # A lightly loaded server with a small model, layers that rotate q and k themselves.
        _case("decode_small_batch", kind="decode", layer="forward", layers=8, hq=16, hkv=8, batch=8,
              lens=101, kv_lo=256, kv_hi=2048),
        # A busy server whose pool has one token per page (per-token slot ids), f16 weights, ragged.
        _case("decode_token_slots", kind="decode", layers=2, dtype="f16", page_size=1, batch=37, lens=7,
              kv_lo=100, kv_hi=6000),
        # Long-context continuous batching: the largest decode, everything is K/V traffic.
        _case("decode_long_context", kind="decode", layer="forward", batch=64, lens=505, kv_lo=4096,
              kv_hi=131072),
        # Gated attention layers with 256-wide heads and a quarter of the head rotated.
        _case("decode_gated_d256", kind="decode", layers=2, hq=16, hkv=2, head_dim=256, rotary=64,
              gate=True, batch=19, lens=11, kv_lo=512, kv_hi=16384),
        # A few short new prompts on an idle server: ragged, nothing cached, per-token slot ids.
        _case("prefill_short_prompts", kind="prefill", layer="forward", layers=8, hq=16, hkv=8,
              page_size=1, batch=6, lens=3, q_lo=17, q_hi=300),
        # Chunked prefill over cached prefixes: the ordinary prefill step.
        _case("prefill_chunked", kind="prefill", layers=2, batch=4, lens=202, kv_hi=4096, q_lo=512,
              q_hi=512),
        # Ragged prompts with ragged prefixes in a pool of per-token slots, f16.
        _case("prefill_token_slots", kind="prefill", layers=2, hq=32, hkv=4, dtype="f16", page_size=1,
              batch=3, lens=5, kv_hi=8000, q_lo=300, q_hi=2000),
        # A chunk of a very long document: the largest prefill, everything is tensor-core work.
        _case("prefill_long_document", kind="prefill", lens=606, kv_lo=32768, kv_hi=32768, q_lo=4096,
              q_hi=4096),
        # Prompts through the gated 256-wide layers.
        _case("prefill_gated_d256", kind="prefill", layers=2, hq=24, hkv=4, head_dim=256, rotary=64,
              gate=True, batch=2, lens=17, kv_hi=1000, q_lo=900, q_hi=2100),
        # A draft layer's block of 16 tokens under a sliding window.
        _case("draft_window_block", kind="prefill", layer="forward", layers=2, batch=16, lens=303,
              kv_lo=8176, kv_hi=8176, q_lo=16, q_hi=16, window=4096),
        # Speculative verification: 8 tokens per request over contexts of very different lengths.
        _case("verify_eight_tokens", kind="verify", layers=2, hkv=4, batch=32, lens=404, kv_lo=1024,
              kv_hi=32768, q_lo=8, q_hi=8),
    ]


def _log(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


HEADS_128 = ((16, 8), (32, 8), (32, 4))
HEADS_256 = ((16, 2), (16, 4), (24, 4), (32, 2))


def draw(rng):
    """A decode step (1 to 128 requests), a prefill step (17 to 4096 new tokens a request), a draft
    layer's window block or a verify step, over the head layouts, types and page sizes above."""
    while True:
        kind = rng.choice(("decode", "decode", "prefill", "prefill", "block", "verify"))
        wide = kind in ("decode", "prefill") and rng.random() < 0.3
        hq, hkv = rng.choice(HEADS_256 if wide else HEADS_128)
        c = dict(layer=rng.choice(("projections", "forward")), layers=rng.choice((1, 2, 4, 8)), hq=hq,
                 hkv=hkv, head_dim=256 if wide else 128, rotary=64 if wide else 0, gate=wide,
                 dtype=rng.choice(("bf16", "bf16", "f16")), page_size=rng.choice((16, 16, 1)),
                 lens=rng.randrange(1, 1 << 20))
        if kind == "decode":
            lo = _log(rng, 64, 32768)
            c.update(kind="decode", batch=_log(rng, 1, 128), kv_lo=lo, kv_hi=_log(rng, lo, 131072))
        elif kind == "prefill":
            q_lo = _log(rng, 17, 2048)
            c.update(kind="prefill", batch=_log(rng, 1, 12), kv_hi=rng.choice((0, 1)) * _log(rng, 64, 32768),
                     q_lo=q_lo, q_hi=_log(rng, q_lo, 4096))
        elif kind == "block":
            kv = _log(rng, 1000, 16384)
            c.update(kind="prefill", batch=_log(rng, 4, 48), kv_lo=kv // 2, kv_hi=kv, q_lo=16, q_hi=16,
                     window=_log(rng, 512, 8192), cross=rng.random() < 0.5)
        else:
            k = rng.randrange(2, 13)
            lo = _log(rng, 256, 8192)
            c.update(kind="verify", batch=_log(rng, 2, 64), kv_lo=lo, kv_hi=_log(rng, lo, 32768), q_lo=k,
                     q_hi=k)
        c = _case(**c)
        w = work(c)
        if w["bytes"] <= MAX_BYTES and w["flops"] <= MAX_FLOPS:
            return c


def _lengths(case):
    """(cached, new) tokens of every request."""
    rng = random.Random(case["lens"])

    def span(lo, hi):
        if lo > 0 and hi > 10 * lo:
            return _log(rng, lo, hi)
        return rng.randint(lo, hi)

    return [(span(case["kv_lo"], case["kv_hi"]), 1 if case["kind"] == "decode" else
             span(case["q_lo"], case["q_hi"])) for _ in range(case["batch"])]


def work(case):
    """Each visible K/V row of the pool is read once per layer, each q, k, v (and gate) once; the
    output, the new pool rows and the normalised, rotated q are written once; 4 D flops per query
    head and visible key."""
    hq, hkv, d, w, ps = case["hq"], case["hkv"], case["head_dim"], case["window"], case["page_size"]
    new = visible = pairs = ids = 0
    for cached, q in _lengths(case):
        total = cached + q
        first = max(0, cached - w + 1) if w > 0 else 0
        new += q
        visible += total - first
        ids += -(-total // ps)
        if case["cross"]:
            pairs += sum(total - max(0, cached + p - w + 1) for p in range(q)) if w > 0 else q * total
        elif w > 0:
            pairs += sum(min(w, cached + p + 1) for p in range(q))
        else:
            pairs += q * cached + q * (q + 1) // 2
    q_rows = 2 + (case["layer"] == "projections") + case["gate"]
    per_layer = 2 * d * (2 * hkv * (visible + new) + q_rows * hq * new)
    return {"bytes": case["layers"] * per_layer + 4 * ids, "flops": case["layers"] * 4.0 * d * hq * pairs}


def tolerance(case):
    """Outputs are rounded to 16 bits, and the probabilities on their way into the second
    contraction are, too."""
    return {"rel": 1e-2 if case["dtype"] == "bf16" else 2e-3}


def prepare(case, seed):
    dev = torch.device("cuda")
    gen = torch.Generator(device=dev).manual_seed(seed)
    dtype, ps, d, hq, hkv = DTYPES[case["dtype"]], case["page_size"], case["head_dim"], case["hq"], case["hkv"]
    lengths = _lengths(case)
    pages = [-(-(cached + q) // ps) for cached, q in lengths]
    num_pages = sum(pages) + sum(pages) // 16 + 8      # a pool that is nearly full
    num_slots = num_pages * ps

    # every request's pages, drawn from all over the pool, as rows of per-token slots
    perm = torch.randperm(num_pages, generator=gen, device=dev).to(torch.int32)
    table = torch.zeros(case["batch"] + 2, max(pages) * ps, dtype=torch.int32, device=dev)
    offs, at, locs, reqs = torch.arange(ps, dtype=torch.int32, device=dev), 0, [], []
    for b, ((cached, q), n) in enumerate(zip(lengths, pages)):
        table[b, : n * ps] = (perm[at:at + n, None] * ps + offs).reshape(-1)
        locs.append(table[b, cached:cached + q])
        reqs.append(Req(table_idx=b, cached_len=cached, device_len=cached + q))
        at += n

    def rand(*shape):
        return torch.empty(*shape, dtype=dtype, device=dev).normal_(generator=gen)

    pool = MHAKVCache(hkv, case["layers"], d, num_slots, dtype, device=dev)
    n = sum(q for _, q in lengths)
    layers = []
    for i in range(case["layers"]):
        pool.k_cache(i).normal_(generator=gen)
        pool.v_cache(i).normal_(generator=gen)
        layers.append(SimpleNamespace(
            q=rand(n, hq, d), k=rand(n, hkv, d), v=rand(n, hkv, d),
            gate=rand(n, hq, d) if case["gate"] else None,
            # q is normalised in place: weights of +-1 leave its size alone, however often it runs
            q_norm=torch.where(rand(d) > 0, 1.0, -1.0).to(dtype), k_norm=1 + 0.1 * rand(d)))
    backend = AttnBackend(SimpleNamespace(head_dim=d, num_kv_heads=hkv), pool, table, page_size=ps)
    phase = {"decode": BatchPhase.DECODE, "prefill": BatchPhase.PREFILL,
             "verify": BatchPhase.TARGET_VERIFY}[case["kind"]]
    batch = Batch(reqs=reqs, phase=phase, out_loc=torch.cat(locs).contiguous())
    return SimpleNamespace(case=case, backend=backend, pool=pool, batch=batch, layers=layers,
                           rotary=case["rotary"] or None)


def run(state):
    case, backend, batch = state.case, state.backend, state.batch
    if case["kind"] == "verify":      # the virtual extend window of a verify step
        batch.attn_metadata = backend.build_prefill_metadata(
            batch.reqs, extend_lens=[r.device_len - r.cached_len for r in batch.reqs],
            kv_lens=[r.device_len for r in batch.reqs])
    else:
        backend.prepare_metadata(batch)
    mask = {}
    if case["window"] or case["cross"]:
        mask = dict(sliding_window_size=case["window"], is_cross_attention=case["cross"])
    outs = []
    if case["layer"] == "projections":
        for i, layer in enumerate(state.layers):
            outs.append(backend.forward_from_projections(
                layer.q, layer.k, layer.v, i, batch, q_norm_weight=layer.q_norm,
                k_norm_weight=layer.k_norm, rope_base=1.0e6, rotary_dim=state.rotary, gate=layer.gate, **mask))
    else:
        for i, layer in enumerate(state.layers):
            outs.append(backend.forward(layer.q, layer.k, layer.v, i, batch, gate=layer.gate, **mask))
    n = len(outs)
    return {"out": outs, "q": [layer.q for layer in state.layers],
            "k_pool": [state.pool.k_cache(i) for i in range(n)],
            "v_pool": [state.pool.v_cache(i) for i in range(n)]}
