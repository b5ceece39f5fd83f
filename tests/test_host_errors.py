"""Errors that the native host module meets reach the caller as Python exceptions: the process goes
on, and a call that found no memory can be made again."""
import subprocess
import sys
from pathlib import Path

import pytest
import torch

from tests.helpers import assert_close_to_oracle

ROOT = Path(__file__).resolve().parent.parent

# Tensors of a CUDA device without a CUDA device behind them: what the module asks of CUDA or of their
# memory throws in C++.
FAKE_CALLS = """
import torch
from torch._subclasses.fake_tensor import FakeTensorMode
from mini_sglang_mlx_b200 import _lib
from mini_sglang_mlx_b200 import kernel as K
with FakeTensorMode():
    def new(*shape, dtype=torch.bfloat16):
        return torch.empty(*shape, dtype=dtype, device="cuda:0")
    q, kc, k = new(1, 2, 128), new(4, 1, 128), new(1, 1, 128)
    two, one = new(2, dtype=torch.int32), new(1, dtype=torch.int32)
    table = new(4, 64, dtype=torch.int32)
calls = [
    lambda: K.paged_decode_attention(q, kc, kc, two, two, one, 0.1, 32),
    lambda: K.paged_prefill_attention(q, kc, kc, two, two, two, one, 0.1, 1),
    lambda: K.paged_decode_attention_p16(q, kc, kc, two, one, one, one, 0.1, 32),
    lambda: K.paged_prefill_attention_p16(q, kc, kc, two, two, one, one, one, 0.1, 1),
    lambda: K.store_kv_cache(kc, kc, one, k, k),
    lambda: K.qk_norm_rope_store(q, k, k, None, None, one, one, kc, kc, rope_base=1e6),
    lambda: K._ops.decode_layer(q, k, k, kc, kc, one, None, two, two, None, 0.1, 32, 1, None),
    lambda: K._ops.prefill_layer(q, k, k, kc, kc, one, None, two, two, two, None, one, 0.1, 1, 1, False, 0, None),
    lambda: K._ops.index_arrays(bytes(12), table, 0, 0, 0, 1, 0, 32, True, None),
]
for call in calls:
    try:
        call()
    except RuntimeError:
        print("raised", flush=True)
"""


def test_what_cpp_throws_is_raised_and_does_not_end_the_process():
    proc = subprocess.run([sys.executable, "-c", FAKE_CALLS], cwd=ROOT, capture_output=True, text=True, timeout=300)
    assert proc.returncode == 0, proc.stderr[-2000:]
    assert proc.stdout.split() == ["raised"] * 9


@pytest.mark.gpu
@pytest.mark.parametrize("layer", [False, True], ids=["operator", "layer"])
def test_a_call_without_memory_raises_and_can_be_made_again(layer):
    from mini_sglang_mlx_b200 import kernel as K
    from oracle import paged_attention_oracle as O
    torch.cuda.set_device(0)
    dev, n, hq, hkv, d = torch.device("cuda:0"), 4096, 32, 8, 128     # 32 MB of q, as much of output
    gen = torch.Generator(device=dev).manual_seed(3)
    q = torch.randn(n, hq, d, generator=gen, device=dev).bfloat16()
    kc = torch.randn(64, hkv, d, generator=gen, device=dev).bfloat16()
    vc = torch.randn(64, hkv, d, generator=gen, device=dev).bfloat16()
    qo = torch.tensor([0, n], dtype=torch.int32, device=dev)
    kv = torch.tensor([0, 64], dtype=torch.int32, device=dev)
    ids = torch.arange(64, dtype=torch.int32, device=dev)
    prefix = torch.tensor([0], dtype=torch.int32, device=dev)
    rows = ids[:1].clone()
    k, v = kc[:1].clone(), vc[:1].clone()      # (what is stored is what the pool holds)
    scale = d ** -0.5

    def call():
        if layer:
            return K._ops.prefill_layer(q, k, v, kc, vc, rows, None, qo, kv, ids, None, prefix, scale, n, 1, True, 0,
                                        None)
        return K.paged_prefill_attention(q, kc, vc, qo, kv, ids, prefix, scale, n, is_cross_attention=True)

    call()                                     # (the scratch is there)
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    total = torch.cuda.get_device_properties(0).total_memory
    try:
        torch.cuda.set_per_process_memory_fraction((torch.cuda.memory_reserved() + (1 << 20)) / total)
        hold = []                              # free places inside the blocks that torch keeps
        with pytest.raises(torch.OutOfMemoryError):
            for _ in range(64):
                hold.append(call())
        with pytest.raises(torch.OutOfMemoryError):
            call()
        hold.clear()
    finally:
        torch.cuda.set_per_process_memory_fraction(1.0)
    out = call()
    ref = O.paged_prefill_attention_oracle(q, kc, vc, qo, kv, ids, prefix, scale, is_cross_attention=True)
    assert_close_to_oracle(out, ref, "after the memory came back")
