"""Calls of several threads on one stream: an attention call can be several launches that hand data over
through the stream's scratch, so each call's launches stay together.

The native host module is built here over CPU tensors: torch's CUDA headers are replaced by a few lines, and
the attention entries of the C ABI by ones that note where a call's launches begin and end."""
import ctypes
import importlib.machinery
import importlib.util
import shutil
import subprocess
import sys
import threading
from pathlib import Path

import pytest
import torch

from mini_sglang_mlx_b200 import build as B

HEADERS = {
    "c10/cuda/CUDAFunctions.h": "#pragma once\nnamespace c10::cuda { inline int current_device() { return -1; } }\n",
    "c10/cuda/CUDAStream.h": """#pragma once
namespace c10::cuda {
struct CUDAStream { long stream() const { return 7; } };
inline CUDAStream getCurrentCUDAStream(int) { return {}; }
}
""",
    # (behind the headers that the module includes: its own tests for a CUDA tensor)
    "on_cpu.h": """#include <Python.h>
#include <ATen/ATen.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>
#include <torch/csrc/utils/object_ptr.h>
#define is_cuda is_cpu
""",
}

# The recorded entries: an argument list of any kind, a begin and an end a millisecond apart, as two launches
# with the host at work between them.
RECORDER = """
#include <unistd.h>
#include <atomic>
#include <cstddef>
#include <cstdint>
namespace {
size_t g_workspace, g_pages;
bool g_have_pages;
std::atomic<int> g_next{0}, g_at{0};
int g_log[4096];
int note() {
  const int call = ++g_next;
  g_log[g_at++ % 4096] = call;
  usleep(1000);
  g_log[g_at++ % 4096] = -call;
  return 0;
}
}
extern "C" {
int recorded(int i) { return i < g_at ? g_log[i] : 0; }
#define ENTRY(name) int name() { return note(); }
ENTRY(msgl_paged_decode_attention_sized)
ENTRY(msgl_paged_decode_attention_p16)
ENTRY(msgl_paged_prefill_attention)
ENTRY(msgl_paged_prefill_attention_gated)
ENTRY(msgl_paged_prefill_attention_p16)
ENTRY(msgl_decode_layer)
// 5 MB of pages for every call of more than 100 query tokens
size_t msgl_prefill_kv_pages_bytes(int, int total_q, int64_t, int, int, int, int, int) {
  return total_q > 100 ? 5000000 : 0;
}
int msgl_prefill_layer_pages(const void*, void*, void*, void*, const void*, const void*, const void*, const void*,
                             const void*, const void*, void*, void*, size_t workspace, void* pages, size_t bytes) {
  g_workspace = workspace;
  g_have_pages = pages != nullptr;
  g_pages = bytes;
  return note();
}
size_t last_workspace() { return g_workspace; }
size_t last_pages() { return g_have_pages ? g_pages : 0; }
}
"""


@pytest.fixture(scope="module")
def host(tmp_path_factory):
    """(module, its recorder)"""
    at = tmp_path_factory.mktemp("host")
    for name, text in {**HEADERS, "recorder.cpp": RECORDER}.items():
        (at / name).parent.mkdir(parents=True, exist_ok=True)
        (at / name).write_text(text)
    lib = at / "_host.so"
    B.build()
    cmd = B._host_command()
    cmd[cmd.index("-O2")] = "-O0"
    first = next(i for i, a in enumerate(cmd) if a.startswith("-I"))
    cmd[first:first] = [f"-I{at}", "-include", str(at / "on_cpu.h")]
    entries = at / "recorder.o"
    subprocess.run([shutil.which("g++") or "g++", "-std=c++17", "-fPIC", "-c", str(at / "recorder.cpp"), "-o",
                    str(entries)], check=True)
    subprocess.run([*cmd, str(entries), "-Wl,-Bsymbolic", f"-Wl,-rpath,{B.PKG_DIR}", "-o", str(lib)], check=True)
    loader = importlib.machinery.ExtensionFileLoader("_host", str(lib))
    module = importlib.util.module_from_spec(importlib.util.spec_from_loader("_host", loader))
    loader.exec_module(module)
    recorder = ctypes.CDLL(str(lib))
    recorder.last_workspace.restype = recorder.last_pages.restype = ctypes.c_size_t
    return module, recorder


def _calls(m):
    q, kc, k = torch.zeros(1, 2, 128).bfloat16(), torch.zeros(64, 1, 128).bfloat16(), torch.zeros(1, 1, 128).bfloat16()
    two, one = torch.zeros(2, dtype=torch.int32), torch.zeros(1, dtype=torch.int32)
    return {
        "decode": lambda: m.decode(q, kc, kc, two, two, one, 0.1, 32, None, 7),
        "decode_paged": lambda: m.decode_paged(q, kc, kc, two, one, one, one, 0.1, 32, 5, None, 7),
        "prefill": lambda: m.prefill(q, kc, kc, two, two, two, one, 0.1, 1, False, 0, None, 7),
        "prefill gated": lambda: m.prefill(q, kc, kc, two, two, two, one, 0.1, 1, False, 0, q, 7),
        "prefill_paged": lambda: m.prefill_paged(q, kc, kc, two, two, one, one, one, 0.1, 1, 5, False, 0, None, 7),
        "decode_layer": lambda: m.decode_layer(q, k, k, kc, kc, one, None, two, two, None, 0.1, 32, 1, None),
        "prefill_layer": lambda: m.prefill_layer(q, k, k, kc, kc, one, None, two, two, two, None, one, 0.1, 1, 1, False,
                                                 0, None),
    }


def test_calls_on_one_stream_queue_their_launches_in_turn(host):
    m, log = host
    m.set_workspace_maker(lambda nbytes, index, stream, kind: torch.zeros(nbytes, dtype=torch.uint8))
    calls = list(_calls(m).values())
    assert all(isinstance(call(), torch.Tensor) for call in calls)
    fails = []

    def work(i):
        try:
            for n in range(6):
                assert calls[(i + n) % len(calls)]() is not None
        except Exception as e:          # noqa: BLE001 - reported by the test's own thread
            fails.append(e)

    before = sys.getswitchinterval()
    sys.setswitchinterval(1e-5)
    try:
        threads = [threading.Thread(target=work, args=(i,)) for i in range(7)]
        for t in threads:
            t.start()
        for t in threads:
            t.join()
    finally:
        sys.setswitchinterval(before)
    assert not fails, fails
    n = len(calls) + 7 * 6
    seen = [log.recorded(i) for i in range(2 * n)]
    assert sorted(seen) == sorted([*range(1, n + 1), *range(-n, 0)])
    assert all(seen[i] > 0 and seen[i + 1] == -seen[i] for i in range(0, 2 * n, 2)), seen


@pytest.mark.parametrize("layer", [False, True], ids=["operator", "layer"])
def test_a_long_prefill_goes_without_page_memory_that_nobody_has(host, monkeypatch, layer):
    """The rows' pages are memory of the call's own: the scratch that stays is the least one, and where the
    pages find no memory the call runs without them (and the next ones do not ask again)."""
    from mini_sglang_mlx_b200 import kernel as K
    m, log = host
    asked, kept = [], []

    def workspace(nbytes, index, stream, kind):
        kept.append(nbytes)
        return torch.zeros(nbytes, dtype=torch.uint8)

    m.set_workspace_maker(workspace)
    n = 200
    q, kc, k = torch.zeros(n, 2, 128).bfloat16(), torch.zeros(64, 1, 128).bfloat16(), torch.zeros(1, 1, 128).bfloat16()
    two, one = torch.zeros(2, dtype=torch.int32), torch.zeros(1, dtype=torch.int32)

    def call():
        if layer:
            return m.prefill_layer(q, k, k, kc, kc, one, None, two, two, two, None, one, 0.1, n, 1, False, 0, None)
        return m.prefill(q, kc, kc, two, two, two, one, 0.1, n, False, 0, None, 7)

    m.set_pages_maker(lambda nbytes, index, stream: asked.append(nbytes) or torch.empty(nbytes, dtype=torch.uint8))
    assert isinstance(call(), torch.Tensor) and asked == [5000000] and log.last_pages() == 5000000
    assert sum(kept) < 1000000 and log.last_workspace() < 1000000

    def none_left(*a, **kw):
        asked.append(a)
        raise torch.OutOfMemoryError("no memory")

    monkeypatch.setattr(torch, "empty", none_left)
    monkeypatch.setattr(K, "_stream_handle", lambda stream, device: 7)
    monkeypatch.setattr(torch.cuda, "is_current_stream_capturing", lambda: False)
    monkeypatch.setattr(K, "_pages_pause", {})
    m.set_pages_maker(lambda nbytes, index, stream: K._make_pages(nbytes, 0, stream))
    asked.clear()
    for _ in range(K._PAGES_PAUSE + 1):
        assert K._make_pages(100, 0, 7) is None
    assert len(asked) == 1
    for asks in (2, 2):
        assert isinstance(call(), torch.Tensor) and len(asked) == asks and log.last_pages() == 0


def test_calls_on_other_streams_do_not_wait(host):
    """Two streams: the second call begins before the first has ended."""
    m, log = host
    m.set_workspace_maker(lambda nbytes, index, stream, kind: torch.zeros(nbytes, dtype=torch.uint8))
    q, kc = torch.zeros(1, 2, 128).bfloat16(), torch.zeros(64, 1, 128).bfloat16()
    two, one = torch.zeros(2, dtype=torch.int32), torch.zeros(1, dtype=torch.int32)
    meet = threading.Barrier(2)

    def work(stream):
        for _ in range(20):
            meet.wait()
            m.decode(q, kc, kc, two, two, one, 0.1, 32, None, stream)

    first = next(i for i in range(4096) if log.recorded(i) == 0)
    threads = [threading.Thread(target=work, args=(s,)) for s in (11, 12)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    seen = [log.recorded(first + i) for i in range(80)]
    assert any(a > 0 and b > 0 for a, b in zip(seen, seen[1:]))
