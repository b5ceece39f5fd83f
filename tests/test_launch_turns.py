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
#include <cstdint>
namespace {
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
ENTRY(msgl_prefill_layer)
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
    recorder = at / "recorder.o"
    subprocess.run([shutil.which("g++") or "g++", "-std=c++17", "-fPIC", "-c", str(at / "recorder.cpp"), "-o",
                    str(recorder)], check=True)
    subprocess.run([*cmd, str(recorder), "-Wl,-Bsymbolic", f"-Wl,-rpath,{B.PKG_DIR}", "-o", str(lib)], check=True)
    loader = importlib.machinery.ExtensionFileLoader("_host", str(lib))
    module = importlib.util.module_from_spec(importlib.util.spec_from_loader("_host", loader))
    loader.exec_module(module)
    return module, ctypes.CDLL(str(lib))


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
