"""The non-allocating bounce filter's first call in a process, inside a stream capture: it is recorded like any other,
and the replayed graph filters what its input holds then. A process of its own for each capture mode, so that
nothing has loaded the kernel before."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

HERE = os.path.dirname(os.path.abspath(__file__))
PROGRAM = """
import ctypes as C, sys
import torch
sys.path.insert(0, sys.argv[1])
import conftest
import dynlight_gb300 as dl
w, h, size = 61, 45, 128
lib = dl.load_library()
src, out = torch.zeros(w * h * 3, device="cuda"), torch.full((w * h * 3,), -1.0, device="cuda")
def call(stream):
    return lib.dl_filter_bounce_window_noalloc(C.c_void_p(src.data_ptr()), C.c_void_p(out.data_ptr()), w, h, 3, 5, size,
                                               C.c_void_p(stream.cuda_stream))
torch.cuda.synchronize()
graph = torch.cuda.CUDAGraph()
with torch.cuda.graph(graph, capture_error_mode=sys.argv[2]):
    status = call(torch.cuda.current_stream())
assert status == 0, lib.dl_last_error()
for seed in (1, 2):
    src.copy_(torch.rand(w * h * 3, generator=torch.Generator().manual_seed(seed)))
    graph.replay()
    torch.cuda.synchronize()
    replayed = out.clone()
    out.fill_(-1.0)
    assert call(torch.cuda.current_stream()) == 0
    torch.cuda.synchronize()
    assert torch.equal(replayed, out) and bool((out >= 0).all()) and bool((out > 0).any())
print("captured")
"""


@pytest.mark.parametrize("mode", ["global", "thread_local", "relaxed"])
def test_the_first_call_may_be_captured(mode):
    pytest.importorskip("torch")
    out = subprocess.run([sys.executable, "-c", PROGRAM, HERE, mode], capture_output=True, text=True, timeout=300,
                         cwd=os.path.dirname(HERE))
    assert out.returncode == 0 and "captured" in out.stdout, out.stdout + out.stderr[-2000:]
