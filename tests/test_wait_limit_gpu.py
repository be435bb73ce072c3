"""A bounded wait that runs out is reported: by the error check of a later call, once, whatever the thread."""
import ctypes as C
import os
import subprocess
import sys
import threading

import pytest
import torch

import candle_vllm_b200 as pkg
from candle_vllm_b200 import _lib

pytestmark = pytest.mark.gpu


def test_a_wait_that_runs_out_is_reported_once():
    L = pkg.lib()
    L.b200_wait_limit_check(C.c_int32(2000), C.c_int64(torch.cuda.current_stream().cuda_stream))
    torch.cuda.synchronize()
    with pytest.raises(pkg.BackendError, match="gave up a wait"):
        _lib.check("any call")
    _lib.check("the next one")
    x = torch.ones(4, 256, device="cuda")
    assert torch.isfinite(pkg.silu_mul(x, x)).all()           # the context is usable


def test_another_thread_sees_it():
    L = pkg.lib()
    L.b200_wait_limit_check(C.c_int32(500), C.c_int64(torch.cuda.current_stream().cuda_stream))
    torch.cuda.synchronize()
    codes = []
    t = threading.Thread(target=lambda: codes.append(L.b200_last_error()))
    t.start()
    t.join()
    assert codes[0] != 0 and L.b200_last_error() == 0


def test_limits_are_checked():
    L = pkg.lib()
    for us in (0, -1, 1000001):
        L.b200_wait_limit_check(C.c_int32(us), C.c_int64(0))
        assert L.b200_last_error() == 1


_FIRST_USE = """
import torch
import candle_vllm_b200 as pkg
x, w = torch.randn(4096, 512, device="cuda").bfloat16(), torch.randn(4096, 512, device="cuda").bfloat16()
op = pkg.Linear(w, None)
out = []
g = torch.cuda.CUDAGraph()
with torch.cuda.graph(g):
    out.append(op.forward(x))                 # the two-SM GEMM: the word is asked for here, in the capture
g.replay()
torch.cuda.synchronize()
ref = x.double() @ w.double().T
assert float((out[0].double() - ref).norm() / ref.norm()) < 2.0 ** -8
pkg.lib().b200_wait_limit_check(__import__("ctypes").c_int32(500), __import__("ctypes").c_int64(0))
torch.cuda.synchronize()
assert pkg.lib().b200_last_error() != 0
print("fine")
"""


def test_the_word_can_be_asked_for_during_a_capture():
    """a process whose first kernel with bounded waits is launched into a graph"""
    r = subprocess.run([sys.executable, "-c", _FIRST_USE], cwd=os.path.dirname(os.path.dirname(os.path.abspath(__file__))), capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and "fine" in r.stdout, r.stderr[-2000:]
