"""The allocation-free Gram product in a captured CUDA graph: after one call on the device of
any size, every size can be captured and replayed on new data (its kernels for both tile
orders, for even and odd K, are loaded by the first call).  In a process of its own, whose
first call is the one below."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PROGRAM = """
import ctypes, sys
sys.path.insert(0, {pkg!r})
import torch
from sdpx_b200.cuda_backend import load_library
lib = load_library()

def gram(P, S, stream):
    rc = lib.sdpx_b200_gram_noalloc(ctypes.c_void_p(P.data_ptr()), ctypes.c_int64(P.shape[1]),
                                    ctypes.c_int32(P.shape[0]), ctypes.c_void_p(S.data_ptr()),
                                    ctypes.c_void_p(stream.cuda_stream))
    assert rc == 0, lib.sdpx_b200_gram_noalloc_error()

def buffers(m, K):
    return (torch.randn(m, K, dtype=torch.float64, device="cuda"),
            torch.zeros(m, m, dtype=torch.float64, device="cuda"))

lib.sdpx_b200_gram_noalloc_error.restype = ctypes.c_char_p
P, S = buffers({m0}, {k0})
gram(P, S, torch.cuda.current_stream())
torch.cuda.synchronize()
for m, K in ((61, 333), (61, 334), (1000, 3000), (1000, 3001), (2048, 500)):
    P, S = buffers(m, K)
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        gram(P, S, torch.cuda.current_stream())
    for _ in range(2):
        P.copy_(torch.randn(m, K, dtype=torch.float64, device="cuda"))
        g.replay()
        torch.cuda.synchronize()
        assert torch.allclose(S, P @ P.T, rtol=0, atol=1e-12 * K), (m, K)
print("captured")
"""


def test_capture_after_one_call():
    code = PROGRAM.format(pkg=os.path.join(ROOT, "sdpx.jl_b200"), m0=24, k0=72)
    out = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, timeout=300)
    assert out.returncode == 0 and "captured" in out.stdout, out.stdout + out.stderr
