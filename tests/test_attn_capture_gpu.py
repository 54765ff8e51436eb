"""The prompt attention's very first call of a process may be a captured one, although it sets up its status word."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CHILD = """
import ctypes as C, importlib, sys
sys.path.insert(0, sys.argv[1])
import torch
lib = importlib.import_module("s2pro-native_b200.capi").load_library()
q, k, v = (torch.randn(*s, device="cuda").bfloat16() for s in ((40, 4096), (8, 64, 128), (8, 64, 128)))
outs = [torch.zeros_like(q) for _ in range(2)]
def attend(out):
    st = C.c_void_p(torch.cuda.current_stream().cuda_stream)
    assert lib.s2pk_attention(*[C.c_void_p(t.data_ptr()) for t in (q, k, v, out)], 40, 32, 8, 128, 3, 64, st) == 0
torch.cuda.synchronize()
g = torch.cuda.CUDAGraph()
with torch.cuda.graph(g):
    attend(outs[0])
assert not outs[0].any()
g.replay()
attend(outs[1])
torch.cuda.synchronize()
assert outs[1].any() and torch.equal(outs[0].view(torch.int16), outs[1].view(torch.int16))
print("same")
"""


def test_first_call_under_capture():
    r = subprocess.run([sys.executable, "-c", CHILD, ROOT], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and "same" in r.stdout, r.stdout + r.stderr
