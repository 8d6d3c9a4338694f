"""GPU: a library call that is the first on its device may come while a stream is being captured, its own or
another: it allocates nothing, so it neither fails nor breaks the capture. Each in a fresh process."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SCRIPT = """
import sys, torch
from dadgpt_b200 import attention as dad
path, where = sys.argv[1:]
BH, S, D = 2, 100, 64
dtype = torch.float32 if path == "f32" else torch.bfloat16
q, k, v = (torch.randn(BH, S, D, device="cuda").to(dtype) for _ in range(3))
out, lse, y = torch.zeros_like(q), torch.empty(BH, S, device="cuda"), torch.zeros(4, device="cuda")

def call():
    f = dad.gpu_flash_attention_forward if path == "f32" else dad.gpu_flash_attention_forward_bf16
    f(out, lse, q, k, v, BH, S, D, 0.125)

if path == "decode":
    cache = dad.KVCacheBF16(1, BH, S, D)
    out = torch.zeros(1, BH, D, device="cuda", dtype=dtype)
    q1, k1, v1 = (torch.randn(1, BH, D, device="cuda").to(dtype) for _ in range(3))
    call = lambda: dad.decode_attention_bf16(out, q1, k1, v1, cache, 0.125)
other = torch.cuda.Stream()
torch.cuda.synchronize()
graph = torch.cuda.CUDAGraph()
with torch.cuda.graph(graph, capture_error_mode="global"):
    y.add_(1.0)
    if where == "own":
        call()
    else:
        with torch.cuda.stream(other):
            call()
if where == "own":
    torch.cuda.synchronize()
    assert not out.any()
graph.replay()
torch.cuda.synchronize()
assert y.eq(1.0).all() and out.any() and out.isfinite().all()
assert dad.device_status() == 0
"""


@pytest.mark.parametrize("path,where", [("f32", "other"), ("f32", "own"), ("bf16", "other"), ("decode", "own")])
def test_first_call_during_a_capture(cuda, path, where):
    r = subprocess.run([sys.executable, "-c", SCRIPT, path, where], cwd=ROOT, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-3000:]
