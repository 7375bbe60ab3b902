"""A process's first call may be one that is recorded in a graph, on a stream that orders itself with the legacy one."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
PROGRAM = """
import ctypes as C, os, sys
sys.path.insert(0, os.path.join(sys.argv[1], "chaos-ultra_gb300"))
import torch
import chaos_gb300 as cg
counts = torch.zeros(64 * 48, dtype=torch.int32, device="cuda:0")
torch.cuda.synchronize()
rt = C.CDLL("libcudart.so.13", mode=C.RTLD_GLOBAL)
def ok(rc):
    assert rc == 0, rc
s, graph, run = C.c_void_p(), C.c_void_p(), C.c_void_p()
ok(rt.cudaStreamCreate(C.byref(s)))
ok(rt.cudaStreamBeginCapture(s, 2))  # relaxed
d = cg.FrameDesc(width=64, height=48, max_iterations=60, samples_per_pixel=1, sample_mode=cg.SAMPLES_CENTER,
                 tier=cg.TIER_F32, arith=cg.ARITH_PARITY, fractal=cg.MANDELBROT, seed=0, center_x=-0.5, center_y=0.0,
                 pixel_size=0.05)
cg.render_frame(d, cg.FrameOut(counts=counts.data_ptr()), stream=s.value, sync=False)
ok(rt.cudaStreamEndCapture(s, C.byref(graph)))
ok(rt.cudaGraphInstantiate(C.byref(run), graph, C.c_ulonglong(0)))
ok(rt.cudaGraphLaunch(run, s))
ok(rt.cudaStreamSynchronize(s))
first = counts.clone()
counts.zero_()
cg.render_frame(d, cg.FrameOut(counts=counts.data_ptr()))
assert int(first.max()) == 60 and torch.equal(first, counts)
print("ok")
"""


def test_first_call_captured(cuda, native):
    out = subprocess.run([sys.executable, "-c", PROGRAM, ROOT], capture_output=True, text=True, timeout=300)
    assert out.returncode == 0 and out.stdout.strip() == "ok", out.stderr[-2000:]
