"""Work-counter slots: a slot goes out again only when the launch that had it has ended, however many launches follow."""
import os
import shutil
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "chaos-ultra_gb300", "csrc")
SLOTS = 4096  # kCounterSlots


def test_slot_ring(tmp_path):
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("no g++")
    exe = str(tmp_path / "slots_check")
    subprocess.run([gxx, "-O2", "-std=c++17", "-pthread", "-I", CSRC, "-o", exe,
                    os.path.join(ROOT, "tests", "slots_check.cpp")], check=True)
    out = subprocess.run([exe], capture_output=True, text=True, timeout=60)
    assert out.returncode == 0 and out.stdout.strip() == "ok", out.stdout


# c = -1.9 on the real axis: the orbit is chaotic and bounded, so one binary64 pixel runs to the limit in one warp
LONG_ITER = 3_000_000


def frame(cg, w, h, tier, max_iter, center=(-0.5, 0.0), pixel_size=0.04, limit=0.0):
    return cg.FrameDesc(width=w, height=h, max_iterations=max_iter, samples_per_pixel=1, sample_mode=cg.SAMPLES_CENTER,
                        tier=tier, arith=cg.ARITH_PARITY, fractal=cg.MANDELBROT, seed=0, center_x=center[0],
                        center_y=center[1], pixel_size=pixel_size, time_limit_s=limit)


@pytest.mark.gpu
def test_launches_beside_a_long_one(cuda, native, oracle):
    """One frame that runs while the ring comes round, then a whole ring of frames: every one complete."""
    import chaos_gb300 as cg
    torch = cuda
    long_s, short_s = torch.cuda.Stream(), torch.cuda.Stream()
    w, h, mi = 70, 50, 60
    kinds = [(cg.TIER_F32, False), (cg.TIER_F64, True)]
    want = [oracle.frame(w, h, mi, 1, 0, wide, cg.ARITH_PARITY, cg.MANDELBROT, 0, (-0.5, 0.0), 0.04) for _, wide in kinds]
    want = [(torch.from_numpy(o["counts"].reshape(-1).view(np.int32).copy()).to("cuda:0"), int(o["total"])) for o in want]
    counts = torch.zeros((SLOTS + 64, w * h), dtype=torch.int32, device="cuda:0")
    totals = torch.zeros(SLOTS + 64, dtype=torch.int64, device="cuda:0")
    lc = torch.zeros(1, dtype=torch.int32, device="cuda:0")
    lt = torch.zeros(1, dtype=torch.int64, device="cuda:0")
    lstatus = torch.zeros(1, dtype=torch.int32, device="cuda:0")
    torch.cuda.synchronize()

    def check():
        torch.cuda.synchronize()
        for k in range(2):
            assert bool((counts[k::2] == want[k][0]).all()), k
            assert bool((totals[k::2] == want[k][1]).all()), k
        counts.zero_()
        totals.zero_()
        torch.cuda.synchronize()

    def ring():
        for k in range(SLOTS + 64):
            cg.render_frame(frame(cg, w, h, kinds[k % 2][0], mi),
                            cg.FrameOut(counts=counts[k].data_ptr(), total_iterations=totals[k:].data_ptr()),
                            stream=short_s, sync=False)

    for k in range(2):  # (a kernel's first launch may wait for the GPU)
        cg.render_frame(frame(cg, w, h, kinds[k][0], mi), cg.FrameOut(counts=counts[k].data_ptr()))
    cg.render_frame(frame(cg, 1, 1, cg.TIER_F64, LONG_ITER, (-1.9, 0.0), 1e-9, limit=20.0),
                    cg.FrameOut(counts=lc.data_ptr(), total_iterations=lt.data_ptr(), status=lstatus.data_ptr()),
                    stream=long_s, sync=False)
    ring()
    short_s.synchronize()
    assert not long_s.query()  # (else the ring did not come round beside it)
    check()
    assert int(lstatus.item()) == 0 and int(lc.item()) == LONG_ITER and int(lt.item()) == LONG_ITER
    ring()
    check()


@pytest.mark.gpu
def test_captured_launches(cuda, native, oracle):
    """A graph's launches keep their counters: replayed after and beside more launches than the ring has slots."""
    import chaos_gb300 as cg
    torch = cuda
    w, h, mi = 70, 50, 60
    o = oracle.frame(w, h, mi, 1, 0, False, cg.ARITH_PARITY, cg.MANDELBROT, 0, (-0.5, 0.0), 0.04)
    want = torch.from_numpy(o["counts"].reshape(-1).view(np.int32).copy()).to("cuda:0")
    a, b, c = (torch.zeros(w * h, dtype=torch.int32, device="cuda:0") for _ in range(3))
    d = frame(cg, w, h, cg.TIER_F32, mi)
    cg.render_frame(d, cg.FrameOut(counts=a.data_ptr()))
    side = torch.cuda.Stream()
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        s = torch.cuda.current_stream()
        cg.render_frame(d, cg.FrameOut(counts=a.data_ptr()), stream=s, sync=False)
        cg.render_frame(d, cg.FrameOut(counts=b.data_ptr()), stream=s, sync=False)
    for k in range(SLOTS + 64):
        cg.render_frame(d, cg.FrameOut(counts=c.data_ptr()), stream=side, sync=False)
        if k % 256 == 0:
            torch.cuda.synchronize()
            a.zero_(), b.zero_()
            g.replay()
            torch.cuda.synchronize()
            assert torch.equal(a, want) and torch.equal(b, want) and torch.equal(c, want), k
            c.zero_()
            torch.cuda.synchronize()
