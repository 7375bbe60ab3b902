"""Work-counter slots that the host gives back (calls that wait) and those that the launch does (calls that do not):
more of both than there are slots, from several threads, every frame complete."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SLOTS = 4096  # kCounterSlots


def test_waiting_and_other_calls(cuda, native, oracle):
    import chaos_gb300 as cg
    torch = cuda
    w, h, mi, n = 66, 46, 60, SLOTS // 2 + 100
    o = oracle.frame(w, h, mi, 1, 0, False, cg.ARITH_PARITY, cg.MANDELBROT, 0, (-0.5, 0.0), 0.04)
    want, total = torch.from_numpy(o["counts"].reshape(-1).view(np.int32).copy()).to("cuda:0"), int(o["total"])
    threads = 4
    counts = torch.zeros((threads, n, w * h), dtype=torch.int32, device="cuda:0")
    totals = torch.zeros((threads, n), dtype=torch.int64, device="cuda:0")
    streams = [torch.cuda.Stream() for _ in range(threads)]
    torch.cuda.synchronize()
    errors = []

    def work(t):
        try:
            for k in range(n):
                limit = 20.0 if k % 3 == 0 and k % 2 == t % 2 else 0.0  # (a status word goes with the slot)
                d = cg.FrameDesc(width=w, height=h, max_iterations=mi, samples_per_pixel=1, tier=cg.TIER_F32,
                                 sample_mode=cg.SAMPLES_CENTER, arith=cg.ARITH_PARITY, fractal=cg.MANDELBROT, seed=0,
                                 center_x=-0.5, center_y=0.0, pixel_size=0.04, time_limit_s=limit)
                cg.render_frame(d, cg.FrameOut(counts=counts[t, k].data_ptr(), total_iterations=totals[t, k:].data_ptr()),
                                stream=streams[t], sync=k % 2 == t % 2)
        except Exception as e:  # noqa: BLE001
            errors.append(e)

    pool = [threading.Thread(target=work, args=(t,)) for t in range(threads)]
    for p in pool:
        p.start()
    for p in pool:
        p.join()
    torch.cuda.synchronize()
    assert not errors
    assert bool((counts == want).all()) and bool((totals == total).all())
