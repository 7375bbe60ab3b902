"""The interior test's edge (|mu| = 1 - 2^-7 about the cardioid, 1 - 2^-6 about the period-2 disc) in the arithmetics and
callers beside the rounded frames of test_gpu_frame32.py: fused frames, contracted reference-mode frames, batches."""
import cmath

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

from oracle.oracle import MANDELBROT  # noqa: E402
from tests.gpu_util import pitched, read_pixels, same_pixels  # noqa: E402

W = H = 48
PS, LIMIT = 2e-4, 1500


def edges(turn):
    mu = (1 - 2.0 ** -7) * cmath.exp(2j * cmath.pi * turn)
    for c in (mu / 2 - mu * mu / 4, -1 + (1 - 2.0 ** -6) / 4 * cmath.exp(2j * cmath.pi * turn)):
        yield c.real, c.imag


@pytest.mark.parametrize("turn", [0.0, 0.01, 0.17, 1 / 3, 0.5])
def test_edge(cuda, native, oracle, turn):
    import chaos_gb300 as cg
    torch = cuda
    for center in edges(turn):
        views = []
        for tier in (cg.TIER_F32, cg.TIER_F64):
            counts = torch.zeros(W * H, dtype=torch.int32, device="cuda:0")
            d = cg.FrameDesc(width=W, height=H, max_iterations=LIMIT, samples_per_pixel=1, sample_mode=cg.SAMPLES_CENTER,
                             tier=tier, arith=cg.ARITH_FMA, fractal=cg.MANDELBROT, seed=0, center_x=center[0],
                             center_y=center[1], pixel_size=PS)
            cg.render_frame(d, cg.FrameOut(counts=counts.data_ptr()))
            o = oracle.frame(W, H, LIMIT, 1, 0, tier == cg.TIER_F64, cg.ARITH_FMA, MANDELBROT, 0, center, PS, smooth=False,
                             pixels=False)
            assert np.array_equal(counts.cpu().numpy().view(np.uint32), o["counts"].ravel()), tier
        rect = (center[0] - W * PS / 2, center[1] - H * PS / 2, center[0] + W * PS / 2, center[1] + H * PS / 2)
        for dbl in (False, True):
            out, pitch = pitched(torch, W, H)
            with cg.Module("mandelbrot") as m:
                m.render_main(out.data_ptr(), pitch, W, H, rect, LIMIT, 1.0, 0, double=dbl, arith=cg.ARITH_CONTRACTED)
            want = oracle.render_main(MANDELBROT, dbl, cg.ARITH_CONTRACTED, W, H, rect, LIMIT, 1.0, 0)
            assert not same_pixels(read_pixels(out, W), want).any(), dbl
        for binary64 in (cg.TIER_F64, cg.TIER_F64_ROUNDED):  # (one of the two in a batch)
            tiers = [cg.TIER_F32, cg.TIER_FLOATFLOAT, binary64]
            views = [torch.zeros(W * H, dtype=torch.int32, device="cuda:0") for _ in tiers]
            b = cg.Batch([cg.Viewport(width=W, height=H, max_iterations=LIMIT, samples_per_pixel=1,
                                      sample_mode=cg.SAMPLES_CENTER, tier=t, seed=0, center_x=center[0],
                                      center_y=center[1], pixel_size=PS, counts=v.data_ptr())
                          for t, v in zip(tiers, views)])
            b.launch()
            torch.cuda.synchronize()
            for t, v in zip(tiers, views):
                o = oracle.batch_viewport(W, H, 1, 0, LIMIT, t, 0, center, PS)
                assert np.array_equal(v.cpu().numpy().view(np.uint32), o["counts"].ravel()), t
            b.close()
