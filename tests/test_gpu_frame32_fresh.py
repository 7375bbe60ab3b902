"""Binary32 frames at the iteration limits where fresh pixels run to the limit (200; 512 where every warp has one batch at
most) and just past them: counts, totals and smooth values like the oracle's."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

from oracle.oracle import JULIA, MANDELBROT  # noqa: E402


@pytest.mark.parametrize("w,h,spp", [(70, 50, 1), (67, 41, 3), (997, 613, 1), (499, 401, 2)])
@pytest.mark.parametrize("max_iter", [1, 33, 200, 201, 512, 513])
@pytest.mark.parametrize("fractal,center,span", [(MANDELBROT, (-1.25, 0.0), 0.2), (JULIA, (0.0, 0.0), 3.0)])
def test_limits(cuda, native, oracle, w, h, spp, max_iter, fractal, center, span):
    import chaos_gb300 as cg
    torch = cuda
    counts = torch.zeros(w * h * spp, dtype=torch.int32, device="cuda:0")
    smooth = torch.zeros(w * h * spp, dtype=torch.float32, device="cuda:0")
    total = torch.zeros(1, dtype=torch.int64, device="cuda:0")
    mode = cg.SAMPLES_JITTER if spp > 1 else cg.SAMPLES_CENTER
    d = cg.FrameDesc(width=w, height=h, max_iterations=max_iter, samples_per_pixel=spp, sample_mode=mode,
                     tier=cg.TIER_F32, arith=cg.ARITH_PARITY, fractal=fractal, seed=9, center_x=center[0],
                     center_y=center[1], pixel_size=span / w, julia_cx=-0.8, julia_cy=0.156)
    cg.render_frame(d, cg.FrameOut(counts=counts.data_ptr(), smooth=smooth.data_ptr(), total_iterations=total.data_ptr()))
    o = oracle.frame(w, h, max_iter, spp, mode, False, cg.ARITH_PARITY, fractal, 9, center, span / w,
                     julia_c=(-0.8, 0.156))
    assert np.array_equal(counts.cpu().numpy().view(np.uint32), o["counts"].ravel())
    assert int(total.item()) == int(o["total"])
    want = o["smooth"].ravel()
    assert (np.abs(smooth.cpu().numpy() - want) <= 2 * np.spacing(np.abs(want)) + 2e-6).all()
