"""The binary64 frame kernel's hand-over from claiming pixels to packing what is left: the warps of a block get there at
different rounds and one of them tells the others, in blocks of every size.  Counts and totals bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

from oracle.oracle import JULIA, MANDELBROT  # noqa: E402
from tests.test_gpu_frame import run_frame  # noqa: E402


# pixels from a part of one warp to several claims a lane; views where few and many orbits are long
@pytest.mark.parametrize("w,h,spp", [(7, 1, 1), (152 * 32, 1, 1), (152 * 32 + 1, 3, 1), (640, 130, 1), (331, 101, 4),
                                     (853, 479, 1)])
@pytest.mark.parametrize("arith", [0, 1])
def test_hand_over(cuda, oracle, w, h, spp, arith):
    import chaos_gb300 as cg
    mode = cg.SAMPLES_JITTER if spp > 1 else cg.SAMPLES_CENTER
    for fractal, center, span, julia_c in ((MANDELBROT, (-0.5, 0.0), 3.0, (0.0, 0.0)),
                                           (MANDELBROT, (-0.7436, 0.1318), 2e-3, (0.0, 0.0)),
                                           (JULIA, (0.0, 0.0), 3.0, (-0.8, 0.156))):
        g = run_frame(cuda, w, h, 700, spp, mode, cg.TIER_F64, arith, fractal=fractal, seed=4, center=center,
                      ps=span / w, julia_c=julia_c)
        o = oracle.frame(w, h, 700, spp, 1 if spp > 1 else 0, True, arith, fractal, 4, center, span / w,
                         julia_c=julia_c)
        assert np.array_equal(g["counts"], o["counts"])
        assert g["total"] == o["total"]
