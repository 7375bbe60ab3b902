"""The binary32 frame kernel's queues and packing, and the interior test at its
edge, against the oracle: escape counts and totals bit for bit."""
import cmath

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

from oracle.oracle import MANDELBROT  # noqa: E402
from tests.test_gpu_frame import check_rgba, check_smooth, run_frame  # noqa: E402


# iteration limits around the fresh share (32 steps after the first), the untested blocks (16) and the rounds (64);
# sizes from one pixel to more batches than warps; views where few, some and nearly all orbits are long
@pytest.mark.parametrize("max_iter", [0, 1, 2, 33, 34, 49, 97, 98, 1000])
@pytest.mark.parametrize("w,h,spp", [(1, 1, 1), (31, 3, 1), (517, 129, 1), (65, 33, 3)])
def test_limits_and_sizes(cuda, oracle, w, h, spp, max_iter):
    import chaos_gb300 as cg
    from chaos_gb300.palette import seeded_palette
    pal = seeded_palette(64, seed=2)
    for arith, center, ps in ((1, (-0.5, 0.0), 3.0 / w), (0, (-0.748, 0.1), 0.01 / w), (1, (-1.7548, 0.0), 0.04 / w)):
        mode = cg.SAMPLES_JITTER if spp > 1 else cg.SAMPLES_CENTER
        g = run_frame(cuda, w, h, max_iter, spp, mode, cg.TIER_F32, arith, seed=9, center=center, ps=ps, palette=pal)
        o = oracle.frame(w, h, max_iter, spp, 1 if spp > 1 else 0, False, arith, MANDELBROT, 9, center, ps,
                         palette=pal)
        assert np.array_equal(g["counts"], o["counts"])
        assert g["total"] == o["total"]
        check_smooth(g["smooth"], o["smooth"])
        check_smooth(g["pixels"]["value"], o["pixels"]["value"])
        check_rgba(g["rgba"], o["rgba"])


def test_more_pixels_than_fixed_batches(cuda, oracle):
    """A frame of several batches a warp, all of them long orbits (the queue fills and drains in between)."""
    import chaos_gb300 as cg
    g = run_frame(cuda, 1999, 301, 400, 1, cg.SAMPLES_CENTER, cg.TIER_F32, 1, center=(-0.7436, 0.1318), ps=2e-5)
    o = oracle.frame(1999, 301, 400, 1, 0, False, 1, MANDELBROT, 0, (-0.7436, 0.1318), 2e-5)
    assert np.array_equal(g["counts"], o["counts"])
    assert g["total"] == o["total"]


@pytest.mark.parametrize("tier", [0, 1])
@pytest.mark.parametrize("turn", [0.0, 0.01, 0.17, 1 / 3, 0.381966, 0.5])
def test_interior_test_edge(cuda, oracle, tier, turn):
    """Windows across the bound |mu| = 1 - 2^-7 of the interior test, and the disc's 1 - 2^-6."""
    import chaos_gb300 as cg
    mu = (1 - 2.0 ** -7) * cmath.exp(2j * cmath.pi * turn)
    for c in (mu / 2 - mu * mu / 4, -1 + (1 - 2.0 ** -6) / 4 * cmath.exp(2j * cmath.pi * turn)):
        center, ps = (c.real, c.imag), 2e-4
        g = run_frame(cuda, 64, 64, 3000, 1, cg.SAMPLES_CENTER, tier, 1, center=center, ps=ps)
        o = oracle.frame(64, 64, 3000, 1, 0, tier == 1, 1, MANDELBROT, 0, center, ps)
        assert np.array_equal(g["counts"], o["counts"])
