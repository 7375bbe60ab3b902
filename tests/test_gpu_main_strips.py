"""Reference-mode frames large enough for strips of several tiles, at limits where the longest strip changes (8, 4, 2
tiles), a ragged last column and row: every record like the oracle's."""
import pytest

pytestmark = pytest.mark.gpu

from oracle.oracle import MANDELBROT  # noqa: E402
from tests.gpu_util import pitched, read_pixels, same_pixels  # noqa: E402


@pytest.mark.parametrize("w,h,max_iter,max_ss", [(3837, 2159, 16, 1.0), (3837, 2159, 64, 1.0), (3837, 2159, 64, 3.0),
                                                 (7677, 4317, 24, 1.0)])
def test_strips(cuda, oracle, w, h, max_iter, max_ss):
    import chaos_gb300 as cg
    rect = (-2.0, -1.5 * h / w, 1.0, 1.5 * h / w)
    out, pitch = pitched(cuda, w, h)
    with cg.Module("mandelbrot") as m:
        m.render_main(out.data_ptr(), pitch, w, h, rect, max_iter, max_ss, 1, arith=cg.ARITH_PARITY)
    want = oracle.render_main(MANDELBROT, False, cg.ARITH_PARITY, w, h, rect, max_iter, max_ss, 1)
    assert not same_pixels(read_pixels(out, w), want).any()
