"""Reference-mode frames whose tiles fit the GPU at once go out in blocks sized to fill the SMs evenly: tile counts where
the block size changes, against the oracle, every record field bit for bit."""
import pytest

pytestmark = pytest.mark.gpu

from oracle.oracle import MANDELBROT  # noqa: E402
from tests.gpu_util import pitched, read_pixels, same_pixels, upload_pixels  # noqa: E402


@pytest.mark.parametrize("dbl", [False, True])
@pytest.mark.parametrize("per_sm,more", [(0, 1), (1, -1), (1, 0), (1, 1), (3, 1), (7, 0), (7, 1), (8, 0), (8, 1), (15, 1), (32, 1)])
def test_tile_counts(cuda, oracle, per_sm, more, dbl):
    import chaos_gb300 as cg
    tiles = per_sm * cuda.cuda.get_device_properties(0).multi_processor_count + more
    rows = max(r for r in (1, 2, 3, 4, 5) if tiles % r == 0)
    w, h = 8 * (tiles // rows) - 3 * (tiles > rows), 4 * rows - 1
    old = (-0.75, 0.099, -0.746, 0.099 + 0.004 * h / w)
    new = (-0.7499, 0.09901, -0.7461, 0.09901 + 0.0038 * h / w)
    out, pitch = pitched(cuda, w, h)
    with cg.Module("mandelbrot") as m:
        m.render_main(out.data_ptr(), pitch, w, h, old, 300, 2.0, 1, double=dbl, arith=cg.ARITH_PARITY)
        first = oracle.render_main(MANDELBROT, dbl, cg.ARITH_PARITY, w, h, old, 300, 2.0, 1)
        assert not same_pixels(read_pixels(out, w), first).any()
        src, src_pitch = upload_pixels(cuda, first)
        flags = cg.FLAG_ADAPTIVE_SS | cg.FLAG_SAMPLE_REUSE | cg.FLAG_IS_ZOOMING | cg.FLAG_ZOOMING_IN
        m.render_advanced(out.data_ptr(), pitch, w, h, new, 300, 2.0, flags, old, src.data_ptr(), src_pitch, (9, 1),
                          double=dbl, arith=cg.ARITH_PARITY)
        second = oracle.render_advanced(MANDELBROT, dbl, cg.ARITH_PARITY, w, h, new, 300, 2.0, flags, old, first, (9, 1))
        assert not same_pixels(read_pixels(out, w), second).any()
