"""Reuse frames in binary64, whose warps' first strips go out without a claim: fewer tiles than warps, a last strip that
does not fill, strips of several tiles, against the drop-in module's fractalRenderAdvancedDouble (one tile a warp)."""
import os

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

from tests.gpu_util import Driver, advanced_params, java_grid, read_pixels, same_pixels, upload_pixels  # noqa: E402


@pytest.mark.parametrize("w,h", [(5, 5), (33, 9), (331, 187), (1235, 801), (2403, 1661)])
@pytest.mark.parametrize("sub,arith", [("DROPIN_PARITY_DIR", 1), ("DROPIN_DIR", 2)])
def test_zoom_out_equals_the_dropin_module(cuda, native, w, h, sub, arith):
    import chaos_gb300 as cg
    torch = cuda
    rng = np.random.default_rng(w)
    prev = np.zeros((h, w), dtype=[("value", "<f4"), ("weight", "<f4"), ("is_reused", "u1"), ("pad", "u1", 3),
                                   ("weight_of_new_samples", "<f4")])
    prev["value"] = rng.integers(0, 300, size=(h, w))
    prev["weight"] = np.where(rng.uniform(size=(h, w)) < 0.99, 2.0, 0.0)  # some pixels hold nothing to reuse
    src, pitch = upload_pixels(torch, prev)
    rect = (-0.7538, 0.1266, -0.7334, 0.1266 + 0.0204 * h / w)
    old = (-0.7536, 0.1268, -0.7336, 0.1268 + 0.02 * h / w)
    flags = cg.FLAG_ADAPTIVE_SS | cg.FLAG_SAMPLE_REUSE | cg.FLAG_IS_ZOOMING
    ours, theirs = torch.zeros_like(src), torch.zeros_like(src)
    m = cg.Module("mandelbrot")
    m.render_advanced(ours.data_ptr(), pitch, w, h, rect, 150, 2.0, flags, old, src.data_ptr(), pitch, (w // 2, h // 2),
                      double=True, arith=arith)
    d = Driver()
    mod = d.load(os.path.join(getattr(cg, sub), "mandelbrot.ptx"))
    grid, block = java_grid(w, h)
    d.launch(d.function(mod, "fractalRenderAdvancedDouble"), grid, block,
             advanced_params(theirs.data_ptr(), pitch, w, h, rect, 150, 2.0, flags, old, src.data_ptr(), pitch,
                             (w // 2, h // 2), True))
    assert not same_pixels(read_pixels(ours, w), read_pixels(theirs, w)).any()
    d.unload(mod)
