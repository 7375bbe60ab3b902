"""Large zoom steps with a foveal region (strips of one group from block-sized pieces, and the fovea's bound by distance)
against the drop-in module's fractalRenderAdvancedFloat, which renders one tile a warp: records bit for bit."""
import os

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

from tests.gpu_util import Driver, advanced_params, java_grid, read_pixels, same_pixels, upload_pixels  # noqa: E402


@pytest.mark.parametrize("w,h,focus", [(2568, 1948, (1284, 974)), (3841, 2161, (3, 2157)), (5000, 1001, (4999, 0))])
@pytest.mark.parametrize("sub,arith", [("DROPIN_PARITY_DIR", 1), ("DROPIN_DIR", 2)])
def test_zoom_step_equals_the_dropin_module(cuda, native, w, h, focus, sub, arith):
    import chaos_gb300 as cg
    torch = cuda
    rng = np.random.default_rng(w)
    prev = np.zeros((h, w), dtype=[("value", "<f4"), ("weight", "<f4"), ("is_reused", "u1"), ("pad", "u1", 3),
                                   ("weight_of_new_samples", "<f4")])
    prev["value"] = rng.integers(0, 300, size=(h, w))
    prev["weight"] = np.where(rng.uniform(size=(h, w)) < 0.999, 2.0, 0.0)  # some pixels hold nothing to reuse
    src, pitch = upload_pixels(torch, prev)
    rect = (-0.7536, 0.1268, -0.7336, 0.1268 + 0.02 * h / w)
    old = (-0.7538, 0.1266, -0.7334, 0.1266 + 0.0204 * h / w)
    flags = (cg.FLAG_ADAPTIVE_SS | cg.FLAG_SAMPLE_REUSE | cg.FLAG_FOVEATION | cg.FLAG_IS_ZOOMING | cg.FLAG_ZOOMING_IN)
    ours, theirs = torch.zeros_like(src), torch.zeros_like(src)
    m = cg.Module("mandelbrot")
    m.render_advanced(ours.data_ptr(), pitch, w, h, rect, 200, 2.0, flags, old, src.data_ptr(), pitch, focus,
                      arith=arith)
    d = Driver()
    mod = d.load(os.path.join(getattr(cg, sub), "mandelbrot.ptx"))
    grid, block = java_grid(w, h)
    d.launch(d.function(mod, "fractalRenderAdvancedFloat"), grid, block,
             advanced_params(theirs.data_ptr(), pitch, w, h, rect, 200, 2.0, flags, old, src.data_ptr(), pitch, focus,
                             False))
    assert not same_pixels(read_pixels(ours, w), read_pixels(theirs, w)).any()
    d.unload(mod)
