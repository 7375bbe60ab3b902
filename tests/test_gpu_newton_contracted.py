"""The Newton modules of the default build (nvcc's contraction on) against the plain loops around the same step
(newton_plain.cu, built the same way): which products nvcc fuses is part of these modules' values."""
import ctypes as C
import os
import shutil
import subprocess

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

from tests.gpu_util import Driver, java_grid, main_params, pitched, read_pixels  # noqa: E402

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
ROOTS = [1, 0, -0.5, 0.86602540378, -0.5, -0.86602540378]


@pytest.fixture(scope="module")
def plain(cuda, tmp_path_factory):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("no nvcc")
    out = str(tmp_path_factory.mktemp("plain") / "newton_plain.cubin")
    subprocess.run([nvcc, "-gencode", "arch=compute_103a,code=sm_103a", "-O3", "-std=c++17", "--expt-relaxed-constexpr",
                    "-cubin", "-o", out, os.path.join(ROOT, "tests", "newton_plain.cu")], check=True)
    drv = Driver()
    return drv, drv.load(out)


@pytest.mark.parametrize("max_iter", [5, 30, 200])
@pytest.mark.parametrize("coeffs", [[-1, 0, 0, 1], [-0.1, 0, 0, 1], [-1.5, 0, 0, 1], [2, -2, 0, 1], [-1, 0.5, 0, 2]])
@pytest.mark.parametrize("kind", ["wired", "generic", "iterations"])
def test_default_build(cuda, plain, kind, coeffs, max_iter):
    import chaos_gb300 as cg
    torch = cuda
    drv, ref = plain
    if kind == "wired" and coeffs != [-1, 0, 0, 1]:
        pytest.skip("the wired module has no coefficients")
    w, h = 640, 360
    r = (-2.1, -1.125, 2.0, 1.18125)
    dev = [torch.tensor(v, dtype=torch.float64, device="cuda:0") for v in (r, coeffs, ROOTS)]
    mod = drv.load(os.path.join(cg.DROPIN_DIR, "newton_" + kind + ".ptx"))
    if kind != "wired":
        drv.write_constant(mod, "coefficients", np.array(coeffs, dtype=np.float64).tobytes())
        drv.write_constant(mod, "roots", np.array(ROOTS, dtype=np.float64).tobytes())
    grid, block = java_grid(w, h)
    for dbl in (False, True):
        want = torch.zeros((h, w), dtype=torch.float32, device="cuda:0")
        torch.cuda.synchronize()
        drv.launch(drv.function(ref, kind + ("_f64" if dbl else "_f32")), ((w + 31) // 32, (h + 7) // 8), (32, 8),
                   [C.c_uint64(want.data_ptr()), C.c_int32(w), C.c_int32(h), C.c_uint64(dev[0].data_ptr()),
                    C.c_uint32(max_iter), C.c_uint64(dev[1].data_ptr()), C.c_uint64(dev[2].data_ptr())])
        buf, pitch = pitched(torch, w, h)
        torch.cuda.synchronize()
        drv.launch(drv.function(mod, "fractalRenderMainDouble" if dbl else "fractalRenderMainFloat"), grid, block,
                   main_params(buf.data_ptr(), pitch, w, h, r, max_iter, 1.0, 0, dbl))
        got = read_pixels(buf, w)["value"]
        assert np.array_equal(got, want.cpu().numpy()), (dbl, int((got != want.cpu().numpy()).sum()))
    drv.unload(mod)
