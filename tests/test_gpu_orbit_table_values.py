"""The perturbation kernels' block tables, as the device makes them, against their definition (orbit_tables_check.cu):
orbits around the table kernel's blocks (64 threads) and the composed blocks (16 and 64 steps), an orbit that passes
near 0 and near |z| = 2, and the whole deep-zoom orbit."""
import os
import shutil
import subprocess

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def program(cuda, tmp_path_factory):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("no nvcc")
    exe = str(tmp_path_factory.mktemp("tables") / "orbit_tables_check")
    subprocess.run([nvcc, "-gencode", "arch=compute_103a,code=sm_103a", "-O2", "-std=c++17", "--expt-relaxed-constexpr",
                    "-I", os.path.join(ROOT, "include"), "-o", exe, os.path.join(ROOT, "tests", "orbit_tables_check.cu")],
                   check=True)
    return exe


def tables(program, centre, bits, limits):
    out = subprocess.run([program, *centre, str(bits)] + [str(n) for n in limits], capture_output=True, text=True,
                         timeout=300)
    assert out.returncode == 0, out.stdout
    return [[int(v) for v in line.split()[1:]] for line in out.stdout.split("\n") if line]


@pytest.mark.parametrize("cx,cy", [(-0.7455, 0.1133), (-1.25, 0.01), (-2.0, 0.0), (0.0, 1.0)])
def test_lengths(cuda, program, cx, cy):
    import chaos_gb300 as cg
    limits = [1, 2, 15, 16, 17, 18, 19, 63, 64, 65, 66, 67, 127, 128, 129, 130, 131, 193, 500]
    got = tables(program, (cg.to_hex_fixed(cx, 192), cg.to_hex_fixed(cy, 192)), 192, limits)
    assert len(got) == len(limits)
    if cx == -1.25:  # no events: a block of 16 starts at every index from 1 that has 17 after it, unless its bound is too low
        assert got[limits.index(17)] == [0, 0] and got[limits.index(500)][0] > 480


def test_deep_zoom_orbit(cuda, program):
    from chaos_gb300.workloads import deep_zoom_centre
    d = deep_zoom_centre()
    (got,) = tables(program, (d["center_x"], d["center_y"]), 1088, [100000])
    assert min(got) > 1500
