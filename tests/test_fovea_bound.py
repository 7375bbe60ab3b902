"""The bound by distance of the foveal region (clear_of_fovea in csrc/chaos_device.cuh) on its own, and the interior
test's constants: both read from the header, so that neither can move without the proof that it needs."""
import os
import re

import numpy as np

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
with open(os.path.join(ROOT, "chaos-ultra_gb300", "csrc", "chaos_device.cuh")) as fh:
    HEADER = fh.read()


def test_no_tile_beyond_the_bound_is_foveal():
    """getFoveationAdvisedSampleCount (gen.cu:209-257): inside means an angle of at most 5.5 degrees (less where
    maxSuperSampling is below 1), seen from 60 cm at 0.02652 cm a pixel.  Every offset of tile corners that the bound
    calls clear has a larger angle, with room for binary32 (a few 2^-24 on each of six operations)."""
    m = re.search(r"fmaf\(dx, dx, dy \* dy\) > (\d+)\.f \* (\d+)\.f", HEADER)
    bound = int(m.group(1))
    assert m.group(1) == m.group(2)
    dx, dy = np.meshgrid(np.arange(0, 2 * bound), np.arange(0, 2 * bound))
    d2 = dx.astype(np.int64) ** 2 + dy.astype(np.int64) ** 2
    clear = d2.astype(np.float32) > np.float32(bound * bound)
    angle = np.degrees(np.arctan(np.sqrt(d2) * 0.02652 / 60.0))
    assert angle[clear].min() > 5.5 * (1 + 1e-5)
    assert angle[~clear & (d2 <= (bound - 2) ** 2)].max() <= 5.5  # and the bound is no wider than it has to be


def test_interior_constants_are_the_proven_ones():
    """tests/test_interior_bound.py proves the interior test for these two bounds."""
    cardioid = float(re.search(r"constexpr float CARDIOID = ([\d.]+)f;", HEADER).group(1))
    disc = float(re.search(r"constexpr float DISC = ([\d.]+)f;", HEADER).group(1))
    with open(os.path.join(ROOT, "tests", "test_interior_bound.py")) as fh:
        proof = fh.read()
    assert f"f({cardioid})" in proof and f"f({disc})" in proof
    assert cardioid > 1 - (1 - 2.0 ** -7) ** 2 and disc < ((1 - 2.0 ** -6) / 4) ** 2
