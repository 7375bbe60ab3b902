"""The pages of a caller's buffer are brought in before the device's copy without a byte of it changing, and an address
that cannot be written is left to the copy."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_populate_pages(tmp_path):
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("no g++")
    exe = str(tmp_path / "hostpages_check")
    subprocess.run([gxx, "-O2", "-std=c++17", "-I", os.path.join(ROOT, "chaos-ultra_gb300", "csrc"), "-o", exe,
                    os.path.join(ROOT, "tests", "hostpages_check.cpp")], check=True)
    out = subprocess.run([exe], capture_output=True, text=True, timeout=60)
    assert out.returncode == 0 and out.stdout.strip() in ("ok", "old kernel"), out.stdout
