"""The Newton loop's groups of four steps at iteration limits near 2^32, on the host: a state that never settles (the
2-cycle of x^3 - 2x + 2) would take minutes to get there on a GPU, and never leave where the sum wraps."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_groups_end_at_the_limit(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("no nvcc")
    exe = str(tmp_path / "newton_group_check")
    subprocess.run([nvcc, "-gencode", "arch=compute_103a,code=sm_103a", "-std=c++17", "--expt-relaxed-constexpr", "-I",
                    os.path.join(ROOT, "chaos-ultra_gb300", "csrc"), "-I", os.path.join(ROOT, "include"), "-o", exe,
                    os.path.join(ROOT, "tests", "newton_group_check.cu")], check=True)
    out = subprocess.run([exe], capture_output=True, text=True, timeout=60)
    assert out.returncode == 0 and out.stdout.strip() == "ok", out.stdout
