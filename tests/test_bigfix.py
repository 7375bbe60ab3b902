"""The multi-word product of the reference orbits, with its two guard columns, equals the full product."""
import os
import subprocess


def test_guarded_product_equals_the_full_one(tmp_path):
    here = os.path.dirname(os.path.abspath(__file__))
    exe = str(tmp_path / "bigfix_check")
    subprocess.run(["g++", "-O2", "-std=c++17", os.path.join(here, "bigfix_check.cpp"), "-o", exe], check=True)
    assert subprocess.run([exe], check=True, capture_output=True, text=True).stdout.strip() == "0"
