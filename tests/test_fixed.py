"""Coordinates as 32-bit fractions of the box (fixed_coord), checked on the host against extended precision
within the roundings that it is made of, and the redraw probability as an integer threshold against the
division of the draw that it stands for."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_fixed_coordinates_and_draw_thresholds(tmp_path):
    if shutil.which("g++") is None:
        pytest.skip("g++ not available")
    exe = str(tmp_path / "fixed_check")
    r = subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-I", os.path.join(ROOT, "oxdna_gb300", "csrc"),
                        os.path.join(ROOT, "tests", "native", "fixed_check.cpp"), "-o", exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([exe, "400000"], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr
