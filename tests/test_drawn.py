"""The redraw test of the Brownian thermostat, drawn(x, draw_threshold(p)), as host and device share it: the same
as (x + 1) / 2^32 < p for every draw, with p = 0, 1 and beyond, and through the threshold's bits."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_thresholds_stand_for_the_division(tmp_path):
    if shutil.which("g++") is None:
        pytest.skip("g++ not available")
    exe = str(tmp_path / "drawn_check")
    r = subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-I", os.path.join(ROOT, "oxdna_gb300", "csrc"),
                        os.path.join(ROOT, "tests", "native", "drawn_check.cpp"), "-o", exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([exe, "300000"], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr
