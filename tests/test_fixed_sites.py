"""Fixed-point sites and their separations, as the first step and the non-bonded kernel form them (fixed_site,
fixed_sep), on the host: the minimum image within the roundings it is made of, across the faces of the box too,
with no undefined arithmetic."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_separations_of_fixed_point_sites(tmp_path):
    if shutil.which("g++") is None:
        pytest.skip("g++ not available")
    exe = str(tmp_path / "fixed_sites_check")
    base = ["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-I", os.path.join(ROOT, "oxdna_gb300", "csrc"),
            os.path.join(ROOT, "tests", "native", "fixed_sites_check.cpp"), "-o", exe]
    r = subprocess.run(base + ["-fsanitize=signed-integer-overflow", "-fno-sanitize-recover=all"], capture_output=True, text=True)
    if r.returncode != 0 and "sanitize" in r.stderr + r.stdout or "ubsan" in r.stderr:
        r = subprocess.run(base, capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([exe, "400000"], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr
