"""The (iIn, IP) of interpSpectrum's general-ratio branch formed point by
point (clblm_gb300/csrc/clblm_interpmap.cuh) equal the reference's steps:
tests/c/interpmap_check.cpp, compiled for the host from the same header, over
random ratios, grids that coincide (spacings of a few digits, small
fractions) and the edges of its ranges."""
import shutil
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]


def test_interpolation_map_equals_the_steps(tmp_path):
    cxx = shutil.which("g++") or shutil.which("c++")
    if not cxx:
        pytest.skip("no C++ compiler")
    exe = tmp_path / "interpmap_check"
    subprocess.run([cxx, "-O2", "-std=c++17", "-ffp-contract=off", "-I", str(ROOT / "clblm_gb300" / "csrc"),
                    str(ROOT / "tests" / "c" / "interpmap_check.cpp"), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr
    assert "mismatches 0" in r.stdout
