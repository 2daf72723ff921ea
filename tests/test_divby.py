"""Division by a divisor known ahead (clblm_gb300/csrc/clblm_fpconv.cuh,
div_by) equals the machine's correctly rounded quotient, and the comparisons
on the bits the machine's own: tests/c/divby_check.cpp, compiled for the host
from the same header."""
import shutil
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]


def test_quotients_and_comparisons(tmp_path):
    cxx = shutil.which("g++") or shutil.which("c++")
    if not cxx:
        pytest.skip("no C++ compiler")
    exe = tmp_path / "divby_check"
    subprocess.run([cxx, "-O2", "-std=c++17", "-ffp-contract=off", "-I", str(ROOT / "clblm_gb300" / "csrc"),
                    str(ROOT / "tests" / "c" / "divby_check.cpp"), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr
    assert "mismatches 0" in r.stdout
