"""The far wings' nodes (clblm_gb300/csrc/clblm_f4nodes.cuh): the error of the
polynomial through them and of whole sums of records through them against
those record by record: tests/c/f4nodes_check.cpp,
compiled for the host from the same header."""
import shutil
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]


def test_nodes(tmp_path):
    cxx = shutil.which("g++") or shutil.which("c++")
    if not cxx:
        pytest.skip("no C++ compiler")
    exe = tmp_path / "f4nodes_check"
    subprocess.run([cxx, "-O2", "-std=c++17", "-ffp-contract=off", "-x", "c++", "-I",
                    str(ROOT / "clblm_gb300" / "csrc"), str(ROOT / "tests" / "c" / "f4nodes_check.cpp"), "-o",
                    str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr
    assert "violations 0" in r.stdout
