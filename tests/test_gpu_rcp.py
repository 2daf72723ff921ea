"""rcp_d (clblm_gb300/csrc/clblm_fpconv.cuh), the reciprocal of the FP64 far
wings, within a unit in the last place of the division: tests/c/rcp_check.cu,
built from the same header with the library's architecture."""
import subprocess
from pathlib import Path

import pytest

from clblm_gb300 import build

pytestmark = pytest.mark.gpu
ROOT = Path(__file__).resolve().parents[1]


def test_reciprocals(tmp_path):
    exe = tmp_path / "rcp_check"
    subprocess.run([build.nvcc(), *build.ARCH, "-O3", "-std=c++17", "-I", str(ROOT / "clblm_gb300" / "csrc"),
                    str(ROOT / "tests" / "c" / "rcp_check.cu"), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr
