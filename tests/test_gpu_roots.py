"""The library's own correctly rounded square root and reciprocals (roots.cuh) on the device, for
every float of the ranges they are used in (tests/cpp/roots_check.cu, built here)."""
import os
import shutil
import subprocess
from pathlib import Path

import pytest

pytestmark = pytest.mark.gpu
REPO = Path(__file__).resolve().parents[1]


def test_every_float(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    assert os.path.exists(nvcc)
    exe = tmp_path / "roots_check"
    r = subprocess.run([nvcc, "-gencode", "arch=compute_103a,code=sm_103a", "-O3", "-std=c++17", "-o", str(exe),
                        str(REPO / "tests" / "cpp" / "roots_check.cu")], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    lines = r.stdout.splitlines()
    assert r.returncode == 0 and len(lines) == 4 and all(x.endswith("differing 0") for x in lines), r.stdout + r.stderr
