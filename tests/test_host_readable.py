"""host_readable.h, the question whether the caller's memory can be read (CPU only)."""
import shutil
import subprocess
from pathlib import Path

import pytest

REPO = Path(__file__).resolve().parents[1]


def test_host_readable(tmp_path):
    if not shutil.which("g++"):
        pytest.skip("no g++")
    exe = tmp_path / "host_readable_test"
    r = subprocess.run(["g++", "-O2", "-Wall", "-Werror", "-std=c++17", str(REPO / "tests" / "cpp" / "host_readable_test.cpp"),
                        "-o", str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0 and r.stdout.strip() == "ok", r.stdout + r.stderr
