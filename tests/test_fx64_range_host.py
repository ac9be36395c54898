"""Host-side check of the fixed-point products at values of 2^62, the end of the range
that the transforms use, compiled for the host by nvcc and checked by
tests/fx64_range_check.cu."""

import shutil
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parent.parent


def test_products_at_the_end_of_the_range(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not Path(nvcc).exists():
        pytest.skip("nvcc not available")
    exe = tmp_path / "fx64_range_check"
    build = subprocess.run([nvcc, "-O2", "-std=c++17", f"-I{ROOT / 'nhqg_gb300' / 'csrc'}",
                            str(ROOT / "tests" / "fx64_range_check.cu"), "-o", str(exe)],
                           capture_output=True, text=True, timeout=600)
    assert build.returncode == 0, build.stderr[-2000:]
    run = subprocess.run([str(exe)], capture_output=True, text=True, timeout=300)
    assert run.returncode == 0, run.stdout + run.stderr
