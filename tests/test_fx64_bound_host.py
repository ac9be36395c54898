"""Host-side check that the fixed-point products' bound of a sequence is one: each
held value's term (fx64.cuh's cterm) is above its size, compiled for the host by
nvcc and checked by tests/fx64_bound_check.cu."""

import shutil
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parent.parent


def test_terms_bound_their_values(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not Path(nvcc).exists():
        pytest.skip("nvcc not available")
    exe = tmp_path / "fx64_bound_check"
    build = subprocess.run([nvcc, "-O2", "-std=c++17", f"-I{ROOT / 'nhqg_gb300' / 'csrc'}",
                            str(ROOT / "tests" / "fx64_bound_check.cu"), "-o", str(exe)],
                           capture_output=True, text=True, timeout=600)
    assert build.returncode == 0, build.stderr[-2000:]
    run = subprocess.run([str(exe)], capture_output=True, text=True, timeout=300)
    assert run.returncode == 0, run.stdout + run.stderr
