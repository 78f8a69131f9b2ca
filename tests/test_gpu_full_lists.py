"""Counters of the bounded device lists past 2^32: what is in use is not handed
out again (tests/native/test_full_lists.cu)."""
import os
import subprocess
from pathlib import Path

import pytest

pytestmark = pytest.mark.gpu
REPO = Path(__file__).resolve().parents[1]


def test_full_lists_stay_full(tmp_path):
    exe = tmp_path / "full_lists"
    nvcc = Path(os.environ.get("CUDA_HOME", "/usr/local/cuda")) / "bin" / "nvcc"
    csrc = REPO / "kami-hair-solver_gb300" / "csrc"
    subprocess.run([str(nvcc), "-gencode", "arch=compute_103a,code=sm_103a", "-O3", "-std=c++17", f"-I{csrc}",
                    f"-I{REPO / 'include'}", str(REPO / "tests" / "native" / "test_full_lists.cu"), "-o", str(exe)], check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    print(out.stdout)
    assert out.returncode == 0 and "PASS" in out.stdout, out.stdout + out.stderr
