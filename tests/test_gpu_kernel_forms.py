"""Kernels that several threads share a result in against their one-thread forms,
bit for bit (tests/native/test_kernel_forms.cu)."""
import os
import subprocess
from pathlib import Path

import pytest

pytestmark = pytest.mark.gpu
REPO = Path(__file__).resolve().parents[1]


def test_shared_forms_match_the_one_thread_forms(tmp_path):
    exe = tmp_path / "kernel_forms"
    nvcc = Path(os.environ.get("CUDA_HOME", "/usr/local/cuda")) / "bin" / "nvcc"
    subprocess.run([str(nvcc), "-gencode", "arch=compute_103a,code=sm_103a", "-O3", "-lineinfo", "-std=c++17", "-Xcompiler",
                    "-ffp-contract=off", f"-I{REPO / 'kami-hair-solver_gb300' / 'csrc'}", f"-I{REPO / 'include'}",
                    str(REPO / "tests" / "native" / "test_kernel_forms.cu"), "-o", str(exe)], check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    print(out.stdout)
    assert out.returncode == 0 and "PASS" in out.stdout, out.stdout + out.stderr
