"""Strands that fail in the FP64 block solve and their neighbours, in every
layout (tests/native/test_block_solve_failures.cu)."""
import os
import subprocess
from pathlib import Path

import pytest

pytestmark = pytest.mark.gpu
REPO = Path(__file__).resolve().parents[1]


def test_failing_strands_are_reported_and_the_others_solved(tmp_path):
    exe = tmp_path / "block_solve_failures"
    nvcc = Path(os.environ.get("CUDA_HOME", "/usr/local/cuda")) / "bin" / "nvcc"
    subprocess.run([str(nvcc), "-gencode", "arch=compute_103a,code=sm_103a", "-O3", "-std=c++17", "-Xcompiler",
                    "-ffp-contract=off", f"-I{REPO / 'kami-hair-solver_gb300' / 'csrc'}",
                    str(REPO / "tests" / "native" / "test_block_solve_failures.cu"), "-o", str(exe)], check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    print(out.stdout)
    assert out.returncode == 0 and "PASS" in out.stdout, out.stdout + out.stderr
