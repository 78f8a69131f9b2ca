"""An element's gradient and Hessian by two threads, one for each end, equal the
one-thread form bit for bit (tests/native/test_element_ends.cpp)."""
import shutil
import subprocess
from pathlib import Path

import pytest

REPO = Path(__file__).resolve().parents[1]


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs g++")
def test_element_by_ends_matches_the_one_thread_form(tmp_path):
    exe = tmp_path / "ends"
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", f"-I{REPO / 'kami-hair-solver_gb300' / 'csrc'}",
                    str(REPO / "tests" / "native" / "test_element_ends.cpp"), "-o", str(exe)], check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True)
    print(out.stdout)
    assert out.returncode == 0 and "PASS" in out.stdout, out.stdout + out.stderr
