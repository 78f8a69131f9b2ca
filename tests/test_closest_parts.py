"""The segment-triangle closest pair with integer comparisons and squared
distances equals the plain floating form bit for bit
(tests/native/test_closest_parts.cpp)."""
import shutil
import subprocess
from pathlib import Path

import pytest

REPO = Path(__file__).resolve().parents[1]


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs g++")
def test_closest_pair_matches_the_plain_form(tmp_path):
    exe = tmp_path / "closest"
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", f"-I{REPO / 'kami-hair-solver_gb300' / 'csrc'}",
                    str(REPO / "tests" / "native" / "test_closest_parts.cpp"), "-o", str(exe)], check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True)
    print(out.stdout)
    assert out.returncode == 0 and "PASS" in out.stdout, out.stdout + out.stderr
