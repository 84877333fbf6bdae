"""Compiles and runs tests/host/test_kquarter.cpp: the quarter-wise K code-word decode of the mma.sync kernel against a
plain per-dim decode, on the CPU, from no outliers at all to nothing else."""
import shutil
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parent.parent


@pytest.mark.parametrize("p_out", [0.0, 0.11, 0.2, 0.35, 0.6, 1.0])
def test_quarter_decode_matches_plain_decode(tmp_path, p_out):
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("no host C++ compiler")
    exe = tmp_path / "test_kquarter"
    subprocess.run([cxx, "-O2", "-std=c++17", "-I", str(ROOT / "bonsai_mojo_1bit_optimization_t4_cuda_b200" / "csrc"),
                    "-o", str(exe), str(ROOT / "tests" / "host" / "test_kquarter.cpp")], check=True)
    res = subprocess.run([str(exe), str(p_out)], capture_output=True, text=True)
    assert res.returncode == 0, res.stdout + res.stderr
    assert res.stdout.startswith("ok")
