"""The training step's sums over the partial rows (csrc/mlp.cuh) at the edges of their chunks of 256 rows,
blocks of 8 columns and vectors of 2,080 values, against a loop in row order: bit equality
(tests/cpp/ordered_sums_check.cu)."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.mark.gpu
def test_sums_are_those_of_a_loop(tmp_path):
    exe = tmp_path / "ordered_sums_check"
    nvcc = "/usr/local/cuda/bin/nvcc" if os.path.exists("/usr/local/cuda/bin/nvcc") else "nvcc"
    cmd = [nvcc, "-O2", "-std=c++17", "-gencode", "arch=compute_100a,code=sm_100a", "-fmad=false", "-ftz=false",
           "-I", os.path.join(ROOT, "liquidsimulation_b200", "csrc"),
           os.path.join(ROOT, "tests", "cpp", "ordered_sums_check.cu"), "-o", str(exe)]
    if os.path.exists("/usr/bin/g++"):
        cmd[1:1] = ["-ccbin", "/usr/bin/g++"]
    subprocess.run(cmd, check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr
    assert "65 shapes, 0 mismatches" in r.stdout, r.stdout
