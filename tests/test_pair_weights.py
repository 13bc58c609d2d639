"""The kernel weights the device computes by arithmetic (csrc/lsp_device.cuh) against the tables
they restate: every float squared distance below the cutoff and beyond, every float distance, and
infinities, NaN and far values, one pair and two pairs at a time; and the two-pair
distance and direction against the IEEE operations. Bit equality
(tests/cpp/pair_weights_check.cu)."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    exe = tmp_path_factory.mktemp("weights") / "pair_weights_check"
    nvcc = "/usr/local/cuda/bin/nvcc" if os.path.exists("/usr/local/cuda/bin/nvcc") else "nvcc"
    cmd = [nvcc, "-O2", "-std=c++17", "-gencode", "arch=compute_100a,code=sm_100a", "-fmad=false",
           "-prec-div=true", "-prec-sqrt=true", "-ftz=false", "-Xcompiler", "-ffp-contract=off",
           "-I", os.path.join(ROOT, "liquidsimulation_b200", "csrc"),
           os.path.join(ROOT, "tests", "cpp", "pair_weights_check.cu"), "-o", str(exe)]
    if os.path.exists("/usr/bin/g++"):
        cmd[1:1] = ["-ccbin", "/usr/bin/g++"]
    subprocess.run(cmd, check=True)
    return exe


@pytest.mark.gpu
@pytest.mark.parametrize("radius,factor", [(0.0125, 3.2), (0.00459375, 3.2), (0.017, 2.688), (0.031, 3.0)])
def test_weights_are_the_tables_entries(program, radius, factor):
    r = subprocess.run([str(program), str(radius), str(factor)], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr
    assert r.stdout.count(" 0 mismatches") == 5, r.stdout
