"""The shared reciprocal of the solver's divisions (csrc/quotient.hpp): its
refinement on the CPU from starts at the edge of what it allows, and the whole
of it on the GPU against CUDA's and the host's division."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "unblending_b200", "csrc")


def run(cmd, exe):
    subprocess.run(cmd, check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout


def test_refinement_from_the_worst_start(tmp_path):
    exe = tmp_path / "reciprocal_check"
    run(["g++", "-std=c++17", "-O2", "-mfma", "-ffp-contract=off", "-I", CSRC,
         os.path.join(ROOT, "tests", "cpp", "reciprocal_check.cpp"), "-o", str(exe)], exe)


@pytest.mark.gpu
def test_reciprocal_and_quotient_on_the_gpu(tmp_path):
    exe = tmp_path / "reciprocal_gpu"
    nvcc = os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "bin", "nvcc")
    run([nvcc, "-std=c++17", "-O3", "--fmad=false", "-gencode", "arch=compute_100a,code=sm_100a", "-I", CSRC,
         os.path.join(ROOT, "tests", "cpp", "reciprocal_gpu.cu"), "-o", str(exe)], exe)
