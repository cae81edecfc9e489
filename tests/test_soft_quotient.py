"""Quotients by a shared divisor on the integer pipes (soft_fp64.cuh quot, mulquot)
against IEEE-754 arithmetic, bit for bit: on the host, and the device build on the GPU."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "code_mge_gb300", "csrc")


def test_host(tmp_path):
    exe = str(tmp_path / "check")
    subprocess.run(["g++", "-std=c++17", "-O2", "-ffp-contract=off", "-fno-fast-math", "-I", CSRC, "-I", HERE,
                    os.path.join(HERE, "soft_quotient_check.cpp"), "-o", exe], check=True)
    r = subprocess.run([exe, "1000000"], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout


@pytest.mark.gpu
def test_device(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    exe = str(tmp_path / "check")
    subprocess.run([nvcc, "-gencode", "arch=compute_103a,code=sm_103a", "-std=c++17", "-O3", "--fmad=false", "-I", CSRC,
                    "-I", HERE, os.path.join(HERE, "soft_quotient_check.cu"), "-o", exe], check=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout
