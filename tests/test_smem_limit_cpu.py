"""Kernels that need more than 48 KB of shared memory raise their limit on every device
that launches them (ciflow_gb300/csrc/smem_limit.cuh), here against a fake runtime of
several devices, and no launch site raises it once per process."""
import glob
import os
import re
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "ciflow_gb300", "csrc")


def test_limit_per_device(tmp_path):
    gxx, nvcc = shutil.which("g++"), shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if gxx is None or not os.path.exists(nvcc):
        pytest.skip("needs g++ and the CUDA headers")
    include = os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(nvcc))), "include")
    exe = str(tmp_path / "test_smem_limit")
    subprocess.run([gxx, "-O1", "-std=c++17", "-I" + include, os.path.join(ROOT, "tests", "cpp", "test_smem_limit.cpp"),
                    "-o", exe], check=True)
    out = subprocess.run([exe], capture_output=True, text=True)
    assert out.returncode == 0, out.stdout


def test_no_limit_is_raised_once_per_process():
    for path in glob.glob(os.path.join(CSRC, "*.cu")):
        text = open(path).read()
        once = re.search(r"static const \w+ \w+ =\s*(?:\[\][^;]*?)?cudaFuncSetAttribute", text)
        assert once is None, (path, once.group(0))
