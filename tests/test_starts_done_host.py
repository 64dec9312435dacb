"""The end of a depth start (photic_starts.cuh): one answer for the lanes of a
group, one group that compares the pixel's records, and barriers around the
first lane's look at them.  The header the kernels compile, built for the
host.  No GPU needed."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_records_are_read_behind_a_barrier(tmp_path):
    cxx = shutil.which("g++") or shutil.which("c++")
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if cxx is None or not os.path.exists(nvcc):
        pytest.skip("no C++ compiler or CUDA headers")
    cuda = os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(nvcc))), "include")
    exe = str(tmp_path / "starts_done_host_check")
    r = subprocess.run([cxx, "-O2", "-std=c++17", "-ffp-contract=off", "-pthread", "-I", cuda,
                        "-I", os.path.join(ROOT, "photic_gb300", "csrc"),
                        os.path.join(ROOT, "tests", "starts_done_host_check.cpp"), "-o", exe],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([exe, "300"], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0 and r.stdout.strip().endswith("OK"), r.stdout + r.stderr
