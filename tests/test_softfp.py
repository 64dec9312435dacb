"""The integer and FP32 forms of double division, square root, product and
comparison (photic_softfp.cuh) and the two-operation constant divisions, bit
for bit against IEEE arithmetic, from the same header the kernels compile."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "photic_gb300", "csrc")


@pytest.fixture(scope="module")
def check(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("softfp") / "softfp_check")
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-I", CSRC, "-o", exe,
                    os.path.join(ROOT, "tests", "softfp_check.cpp")], check=True)
    return exe


@pytest.mark.parametrize("seed", [1, 2, 3])
def test_soft_operations_give_the_ieee_bits(check, seed):
    r = subprocess.run([check, "2000000", str(seed)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
