"""The single-scene kernels' Nelder-Mead (photic_nmpixel.cuh), compiled for the
host from the same source, reproduces the oracle's nelmin (the restatement of
model/asa047.c:10-502) bit for bit, its integer centroid sums the double ones.
No GPU needed."""
import pytest

from test_nm_host import _build, _run_ok


@pytest.mark.parametrize("seed", [1, 2])
def test_pixel_state_machine_matches_oracle_nelmin(tmp_path, port, seed):
    _run_ok(_build(tmp_path, "nmpixel_host_check.cpp"), "600", str(seed))
