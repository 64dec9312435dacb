"""Packing a grid whose minimum is zero, of both signs: the offset is the first
zero of the grid, as compress_2d's comparisons leave it, to the bit."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

SPVAL = -9999.0


def _check(port, g):
    from photic_gb300 import ncgrid as N
    want, off, sc, _ = port.nc_compress(g.reshape(1, -1), SPVAL)
    packed, info = N.pack(torch.from_numpy(g).cuda(), SPVAL)
    got = np.frombuffer(packed.cpu().numpy().tobytes(), dtype=">i2").astype(np.int16)
    np.testing.assert_array_equal(got, want.reshape(-1))
    assert np.float32(info["add_offset"]).tobytes() == np.float32(off).tobytes()
    assert np.float32(info["scale_factor"]).tobytes() == np.float32(sc).tobytes()


@pytest.mark.parametrize("signs", [(0.0, -0.0), (-0.0, 0.0), (-0.0, -0.0), (0.0, 0.0)])
@pytest.mark.parametrize("at", [(0, 1), (3, 259), (5000, 5001), (5000, 5256), (70000, 90001)])
@pytest.mark.parametrize("falling", [False, True])
def test_first_zero(gpu, port, signs, at, falling):
    g = np.random.default_rng(5).uniform(1.0, 40.0, 90003).astype(np.float32)
    if falling:  # the general kernels
        g = np.linspace(99.0, 1.0, 90003).astype(np.float32)
    g[list(at)] = signs
    _check(port, g)


@pytest.mark.parametrize("signs", [(0.0, -0.0), (-0.0, 0.0)])
def test_two_cells(gpu, port, signs):
    _check(port, np.array(signs, np.float32))
