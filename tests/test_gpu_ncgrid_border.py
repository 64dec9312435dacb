"""Packing a grid that begins with cells without data, a scene's border: the
oracle's compress_2d bit for bit, in little more time than without the border."""
import time

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

SPVAL = -9999.0


@pytest.mark.parametrize("behind", ["random", "run", "ends", "largest_first", "equal", "none",
                                    "negative", "infinite"])
@pytest.mark.parametrize("border", [4000, 4095, 4096, 4097, 70001])
@pytest.mark.parametrize("nan", [False, True])
def test_borders(gpu, port, border, behind, nan):
    from photic_gb300 import ncgrid as N
    rng = np.random.default_rng(border)
    n = border + 6007
    g = np.full(n, np.nan if nan else SPVAL, np.float32)
    v = rng.uniform(0.0, 40.0, 6007).astype(np.float32)
    if behind in ("run", "ends"):
        v = np.linspace(90.0, -30.0, 6007).astype(np.float32)
        if behind == "ends":
            v[-1] = 89.0
    elif behind == "largest_first":
        v[0] = 60.0
    elif behind == "equal":
        v[:] = 3.25
    elif behind == "none":
        v[:] = SPVAL
    elif behind == "negative":
        v = -v - 1.0
    elif behind == "infinite":
        v[0], v[50] = np.inf, -np.inf
    g[border:] = v
    want, off, sc, _ = port.nc_compress(g.reshape(1, n), SPVAL)
    packed, info = N.pack(torch.from_numpy(g).cuda(), SPVAL)
    got = np.frombuffer(packed.cpu().numpy().tobytes(), dtype=">i2").astype(np.int16)
    np.testing.assert_array_equal(got, want.reshape(-1))
    assert np.float32(info["add_offset"]).tobytes() == np.float32(off).tobytes()
    assert np.float32(info["scale_factor"]).tobytes() == np.float32(sc).tobytes()


def test_a_border_costs_little(gpu):
    """4096 x 4096 cells, the first 64 rows missing: another look at the grid's
    beginning, not another four passes (which took five times the time)."""
    from photic_gb300 import ncgrid as N
    g = torch.rand(4096, 4096, generator=torch.Generator(device="cuda").manual_seed(1),
                   device="cuda") * 40
    b = g.clone()
    b[:64] = SPVAL

    def seconds(x):
        t = []
        for _ in range(15):
            torch.cuda.synchronize()
            t0 = time.perf_counter()
            N.pack(x, SPVAL)
            t.append(time.perf_counter() - t0)
        return np.median(t[3:])

    plain, border = seconds(g), seconds(b)
    assert border < 2.5 * plain, (plain, border)
