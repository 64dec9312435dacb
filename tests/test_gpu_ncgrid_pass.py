"""Packing in one pass over the grid (nc_range_kernel) where its rule about the
leading decreasing run of cells matters, and the wide loads and stores of the
packing and unpacking kernels at odd sizes and odd addresses: bit for bit
against the oracle's compress_2d / decompress_2d."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SPVAL = -9999.0


def _grid(kind, n):
    rng = np.random.default_rng(n)
    g = np.linspace(90.0, -30.0, n).astype(np.float32)  # strictly decreasing
    if kind == "ends":  # the run ends at the last cell
        g[-1] = 95.0
    elif kind == "later_max":
        g[n // 2:] = rng.uniform(-40.0, 20.0, n - n // 2)
    elif kind == "gaps":
        g[rng.random(n) < 0.4] = SPVAL
        g[rng.random(n) < 0.1] = np.nan
    elif kind == "equal":
        g[:] = 3.25
    elif kind == "infinite":
        g[n // 3] = np.inf
    return g


@pytest.mark.parametrize("kind", ["run", "ends", "later_max", "gaps", "equal", "infinite"])
@pytest.mark.parametrize("n", [1, 33, 4095, 4096, 4097, 20011])
def test_leading_runs(gpu, port, kind, n):
    import torch
    from photic_gb300 import ncgrid as N
    g = _grid(kind, n)
    want, off, sc, _ = port.nc_compress(g.reshape(1, n), SPVAL)
    packed, info = N.pack(torch.from_numpy(g).cuda(), SPVAL)
    got = np.frombuffer(packed.cpu().numpy().tobytes(), dtype=">i2").astype(np.int16)
    np.testing.assert_array_equal(got, want.reshape(-1))
    assert np.float32(info["add_offset"]).tobytes() == np.float32(off).tobytes()
    assert np.float32(info["scale_factor"]).tobytes() == np.float32(sc).tobytes()


@pytest.mark.parametrize("n", [7, 4099, 30001])
def test_unaligned_grid_packs_as_the_aligned_one(gpu, n):
    import torch
    from photic_gb300 import ncgrid as N
    g = torch.rand(n + 1, device="cuda") * 40 - 5
    a, ia = N.pack(g[1:], SPVAL)          # on a 4-byte boundary
    b, ib = N.pack(g[1:].clone(), SPVAL)  # on a 256-byte one
    assert torch.equal(a, b) and ia == ib


@pytest.mark.parametrize("nb", [4, 8])
@pytest.mark.parametrize("shift", [0, 2, 4])
@pytest.mark.parametrize("npix", [1, 2, 4097])
def test_unpack_at_odd_sizes_and_addresses(gpu, port, nb, shift, npix):
    import torch
    from photic_gb300 import ncgrid as N
    rng = np.random.default_rng(nb + npix)
    packed, infos, want = [], [], []
    for b in range(nb):
        p = rng.integers(-32768, 32768, npix).astype(np.int16)
        off, sc = float(rng.uniform(-1, 1)), float(rng.uniform(1e-5, 1e-3))
        want.append(port.nc_decompress(p, off, sc, -32768, SPVAL)[0])
        buf = torch.zeros(2 * npix + shift, dtype=torch.uint8, device="cuda")
        buf[shift:] = torch.from_numpy(np.frombuffer(p.astype(">i2").tobytes(), dtype=np.uint8).copy())
        packed.append(buf[shift:])
        infos.append({"ncols": npix, "nrows": 1, "add_offset": off, "scale_factor": sc,
                      "missing_value": -32768, "spval": SPVAL})
    got = N.unpack_bands(packed, infos, npix).cpu().numpy()
    for b in range(nb):
        assert got[:, b].tobytes() == want[b].tobytes(), b
