"""The work that a user of photic_gb300 has it do, as sized cases.

Every kind goes through a public entry point of ``photic_gb300``; the listed
cases are one size each of the ranges that ``draw`` covers:

* ``invert``: the plain per-pixel fit of a scene, from the few hundred pixels
  of a point query to a 1024 x 320 coastal scene; four or eight bands.
* ``seeded``: the warm start of a tile (polished seeds, cold fallbacks first).
* ``joint``: the temporal fit of a stack of two to eight scenes, both layouts.
* ``region``: 3 x 3 neighbourhoods, with one bottom type or with the three that
  the reference mixes by default.
* ``lut`` / ``region_lut``: the reference's pixel loop with its lookup table
  over a coherent scene, at the reference's tolerances.
* ``grads``: one gradient of the warm-start network over a mini-batch.
* ``ncgrid``: a scene's grids packed to the reference's shorts and back.

Sizes are odd where real scenes are: a coast, a tile's edge or a mask leaves no
multiple of a block.
"""
import math

import numpy as np
import torch

import photic_gb300 as pg
from photic_gb300 import ncgrid
from photic_gb300 import surrogate as sg

WL4 = (443.0, 482.0, 561.0, 655.0)
WL8 = (412.5, 442.5, 490.0, 510.0, 560.0, 620.0, 665.0, 708.75)
SPVAL = -9999.0

# cost evaluations a fitted pixel takes, from counting them over these
# distributions; FP64 operations of one evaluation (each exp, division and
# square root as one): 43 a band term and 9 for the rest
EVALS = {"invert": 1100.0, "seeded": 370.0, "joint": 2200.0, "region1": 12000.0,
         "region3": 7600.0, "lut": 470.0, "region_lut": 7600.0}


def _band_flops(terms):
    return 43.0 * terms + 9.0


def listed():
    return [
        # a point query or a validation transect: a few hundred soundings
        {"name": "invert_256", "kind": "invert", "npix": 256, "bands": 4},
        # a whole coastal scene, 15 % of it land or cloud
        {"name": "invert_1024x320", "kind": "invert", "npix": 1024 * 320, "bands": 4},
        # an eight-band sensor's strip
        {"name": "invert_8band", "kind": "invert", "npix": 20011, "bands": 8},
        # one tile of a large scene through the warm start
        {"name": "seeded_tile", "kind": "seeded", "npix": 701 * 997},
        # a temporal stack, the reference's shared bottom
        {"name": "joint_reference", "kind": "joint", "npix": 8009, "layout": "reference"},
        # the same with each scene's own bottom albedo
        {"name": "joint_scene_b", "kind": "joint", "npix": 3001, "layout": "scene_b"},
        # the reference's default call: 3 x 3 regions, sand, seagrass, coral
        {"name": "region_mixture", "kind": "region", "nrows": 41, "ncols": 29, "bottoms": 3},
        # 3 x 3 regions on sand at the plain tolerance
        {"name": "region_sand", "kind": "region", "nrows": 19, "ncols": 23, "bottoms": 1},
        # the reference's pixel loop over a coherent scene
        {"name": "lut_loop", "kind": "lut", "nrows": 509, "ncols": 400},
        # the same loop in the reference's default configuration
        {"name": "region_lut_loop", "kind": "region_lut", "nrows": 24, "ncols": 27},
        # a training step's gradient of the warm-start network
        {"name": "surrogate_grads", "kind": "grads", "rows": 8192},
        # four band grids of a large scene to the file format's shorts and back
        {"name": "ncgrid_4096", "kind": "ncgrid", "nrows": 4096, "ncols": 4096, "bands": 4},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["invert", "invert", "seeded", "joint", "region", "lut", "region_lut",
                       "grads", "ncgrid"])
    if kind == "invert":
        bands = rng.choice([4, 4, 8])
        return {"kind": kind, "npix": _log_int(rng, 200, 327680 if bands == 4 else 50000),
                "bands": bands}
    if kind == "seeded":
        return {"kind": kind, "npix": _log_int(rng, 2000, 700000)}
    if kind == "joint":
        return {"kind": kind, "npix": _log_int(rng, 200, 9000),
                "layout": rng.choice(["reference", "scene_b"])}
    if kind == "region":
        return {"kind": kind, "nrows": rng.randint(7, 41), "ncols": rng.randint(7, 29),
                "bottoms": rng.choice([1, 2, 3])}
    if kind == "lut":
        return {"kind": kind, "nrows": rng.randint(64, 512), "ncols": rng.randint(64, 512)}
    if kind == "region_lut":
        return {"kind": kind, "nrows": rng.randint(9, 30), "ncols": rng.randint(9, 30)}
    if kind == "grads":
        return {"kind": kind, "rows": _log_int(rng, 256, 65536)}
    return {"kind": kind, "nrows": _log_int(rng, 120, 4096), "ncols": _log_int(rng, 120, 4096),
            "bands": rng.choice([1, 3, 4, 4, 8])}


# ---------------------------------------------------------------------------
# Inputs
# ---------------------------------------------------------------------------
def _mlp_params(seed):
    """Weights of the 6-128-128-128-5 network (inputs padded to 16 columns,
    outputs to 16 rows), in the order the framework keeps them: each layer's
    weights, then its biases."""
    r = np.random.RandomState(seed % (2 ** 32))
    parts = []
    for rows, cols, vr, vc in ((128, 16, 128, 6), (128, 128, 128, 128), (128, 128, 128, 128),
                               (16, 128, 5, 128)):
        a = 1.0 / math.sqrt(vc)
        w = np.zeros((rows, cols), np.float32)
        w[:vr, :vc] = r.uniform(-a, a, (vr, vc))
        b = np.zeros(rows, np.float32)
        b[:vr] = r.uniform(-0.05, 0.05, vr)
        parts += [w.ravel(), b]
    return np.concatenate(parts)


def _mlp_batch(rows, seed):
    """Spectra and targets with the prior's spread."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    u = torch.rand(rows, 9, generator=g, device="cuda")
    x = torch.empty(rows, 6, device="cuda")
    x[:, :4] = 0.002 + 0.02 * u[:, :4]
    x[:, 4] = 35.0
    x[:, 5] = 0.0
    t = torch.stack([-5.3 + 3.0 * u[:, 4], -5.3 + 3.7 * u[:, 5], -6.9 + 3.9 * u[:, 6],
                     0.05 + 0.45 * u[:, 7], 0.5 + 24.5 * u[:, 8]], 1)
    return x, t.contiguous()


def _grids(case, seed):
    """Band grids [nrows, ncols] of a smooth scene with noise and 10 % missing
    cells, as reflectances."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    nr, nc = case["nrows"], case["ncols"]
    y = torch.linspace(0, 6.0, nr, device="cuda")[:, None]
    x = torch.linspace(0, 9.0, nc, device="cuda")[None, :]
    out = []
    for b in range(case["bands"]):
        ph = torch.rand(2, generator=g, device="cuda") * 6.0
        v = 0.012 + 0.008 * torch.sin(x + ph[0]) * torch.cos(y + ph[1])
        v = v + 2e-4 * torch.randn(nr, nc, generator=g, device="cuda")
        v[torch.rand(nr, nc, generator=g, device="cuda") < 0.1] = SPVAL
        out.append(v.contiguous())
    return out


def _stacks(npix, seed, cfg):
    """Stacks of 2..8 scenes: each count as often as the others, in a random
    order of the pixels, the scenes those of the generator's stacks of 8."""
    _, theta, rrs, _ = pg.generate_joint(npix, seed=seed, config=cfg, kmin=8, kmax=8)
    g = torch.Generator(device="cuda").manual_seed(seed)
    k = (2 + torch.arange(npix, device="cuda") % 7)[torch.randperm(npix, generator=g,
                                                                   device="cuda")]
    offsets = torch.zeros(npix + 1, dtype=torch.int32, device="cuda")
    offsets[1:] = torch.cumsum(k, 0, dtype=torch.int32)
    keep = (torch.arange(8, device="cuda")[None, :] < k[:, None]).view(-1)
    return {"offsets": offsets, "theta": theta[keep].contiguous(), "rrs": rrs[keep].contiguous()}


def _loop_outputs(out, npix):
    """The loop's outputs, the order and the chains' statistics (as long as
    the scene's unmasked pixels are many) filled up to the pixel count."""
    for k in ("order", "chain_stats"):
        v = out[k]
        full = torch.full((npix,) + v.shape[1:], -1, dtype=v.dtype, device=v.device)
        full[:v.shape[0]] = v
        out[k] = full
    return out


def prepare(case, seed):
    kind = case["kind"]
    s = {"case": case}
    if kind == "invert":
        s["cfg"] = pg.Config(wavelengths=WL4 if case["bands"] == 4 else WL8)
        s["rrs"], _ = pg.generate_scene(case["npix"], seed=seed, config=s["cfg"],
                                        with_truth=False)
    elif kind == "seeded":
        s["cfg"] = pg.Config(seed_step_scale=0.1)
        s["rrs"], _ = pg.generate_scene(case["npix"], seed=seed, config=s["cfg"],
                                        with_truth=False)
    elif kind == "joint":
        s["cfg"] = pg.Config(layout=case["layout"])
        s.update(_stacks(case["npix"], seed, s["cfg"]))
    elif kind in ("region", "region_lut", "lut"):
        s["cfg"] = pg.Config() if kind == "region" and case["bottoms"] == 1 else \
            pg.Config.reference_default()
        nr, nc = case["nrows"], case["ncols"]
        rrs, _ = pg.generate_field(nr, nc, seed=seed, config=s["cfg"], with_truth=False)
        s["rrs"] = rrs if kind == "lut" else rrs.view(nr, nc, 4)
    elif kind == "grads":
        s["net"] = sg.Surrogate(seed=1)
        s["net"].set_params(_mlp_params(seed))
        s["x"], s["t"] = _mlp_batch(case["rows"], seed)
    else:
        s["grids"] = _grids(case, seed)
    return s


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "invert":
        return pg.invert(state["rrs"], state["cfg"])
    if kind == "seeded":
        seeds, resid = sg.heuristic_seeds(state["rrs"], state["cfg"])
        out = pg.invert(state["rrs"], state["cfg"], seeds=seeds, order=pg.fallbacks_first(seeds))
        return {"fit": out, "seeds": seeds, "resid": resid}
    if kind == "joint":
        return pg.joint_invert(state["offsets"], state["theta"], state["rrs"], state["cfg"])
    if kind == "region":
        return pg.region_fit(state["rrs"], state["cfg"], n_spatial=2, n_bottoms=case["bottoms"])
    if kind == "lut":
        return _loop_outputs(pg.lut_invert(state["rrs"], state["cfg"]), state["rrs"].shape[0])
    if kind == "region_lut":
        return _loop_outputs(pg.region_lut_invert(state["rrs"], state["cfg"]),
                             case["nrows"] * case["ncols"])
    if kind == "grads":
        g, loss = state["net"].grads(state["x"], state["t"])
        return {"grad": g, "loss": loss}
    packed, infos = [], []
    for grid in state["grids"]:
        p, i = ncgrid.pack(grid, SPVAL)
        packed.append(p)
        infos.append(i)
    rrs = ncgrid.unpack_bands(packed, infos, case["nrows"] * case["ncols"])
    return {"packed": packed, "rrs": rrs,
            "offset": [i["add_offset"] for i in infos],
            "scale": [i["scale_factor"] for i in infos]}


def work(case):
    kind = case["kind"]
    if kind in ("invert", "seeded"):
        nb = case.get("bands", 4)
        fits = 0.85 * case["npix"] * EVALS[kind]
        # spectra in; ten products and six parameters out (and the seeds)
        b = case["npix"] * (4 * nb + 56 + 48 + (52 if kind == "seeded" else 0))
        return {"bytes": b, "flops": fits * _band_flops(nb)}
    if kind == "joint":
        n_obs = 5 * case["npix"]
        return {"bytes": n_obs * (16 + 8 + 12) + case["npix"] * 52,
                "flops": case["npix"] * EVALS["joint"] * _band_flops(20)}
    if kind in ("region", "region_lut", "lut"):
        n = case["nrows"] * case["ncols"]
        if kind == "lut":
            return {"bytes": n * (16 + 56 + 48 + 16), "flops": 0.9 * n * EVALS["lut"] * _band_flops(4)}
        key = "region_lut" if kind == "region_lut" else ("region1" if case["bottoms"] == 1 else "region3")
        return {"bytes": n * (16 + 72), "flops": 0.9 * n * EVALS[key] * _band_flops(36)}
    if kind == "grads":
        mac = 6 * 128 + 2 * 128 * 128 + 5 * 128
        return {"bytes": case["rows"] * 44 + 37000 * 4 * 2,
                "flops": case["rows"] * 2.0 * (2 * mac + 2 * 128 * 128 + 5 * 128)}
    n = case["nrows"] * case["ncols"] * case["bands"]
    return {"bytes": n * (4 + 2 + 2 + 4), "flops": 6.0 * n}


# ---------------------------------------------------------------------------
# 64-bit values
# ---------------------------------------------------------------------------
def _exact_grads(case, seed):
    p = _mlp_params(seed)
    x, t = _mlp_batch(case["rows"], seed)
    x, t = x.double(), t.double()
    dev = x.device
    mean = torch.tensor([0.011, 0.012, 0.010, 0.0035, 35.0, 0.0], dtype=torch.float64, device=dev)
    std = torch.tensor([0.006, 0.007, 0.007, 0.004, 10.0, 10.0], dtype=torch.float64, device=dev)
    omean = torch.tensor([-3.80, -3.45, -4.95, 0.275, 12.75], dtype=torch.float64, device=dev)
    ostd = torch.tensor([0.865, 1.065, 1.129, 0.130, 7.07], dtype=torch.float64, device=dev)
    shapes = ((128, 16), (128, 128), (128, 128), (16, 128))
    leaves, o = [], 0
    for r, c in shapes:
        leaves.append(torch.tensor(p[o:o + r * c], dtype=torch.float64, device=dev).view(r, c)
                      .requires_grad_())
        o += r * c
        leaves.append(torch.tensor(p[o:o + r], dtype=torch.float64, device=dev).requires_grad_())
        o += r
    a = torch.zeros(x.shape[0], 16, dtype=torch.float64, device=dev)
    a[:, :6] = (x - mean) / std
    for k in range(4):
        a = a @ leaves[2 * k].T + leaves[2 * k + 1]
        if k < 3:
            a = torch.nn.functional.silu(a)
    loss = ((a[:, :5] - (t - omean) / ostd) ** 2).mean()
    loss.backward()
    return {"grad": torch.cat([v.grad.reshape(-1) for v in leaves]),
            "loss": loss.detach().reshape(1)}


def _exact_ncgrid(case, seed):
    """Scale, offset and the unpacked cells; the packed bytes are whole."""
    cells, offs, scales = [], [], []
    for grid in _grids(case, seed):
        v = grid.double()
        ok = grid != SPVAL
        lo, hi = v[ok].min(), v[ok].max()
        scale = (hi - lo) / 32767.0
        q = torch.round((v - lo) / scale)
        cells.append(torch.where(ok, q * scale + lo, torch.full_like(v, SPVAL)).view(-1))
        offs.append(float(lo))
        scales.append(float(scale))
    return {"packed": [None] * len(cells), "rrs": torch.stack(cells, 1),
            "offset": offs, "scale": scales}


def exact(case, seed):
    """The fits have no value in plain 64-bit torch: each is the end of a
    Nelder-Mead path of hundreds to thousands of dependent evaluations."""
    if case["kind"] == "grads":
        return _exact_grads(case, seed)
    if case["kind"] == "ncgrid":
        return _exact_ncgrid(case, seed)
    return None
