"""The inversion with every depth start a queue position of its own (the
allocating entry points: a group of lanes a start, or a lane a start for
more) against the sequential loop over a pixel's starts
(the allocation-free one): the same bits, at sizes around a warp and a block,
with seeds, an early exit at the first start, one that is never met, and the
largest number of starts."""
import ctypes as C

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

WL8 = (412.5, 442.5, 490.0, 510.0, 560.0, 620.0, 665.0, 708.75)
FIELDS = ("depth_f64", "P", "G", "X", "bottom_albedo", "model_error", "rrs_error", "K_min", "iod",
          "evals", "evals_kept", "status", "params")


def _noalloc(gpu, rrs, cfg, seeds):
    from photic_gb300 import _lib as L
    out = gpu.alloc_outputs(rrs.shape[0], rrs.device, FIELDS)
    o = gpu.api._outputs_struct(out)
    c = cfg.to_c()
    L.check(L.lib().photic_invert_batch_noalloc(
        C.byref(c), rrs.data_ptr(), rrs.shape[0], rrs.shape[1], 1,
        None if seeds is None else seeds.data_ptr(), C.byref(o),
        torch.cuda.current_stream().cuda_stream))
    torch.cuda.synchronize()
    return out


@pytest.mark.parametrize("npix,kw,seeded", [
    (1, {}, False),
    (31, {}, True),
    (257, {"early_exit_per_scene": 1e-30}, False),
    (500, {"early_exit_per_scene": 1e9}, False),
    (700, {"hstarts": (10.0,)}, False),
    (300, {"hstarts": tuple(0.7 * (i + 1) for i in range(32)), "kcount": 120}, False),
    (3001, {"seed_step_scale": 0.1}, True),
    (2000, {"precision": "df64"}, False),
    # two and eight bands, a lane a start beyond the groups' sizes
    (90, {"wavelengths": (482.0, 561.0)}, False),
    (130, {"wavelengths": WL8}, False),
    (11003, {}, False),
    (40, {"block_threads": 64}, False),
    # both sides of the line between groups of lanes and lanes (152 SMs)
    (1824, {}, False),
    (1825, {}, False),
    (4865, {"wavelengths": WL8}, False),
    (14593, {"seed_step_scale": 0.1}, True),
    # starts that warps hand on at the end of a launch: eight bands, seeds,
    # and a scene whose first pixels run their starts in sequence
    (20011, {"wavelengths": WL8}, False),
    (60007, {"seed_step_scale": 0.1}, True),
    (530001, {"hstarts": tuple(0.7 * (i + 1) for i in range(32)), "kcount": 30}, False),
])
def test_starts_in_parallel_match_the_sequence(gpu, npix, kw, seeded):
    cfg = gpu.Config(**kw)
    rrs, _ = gpu.generate_scene(npix, seed=91 + npix, config=cfg)
    seeds = None
    if seeded:
        from photic_gb300 import surrogate as S
        seeds, _ = S.heuristic_seeds(rrs, cfg)
        seeds[::3, 0] = float("nan")
    ref = _noalloc(gpu, rrs, cfg, seeds)
    got = gpu.invert(rrs, cfg, seeds=seeds, fields=FIELDS)
    torch.cuda.synchronize()
    for f in FIELDS:
        np.testing.assert_array_equal(got[f].cpu().numpy(), ref[f].cpu().numpy(), err_msg=f)
