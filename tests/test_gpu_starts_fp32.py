"""The single-precision inversion with every depth start a queue position of
its own against its sequential loop over a pixel's starts: beyond 523 266
pixels (32 starts, 1 GiB of records) the first ones of a call run in sequence,
and as a call of their own in parallel.  The same bits."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

WL8 = (412.5, 442.5, 490.0, 510.0, 560.0, 620.0, 665.0, 708.75)
STARTS = tuple(0.7 * (i + 1) for i in range(32))
FIELDS = ("depth_f64", "P", "G", "X", "bottom_albedo", "model_error", "rrs_error", "K_min", "iod",
          "evals", "evals_kept", "status", "params")
IN_PARALLEL = (1 << 30) // (32 * 64 + 4)


@pytest.mark.parametrize("npix,kw,seeded", [
    (1, {}, False),
    (6000, {}, False),
    (6000, {"seed_step_scale": 0.1}, True),
    (3001, {"wavelengths": WL8}, False),
    (2000, {"early_exit_per_scene": 1e9}, False),
])
def test_starts_in_parallel_match_the_sequence(gpu, npix, kw, seeded):
    cfg = gpu.Config(precision="fp32", kcount=60, hstarts=STARTS, **kw)
    rrs, _ = gpu.generate_scene(IN_PARALLEL + npix, seed=91 + npix, config=cfg)
    seeds = part = None
    if seeded:
        from photic_gb300 import surrogate as S
        seeds, _ = S.heuristic_seeds(rrs, cfg)
        seeds[::3, 0] = float("nan")
        part = seeds[:npix].contiguous()
    ref = gpu.invert(rrs, cfg, seeds=seeds, fields=FIELDS)
    got = gpu.invert(rrs[:npix].contiguous(), cfg, seeds=part, fields=FIELDS)
    torch.cuda.synchronize()
    for f in FIELDS:
        np.testing.assert_array_equal(got[f].cpu().numpy(), ref[f][:npix].cpu().numpy(), err_msg=f)
