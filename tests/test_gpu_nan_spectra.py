"""Pixels whose spectrum has a NaN (the reference masks its nodata value and
negative cells, not those): their cost is NaN at every point, so every start
runs to its evaluation limit.  The oracle's evaluations, depths and statuses,
in no more time an evaluation than others take."""
import numpy as np
import pytest
import torch

from test_gpu_starts import _noalloc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("noalloc", [False, True])
@pytest.mark.parametrize("npix,kcount", [(40, 2000), (9000, 150)])
def test_single_scene_matches_the_oracle(gpu, port, noalloc, npix, kcount):
    cfg = gpu.Config(kcount=kcount)
    rrs, _ = gpu.generate_scene(npix, seed=6, config=cfg, mask_frac=0.1)
    clean = rrs.clone()
    at = torch.arange(0, npix, 7)
    for b in range(4):
        rrs[at[b::4], b] = float("nan")
    run = (lambda r: _noalloc(gpu, r, cfg, None)) if noalloc else (lambda r: gpu.invert(r, cfg))
    out = {k: v.cpu().numpy() for k, v in run(rrs).items()}
    ref = {k: v.cpu().numpy() for k, v in run(clean).items()}
    odd = np.zeros(npix, dtype=bool)
    odd[at.numpy()] = True
    for k in out:  # the other pixels do not notice
        if k != "depth":
            np.testing.assert_array_equal(out[k][~odd], ref[k][~odd], err_msg=k)
    want = port.invert_batch(rrs.cpu().numpy()[odd], kcount=kcount)
    fit = (out["status"][odd] & 0xFF) == 0
    assert fit.any()
    np.testing.assert_array_equal(out["evals"][odd][fit], want[fit, 7].astype(np.int32))
    np.testing.assert_array_equal(out["depth_f64"][odd][fit], want[fit, 0])
    assert np.isnan(out["model_error"][odd][fit]).all()
    assert np.isnan(want[fit, 2]).all()


@pytest.mark.parametrize("what", ["temporal", "temporal_8_bands", "general"])
def test_every_start_runs_to_its_limit(gpu, what):
    """The evaluations of a pixel are those of one start times the starts, and
    its neighbours are as they are without it."""
    starts = (40.0, 10.0, 2.5)
    kw = {"kcount": 200}
    if what == "temporal_8_bands":
        kw["wavelengths"] = (412.5, 442.5, 490.0, 510.0, 560.0, 620.0, 665.0, 708.75)

    def fit(hstarts, nan):
        cfg = gpu.Config(hstarts=hstarts, **kw)
        if what == "general":
            g = gpu.generate_field(9, 9, seed=3, config=cfg, mask_frac=0.0)[0].view(9, 9, 4)
            if nan:
                g[4, 4, 1] = float("nan")
            out = gpu.region_fit(g.contiguous(), cfg, n_spatial=1, n_bottoms=2)
        else:
            off, theta, rrs, _ = gpu.generate_joint(81, seed=3, config=cfg)
            if nan:
                rrs[int(off[40]), 1] = float("nan")
            out = gpu.joint_invert(off, theta, rrs, cfg)
        return {k: out[k].cpu().numpy() for k in ("evals", "depth_f64", "model_error", "status")}

    one, all_, clean = fit(starts[:1], True), fit(starts, True), fit(starts, False)
    assert one["evals"][40] >= 200
    assert all_["evals"][40] == 3 * one["evals"][40]
    assert np.isnan(all_["model_error"][40])
    for k in clean:
        np.testing.assert_array_equal(np.delete(all_[k], 40), np.delete(clean[k], 40), err_msg=k)


def test_a_nan_evaluation_costs_what_another_does(gpu):
    """One pixel alone, its eight starts in sequence, run to their limits: with
    a NaN, and without (no early exit, a variance limit that is never met).  An
    evaluation that is NaN in every term takes the terms once."""

    def microseconds(nan):
        cfg = gpu.Config(kcount=800, reqmin=1e-300, early_exit_per_scene=0.0)
        rrs, _ = gpu.generate_scene(1, seed=3, config=cfg, mask_frac=0.0)
        if nan:
            rrs[0, 2] = float("nan")
        t = []
        for _ in range(5):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record()
            out = _noalloc(gpu, rrs, cfg, None)
            b.record()
            torch.cuda.synchronize()
            t.append(a.elapsed_time(b))
        return 1e3 * np.median(t) / out["evals"].item()

    clean, nan = microseconds(False), microseconds(True)
    assert nan < 1.2 * clean, (nan, clean)
