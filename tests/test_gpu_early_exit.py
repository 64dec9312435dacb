"""Depth starts that run as work items of their own, with an early exit that
about half of the starts meet: starts under way are given up while other warps
still lower the word that says so.  The reference is built from fits of one
start each (a plain fit of one pixel), taken together on the host in the order
of the starts as samodel_optimise_one_bottom_combination does
(model/samodel.c:2380-2405): the same depths, evaluation counts and statuses,
bit for bit."""
import dataclasses

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

WL8 = (412.5, 442.5, 490.0, 510.0, 560.0, 620.0, 665.0, 708.75)
STARTS = (40.0, 30.0, 20.0, 15.0, 10.0, 7.5, 2.5, 1.0)
FIELDS = ("depth_f64", "model_error", "evals", "evals_kept", "status")


def _host(out):
    torch.cuda.synchronize()
    return {k: out[k].cpu().numpy() for k in FIELDS}


def _compare(fit, cfg, scenes, low_share, high_share):
    """fit(cfg) against single-start fits under the median start's cost."""
    one = [_host(fit(dataclasses.replace(cfg, hstarts=(h,), early_exit_per_scene=1e-30)))
           for h in STARTS]
    fitted = (one[0]["status"] & 0xFF) == 0
    me = np.stack([o["model_error"].astype(np.float64) for o in one])
    per_scene = float(np.median((me / scenes)[:, fitted]))
    early = per_scene * scenes.astype(np.float64)
    got = _host(fit(dataclasses.replace(cfg, hstarts=STARTS, early_exit_per_scene=per_scene)))

    n = fitted.size
    lowest, kept = np.full(n, 1.0e4), np.zeros(n, dtype=np.int64)
    total, open_ = np.zeros(n, dtype=np.int64), np.ones(n, dtype=bool)
    sure = fitted.copy()  # model_error is the cost rounded to float: leave ties out
    for k, o in enumerate(one):
        sure &= ~(open_ & ((np.abs(me[k] - early) < 1e-6 * early) |
                           (np.abs(me[k] - lowest) < 1e-6 * lowest)))
        total[open_] += o["evals"][open_]
        better = open_ & (me[k] < lowest)
        lowest[better], kept[better] = me[k][better], k
        open_ &= ~(better & (lowest < early))
    left = open_[sure].mean()
    assert low_share < left < high_share, left  # some pixels exit, some never do
    assert sure.mean() > 0.5 * fitted.mean()
    at = np.arange(n)
    for f in ("depth_f64", "model_error", "evals_kept"):
        want = np.stack([o[f] for o in one])[kept, at]
        if f == "evals_kept":
            want = np.stack([o["evals"] for o in one])[kept, at]
        np.testing.assert_array_equal(got[f][sure], want[sure], err_msg=f)
    np.testing.assert_array_equal(got["evals"][sure], total[sure])
    np.testing.assert_array_equal((got["status"][sure] >> 16) & 0xFF, kept[sure])
    np.testing.assert_array_equal(got["status"][~fitted], one[0]["status"][~fitted])


# groups of lanes a start, lanes a start, and groups that finish what lanes
# have handed on
@pytest.mark.parametrize("npix,kw", [(300, {}), (150, {"wavelengths": WL8}), (11003, {}),
                                     (20011, {"wavelengths": WL8})])
def test_inversion(gpu, npix, kw):
    cfg = gpu.Config(kcount=400, **kw)
    rrs, _ = gpu.generate_scene(npix, seed=17 + npix, config=cfg, mask_frac=0.1)
    _compare(lambda c: gpu.invert(rrs, c, fields=FIELDS), cfg, np.ones(npix), 0.005, 0.995)


@pytest.mark.parametrize("layout", ["reference", "scene_b"])
@pytest.mark.parametrize("npix", [130, 3001])
def test_temporal(gpu, layout, npix):
    cfg = gpu.Config(layout=layout, kcount=300)
    off, theta, rrs, _ = gpu.generate_joint(npix, seed=5 + npix, config=cfg, mask_frac=0.1)
    k = np.diff(off.cpu().numpy())
    _compare(lambda c: gpu.joint_invert(off, theta, rrs, c, fields=FIELDS), cfg, k, 0.005, 0.995)


@pytest.mark.parametrize("kw", [{"n_spatial": 1, "n_bottoms": 1}, {"n_spatial": 2, "n_bottoms": 1},
                                {"n_spatial": 2, "n_bottoms": 3}])
def test_general(gpu, kw):
    cfg = gpu.Config(kcount=300)
    grid = gpu.generate_field(17, 19, seed=23, config=cfg)[0].view(17, 19, 4)
    _compare(lambda c: gpu.region_fit(grid, c, fields=FIELDS, **kw), cfg, np.ones(17 * 19),
             0.005, 0.995)
