"""The lookup-table loops with a chain for every pixel (the default for scenes
of few pixels), which run as plain fits with their starts in parallel, against
the chain kernels: an empirical depth grid without a depth keeps those, and
changes nothing but the order of the chains."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _same(a, b):
    for k in a:
        if k in ("order", "chain_stats"):
            continue
        np.testing.assert_array_equal(a[k].cpu().numpy(), b[k].cpu().numpy(), err_msg=k)
    sa = a["chain_stats"][torch.argsort(a["order"])].cpu().numpy()
    sb = b["chain_stats"][torch.argsort(b["order"])].cpu().numpy()
    np.testing.assert_array_equal(sa, sb)


@pytest.mark.parametrize("shape", [(1, 1), (5, 9), (33, 65)])
def test_plain_loop(gpu, shape):
    cfg = gpu.Config.reference_default()
    f, _ = gpu.generate_field(*shape, seed=3, config=cfg)
    none = torch.full((f.shape[0],), -9999.0, device="cuda")
    _same(gpu.lut_invert(f, cfg), gpu.lut_invert(f, cfg, empirical=none))


@pytest.mark.parametrize("kw", [{"n_spatial": 2, "n_bottoms": 3}, {"n_spatial": 1, "n_bottoms": 2},
                                {"n_spatial": 2, "n_bottoms": 1, "scenes": 2}])
def test_general_loop(gpu, kw):
    kw = dict(kw)
    cfg = gpu.Config.reference_default(kcount=600)
    S = kw.pop("scenes", 1)
    g = torch.stack([gpu.generate_field(7, 9, seed=4 + s, config=cfg)[0].view(7, 9, 4)
                     for s in range(S)])
    none = torch.full((63,), -9999.0, device="cuda")
    _same(gpu.region_lut_invert(g, cfg, **kw), gpu.region_lut_invert(g, cfg, empirical=none, **kw))
