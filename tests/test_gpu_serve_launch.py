"""A batch of the serving loop is launched without waiting for it: the loop
sees arrivals and other batches' completions while it runs."""
import time

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def test_launch_does_not_wait(gpu):
    from photic_gb300 import serve as S
    ex = S.GpuTileExecutor(config=gpu.Config())
    sides = (640, 31, 300)

    def tiles(seed):
        reqs = [S.TileRequest(rid=i, side=n, arrival=0.0, seed=seed + i)
                for i, n in enumerate(sides)]
        for r in reqs:
            ex.admit(r)
        torch.cuda.synchronize()
        return reqs

    warm = tiles(1)  # kernels loaded, memory at hand
    ex.collect(ex.launch(warm), warm)
    ex.n_launched = 0  # the same stream, whose memory torch keeps apart
    reqs = tiles(2)
    t0 = time.perf_counter()
    torch.cuda.set_sync_debug_mode("error")  # an operation that waits raises
    try:
        tok = ex.launch(reqs)
    finally:
        torch.cuda.set_sync_debug_mode("default")
    t1 = time.perf_counter()
    running = not ex.done(tok)
    ex.collect(tok, reqs)
    t2 = time.perf_counter()
    # 500 000 cold fits take a few hundred milliseconds
    assert running and t1 - t0 < 0.5 * (t2 - t0), (t1 - t0, t2 - t0)
    for r in reqs:
        rrs, _ = gpu.generate_scene(r.npix, seed=r.seed, config=ex.cfg, mask_frac=ex.mask_frac,
                                    with_truth=False)
        out = gpu.invert(rrs, ex.cfg, fields=("depth", "status"))
        st = out["status"].cpu().numpy()
        fitted = (st & 0xFF) == 0
        np.testing.assert_array_equal(r.state["depth"].numpy(), out["depth"].cpu().numpy())
        assert r.fitted == fitted.sum()
        assert r.converged == (fitted & ((st >> 8) & 1).astype(bool)).sum()
