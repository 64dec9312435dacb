"""The temporal fit captured as a graph on a device with less memory left than
its records of depth starts would take (374 MB here): the graph is captured
without them and replays, with the same bits."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

FREE = 300 << 20
FIELDS = ("depth_f64", "status", "evals")


def test_captured_with_little_memory(gpu):
    cfg = gpu.Config(kcount=40)
    off, theta, rrs, _ = gpu.generate_joint(200_000, seed=8, config=cfg)
    want = {k: v.cpu().numpy() for k, v in
            gpu.joint_invert(off, theta, rrs, cfg, fields=FIELDS).items()}
    gpu.sync()
    torch.cuda.empty_cache()
    gpu.release_workspace()
    held = []
    try:
        while True:
            room = torch.cuda.mem_get_info()[0] - FREE
            if room < (64 << 20):
                break
            held.append(torch.empty(min(room, 16 << 30), dtype=torch.uint8, device="cuda"))
        g = gpu.JointGraph(200_000, rrs.shape[0], cfg, fields=FIELDS)
        got = {k: v.cpu().numpy() for k, v in g.run(off, theta, rrs).items()}
        gpu.sync()
    finally:
        del held
        torch.cuda.empty_cache()
    for k in want:
        np.testing.assert_array_equal(got[k], want[k], err_msg=k)
    # and with memory at hand, records and all
    g = gpu.JointGraph(200_000, rrs.shape[0], cfg, fields=FIELDS)
    got = {k: v.cpu().numpy() for k, v in g.run(off, theta, rrs).items()}
    gpu.sync()
    for k in want:
        np.testing.assert_array_equal(got[k], want[k], err_msg=k)
