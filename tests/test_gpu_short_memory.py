"""The fits on a device with less memory left than their records of depth
starts would take (1 GiB here): fewer records or none, the same bits.

The rest of the device is held by tensors; 900 MB stay free, ample for
anything but the records."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

FREE = 900 << 20
MANY = tuple(0.7 * (i + 1) for i in range(32))


def _plain(gpu):
    # 2 052 B a pixel: 523 000 pixels' records are 1 GiB
    cfg = gpu.Config(kcount=20, hstarts=MANY)
    rrs, _ = gpu.generate_scene(530_001, seed=8, config=cfg)
    return lambda: gpu.invert(rrs, cfg, fields=("depth_f64", "status", "evals"))


def _temporal(gpu):
    # 1 872 B a stack, all or none
    cfg = gpu.Config(kcount=40)
    off, theta, rrs, _ = gpu.generate_joint(560_000, seed=8, config=cfg)
    return lambda: gpu.joint_invert(off, theta, rrs, cfg, fields=("depth_f64", "status", "evals"))


def _general(gpu):
    # 4 368 B a pixel: 245 000 pixels' records are 1 GiB
    cfg = gpu.Config(kcount=70)
    grid = gpu.generate_field(500, 520, seed=8, config=cfg)[0].view(500, 520, 4)
    return lambda: gpu.region_fit(grid, cfg, fields=("depth_f64", "status", "evals"))


@pytest.mark.parametrize("make", [_plain, _temporal, _general])
def test_same_bits_with_little_memory(gpu, make):
    call = make(gpu)
    want = {k: v.cpu().numpy() for k, v in call().items()}
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
        got = {k: v.cpu().numpy() for k, v in call().items()}
        gpu.sync()
    finally:
        del held
        torch.cuda.empty_cache()
    for k in want:
        np.testing.assert_array_equal(got[k], want[k], err_msg=k)
