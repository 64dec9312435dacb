"""The temporal fit's launch bounds the blocks resident on an SM for few
pixels (one block, two, three, none): the bound never reaches the results.
Pixel counts on both sides of each of its lines, against a launch whose shape
is given (no bound); the same bits, for both layouts."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("layout", ["reference", "scene_b"])
@pytest.mark.parametrize("per_sm", [1, 5, 48, 160])
def test_bounded_residency_same_bits(gpu, layout, per_sm):
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    for npix in (per_sm * sms, per_sm * sms + 1):
        # a small budget of evaluations: the lines are of the launch only
        kw = dict(layout=layout, kcount=60)
        off, theta, rrs, _ = gpu.generate_joint(npix, seed=7 + npix, config=gpu.Config(**kw),
                                                mask_frac=0.1)
        got = gpu.joint_invert(off, theta, rrs, gpu.Config(**kw))
        ref = gpu.joint_invert(off, theta, rrs, gpu.Config(blocks_per_sm=32, **kw))
        torch.cuda.synchronize()
        for f in ref:
            np.testing.assert_array_equal(got[f].cpu().numpy(), ref[f].cpu().numpy(), err_msg=f)
