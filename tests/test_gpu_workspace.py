"""The scratch pool: what it keeps between calls can be given back."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def test_release_workspace_gives_the_memory_back(gpu):
    """The records of 700 000 pixels' eight starts are 361 MB, below the bound
    that the pool keeps."""
    cfg = gpu.Config(kcount=10)
    rrs, _ = gpu.generate_scene(700_000, seed=2, config=cfg)
    gpu.invert(rrs, cfg, fields=("depth",))
    gpu.sync()
    held = torch.cuda.mem_get_info()[0]
    gpu.release_workspace()
    assert torch.cuda.mem_get_info()[0] - held >= 361_000_000
    a = gpu.invert(rrs[:1000].contiguous(), cfg, fields=("depth",))  # and takes new scratch
    gpu.sync()
    assert torch.isfinite(a["depth"]).all()
