"""The network's gradients through the operands that the GEMM transposes as it
stages them, at batches around its tiles and chunks, against the FP64
restatement in plain numpy: the biases' and weights' sums over the rows, which
those products and the column sums form."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows", [1, 127, 128, 129, 4096, 8191])
def test_gradients_scale_with_repeated_rows(gpu, rows):
    """A batch of one row repeated has the gradient of that row: every sum over
    rows is rows x (1 / rows) of the same BF16 terms, so the two agree to the
    FP32 sums' rounding (rows x 2^-24 at worst, 2^-24 log2 rows for the split
    and tree sums; 1e-4 covers both) and to the BF16 rounding of 1 / rows,
    which is exact for powers of two and 2^-9 otherwise."""
    from photic_gb300 import surrogate as S
    net = S.Surrogate(seed=5)
    g = torch.Generator(device="cuda").manual_seed(rows)
    x = 0.002 + 0.02 * torch.rand(1, 6, generator=g, device="cuda")
    x[:, 4:] = torch.tensor([35.0, 0.0], device="cuda")
    t = torch.tensor([[-4.0, -3.0, -5.0, 0.3, 12.0]], device="cuda")
    one, _ = net.grads(x, t)
    many, _ = net.grads(x.repeat(rows, 1).contiguous(), t.repeat(rows, 1).contiguous())
    a, b = one.double().cpu().numpy(), many.double().cpu().numpy()
    tol = 1e-4 if rows & (rows - 1) == 0 else 3 * 2.0 ** -8
    assert np.linalg.norm(a - b) <= tol * np.linalg.norm(a)
    net.close()
