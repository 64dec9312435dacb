"""The network's gradients at batches around the tiles and chunks of their
products, row by row: the weights' and biases' sums run over the rows of two
operands that are transposed as they are staged and cut into slices.

* every row's outputs are its targets but one row's: the gradient is that row's
  alone, so a row that is lost, taken twice or paired with another shows whole;
* distinct rows and targets, against the restatement in 64 bits with the same
  BF16 roundings (oracle/surrogate_ref.py)."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _batch(S, rows):
    x, t = S.training_data(2 * rows + 64, 0, seed=31 + rows)
    assert x.shape[0] >= rows
    return x[:rows].contiguous(), t[:rows].contiguous()


@pytest.mark.parametrize("rows", [1, 127, 128, 129, 4095, 8191])
def test_one_row_counts(gpu, rows):
    """The row's error is some 30 in standardised units, the others' what their
    targets lose in single precision, at most 2e-6 each: 8 191 of them below
    1e-3 of it.  The row's own gradient in 64 bits differs by dY's and the
    three dZ's rounding to BF16, 2^-9 on either side for each."""
    from oracle import surrogate_ref as R
    from photic_gb300 import surrogate as S
    net = S.Surrogate(seed=5)
    x, _ = _batch(S, rows)
    own = net.infer(x)
    p = net.params().astype(np.float64)
    std = torch.tensor(R.OUT_STD, device="cuda")
    for j in sorted({0, 7, 8, 63, 64, 127, 128, rows // 2, rows - 1}):
        if j >= rows:
            continue
        t = own.clone()
        t[j] += 30.0 * std
        got = net.grads(x, t)[0].double().cpu().numpy() * rows
        want, _ = R.grads(p, x[j:j + 1].cpu().numpy(), t[j:j + 1].cpu().numpy())
        for k, (o, n) in R.OFF.items():
            d = np.linalg.norm(got[o:o + n] - want[o:o + n])
            assert d <= (4 * 2.0 ** -8 + 1e-3) * np.linalg.norm(want[o:o + n]), (j, k)
    net.close()


@pytest.mark.parametrize("rows", [1, 127, 128, 129, 4095, 8191])
def test_distinct_rows_match_the_restatement(gpu, rows):
    """Single-precision sums of 128 products move a value by at most 2^-17,
    which takes one in 2^8 to the next BF16 number, 2^-8 away: 2^-12 of a
    tensor's norm for each of the eight roundings on the way to a gradient.
    2^-6 leaves a factor of eight for gradients that cancel over the rows."""
    from oracle import surrogate_ref as R
    from photic_gb300 import surrogate as S
    net = S.Surrogate(seed=5)
    x, t = _batch(S, rows)
    got = net.grads(x, t)[0].double().cpu().numpy()
    want, _ = R.grads(net.params().astype(np.float64), x.cpu().numpy(), t.cpu().numpy())
    for k, (o, n) in R.OFF.items():
        d = np.linalg.norm(got[o:o + n] - want[o:o + n])
        assert d <= 2.0 ** -6 * np.linalg.norm(want[o:o + n]), (k, d)
    net.close()
