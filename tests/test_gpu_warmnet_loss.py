"""The training loss where FP32 sums end: FP64 sums of FP32 squares (four at a
time), element by element in FP64 for a target that is not 16-byte aligned.
With all parameters zero the network's output is x."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _loss(ginf, d, aligned=True):
    """The loss of x = 0 against the target -d."""
    import torch
    n, h, w, L = d.shape
    buf = torch.empty(d.size + 1, device="cuda")
    target = (buf[:-1] if aligned else buf[1:]).view(d.shape)
    target.copy_(torch.from_numpy(-d))
    with ginf.WarmNet(L, 32, seed=1) as net:
        net.set_params(np.zeros(net.num_params(), np.float32))
        return net.gradients(torch.zeros(d.shape, device="cuda"), target)[0]


@pytest.mark.parametrize("L", [16, 32, 64])
@pytest.mark.parametrize("aligned", [True, False])
def test_sum_beyond_fp32(ginf, L, aligned):
    """Squares whose sum exceeds FP32's range and whose mean does not: the
    FP32 squares are off by a unit roundoff each at most (four of them and
    three additions: 7 * 2^-24), and so is the result."""
    d = np.full((2, 9, 140, L), 2e18, np.float32) * np.linspace(0.5, 1, L, dtype=np.float32)
    want = np.mean(d.astype(np.float64) ** 2)
    assert abs(_loss(ginf, d, aligned) - want) <= 8 * 2.0 ** -24 * want


@pytest.mark.parametrize("L", [16, 64])
def test_infinite_and_nan_residuals(ginf, L):
    for aligned in (True, False):
        d = np.ones((1, 5, 40, L), np.float32)
        d[0, 2, 7, 3] = np.inf
        assert _loss(ginf, d, aligned) == np.inf
        d[0, 2, 7, 3] = np.nan
        assert np.isnan(_loss(ginf, d, aligned))
    d[0, 2, 7, 3] = 1e20  # its FP32 square is infinite
    assert _loss(ginf, d) == np.inf


def test_unaligned_target_in_fp64(ginf):
    d = np.zeros((1, 4, 40, 64), np.float32)
    d[0, 1, 2, 3] = 1e20
    want = float(np.float32(1e20)) ** 2 / d.size
    assert abs(_loss(ginf, d, aligned=False) - want) <= 1.01 * 2.0 ** -24 * want
    # Squares that vanish beside their neighbour's in FP32.
    d = np.full((1, 3, 33, 16), 2.0 ** -12.1, np.float32)
    d[..., ::4] = 1
    want = np.mean(d.astype(np.float64) ** 2)
    assert abs(_loss(ginf, d, aligned=False) - want) <= 1.01 * 2.0 ** -24 * want
