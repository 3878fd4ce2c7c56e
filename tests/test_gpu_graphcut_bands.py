"""Alpha-beta swap on wide low grids, whose bands have two rows: a last band of
one row (2700x9: 2, 2, 2, 2, 1, the remaining CTAs idle), of two, and a height
that one band holds."""
import numpy as np
import pytest

from gridinfcuda_gb300 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("W,H", [(2700, 9), (2701, 10), (2700, 11), (2400, 3), (1500, 9)])
def test_short_last_bands(ginf, orc, W, H):
    P = synth.random_problem(W, H, 2, W + H, model=synth.TRUNC_LINEAR, scale=5, trunc=20, dtype=np.int32, cost_max=20)
    init = P.D.argmin(0).astype(np.int32)
    want = orc.alpha_beta(P.D, P.V, init, 1)
    assert (want != init).any()
    assert np.array_equal(ginf.decode_alpha_beta(P.D, P.V, P.model, init, 1), want)
