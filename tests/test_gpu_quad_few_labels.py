"""Truncated-quadratic messages of few labels, where the window of the
transform is as wide as the label range: every radius, the window form against
the O(L^2) min-convolution of the same table, bit for bit."""
import numpy as np
import pytest

from gridinfcuda_gb300 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("store", [0, 1])
@pytest.mark.parametrize("norm", [0, 1])
@pytest.mark.parametrize("scale", [1.0, 0.3, 2.5])
def test_window_messages_equal_min_convolution(ginf, store, norm, scale):
    for L in range(2, 17):
        for radius in sorted({1, 4, 5, L - 2, L - 1} & set(range(1, min(L - 1, 8) + 1))):
            # V(0, radius) < trunc <= V(0, radius + 1)
            P = synth.random_problem(37, 13, L, 10 * L + radius, model=synth.TRUNC_QUAD, scale=scale,
                                     trunc=scale * (radius * radius + radius + 0.5), cost_max=30.0)
            # The FP16 store's exactly quadratic tables of radius up to 4 take another form.
            V = P.V + np.float32(0.5) if store else P.V
            opt = dict(want_msgs=True, rule=ginf.RULE_STANDARD, normalize=norm, store=store)
            lq, mq = ginf.decode_hbp(P.D, V, synth.TRUNC_QUAD, 2, 4, **opt)
            lb, mb = ginf.decode_hbp(P.D, V, synth.EXPLICIT, 2, 4, **opt)
            assert np.array_equal(lq, lb), (L, radius)
            assert np.array_equal(mq.view(np.uint8), mb.view(np.uint8)), (L, radius)
