"""Alpha-beta swap on a thread-block cluster against the CPU oracle, bit for
bit: heights around the bands' edges (one to sixteen bands of up to 32 rows,
short last bands), odd and even widths, and a grid too large for the cluster
(one CTA in global memory)."""
import numpy as np
import pytest

from gridinfcuda_gb300 import synth

pytestmark = pytest.mark.gpu


def _check(ginf, orc, W, H, L, seed, iters=1, trunc=20, cost_max=20):
    P = synth.random_problem(W, H, L, seed, model=synth.TRUNC_LINEAR, scale=5, trunc=trunc, dtype=np.int32,
                             cost_max=cost_max)
    init = P.D.argmin(0).astype(np.int32)
    want = orc.alpha_beta(P.D, P.V, init, iters)
    got = ginf.decode_alpha_beta(P.D, P.V, P.model, init, iters)
    assert np.array_equal(got, want), (W, H, L)
    assert H < 3 or (want != init).any()  # energies count interior nodes only


@pytest.mark.parametrize("H", [1, 2, 31, 32, 33, 63, 64, 65, 70, 127, 129, 200, 257, 300])
def test_band_edges(ginf, orc, H):
    for W in (17, 40):
        _check(ginf, orc, W, H, 3, H * 3 + W)


def test_several_passes_and_signed_costs(ginf, orc):
    _check(ginf, orc, 61, 90, 5, 5, iters=3)
    P = synth.random_problem(50, 70, 4, 8, model=synth.POTTS, scale=3, dtype=np.int32, cost_max=12)
    D = P.D - 6  # negative costs: excesses and sink residues of either sign
    init = np.zeros((70, 50), np.int32)
    assert np.array_equal(ginf.decode_alpha_beta(D, P.V, P.model, init, 2), orc.alpha_beta(D, P.V, init, 2))


def test_wide_full_cluster_and_beyond(ginf, orc):
    _check(ginf, orc, 384, 288, 3, 1)
    _check(ginf, orc, 1100, 60, 3, 2)   # columns beyond the 31 chunk masks
    _check(ginf, orc, 420, 320, 2, 3)   # 16 bands do not hold it


def test_labels_outside_the_range_are_reported(ginf):
    P = synth.random_problem(30, 20, 4, 1, dtype=np.int32)
    for v in (-1, 4, 300):
        init = np.zeros((20, 30), np.int32)
        init[7, 11] = v
        with pytest.raises(ginf.GinfError) as e:
            ginf.decode_alpha_beta(P.D, P.V, P.model, init, 1)
        assert e.value.status == ginf.ERR_INVALID_ARGUMENT
