"""Half-sweeps whose table holds a -0, a -infinity or a NaN, which take the
reference's comparisons in order: at the edges of the kernels' label ranges, and
not out of proportion slower than other tables."""
import numpy as np
import pytest

from gridinfcuda_gb300 import synth

pytestmark = pytest.mark.gpu

EDGES = [2, 3, 5, 8, 9, 15, 16, 23, 32, 33, 47, 64, 65, 77, 100, 127, 128]


@pytest.mark.parametrize("rule", [0, 1])
@pytest.mark.parametrize("store", [0, 1])
def test_signed_zeros_equal_zeros(ginf, rule, store):
    """A table's zeros as -0 change the form and the zeros' signs alone."""
    for L in EDGES:
        P = synth.random_problem(37, 13, L, 10 + L, model=synth.EXPLICIT, cost_max=4.0)
        V = P.V.copy()
        V[::L + 1] = 0
        W = V.copy()
        W[::L + 1] = np.float32(-0.0)
        opt = dict(want_msgs=True, rule=rule, store=store)
        want, mw = ginf.decode_hbp(P.D, V, P.model, 2, 3, **opt)
        got, mg = ginf.decode_hbp(P.D, W, P.model, 2, 3, **opt)
        assert np.array_equal(got, want) and np.array_equal(mg, mw), L


@pytest.mark.parametrize("value", [-0.0, -np.inf, np.nan])
def test_reference_rule_vs_oracle(ginf, orc, value):
    for L in EDGES:
        P = synth.random_problem(37, 13, L, 30 + L, model=synth.EXPLICIT, cost_max=4.0)
        V = P.V.copy()
        V[L // 2 + L * (L - 1)] = value
        _, want = orc.hbp(P.D, V, P.model, 1, 3, want_msgs=True)
        _, got = ginf.decode_hbp(P.D, V, P.model, 1, 3, want_msgs=True)
        nan = np.isnan(want)
        assert np.array_equal(np.isnan(got), nan), L
        assert np.array_equal(got.view(np.uint32)[~nan], want.view(np.uint32)[~nan]), L


@pytest.mark.parametrize("rule,store,L", [(0, 0, 128), (1, 0, 64), (1, 1, 64)])
def test_time_of_a_table_with_signed_zeros(ginf, rule, store, L):
    """At most ten times the time of the same table with ordinary zeros (three
    to four times; a lane per message with its vector in local memory took
    twenty-five and more)."""
    import torch
    D = torch.rand((L, 240, 320), device="cuda") * 4
    ws, times = ginf.Workspace(), []
    for zero in (0.0, -0.0):
        V = torch.rand((L * L,), device="cuda") + 0.1
        V[::L + 1] = zero
        best = float("inf")
        for _ in range(4):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            torch.cuda.synchronize()
            a.record()
            ginf.decode_hbp(D, V, synth.EXPLICIT, 1, 6, workspace=ws, rule=rule, store=store)
            b.record()
            torch.cuda.synchronize()
            best = min(best, a.elapsed_time(b))
        times.append(best)
    assert times[1] < 10 * times[0], times
