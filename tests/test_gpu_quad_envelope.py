"""Truncated-quadratic messages whose radius exceeds the window: the lower
envelope, around the kernels' label ranges, against the FP64 oracle, and in time
against the O(L^2) min-convolution of the same table."""
import numpy as np
import pytest

from gridinfcuda_gb300 import synth

pytestmark = pytest.mark.gpu

EDGES = [11, 12, 15, 16, 17, 24, 31, 32, 33, 48, 63, 64, 65, 100, 127, 128]


def _problem(L, scale, trunc):
    return synth.random_problem(37, 13, L, L, model=synth.TRUNC_QUAD, scale=scale, trunc=trunc, cost_max=30.0)


@pytest.mark.parametrize("norm", [0, 1])
@pytest.mark.parametrize("scale,trunc", [(1.0, 90.0), (0.3, 60.0), (1.0, 1e6)])
def test_messages_vs_fp64_oracle(ginf, orc, norm, scale, trunc):
    """FP64 within 1e-12 of the oracle.  FP32, three half-sweeps: an output's
    few roundings are of 2^-24 of the largest value each (at most eight), a
    border between two parabolas is off by 2^-24 of the numerator's terms (up to
    s L^2), which the outputs beside it carry at most twice, and a half-sweep
    sums three messages (1 + 3 + 9)."""
    for L in EDGES:
        P = _problem(L, scale, trunc)
        want, mw = orc.hbp_f64_std(P.D, P.V, P.model, 1, 3, norm=norm, want_msgs=True)
        opt = dict(want_msgs=True, rule=ginf.RULE_STANDARD, normalize=norm)
        got, mg = ginf.decode_hbp(P.D, P.V, P.model, 1, 3, compute_type=ginf.F64, **opt)
        assert np.abs(mg - mw).max() <= 1e-12 * np.abs(mw).max(), L
        assert np.array_equal(got[1:-1, 1:-1], want[1:-1, 1:-1]), L
        _, m32 = ginf.decode_hbp(P.D, P.V, P.model, 1, 3, **opt)
        big = max(np.abs(mw).max(), P.D.max(), P.V.max() if trunc < 1e5 else 0.0)
        tol = 13 * 2.0 ** -24 * (8 * big + 2 * scale * L * L)
        assert np.abs(m32 - mw).max() <= tol, L


def test_fp16_store_vs_fp64_oracle(ginf, orc):
    """Within 5e-3 of the largest message, the FP16 store's bound elsewhere."""
    for L in EDGES:
        P = _problem(L, 1.0, 90.0)
        _, mw = orc.hbp_f64_std(P.D, P.V, P.model, 1, 4, norm=1, want_msgs=True)
        _, mg = ginf.decode_hbp(P.D, P.V, P.model, 1, 4, want_msgs=True, rule=ginf.RULE_STANDARD, store=ginf.STORE_F16)
        assert np.abs(mg - mw).max() <= 5e-3 * np.abs(mw).max(), L


@pytest.mark.parametrize("store,L", [(0, 64), (0, 128), (1, 128)])
def test_time_beside_the_min_convolution(ginf, store, L):
    """At most four times the min-convolution's time (two and a half to three
    times; with every stack array in local memory and generic label counts four
    to seven)."""
    import torch
    D = torch.rand((L, 240, 320), device="cuda") * 20
    i = torch.arange(L, device="cuda", dtype=torch.float32)
    V = torch.clamp((i[:, None] - i[None, :]) ** 2, max=200.0).reshape(-1).contiguous()
    ws, times = ginf.Workspace(), []
    for model in (synth.EXPLICIT, synth.TRUNC_QUAD):
        best = float("inf")
        for _ in range(4):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            torch.cuda.synchronize()
            a.record()
            ginf.decode_hbp(D, V, model, 1, 6, workspace=ws, rule=ginf.RULE_STANDARD, store=store)
            b.record()
            torch.cuda.synchronize()
            best = min(best, a.elapsed_time(b))
        times.append(best)
    assert times[1] < 4 * times[0], times
