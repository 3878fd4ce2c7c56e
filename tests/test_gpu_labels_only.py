"""The last half-sweep without messages, and the stereo cost kernels' ranges."""
import numpy as np
import pytest

from gridinfcuda_gb300 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("model,opt", [
    (synth.TRUNC_LINEAR, {}), (synth.TRUNC_LINEAR, {"store": 1}), (synth.TRUNC_LINEAR, {"compute_type": 2}),
    (synth.TRUNC_QUAD, {"rule": 1}), (synth.EXPLICIT, {}), (synth.EXPLICIT, {"rule": 1, "store": 1})])
def test_labels_equal_the_full_half_sweep(ginf, model, opt):
    """Asking for the messages keeps the full last half-sweep: same labels
    either way, at the edges of the four-lane partition and of the split
    kernel's halves, odd widths, one to three half-sweeps, two levels, with
    tied and infinite costs."""
    for L in (2, 3, 8, 17, 64, 65, 80, 81, 100, 127, 128):
        for W, H, iters in ((37, 13, 3), (3, 5, 2), (130, 4, 1)):
            P = synth.random_problem(W, H, L, 300 + L, model=model, scale=1.0, trunc=14.0)
            D = np.round(P.D * 2) / 2
            D = D.astype(np.float32)
            D[L // 2, 1::3, 2::5] = np.inf
            want, _ = ginf.decode_hbp(D, P.V, model, 2, iters, want_msgs=True, **opt)
            got = ginf.decode_hbp(D, P.V, model, 2, iters, **opt)
            assert np.array_equal(got, want), (L, W, H, iters)


@pytest.mark.parametrize("W,H,L", [(1, 1, 1), (257, 5, 17), (300, 3, 16), (1, 70000, 3), (2, 1, 2000)])
def test_stereo_cost_ranges(ginf, W, H, L):
    import torch
    rs = np.random.RandomState(W + L)
    left, right = (rs.uniform(0, 255, (H, W)).astype(np.float32) for _ in range(2))
    pair = synth.StereoPair(left, right, np.zeros((H, W), np.int32))
    out = torch.full((L, H, W), -1.0, device="cuda")
    ginf.stereo_costs(torch.from_numpy(left).cuda(), torch.from_numpy(right).cuda(), L, 0.07, 15.0, out)
    assert np.array_equal(out.cpu().numpy(), synth.cost_volume(pair, L, 0.07, 15.0))
    l8, r8 = left.astype(np.uint8), right.astype(np.uint8)
    out = torch.full((L, H, W), -1, dtype=torch.int32, device="cuda")
    ginf.stereo_costs_u8(torch.from_numpy(l8).cuda(), torch.from_numpy(r8).cuda(), L, 20, out)
    want = np.zeros((L, H, W), np.int32)
    for k in range(L):
        if W > L - 1:
            want[k, :, L - 1:] = np.minimum(np.abs(l8[:, L - 1:].astype(int) - r8[:, L - 1 - k:W - k].astype(int)), 20)
    assert np.array_equal(out.cpu().numpy(), want)
