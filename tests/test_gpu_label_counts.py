"""Half-sweep kernels at the edges of their label buckets (multiples of 8 up to
64 labels, of 16 above): the first and last label count of each, where the
labels whose existence is tested at run time begin and end."""
import numpy as np
import pytest

from gridinfcuda_gb300 import synth

pytestmark = pytest.mark.gpu

EDGES = [2, 7, 8, 9, 15, 17, 23, 24, 25, 31, 33, 40, 41, 48, 49, 56, 57, 63, 65, 79, 80, 81, 96, 97, 111, 112, 113,
         127]


@pytest.mark.parametrize("dtype", ["float32", "int32"])
def test_linear_messages_vs_oracle(ginf, orc, dtype):
    """Labels and messages bit for bit, mean and (FP32) two pyramid levels; a
    37-wide grid leaves a partial last tile."""
    dt = np.dtype(dtype).type
    for L in EDGES:
        P = synth.random_problem(37, 23, L, 500 + L, dtype=dt, scale=1.0 if dt is np.float32 else 10,
                                 trunc=1.7 if dt is np.float32 else 20, cost_max=4.0 if dt is np.float32 else 40)
        want, mw = orc.hbp(P.D, P.V, P.model, 2, 5, want_msgs=True)
        got, mg = ginf.decode_hbp(P.D, P.V, P.model, 2, 5, want_msgs=True)
        assert np.array_equal(got, want), L
        assert np.array_equal(mg.view(np.uint32), mw.view(np.uint32)), L


@pytest.mark.parametrize("W,H,L", [(390, 290, 16), (401, 263, 13), (760, 560, 16), (1032, 640, 16), (1029, 641, 10),
                                   (230, 170, 8), (230, 170, 32), (203, 177, 26)])
def test_warp_half_sweep_block_shapes_vs_oracle(ginf, orc, W, H, L):
    """Grids on either side of the lines between the warp half-sweep's block
    shapes (8, 32 labels; at 16 up to 12288, up to 40960 and above of tiles)."""
    P = synth.random_problem(W, H, L, 77, scale=1.0, trunc=1.7, cost_max=4.0)
    want, mw = orc.hbp(P.D, P.V, P.model, 1, 3, want_msgs=True)
    got, mg = ginf.decode_hbp(P.D, P.V, P.model, 1, 3, want_msgs=True)
    assert np.array_equal(got, want)
    assert np.array_equal(mg.view(np.uint32), mw.view(np.uint32))


@pytest.mark.parametrize("store", [0, 1])
@pytest.mark.parametrize("norm", [0, 1])
@pytest.mark.parametrize("trunc", [25.0, 50.0])
def test_window_messages_equal_min_convolution(ginf, store, norm, trunc):
    """The windowed quadratic transform (radius 4 and 7) against the O(L^2)
    min-convolution of the same table, bit for bit; the FP16 cases' table is
    offset so that it stays on the window form."""
    for L in (9, 17, 24, 33, 48, 57, 65, 80, 81, 100, 112, 113, 127):
        P = synth.random_problem(37, 23, L, 700 + L, model=synth.TRUNC_QUAD, scale=1.0, trunc=trunc, cost_max=30.0)
        V = P.V + np.float32(0.5) if store else P.V
        opt = dict(want_msgs=True, rule=ginf.RULE_STANDARD, normalize=norm, store=store)
        lq, mq = ginf.decode_hbp(P.D, V, synth.TRUNC_QUAD, 2, 4, **opt)
        lb, mb = ginf.decode_hbp(P.D, V, synth.EXPLICIT, 2, 4, **opt)
        assert np.array_equal(lq, lb), L
        assert np.array_equal(mq.view(np.uint8), mb.view(np.uint8)), L


def test_fp16_linear_and_pass_form_vs_fp64(ginf, orc):
    """FP16 store: messages after four half-sweeps within 5e-3 of the largest
    FP64 message (an FP16 message is off by at most 2^-11 of it per half-sweep,
    and each half-sweep sums three of them: (3^4 - 1) / 2 * 2^-11 = 2e-2 if
    every rounding added up; a tenth of that is allowed for, rounded to the
    bound the FP16 store has elsewhere), the minimum subtracted."""
    for model, trunc in ((synth.TRUNC_LINEAR, 1.7), (synth.TRUNC_QUAD, 14.0)):
        for L in (7, 9, 24, 41, 65, 81, 100, 127):
            P = synth.random_problem(37, 23, L, 900 + L, model=model, scale=1.0, trunc=trunc, cost_max=4.0)
            _, want = orc.hbp_f64_std(P.D, P.V, P.model, 1, 4, norm=1, want_msgs=True)
            _, got = ginf.decode_hbp(P.D, P.V, P.model, 1, 4, want_msgs=True, rule=ginf.RULE_STANDARD,
                                     store=ginf.STORE_F16)
            assert np.abs(got - want).max() <= 5e-3 * np.abs(want).max(), (model, L)


def test_batch_label_buckets_equal_single_grid_solves(ginf):
    """One batch over every bucket's edge label counts."""
    import torch
    problems = []
    for L in (2, 8, 9, 17, 25, 33, 40, 41, 49, 56, 57, 63):
        P = synth.random_problem(37, 23, L, 40 + L, trunc=2.5)
        problems.append((torch.from_numpy(P.D).cuda(), torch.from_numpy(P.V).cuda(), P.model))
    want = [ginf.decode_hbp(D, V, m, 1, 7).cpu().numpy() for D, V, m in problems]
    for tile in (8, 16, 32):
        labels = [torch.zeros((23, 37), dtype=torch.int32, device="cuda") for _ in problems]
        with ginf.Batch(problems, labels, 7, tile_nodes=tile, sweeps_per_launch=1) as b:
            b.run()
        for lab, w in zip(labels, want):
            assert np.array_equal(lab.cpu().numpy(), w), tile
