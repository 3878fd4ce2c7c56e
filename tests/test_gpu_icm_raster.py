"""Raster-order ICM in one launch against the oracle, label for label: grids
around the four-row strips and the four-step chunks, label counts around the
lanes' chunks and beyond the kernel (130: one launch per diagonal), several
iterations (neighbouring strips' mailboxes reused)."""
import numpy as np
import pytest

from gridinfcuda_gb300 import synth

pytestmark = pytest.mark.gpu


def _run(ginf, orc, W, H, L, iters, dt=np.float32, model=synth.TRUNC_LINEAR, **opt):
    P = synth.random_problem(W, H, L, 7 * W + H + L, model=model, dtype=dt, scale=1.0 if dt is np.float32 else 10,
                             trunc=2.5 if dt is np.float32 else 20, cost_max=4.0 if dt is np.float32 else 40)
    init = np.random.RandomState(W * H + L).randint(0, L, (H, W)).astype(np.int32)
    want = orc.icm(P.D, P.V, init, iters, asynchronous=True)
    got = ginf.decode_icm(P.D, P.V, P.model, init, iters, asynchronous=True, **opt)
    assert np.array_equal(got, want), (W, H, L, iters)


@pytest.mark.parametrize("H", [3, 4, 5, 6, 7, 10, 11, 35])
def test_strip_and_chunk_edges(ginf, orc, H):
    for W in (3, 4, 5, 6, 9, 10, 33):
        for iters in (1, 2, 5):
            _run(ginf, orc, W, H, 8, iters)


@pytest.mark.parametrize("L", [2, 5, 16, 31, 32, 33, 64, 65, 100, 128, 130])
def test_label_counts_and_types(ginf, orc, L):
    _run(ginf, orc, 41, 23, L, 3)
    _run(ginf, orc, 41, 23, L, 3, dt=np.int32)
    _run(ginf, orc, 41, 23, L, 3, model=synth.EXPLICIT)
    if L <= 65:
        _run(ginf, orc, 41, 23, L, 2, compute_type=ginf.F64, dt=np.int32)


def test_many_strips(ginf, orc):
    _run(ginf, orc, 150, 700, 16, 4)
    _run(ginf, orc, 700, 90, 20, 4, dt=np.int32)


def test_bad_labels_are_reported(ginf):
    P = synth.random_problem(12, 9, 4, 1)
    for y, x in ((0, 5), (8, 5), (4, 0), (4, 11), (4, 5)):
        init = np.zeros((9, 12), np.int32)
        init[y, x] = 4
        with pytest.raises(ginf.GinfError) as e:
            ginf.decode_icm(P.D, P.V, P.model, init, 2, asynchronous=True)
        assert e.value.status == ginf.ERR_INVALID_ARGUMENT


@pytest.mark.parametrize("where", ["cost inf", "cost -inf", "table inf", "table -inf", "cost -0"])
def test_extreme_costs(ginf, orc, where):
    """Infinite costs and table entries (no sum is NaN) and signed zeros: -inf
    leaves the kernel's fast form for the chunks that hold it."""
    for L in (7, 32, 70):
        P = synth.random_problem(37, 21, L, L)
        D, V = np.round(P.D).astype(np.float32), P.V.copy()
        value = np.float32({"inf": np.inf, "-inf": -np.inf, "-0": -0.0}[where.split()[1]])
        if where.startswith("cost"):
            D[::3, 2::5, 1::4] = value
            if value == np.inf:
                D[:, 4, 6] = value  # a node with no finite label
        else:
            V[3 + L * 2] = value
        init = np.random.RandomState(L).randint(0, L, (21, 37)).astype(np.int32)
        want = orc.icm(D, V, init, 3, asynchronous=True)
        assert np.array_equal(ginf.decode_icm(D, V, synth.EXPLICIT, init, 3, asynchronous=True), want), L
