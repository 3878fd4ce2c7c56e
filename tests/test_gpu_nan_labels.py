"""Labels of nodes whose costs hold NaN.  A node's label comes from four lanes
that take its labels in 16-byte message chunks in turn (with 128 labels in the
split kernel four lanes for each half), each keeping its first value or a
strictly smaller one, then from a pairwise combine; with NaN that partition
decides the label, so the kernels must share it."""
import numpy as np
import pytest

from gridinfcuda_gb300 import synth

pytestmark = pytest.mark.gpu

NONE = 0x7fffffff


def _scan(b, labels):
    """First value, then strictly smaller ones, over the given labels."""
    n = len(b)
    best, label = np.full(n, np.inf, b.dtype), np.full(n, NONE)
    for i in labels:
        take = (label == NONE) | (b[:, i] < best)
        best, label = np.where(take, b[:, i], best), np.where(take, i, label)
    return best, label


def _combine(parts):
    """Butterfly over the lanes' (value, label)."""
    off = 1
    while off < len(parts):
        new = []
        for k in range(len(parts)):
            (b, l), (ob, ol) = parts[k], parts[k ^ off]
            take = (ol != NONE) & ((l == NONE) | (ob < b) | (~(b < ob) & (ol < l)))
            new.append((np.where(take, ob, b), np.where(take, ol, l)))
        parts, off = new, 2 * off
    return parts[0]


def _lanes(b, begin, end, chunk, lanes=4):
    return _combine([_scan(b, [i for i in range(begin, end) if (i - begin) // chunk % lanes == k])
                     for k in range(lanes)])


FORMS = {
    "linear": (synth.TRUNC_LINEAR, {}, 4),
    "linear f16": (synth.TRUNC_LINEAR, {"store": 1}, 8),
    "linear f64": (synth.TRUNC_LINEAR, {"compute_type": 2}, 2),
    "quadratic": (synth.TRUNC_QUAD, {"rule": 1}, 4),
    "quadratic f16": (synth.TRUNC_QUAD, {"rule": 1, "store": 1}, 8),
    "table, reference rule": (synth.EXPLICIT, {}, 4),
    "table, standard rule": (synth.EXPLICIT, {"rule": 1}, 4),
    "table, reference rule f16": (synth.EXPLICIT, {"store": 1}, 8),
    "table, standard rule f16": (synth.EXPLICIT, {"rule": 1, "store": 1}, 8),
}


@pytest.mark.parametrize("form", FORMS)
def test_labels_with_nan_costs(ginf, form):
    """One half-sweep from zero messages, where beliefs are the costs: the full
    kernel (messages asked for) and the labels-only one."""
    model, opt, chunk = FORMS[form]
    W, H = 37, 11
    ys, xs = np.mgrid[1:H - 1, 1:W - 1]
    first = (xs - ((ys & 1) + 1)) % 2 == 0
    for L in (5, 16, 20, 33, 64, 65, 72, 80, 81, 100, 127, 128):
        P = synth.random_problem(W, H, L, 400 + L, model=model, scale=1.0, trunc=14.0)
        D = P.D.copy()
        D[np.random.RandomState(L).rand(*D.shape) < 0.2] = np.nan
        b = D[:, ys[first], xs[first]].T
        if form == "quadratic" and L == 128:
            want = _combine([_lanes(b, 0, 64, 4), _lanes(b, 64, 128, 4)])[1]
        else:
            want = _lanes(b, 0, L, chunk)[1]
        full, _ = ginf.decode_hbp(D, P.V, model, 1, 1, want_msgs=True, **opt)
        only = ginf.decode_hbp(D, P.V, model, 1, 1, **opt)
        assert np.array_equal(full[ys[first], xs[first]], want), L
        assert np.array_equal(only[ys[first], xs[first]], want), L


@pytest.mark.parametrize("form", FORMS)
def test_labels_only_equals_the_full_half_sweep_with_nan(ginf, form):
    model, opt, _ = FORMS[form]
    for L in (5, 24, 64, 65, 100, 128):
        for W, H, iters in ((37, 13, 3), (130, 4, 2)):
            P = synth.random_problem(W, H, L, 300 + L, model=model, scale=1.0, trunc=14.0)
            D = P.D.copy()
            D[L // 3, ::3, 1::4] = np.nan
            D[0, ::4, ::3] = np.nan
            want, _ = ginf.decode_hbp(D, P.V, model, 1, iters, want_msgs=True, **opt)
            got = ginf.decode_hbp(D, P.V, model, 1, iters, **opt)
            assert np.array_equal(got, want), (L, W, H, iters)


@pytest.mark.parametrize("where", ["cost", "table"])
@pytest.mark.parametrize("compute_type,dtype", [(0, np.float32), (2, np.float64)])
def test_raster_icm_with_nan(ginf, where, compute_type, dtype):
    """Raster order, node by node: eight lanes take a node's labels in 16-byte
    cost chunks in turn."""
    W, H, iters, chunk = 19, 14, 2, 16 // np.dtype(dtype).itemsize
    for L in (7, 32, 60):
        P = synth.random_problem(W, H, L, 20 + L)
        rs = np.random.RandomState(L)
        D, V = P.D.copy(), P.V.copy()
        if where == "cost":
            D[rs.rand(*D.shape) < 0.1] = np.nan
        else:
            V[rs.rand(*V.shape) < 0.1] = np.nan
        init = rs.randint(0, L, (H, W)).astype(np.int32)
        got = ginf.decode_icm(D, V, synth.EXPLICIT, init, iters, asynchronous=True, compute_type=compute_type)
        d, v, lab = D.astype(dtype), V.astype(dtype).reshape(L, L), init.copy()
        for _ in range(iters):
            for y in range(1, H - 1):
                for x in range(1, W - 1):
                    c = d[:, y, x]
                    for f in (lab[y + 1, x], lab[y, x + 1], lab[y - 1, x], lab[y, x - 1]):
                        c = c + v[f]
                    lab[y, x] = _lanes(c[None, :], 0, L, chunk, 8)[1][0]
        assert np.array_equal(got, lab), L
