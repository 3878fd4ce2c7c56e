"""Half-sweeps with an explicit table (min-convolutions): the reference rule
against the oracle and the standard rule against a float32 numpy restatement,
bit for bit, at the edges of the kernels' label ranges and with the values
that leave the fast form (signed zeros, infinities, NaN)."""
import numpy as np
import pytest

from gridinfcuda_gb300 import synth

pytestmark = pytest.mark.gpu

EDGES = [2, 4, 5, 8, 9, 16, 24, 25, 32, 33, 40, 48, 63, 64, 65, 72, 100, 127, 128]


def _rmin(a, b):
    return np.where(a < b, a, b)  # the second operand on a tie or a NaN


def _standard(D, V, iters, norm_min=False):
    """Standard-rule half-sweeps in D's type: messages [H][W][4][L], slot d
    from the neighbour in direction d, the reference's order of operations."""
    L, H, W = D.shape
    T = D.dtype.type
    D = D.transpose(1, 2, 0)
    V = V.reshape(L, L)  # row j: V(i, j) over i
    m = np.zeros((H, W, 4, L), D.dtype)
    step = ((0, 1), (1, 0), (0, -1), (-1, 0))  # (dx, dy) of S, E, N, W
    ys, xs = np.mgrid[1:H - 1, 1:W - 1]
    for it in range(iters):
        sel = (xs - (((ys + it) & 1) + 1)) % 2 == 0
        y, x = ys[sel], xs[sel]
        b = D[y, x]
        for d in range(4):
            b = b + m[y, x, d]
        for d, (dx, dy) in enumerate(step):
            h = b - m[y, x, d]
            out = V[0][None, :] + h[:, :1]
            for j in range(1, L):
                out = _rmin(out, V[j][None, :] + h[:, j:j + 1])
            if norm_min:
                val = out[:, 0]
                for i in range(1, L):
                    val = _rmin(val, out[:, i])
            else:
                val = np.zeros(len(out), D.dtype)
                for i in range(L):
                    val = val + out[:, i]
                val = val / T(L) if T is np.float32 else np.trunc(val / float(L)).astype(np.int32)
            out = out - val[:, None]
            keep = (y + dy >= 1) & (y + dy <= H - 2) & (x + dx >= 1) & (x + dx <= W - 2)
            m[(y + dy)[keep], (x + dx)[keep], (d + 2) % 4] = out[keep]
    return m


def _inner(m):
    return m[1:-1, 1:-1]


def _problem(L, dtype, seed):
    dt = np.dtype(dtype).type
    return synth.random_problem(37, 13, L, seed, model=synth.EXPLICIT, dtype=dt,
                                cost_max=4.0 if dt is np.float32 else 40)


@pytest.mark.parametrize("dtype", ["float32", "int32"])
def test_reference_rule_vs_oracle(ginf, orc, dtype):
    for L in EDGES:
        P = _problem(L, dtype, 10 + L)
        want, mw = orc.hbp(P.D, P.V, P.model, 2, 3, want_msgs=True)
        got, mg = ginf.decode_hbp(P.D, P.V, P.model, 2, 3, want_msgs=True)
        assert np.array_equal(got, want), L
        assert np.array_equal(mg.view(np.uint32), mw.view(np.uint32)), L


@pytest.mark.parametrize("dtype", ["float32", "int32"])
@pytest.mark.parametrize("norm", [0, 1])
def test_standard_rule_vs_restatement(ginf, dtype, norm):
    for L in EDGES:
        P = _problem(L, dtype, 60 + L)
        want = _standard(P.D, P.V, 3, norm_min=norm == 1)
        _, got = ginf.decode_hbp(P.D, P.V, P.model, 1, 3, want_msgs=True, rule=ginf.RULE_STANDARD, normalize=norm)
        assert np.array_equal(_inner(got).view(np.uint32), _inner(want).view(np.uint32)), L


@pytest.mark.parametrize("rule", [0, 1])
@pytest.mark.parametrize("odd", ["table -0", "table inf", "table -inf", "table nan", "cost inf", "cost -0",
                                 "cost -inf", "cost nan"])
def test_values_outside_the_fast_form(ginf, orc, rule, odd):
    """One odd table entry or a scatter of odd costs; NaN positions must match
    and every other value, the sign of zero included."""
    L = 20
    P = _problem(L, "float32", 5)
    value = np.float32({"-0": -0.0, "inf": np.inf, "-inf": -np.inf, "nan": np.nan}[odd.split()[1]])
    D, V = P.D.copy(), P.V.copy()
    if odd.startswith("table"):
        V[7 + L * 3] = value
        if odd == "table -0":
            D[:, ::2] = np.float32(-0.0)
            V[::3] = value
    else:
        D[3::5, 2::7, 1::9] = value
    if rule == 0:
        _, want = orc.hbp(D, V, P.model, 1, 3, want_msgs=True)
    else:
        with np.errstate(invalid="ignore"):
            want = _standard(D, V, 3)
    _, got = ginf.decode_hbp(D, V, P.model, 1, 3, want_msgs=True, rule=rule)
    got, want = _inner(got), _inner(want)
    nan = np.isnan(want)
    assert np.array_equal(np.isnan(got), nan)
    assert np.array_equal(got.view(np.uint32)[~nan], want.view(np.uint32)[~nan])


def test_fp16_store_standard_rule(ginf, orc):
    """FP16 messages: FP32 min-convolution of the widened messages, minimum
    subtracted, rounded once -- within 5e-3 of the largest FP64 message after
    four half-sweeps (the bound of the FP16 store elsewhere)."""
    for L in (5, 16, 24, 33, 64, 100, 128):
        P = synth.random_problem(37, 13, L, 80 + L, model=synth.TRUNC_LINEAR, scale=1.0, trunc=3.0)
        _, want = orc.hbp_f64_std(P.D, P.V, synth.TRUNC_LINEAR, 1, 4, norm=1, want_msgs=True)
        _, got = ginf.decode_hbp(P.D, P.V, synth.EXPLICIT, 1, 4, want_msgs=True, rule=ginf.RULE_STANDARD,
                                 store=ginf.STORE_F16)
        assert np.abs(got - want).max() <= 5e-3 * np.abs(want).max(), L


def test_restatement_equals_oracle_on_a_linear_table(orc):
    """The numpy restatement against the oracle where both are defined: a
    truncated-linear table, whose standard and reference rules agree up to the
    rounding of the linear update's scans."""
    P = synth.random_problem(21, 13, 9, 4)
    _, want = orc.hbp(P.D, P.V, P.model, 1, 3, want_msgs=True)
    got = _standard(P.D, P.V, 3)
    assert np.abs(_inner(got) - _inner(want)).max() < 1e-5
