"""The warm-start network's tensor-core kernels against the CPU oracle
(forward and every parameter gradient), its training step and checkpoints,
and the learned hierarchical BP solve with its fallback."""
import numpy as np
import pytest

from gridinfcuda_gb300 import synth
from oracle import warmnet_ref as REF

pytestmark = pytest.mark.gpu


def _rel(a, b):
    a, b = np.asarray(a, np.float64), np.asarray(b, np.float64)
    return np.linalg.norm(a - b) / max(np.linalg.norm(b), 1e-30)


@pytest.mark.parametrize("L", [16, 32, 64])
def test_forward_matches_oracle(ginf, L):
    import torch
    params = REF.init_params(L, seed=L)
    rng = np.random.default_rng(L)
    x = rng.uniform(0, 1, (2, 9, 7, L)).astype(np.float32)
    with ginf.WarmNet(L, 32) as net:
        net.set_params(params)
        y = net.forward(torch.from_numpy(x).cuda()).cpu().numpy()
    want, _ = REF.forward(params, x, L)
    assert _rel(y, want) < 1e-4


@pytest.mark.parametrize("L", [16, 64])
def test_gradients_match_oracle(ginf, L):
    """Gradient check: loss within 1e-5 and every layer's weight and bias
    gradients within 5e-3 (norm-relative) of the float64 oracle that rounds
    to BF16 at the same points."""
    import torch
    params = REF.init_params(L, seed=7)
    rng = np.random.default_rng(11)
    x = rng.uniform(0, 1, (3, 10, 13, L)).astype(np.float32)
    t = (x + rng.normal(0, 0.2, x.shape)).astype(np.float32)
    with ginf.WarmNet(L, 32) as net:
        net.set_params(params)
        loss, g = net.gradients(torch.from_numpy(x).cuda(), torch.from_numpy(t).cuda())
    want_loss, want_g = REF.gradients(params, x, t, L)
    assert abs(loss - want_loss) <= 1e-5 * abs(want_loss)
    off = 0
    for cin, cout in REF.shapes(L):
        nw = cout * 9 * cin
        assert _rel(g[off:off + nw], want_g[off:off + nw]) < 5e-3, ("weights", cin, cout)
        assert _rel(g[off + nw:off + nw + cout], want_g[off + nw:off + nw + cout]) < 5e-3, ("bias", cin, cout)
        off += nw + cout


def test_training_lowers_the_loss(ginf):
    import torch
    rng = np.random.default_rng(5)
    x = torch.from_numpy(rng.uniform(0, 1, (8, 12, 16, 16)).astype(np.float32)).cuda()
    t = x + 0.3 * torch.roll(x, 1, dims=3)
    with ginf.WarmNet(16, 32, seed=3) as net:
        first = net.train_step(x, t, 3e-3)
        for _ in range(60):
            last = net.train_step(x, t, 3e-3)
    assert last < 0.5 * first


def test_checkpoint_resume_is_exact(ginf, tmp_path):
    import torch
    rng = np.random.default_rng(9)
    x = torch.from_numpy(rng.uniform(0, 1, (4, 8, 8, 32)).astype(np.float32)).cuda()
    t = x * 1.5 - 0.2
    with ginf.WarmNet(32, 32, seed=1) as a:
        for _ in range(10):
            a.train_step(x, t, 1e-3)
        straight = a.get_params()
    with ginf.WarmNet(32, 32, seed=1) as b:
        for _ in range(5):
            b.train_step(x, t, 1e-3)
        b.save(tmp_path / "ck.bin")
    with ginf.WarmNet(path=tmp_path / "ck.bin") as c:
        for _ in range(5):
            c.train_step(x, t, 1e-3)
        resumed = c.get_params()
    assert np.array_equal(straight.view(np.uint32), resumed.view(np.uint32))
    raw = bytearray(open(tmp_path / "ck.bin", "rb").read())
    raw[100] ^= 0xFF
    open(tmp_path / "bad.bin", "wb").write(bytes(raw))
    with pytest.raises(ginf.GinfError) as e:
        ginf.WarmNet(path=tmp_path / "bad.bin")
    assert b"checksum" in str(e.value).encode()


def test_level_state_inputs_and_beliefs(ginf, orc):
    import torch
    P = synth.random_problem(45, 37, 16, 2)
    D, V = torch.from_numpy(P.D).cuda(), torch.from_numpy(P.V).cuda()
    x, b = ginf.level_state(D, V, P.model, 3, 0, 2)
    d = orc.pyramid(orc.pyramid(P.D))                   # (L, H2, W2)
    want = np.transpose(d, (1, 2, 0)) / 16.0
    assert np.array_equal(x.cpu().numpy(), want.astype(np.float32))
    assert torch.equal(x, b)                            # no sweeps: beliefs are the costs
    _, b2 = ginf.level_state(D, V, P.model, 3, 6, 2)
    assert not torch.equal(x, b2)


def _stereo(W=160, H=120, L=16, seed=4):
    import torch
    P = synth.stereo_problem(W, H, L, seed=seed, n_regions=6, sigma=2.0, planar=True, coef=0.07, cap=15.0,
                             model=synth.TRUNC_LINEAR, scale=1.0, trunc=2.0)
    return P, torch.from_numpy(P.D).cuda(), torch.from_numpy(P.V).cuda()


def test_learned_solve_with_zero_network(ginf):
    """A network that predicts zero messages: the warm level starts from zero
    messages, i.e. a shorter pyramid.  The labels equal one of the two plain
    schedules exactly, the one the fallback rule picks."""
    P, D, V = _stereo()
    with ginf.WarmNet(16, 32) as net:
        net.set_params(np.zeros(net.num_params(), np.float32))
        lab, st = ginf.decode_hbp_learned(D, V, P.model, 4, 6, 2, net, want_stats=True)
    lab = lab.cpu().numpy()
    short = ginf.decode_hbp(P.D, P.V, P.model, 3, 6)
    full = ginf.decode_hbp(P.D, P.V, P.model, 4, 6)
    want = short if st["warm_start_used"] else full
    assert np.array_equal(lab[1:-1, 1:-1], want[1:-1, 1:-1])


def test_learned_solve_falls_back_from_a_bad_network(ginf):
    """Wild predictions and one half-sweep per level: the seeded result is
    worse than the cold coarse labelling, so the cold schedule resumes and
    the result equals plain HBP exactly."""
    P, D, V = _stereo(seed=8)
    with ginf.WarmNet(16, 32, seed=5) as net:
        p = net.get_params()
        p *= 1000.0
        net.set_params(p)
        lab, st = ginf.decode_hbp_learned(D, V, P.model, 4, 1, 2, net, want_stats=True)
    assert st["warm_start_used"] == 0
    full = ginf.decode_hbp(P.D, P.V, P.model, 4, 1)
    assert np.array_equal(lab.cpu().numpy()[1:-1, 1:-1], full[1:-1, 1:-1])


def _block_target(orc, D, M, t):
    """(D_t + block mean of the level-0 incoming-message sums) / 4^t in
    float32, accumulated in the kernel's order: block rows, block columns,
    then directions S, E, N, W."""
    L, H, W = D.shape
    Dt = D
    for _ in range(t):
        Dt = orc.pyramid(Dt)
    _, Ht, Wt = Dt.shape
    bs = 1 << t
    out = np.zeros((Ht, Wt, L), np.float32)
    for Y in range(Ht):
        for X in range(Wt):
            acc = np.zeros(L, np.float32)
            cnt = 0
            for y in range(Y * bs, min(H, (Y + 1) * bs)):
                for x in range(X * bs, min(W, (X + 1) * bs)):
                    for d in range(4):
                        acc = (acc + M[y, x, d]).astype(np.float32)
                    cnt += 1
            mean = (acc / np.float32(cnt)).astype(np.float32)
            out[Y, X] = ((Dt[:, Y, X] + mean).astype(np.float32) / np.float32(bs * bs)).astype(np.float32)
    return out


def test_level_state_fine_target(ginf, orc):
    """target 1: the level-0 messages of the whole schedule, averaged per
    level-t block, plus the level-t costs, over 4^t -- bit for bit."""
    import torch
    P = synth.random_problem(37, 29, 16, 2)
    D, V = torch.from_numpy(P.D).cuda(), torch.from_numpy(P.V).cuda()
    for t in (1, 2):
        x, y = ginf.level_state(D, V, P.model, 3, 5, t, target=1)
        _, M = ginf.decode_hbp(P.D, P.V, P.model, 3, 5, want_msgs=True)
        want = _block_target(orc, P.D, M, t)
        assert np.array_equal(y.cpu().numpy(), want), t


def test_seed_of_zero_messages_is_a_shorter_pyramid(ginf):
    """decode_hbp_warm with y = x (zero messages) at level t, no fallback,
    warm_iters = iters: exactly plain HBP with t + 1 levels."""
    import torch
    P, D, V = _stereo(seed=3)
    for t in (1, 2):
        x, _ = ginf.level_state(D, V, P.model, 4, 0, t, want_beliefs=False)
        lab = ginf.decode_hbp_warm(D, V, P.model, 4, 5, t, x, warm_iters=5, fallback=False)
        want = ginf.decode_hbp(P.D, P.V, P.model, t + 1, 5)
        assert np.array_equal(lab.cpu().numpy()[1:-1, 1:-1], want[1:-1, 1:-1]), t
    with pytest.raises(ValueError):
        ginf.decode_hbp_warm(D, V, P.model, 4, 5, 1, torch.zeros((3, 3, 16), device="cuda"))


def test_converged_seed_is_kept_and_converges_fast(ginf):
    """Seeding level 1 with the converged fine-level messages: the fallback
    keeps it and two half-sweeps at level 0 land within 0.5 % of the
    converged energy, where the cold start with two is far off."""
    P, D, V = _stereo(W=320, H=240, L=16, seed=6)
    lab = ginf.decode_hbp(D, V, P.model, 5, 50)
    e_star = ginf.energy(D, V, P.model, lab)
    _, y = ginf.level_state(D, V, P.model, 5, 40, 1, target=1)
    lab, st = ginf.decode_hbp_warm(D, V, P.model, 5, 2, 1, y, warm_iters=0, mid_iters=0, want_stats=True)
    assert st["warm_start_used"] == 1
    e_warm = ginf.energy(D, V, P.model, lab)
    e_cold = ginf.energy(D, V, P.model, ginf.decode_hbp(D, V, P.model, 5, 2))
    assert e_warm <= 1.005 * e_star < e_cold


def test_bad_seed_falls_back_to_plain_hbp(ginf):
    """A seed of zero messages at level 1 with two half-sweeps at level 0 is
    worse than the cold level-2 labelling: the result is plain HBP."""
    P, D, V = _stereo(W=320, H=240, L=16, seed=6)
    x, _ = ginf.level_state(D, V, P.model, 5, 0, 1, want_beliefs=False)
    lab, st = ginf.decode_hbp_warm(D, V, P.model, 5, 2, 1, x, warm_iters=0, mid_iters=0, want_stats=True)
    want = ginf.decode_hbp(P.D, P.V, P.model, 5, 2)
    assert st["warm_start_used"] == 0
    assert np.array_equal(lab.cpu().numpy()[1:-1, 1:-1], want[1:-1, 1:-1])


def test_trained_network_beats_the_network_free_guess(ginf):
    """What the trained network gains over the method without it.  Trained
    with this library's kernels on BP's own converged messages of 48 seeded
    256x192x64 planar-stereo grids (40 epochs), it predicts the converged
    level-1 beliefs (costs plus the finest level's converged incoming
    messages, block-averaged) of 4 held-out grids with a mean squared error
    below 0.93 of the network-free guess (the costs alone, y = x); measured
    0.855.  (Fewer level-0 half-sweeps do not follow: on 1920x1080 grids the
    prescribed network's seeds still need 7-10 half-sweeps per level against
    8 for the cold start, because its errors are whole coherent regions.)"""
    from gridinfcuda_gb300 import warmstart as W
    X, Y = W.make_training_set(n=48, W=256, H=192, seed0=700000, processes=1, target_iters=30)
    Xh, Yh = W.make_training_set(n=4, W=256, H=192, seed0=800000, processes=1, target_iters=30)
    with ginf.WarmNet(64, 32, seed=2) as net:
        hist = W.train(net, X, Y, epochs=40, batch=8, lr=1e-3)
        pred = net.forward(Xh)
    base = float(((Xh - Yh) ** 2).mean())
    got = float(((pred - Yh) ** 2).mean())
    assert hist[-1] < hist[0]
    assert got < 0.93 * base, (got, base)


def _torch_forward(params, x, L):
    """Plain PyTorch float64 forward of the network, rounding to BF16 where
    the library does: x, the weights and the three hidden activations.  x is
    (n, h, w, L) on the GPU; returns y = x + net(x), (n, h, w, L)."""
    import torch
    bf = lambda t: t.to(torch.bfloat16).to(torch.float64)
    p = torch.from_numpy(np.asarray(params, np.float64)).cuda()
    a = bf(x.double()).permute(0, 3, 1, 2)
    off = 0
    for layer, (cin, cout) in enumerate(REF.shapes(L)):
        nw = cout * 9 * cin
        w = bf(p[off:off + nw].reshape(cout, 3, 3, cin).permute(0, 3, 1, 2).contiguous())
        b = p[off + nw:off + nw + cout]
        off += nw + cout
        a = torch.nn.functional.conv2d(a, w, b, padding=1)
        if layer < 3:
            a = bf(torch.relu(a))
    return x.double() + a.permute(0, 2, 3, 1)


@pytest.mark.parametrize("L", [16, 32, 64])
@pytest.mark.parametrize("shape", [(2, 720, 256), (1, 37, 300), (200, 5, 20)])
def test_tcgen05_convolutions_at_scale(ginf, L, shape):
    """The tcgen05 convolutions against a plain PyTorch float64 reference at
    sizes the small oracle tests do not reach: 2 x 720 x 256 gives each CTA
    more rows than either accumulator ring holds (8 slots at COUT 16 / 32, 4
    at 64), so the ring wraps; 1 x 37 x 300 ends in a 44-pixel band; 200
    images of 5 x 20 give more work items than CTA slots, so CTAs carry their
    tile and row-copy counters across items.  Forward within 1e-4
    (norm-relative), as the oracle test; the data-gradient path (the same
    kernel with flipped weights and FP32 output) is exercised through
    `gradients` and checked for finiteness and agreement between two runs."""
    import torch
    n, h, w = shape
    params = REF.init_params(L, seed=3 + L)
    gen = torch.Generator(device="cuda").manual_seed(n * h + w + L)
    x = torch.rand((n, h, w, L), device="cuda", generator=gen)
    with ginf.WarmNet(L, 32) as net:
        net.set_params(params)
        y = net.forward(x)
        t = x + 0.05 * torch.rand(x.shape, device="cuda", generator=gen)
        loss1, g1 = net.gradients(x, t)
        loss2, g2 = net.gradients(x, t)
    want = _torch_forward(params, x, L)
    assert _rel(y.cpu().numpy(), want.cpu().numpy()) < 1e-4
    assert np.isfinite(loss1) and np.all(np.isfinite(g1))
    assert loss1 == loss2 and np.array_equal(g1, g2)


def test_forward_in_place(ginf):
    """ginf_warmnet_forward with y == x, which the header allows: the last
    layer reads each residual element before the same thread writes it, so
    the result equals a forward into a separate buffer, bit for bit."""
    import torch
    L = 32
    params = REF.init_params(L, seed=5)
    gen = torch.Generator(device="cuda").manual_seed(9)
    x = torch.rand((2, 40, 150, L), device="cuda", generator=gen)
    with ginf.WarmNet(L, 32) as net:
        net.set_params(params)
        y = net.forward(x)
        z = x.clone()
        ginf.check(ginf.lib().ginf_warmnet_forward(net.handle, z.data_ptr(), 2, 40, 150, z.data_ptr(), None))
    assert torch.equal(y, z)


@pytest.mark.parametrize("L,shape", [(16, (1, 9, 7)), (32, (2, 5, 131)), (64, (3, 33, 129)), (64, (1, 1, 1))])
def test_gradients_at_ragged_sizes_vs_torch_float64(ginf, L, shape):
    """Loss and gradients where bands end inside a warp or a warp lies beyond
    the image, against PyTorch float64 with the network's BF16 rounding points
    (within 5e-3, norm-relative, as the oracle's check), and the same from a
    target that is not 16-byte aligned."""
    import torch
    n, h, w = shape
    g = torch.Generator(device="cuda").manual_seed(L + w)
    x = torch.rand((n, h, w, L), generator=g, device="cuda")
    buf = torch.empty(x.numel() + 1, device="cuda")
    target = x + 0.5 * torch.randn(x.shape, generator=g, device="cuda")
    with ginf.WarmNet(L, 32, seed=3) as net:
        loss, grads = net.gradients(x, target)
        params = net.get_params()
        odd = buf[1:].view(x.shape)
        odd.copy_(target)
        loss2, grads2 = net.gradients(x, odd)
    assert loss2 == loss and np.array_equal(grads2, grads)

    def bf(a):
        return a.to(torch.bfloat16).to(torch.float64)

    def conv(a, wt):
        return torch.nn.functional.conv2d(a.permute(0, 3, 1, 2), wt.permute(0, 3, 1, 2), padding=1).permute(0, 2, 3, 1)

    chans = [L, 32, 32, 32, L]
    ws, bs, off = [], [], 0
    for k in range(4):
        c = chans[k + 1] * 9 * chans[k]
        ws.append(bf(torch.from_numpy(params[off:off + c]).cuda()).view(chans[k + 1], 3, 3, chans[k]))
        bs.append(torch.from_numpy(params[off + c:off + c + chans[k + 1]]).cuda().double())
        off += c + chans[k + 1]
    acts = [bf(x)]
    for k in range(3):
        acts.append(bf(torch.relu(conv(acts[-1], ws[k]) + bs[k])))
    d = conv(acts[3], ws[3]) + bs[3] + x.double() - target.double()
    want_loss = float((d ** 2).mean())
    grad = 2.0 / d.numel() * d
    parts = []
    for k in (3, 2, 1, 0):
        gb = bf(grad)
        a = acts[k].permute(0, 3, 1, 2)
        dw = torch.nn.grad.conv2d_weight(a, (chans[k + 1], chans[k], 3, 3), gb.permute(0, 3, 1, 2), padding=1)
        parts.insert(0, torch.cat([dw.permute(0, 2, 3, 1).reshape(-1), grad.sum((0, 1, 2))]))
        if k:
            back = torch.nn.functional.conv_transpose2d(gb.permute(0, 3, 1, 2), ws[k].permute(0, 3, 1, 2), padding=1)
            grad = back.permute(0, 2, 3, 1) * (acts[k] > 0)
    want = torch.cat(parts).cpu().numpy()
    assert abs(loss - want_loss) <= 1e-5 * want_loss
    off = 0
    for k in range(4):
        for c in (chans[k + 1] * 9 * chans[k], chans[k + 1]):
            assert _rel(grads[off:off + c], want[off:off + c]) < 5e-3, (k, c)
            off += c
