"""The calls whose speed this framework is judged by, one dict per case.

A case names the call and its sizes; `prepare` makes what a program has in hand
before the call (inputs on the GPU unless the call takes host buffers, plus the
workspace, plan or network such a program keeps), `run` makes the call through
gridinfcuda_gb300.capi and returns its outputs, `work` counts what the call
cannot do without, and `exact` gives the outputs that are computed numbers in
64 bits.  Labellings are whole numbers and have no 64-bit value; neither has
the energy of a labelling that the call itself found.

Kinds
  frame    two images -> cost volume -> hierarchical BP + ICM + energy: the
           per-frame work of a stereo program, everything on the GPU
  host     the same solve on a cost volume in host memory, as the C++ drop-in
           API's callers have it
  bp       loopy BP labels from costs on the GPU (float32 or int32)
  table    loopy BP with a table the linear update does not cover (an explicit
           or truncated-quadratic table), reference or standard message rule
  quad     standard-rule BP with a truncated-quadratic table, FP32 or FP16
           message store
  icm      ICM from an initial labelling, raster order or Jacobi
  swap     the reference example's integer problem: 8-bit images -> integer
           costs -> 30 BP half-sweeps -> one alpha-beta-swap pass
  batch    a kept plan over many grids of mixed sizes and label counts
  forward  the warm-start network's forward pass
  train    the warm-start network's loss and gradients (forward and backward)
"""
import random

import numpy as np
import torch

from gridinfcuda_gb300 import capi

POTTS, LINEAR, QUAD, EXPLICIT = capi.POTTS, capi.TRUNC_LINEAR, capi.TRUNC_QUAD, capi.EXPLICIT
HIDDEN = 32  # the warm-start network's hidden channels

# Twelve grids between 200x150 and 1280x720 with 16, 32 or 64 labels, the
# mix of a batch server; one has a label count between the compiled ones.
BATCH = ("1280x720x64 1047x611x16 913x402x32 640x480x64 733x655x16 311x288x32 "
         "505x197x64 1201x350x32 200x150x16 450x375x48 868x540x16 384x288x32")


def listed():
    return [
        # A thumbnail-sized frame: launches and latency are all there is.
        {"name": "frame-160x120x16", "kind": "frame", "w": 160, "h": 120, "labels": 16, "levels": 3, "iters": 8,
         "icm": 2},
        # The headline workload: a full-HD frame, 64 disparities.
        {"name": "frame-1920x1080x64", "kind": "frame", "w": 1920, "h": 1080, "labels": 64, "levels": 5, "iters": 10,
         "icm": 5},
        # A drop-in caller: odd sizes, a label count between the powers of two, costs in host memory.
        {"name": "host-1001x563x48", "kind": "host", "w": 1001, "h": 563, "labels": 48, "levels": 4, "iters": 10,
         "icm": 3},
        # Plain loopy BP at the reference example's size, fifty iterations: the L2-resident middle of the range.
        {"name": "bp-384x288x16", "kind": "bp", "w": 384, "h": 288, "labels": 16, "iters": 50, "model": LINEAR,
         "dtype": "float32"},
        # A hand-made smoothness table through the reference's rule (the default).
        {"name": "table-640x480x32", "kind": "table", "w": 640, "h": 480, "labels": 32, "iters": 10,
         "model": EXPLICIT, "dtype": "float32", "rule": "reference"},
        # Truncated-quadratic smoothness at 128 labels, the two message stores.
        {"name": "quad-f32-1280x720x128", "kind": "quad", "w": 1280, "h": 720, "labels": 128, "iters": 16,
         "trunc": 25.0, "store": "native"},
        {"name": "quad-f16-1280x720x128", "kind": "quad", "w": 1280, "h": 720, "labels": 128, "iters": 16,
         "trunc": 25.0, "store": "f16"},
        # Raster-order ICM on an integer grid, from the labels of lowest cost.
        {"name": "icm-raster-640x480x32", "kind": "icm", "w": 640, "h": 480, "labels": 32, "iters": 5,
         "raster": True, "dtype": "int32"},
        # The reference example end to end with its graph cut.
        {"name": "swap-384x288x16", "kind": "swap", "w": 384, "h": 288, "labels": 16, "iters": 1},
        # A batch server's plan.
        {"name": "batch-12", "kind": "batch", "grids": BATCH, "iters": 30},
        # The warm-start network at the level it seeds for a full-HD frame, and one training batch.
        {"name": "forward-960x540x64", "kind": "forward", "n": 1, "w": 960, "h": 540, "labels": 64},
        {"name": "train-16x256x192x64", "kind": "train", "n": 16, "w": 256, "h": 192, "labels": 64},
    ]


# ---------------------------------------------------------------- drawn cases

def _log(rng, lo, hi):
    """A whole number spread evenly over the logarithm of [lo, hi]."""
    return int(round(lo * (hi / lo) ** rng.random()))


def _grid(rng, most, w=(64, 1920), h=(48, 1080), labels=(4, 128)):
    """Width, height and label count with w * h * labels <= most."""
    while True:
        g = {"w": _log(rng, *w), "h": _log(rng, *h), "labels": _log(rng, *labels)}
        if g["w"] * g["h"] * g["labels"] <= most:
            return g


def draw(rng):
    kind = rng.choice(["frame", "host", "bp", "table", "quad", "icm", "swap", "batch", "forward", "train"])
    if kind == "frame":
        return {"kind": kind, **_grid(rng, 130_000_000), "levels": rng.randint(1, 5), "iters": rng.randint(4, 12),
                "icm": rng.randint(0, 6)}
    if kind == "host":
        return {"kind": kind, **_grid(rng, 30_000_000), "levels": rng.randint(1, 5), "iters": rng.randint(4, 12),
                "icm": rng.randint(0, 6)}
    if kind == "bp":
        return {"kind": kind, **_grid(rng, 60_000_000), "iters": rng.randint(5, 50),
                "model": rng.choice([LINEAR, POTTS]), "dtype": rng.choice(["float32", "int32"])}
    if kind == "table":
        return {"kind": kind, **_grid(rng, 10_000_000), "iters": rng.randint(4, 12),
                "model": rng.choice([EXPLICIT, EXPLICIT, QUAD]), "dtype": rng.choice(["float32", "int32"]),
                "rule": rng.choice(["reference", "standard"])}
    if kind == "quad":
        return {"kind": kind, **_grid(rng, 120_000_000, labels=(16, 128)), "iters": rng.randint(4, 16),
                "trunc": rng.choice([6.0, 14.0, 25.0, 45.0]), "store": rng.choice(["native", "f16"])}
    if kind == "icm":
        return {"kind": kind, **_grid(rng, 40_000_000), "iters": rng.randint(1, 8), "raster": rng.random() < 0.5,
                "dtype": rng.choice(["float32", "int32"])}
    if kind == "swap":
        return {"kind": kind, "w": _log(rng, 32, 200), "h": _log(rng, 32, 150), "labels": rng.randint(3, 12),
                "iters": 1}
    if kind == "batch":
        grids = []
        for _ in range(rng.randint(2, 12)):
            g = (_log(rng, 200, 1280), _log(rng, 150, 720), rng.choice([16, 32, 64, 64, 32, 16, rng.randint(5, 64)]))
            grids.append("%dx%dx%d" % g)
        return {"kind": kind, "grids": " ".join(grids), "iters": rng.randint(5, 30)}
    n = 1 if kind == "forward" else _log(rng, 1, 16)
    return {"kind": kind, "n": n, "w": _log(rng, 30, 960 if kind == "forward" else 256),
            "h": _log(rng, 30, 540 if kind == "forward" else 192), "labels": rng.choice([16, 32, 64])}


# ---------------------------------------------------------------- inputs

def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _pair(w, h, labels, seed, regions=24, sigma=3.0):
    """A rectified pair of smooth random textures, float32 (h, w) in about
    [0, 255]: the left image is the right one shifted by slanted planes over
    random rectangles, plus noise."""
    g, rng = _generator(seed), random.Random(seed)
    right = torch.rand((1, 1, h, w), generator=g, device="cuda") * 255.0
    right = torch.nn.functional.avg_pool2d(right, 3, 1, 1, count_include_pad=False)[0, 0]
    xs = torch.arange(w, device="cuda", dtype=torch.float32)[None, :].expand(h, w)
    ys = torch.arange(h, device="cuda", dtype=torch.float32)[:, None].expand(h, w)
    disp = torch.full((h, w), float(min(2, labels - 1)), device="cuda")
    for _ in range(regions):
        x0, x1 = sorted((rng.randrange(w), rng.randrange(w)))
        y0, y1 = sorted((rng.randrange(h), rng.randrange(h)))
        a, b, c = rng.uniform(-0.02, 0.02), rng.uniform(-0.02, 0.02), rng.uniform(0, labels - 1)
        box = (slice(y0, y1 + 1), slice(x0, x1 + 1))
        disp[box] = torch.clamp(torch.round(a * xs[box] + b * ys[box] + c), 0, labels - 1)
    src = torch.clamp(xs - disp, min=0).long()
    left = torch.gather(right, 1, src) + sigma * torch.randn((h, w), generator=g, device="cuda")
    return left.contiguous(), right.contiguous()


def _costs(w, h, labels, seed, dtype="float32", coef=0.07, cap=15.0):
    """Label-planar stereo costs (labels, h, w): coef * min(|difference|, cap)
    in float32, the whole-number difference capped at 20 in int32."""
    left, right = _pair(w, h, labels, seed)
    out = torch.empty((labels, h, w), dtype=torch.float32 if dtype == "float32" else torch.int32, device="cuda")
    xs = torch.arange(w, device="cuda")
    for k in range(labels):
        diff = (left - right[:, torch.clamp(xs - k, min=0)]).abs()
        out[k] = coef * torch.clamp(diff, max=cap) if dtype == "float32" else torch.clamp(diff, max=20.0).to(torch.int32)
    return out


def _table(labels, model, dtype="float32", scale=1.0, trunc=4.0, seed=0):
    """Flat smoothness table V(fp, fq) at fp + labels * fq."""
    i = torch.arange(labels, device="cuda", dtype=torch.float32)
    d = (i[None, :] - i[:, None]).abs()
    if dtype == "int32":
        scale, trunc = 10.0, 20.0 if model != QUAD else 90.0
    if model == POTTS:
        v = scale * (d > 0).float()
    elif model == QUAD:
        v = torch.clamp(scale * d * d, max=trunc)
    else:
        v = torch.clamp(scale * d, max=trunc)
        if model == EXPLICIT:  # a linear table with label-dependent weights, as a hand-made one has
            v = v * (0.75 + 0.5 * torch.rand((labels, labels), generator=_generator(seed + 77), device="cuda"))
    return (v if dtype == "float32" else torch.round(v).to(torch.int32)).contiguous().reshape(-1)


def _params(labels, seed):
    """The network's flat parameter vector: He-uniform weights, the last layer
    a tenth of that, small biases."""
    rs = np.random.RandomState(seed % (2 ** 31))
    ch = [labels, HIDDEN, HIDDEN, HIDDEN, labels]
    parts = []
    for k in range(4):
        bound = (6.0 / (9 * ch[k])) ** 0.5 * (0.1 if k == 3 else 1.0)
        parts.append(rs.uniform(-bound, bound, ch[k + 1] * 9 * ch[k]))
        parts.append(rs.uniform(-0.02, 0.02, ch[k + 1]))
    return np.concatenate(parts).astype(np.float32)


def _net_inputs(case, seed):
    """x: costs per fine node, (n, h, w, labels) in [0, 1.05]; target: x plus a
    smooth message sum."""
    n, h, w, L = case["n"], case["h"], case["w"], case["labels"]
    g = _generator(seed)
    x = torch.empty((n, h, w, L), device="cuda")
    target = torch.empty_like(x)
    for k in range(n):
        x[k] = 0.07 * torch.clamp(30.0 * torch.rand((h, w, L), generator=g, device="cuda"), max=15.0)
        m = torch.randn((1, L, h, w), generator=g, device="cuda")
        target[k] = x[k] + 2.0 * torch.nn.functional.avg_pool2d(m, 5, 1, 2)[0].permute(1, 2, 0)
    return x, target


def _shapes(text):
    return [tuple(int(v) for v in item.split("x")) for item in text.split()]


def prepare(case, seed):
    kind, st = case["kind"], {"case": case}
    if kind in ("forward", "train"):
        st["x"], st["target"] = _net_inputs(case, seed)
        st["net"] = capi.WarmNet(case["labels"], HIDDEN, 0)
        st["net"].set_params(_params(case["labels"], seed))
    elif kind == "batch":
        st["problems"], st["labels"] = [], []
        for k, (w, h, L) in enumerate(_shapes(case["grids"])):
            st["problems"].append((_costs(w, h, L, seed + 1000 * k), _table(L, LINEAR, trunc=1.7), LINEAR))
            st["labels"].append(torch.zeros((h, w), dtype=torch.int32, device="cuda"))
        st["plan"] = capi.Batch(st["problems"], st["labels"], case["iters"], tile_nodes=16, sweeps_per_launch=1)
    else:
        w, h, L = case["w"], case["h"], case["labels"]
        st["ws"] = capi.Workspace()
        st["labels"] = torch.zeros((h, w), dtype=torch.int32, device="cuda")
        if kind == "frame":
            st["left"], st["right"] = _pair(w, h, L, seed)
            st["D"] = torch.empty((L, h, w), device="cuda")
            st["V"] = _table(L, LINEAR)
        elif kind == "host":
            st["D"] = _costs(w, h, L, seed).cpu().numpy()
            st["V"] = _table(L, LINEAR).cpu().numpy()
            st["labels"] = np.zeros((h, w), np.int32)
        elif kind in ("bp", "table"):
            st["D"] = _costs(w, h, L, seed, case["dtype"])
            trunc = 16.0 if case["model"] == QUAD else (1.7 if kind == "bp" else 4.0)
            st["V"] = _table(L, case["model"], case["dtype"], trunc=trunc, seed=seed)
        elif kind == "quad":
            st["D"] = _costs(w, h, L, seed, coef=0.05, cap=20.0)
            st["V"] = _table(L, QUAD, trunc=case["trunc"])
        elif kind == "icm":
            st["D"] = _costs(w, h, L, seed, case["dtype"])
            st["V"] = _table(L, LINEAR, case["dtype"])
            st["initial"] = st["D"].argmin(0).to(torch.int32)
        elif kind == "swap":
            left, right = _pair(w, h, L, seed, regions=12, sigma=2.0)
            st["left"], st["right"] = (torch.clamp(torch.round(v), 0, 255).to(torch.uint8) for v in (left, right))
            st["D"] = torch.empty((L, h, w), dtype=torch.int32, device="cuda")
            st["V"] = _table(L, LINEAR, "int32")
        else:
            raise ValueError(kind)
    torch.cuda.synchronize()
    return st


# ---------------------------------------------------------------- the calls

def run(st):
    case = st["case"]
    kind = case["kind"]
    if kind == "frame":
        capi.stereo_costs(st["left"], st["right"], case["labels"], 0.07, 15.0, st["D"])
        return list(capi.solve(st["D"], st["V"], LINEAR, case["levels"], case["iters"], case["icm"],
                               labels=st["labels"], workspace=st["ws"]))
    if kind == "host":
        return list(capi.solve(st["D"], st["V"], LINEAR, case["levels"], case["iters"], case["icm"],
                               labels=st["labels"], workspace=st["ws"]))
    if kind == "bp":
        return capi.decode_hbp(st["D"], st["V"], case["model"], 1, case["iters"], labels=st["labels"],
                               workspace=st["ws"])
    if kind == "table":
        rule = capi.RULE_REFERENCE if case["rule"] == "reference" else capi.RULE_STANDARD
        return capi.decode_hbp(st["D"], st["V"], case["model"], 1, case["iters"], labels=st["labels"],
                               workspace=st["ws"], rule=rule)
    if kind == "quad":
        store = capi.STORE_F16 if case["store"] == "f16" else capi.STORE_NATIVE
        return capi.decode_hbp(st["D"], st["V"], QUAD, 1, case["iters"], labels=st["labels"], workspace=st["ws"],
                               rule=capi.RULE_STANDARD, store=store)
    if kind == "icm":
        return capi.decode_icm(st["D"], st["V"], LINEAR, st["initial"], case["iters"], asynchronous=case["raster"],
                               workspace=st["ws"])
    if kind == "swap":
        capi.stereo_costs_u8(st["left"], st["right"], case["labels"], 20, st["D"])
        first = capi.decode_hbp(st["D"], st["V"], LINEAR, 1, 30, labels=st["labels"], workspace=st["ws"])
        return [first, capi.decode_alpha_beta(st["D"], st["V"], LINEAR, first, case["iters"], workspace=st["ws"])]
    if kind == "batch":
        st["plan"].run()
        return st["labels"]
    if kind == "forward":
        return st["net"].forward(st["x"])
    if kind == "train":
        return list(st["net"].gradients(st["x"], st["target"]))
    raise ValueError(kind)


# ---------------------------------------------------------------- what a call cannot do without

def _bp_flops(w, h, per_label_node, levels, iters):
    """Arithmetic of `iters` half-sweeps (half the interior nodes each) on
    every level."""
    total = 0.0
    for _ in range(levels):
        total += max(w - 2, 0) * max(h - 2, 0) / 2.0 * iters * per_label_node
        w, h = (w + 1) // 2, (h + 1) // 2
    return total


def work(case):
    kind = case["kind"]
    if kind in ("forward", "train"):
        pix, L = case["n"] * case["h"] * case["w"], case["labels"]
        ch = [L, HIDDEN, HIDDEN, HIDDEN, L]
        macs = [9 * ch[k] * ch[k + 1] for k in range(4)]
        params = sum(macs) + sum(ch[1:])
        if kind == "forward":
            return {"bytes": 8.0 * pix * L + 4.0 * params, "flops": 2.0 * pix * sum(macs)}
        # Backward: every layer's weight gradient, and the data gradient of all but the first.
        return {"bytes": 8.0 * pix * L + 8.0 * params, "flops": 2.0 * pix * (3 * sum(macs) - macs[0])}
    # A belief and four linear messages take about 40 operations a label.
    if kind == "batch":
        shapes = _shapes(case["grids"])
        return {"bytes": float(sum(w * h * (4 * L + 4) + 4 * L * L for w, h, L in shapes)),
                "flops": sum(_bp_flops(w, h, 40 * L, 1, case["iters"]) for w, h, L in shapes)}
    w, h, L = case["w"], case["h"], case["labels"]
    n = w * h
    costs, table, labels = 4.0 * n * L, 4.0 * L * L, 4.0 * n
    if kind == "frame":
        return {"bytes": 8.0 * n + table + labels,
                "flops": _bp_flops(w, h, 40 * L, case["levels"], case["iters"]) + n * L * (4 + 5 * case["icm"])}
    if kind == "host":
        return {"bytes": costs + table + labels,
                "flops": _bp_flops(w, h, 40 * L, case["levels"], case["iters"]) + n * L * 5 * case["icm"]}
    if kind == "bp":
        return {"bytes": costs + table + labels, "flops": _bp_flops(w, h, 40 * L, 1, case["iters"])}
    if kind == "table":
        # One min-convolution a node (reference rule), or one a message.
        per = L * (4 + 2 * L) if case["rule"] == "reference" else L * (4 + 4 * (3 + 2 * L))
        return {"bytes": costs + table + labels, "flops": _bp_flops(w, h, per, 1, case["iters"])}
    if kind == "quad":
        return {"bytes": costs + table + labels, "flops": _bp_flops(w, h, 60 * L, 1, case["iters"])}
    if kind == "icm":
        return {"bytes": costs + table + 2 * labels, "flops": 5.0 * n * L * case["iters"]}
    if kind == "swap":
        # BP, then for every label pair the graph, its flow and the energy.
        pairs = L * (L - 1) // 2
        return {"bytes": 2.0 * n + table + 2 * labels, "flops": _bp_flops(w, h, 40 * L, 1, 30) + 20.0 * n * pairs}
    raise ValueError(kind)


# ---------------------------------------------------------------- 64-bit values

def _conv(x, weight, bias):
    """3x3 convolution with zero padding, NHWC, weight (cout, 3, 3, cin)."""
    n, h, w, c = x.shape
    padded = torch.nn.functional.pad(x, (0, 0, 1, 1, 1, 1))
    out = bias
    for dy in range(3):
        for dx in range(3):
            out = out + padded[:, dy:dy + h, dx:dx + w, :].reshape(-1, c) @ weight[:, dy, dx, :].t()
    return out.reshape(n, h, w, -1)


def _net(x, params, labels):
    """x + net(x) with the flat parameter vector `params`."""
    ch = [labels, HIDDEN, HIDDEN, HIDDEN, labels]
    a, off = x, 0
    for k in range(4):
        count = ch[k + 1] * 9 * ch[k]
        weight = params[off:off + count].reshape(ch[k + 1], 3, 3, ch[k])
        bias = params[off + count:off + count + ch[k + 1]]
        off += count + ch[k + 1]
        a = _conv(a, weight, bias)
        if k < 3:
            a = torch.relu(a)
    return x + a


def exact(case, seed):
    kind, L = case["kind"], case.get("labels")
    if kind == "forward":
        x, _ = _net_inputs(case, seed)
        with torch.no_grad():
            return _net(x.double(), torch.from_numpy(_params(L, seed)).cuda().double(), L)
    if kind == "train":
        # One image at a time: the loss is a mean over all of them.
        x, target = _net_inputs(case, seed)
        params = torch.from_numpy(_params(L, seed)).cuda().double().requires_grad_(True)
        loss, grad = 0.0, torch.zeros_like(params)
        for k in range(case["n"]):
            part = ((_net(x[k:k + 1].double(), params, L) - target[k:k + 1].double()) ** 2).sum() / x.numel()
            grad += torch.autograd.grad(part, params)[0]
            loss += float(part)
        return [loss, grad.detach().cpu().numpy()]
    return None
