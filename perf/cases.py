"""Performance cases: the work users have this library do, through its public entry points.

Nine kinds of work, each over the sizes it meets in use (`draw` spreads over them):

* ``features``  inference through a trained 2-layer network (DoG, rank code, two fused layers, global pool): one image
  of a live stream up to a data set's batch;
* ``train``     unsupervised STDP training step of one or two fused layers, from 16 images to the 4096 of the benchmark;
* ``textures``  large-image feature extraction (Gabor bank, T = 30, 64 and 256 maps, no learning);
* ``ops``       the same training step written op by op at the default precision, as programs ported from the
  reference's examples have it (conv, threshold, inhibit, fire, convwta, stdp, pool);
* ``backprop``  temporal backprop through first-spike layers (forward, loss, gradients);
* ``sparse``    the event-list training step at 1-5 % input density;
* ``rstdp``     the reward-modulated step of the 3-layer network (op by op on the tensor-core potentials);
* ``sweep``     many networks trained side by side on images of uneven size, replayed as a CUDA graph.

A training case starts every pass from the weights in its state's snapshot, so that each pass does the same work however
many passes came before it.
"""

from __future__ import annotations

import math

import numpy
import torch
import torch.nn.functional as F

import spyker_b200 as sp
from spyker_b200 import rstdp, sparse, sweep, temporal

C1, C2 = 30, 100  # maps of the 2-layer network
TH1, TH2 = 15.0, 10.0
RATES = (0.004, -0.003)


def listed():
    return [
        # one image of a stream, trained network: the latency of a decision
        {"name": "features_1", "kind": "features", "batch": 1, "side": 28, "time": 15, "precision": "bf16x3"},
        # the small training step of the benchmark (one layer, 64 images)
        {"name": "train_64", "kind": "train", "layers": 1, "batch": 64, "side": 28, "time": 15, "precision": "bf16x3"},
        # the last, ragged batch of a data set, odd image side, the two-term split
        {"name": "train_333_odd", "kind": "train", "layers": 2, "batch": 333, "side": 33, "time": 12,
         "precision": "bf16x2"},
        # the benchmark's headline step
        {"name": "train_4096", "kind": "train", "layers": 2, "batch": 4096, "side": 28, "time": 15,
         "precision": "bf16x3"},
        # large images, 64 and 256 maps
        {"name": "textures_8", "kind": "textures", "batch": 8, "side": 256, "time": 30, "precision": "bf16x3"},
        # a program ported from the reference, op by op, default precision
        {"name": "ops_128", "kind": "ops", "batch": 128, "side": 28, "time": 15},
        # the temporal-backprop benchmark, and a small odd one
        {"name": "backprop_256", "kind": "backprop", "batch": 256, "side": 28, "time": 64, "precision": "bf16x3"},
        {"name": "backprop_37", "kind": "backprop", "batch": 37, "side": 28, "time": 30, "precision": "bf16x3"},
        # event lists: the benchmark's middle density, and a small dense one
        {"name": "sparse_4096", "kind": "sparse", "batch": 4096, "side": 28, "time": 15, "density": 0.02},
        {"name": "sparse_200", "kind": "sparse", "batch": 200, "side": 28, "time": 15, "density": 0.05},
        # the reward-modulated layer of the 3-layer network
        {"name": "rstdp_200", "kind": "rstdp", "batch": 200, "side": 28, "precision": "bf16x3"},
        # a hyperparameter sweep, sizes 20 / 28 / 40 / 64 mixed
        {"name": "sweep_8", "kind": "sweep", "nets": 8, "images": 96},
    ]


def draw(rng):
    def log(lo, hi):
        return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))

    kind = rng.choice(["features", "train", "train", "textures", "ops", "backprop", "sparse", "rstdp", "sweep"])
    case = {"kind": kind}
    if kind in ("features", "train"):
        side = rng.randint(20, 64)
        case.update(batch=log(1 if kind == "features" else 16, min(4096, 4096 * 784 // side ** 2)), side=side,
                    time=rng.randint(8, 30 if kind == "features" else 16), precision=rng.choice(["bf16x3", "bf16x2"]))
        if kind == "train":
            case["layers"] = rng.choice([1, 2])
    elif kind == "textures":
        side = rng.randint(97, 256)
        case.update(batch=log(1, 8), side=side, time=rng.randint(15, 30), precision="bf16x3")
    elif kind == "ops":
        side = rng.randint(20, 40)
        case.update(batch=log(4, 128 * 784 // max(784, side ** 2)), side=side, time=rng.randint(8, 15))
    elif kind == "backprop":
        case.update(batch=log(16, 250), side=rng.randint(20, 28), time=rng.randint(16, 64),
                    precision=rng.choice(["bf16x3", "bf16x2"]))
    elif kind == "sparse":
        side = rng.randint(20, 36)
        case.update(batch=log(64, 4096 * 784 // max(784, side ** 2)), side=side, time=rng.randint(8, 15),
                    density=round(rng.uniform(0.01, 0.05), 3))
    elif kind == "rstdp":
        case.update(batch=log(8, 200), side=rng.randint(22, 28), precision=rng.choice(["bf16x3", "bf16x2"]))
    else:
        case.update(nets=rng.randint(2, 8), images=log(16, 95))
    return case


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------


def _gen(seed, salt):
    return torch.Generator("cuda").manual_seed((int(seed) * 1000003 + salt) % (1 << 62))


def _uniform(g, lo, hi, *size):
    return torch.rand(size, generator=g, device="cuda", dtype=torch.float64) * (hi - lo) + lo


def _strokes(n, side, seed):
    """Images [n, 1, side, side] F32 in [0, 1] (multiples of 1 / 255): 1-4 anti-aliased line or arc strokes, 2-3 px wide,
    level 180-255, on a zero background."""
    g = _gen(seed, 1)
    p = torch.arange(side, device="cuda", dtype=torch.float64) + 0.5
    py, px = p[:, None], p[None, :]
    count = torch.randint(1, 5, (n, 1, 1), generator=g, device="cuda")
    img = torch.zeros((n, side, side), dtype=torch.float64, device="cuda")
    for k in range(4):
        width, level = _uniform(g, 2, 3, n, 1, 1), _uniform(g, 180, 255, n, 1, 1)
        y0, x0, y1, x1 = (_uniform(g, 0.15 * side, 0.85 * side, n, 1, 1) for _ in range(4))
        dy, dx = y1 - y0, x1 - x0
        t = (((py - y0) * dy + (px - x0) * dx) / (dy * dy + dx * dx).clamp_min(1e-9)).clamp(0, 1)
        line = torch.hypot(py - (y0 + t * dy), px - (x0 + t * dx))
        cy, cx = (_uniform(g, 0.3 * side, 0.7 * side, n, 1, 1) for _ in range(2))
        r, a0 = _uniform(g, 0.12 * side, 0.35 * side, n, 1, 1), _uniform(g, 0, 2 * math.pi, n, 1, 1)
        span = _uniform(g, 0.5 * math.pi, 1.6 * math.pi, n, 1, 1)
        inside = torch.remainder(torch.atan2(py - cy, px - cx) - a0, 2 * math.pi) <= span
        ring = (torch.hypot(py - cy, px - cx) - r).abs()
        ends = [torch.hypot(py - (cy + r * torch.sin(a)), px - (cx + r * torch.cos(a))) for a in (a0, a0 + span)]
        arc = torch.where(inside, ring, torch.minimum(*ends))
        d = torch.where(_uniform(g, 0, 1, n, 1, 1) < 0.5, line, arc)
        cover = (width / 2 + 0.5 - d).clamp(0, 1) * level
        img = torch.where(k < count, torch.maximum(img, cover), img)
    return (img.round().clamp(0, 255) / 255).float()[:, None].contiguous()


def _textures(n, side, seed):
    """Images [n, 1, side, side] F32 in [0, 1]: 1/f noise plus 8-32 Gaussian blobs."""
    g = _gen(seed, 2)
    fy = torch.fft.fftfreq(side, device="cuda", dtype=torch.float64)[:, None]
    fx = torch.fft.rfftfreq(side, device="cuda", dtype=torch.float64)[None, :]
    f = torch.hypot(fy, fx)
    amp = torch.where(f > 0, 1 / f.clamp_min(1e-12), torch.zeros_like(f))
    img = torch.fft.irfft2(torch.polar(amp.expand(n, -1, -1).contiguous(), _uniform(g, 0, 2 * math.pi, n, *f.shape)),
                           s=(side, side))
    lo, hi = img.amin((1, 2), keepdim=True), img.amax((1, 2), keepdim=True)
    img = 0.5 * (img - lo) / (hi - lo)
    p = torch.arange(side, device="cuda", dtype=torch.float64)
    count = torch.randint(8, 33, (n, 1, 1), generator=g, device="cuda")
    for k in range(32):
        cy, cx = (_uniform(g, 0, side, n, 1, 1) for _ in range(2))
        s, a = _uniform(g, 2, 12, n, 1, 1), _uniform(g, 0.3, 1, n, 1, 1)
        blob = a * torch.exp(-((p[:, None] - cy) ** 2 + (p[None, :] - cx) ** 2) / (2 * s * s))
        img = torch.where(k < count, img + blob, img)
    lo, hi = img.amin((1, 2), keepdim=True), img.amax((1, 2), keepdim=True)
    return ((img - lo) / (hi - lo)).float()[:, None].contiguous()


def _fresh(seed, salt, *size):
    """Weights at the start of a training: N(0.8, 0.05) in [0, 1]."""
    g = _gen(seed, salt)
    return (torch.randn(size, generator=g, device="cuda") * 0.05 + 0.8).clamp(0, 1)


def _trained(seed, salt, *size, share=0.3):
    """Weights after a training: STDP has driven most of them near 0 or near 1 (`share` of them)."""
    g = _gen(seed, salt)
    return torch.sigmoid(torch.randn(size, generator=g, device="cuda") * 3
                         + torch.where(torch.rand(size, generator=g, device="cuda") < share, 4.0, -4.0))


def _events(case, seed):
    """First-spike times [n, 2, side, side] F32 (`time` = never) with a share `density` of spiking inputs."""
    g, s, n, t = _gen(seed, 3), case["side"], case["batch"], case["time"]
    when = torch.randint(0, t, (n, 2, s, s), generator=g, device="cuda")
    fires = torch.rand((n, 2, s, s), generator=g, device="cuda") < case["density"]
    return torch.where(fires, when, torch.full_like(when, t)).float()


def _sparse_thresholds(case):
    return max(1.0, TH1 * case["density"] / 0.2), TH2


DOG = ((1, 2), (2, 1))
DOG6 = tuple((a / 9, b / 9) for a, b in ((3, 6), (6, 3), (7, 14), (14, 7), (13, 26), (26, 13)))
GABOR = tuple((2.5, th, 0.5, lam, 0.0) for th in (0, 45, 90, 135) for lam in (5.0, 10.0))


def _weights(case, seed):
    """The case's weights, first layer first."""
    kind = case["kind"]
    if kind == "features":
        return [_trained(seed, 11, C1, 2, 5, 5, share=0.5), _trained(seed, 12, C2, C1, 5, 5)]
    if kind == "textures":
        return [_fresh(seed, 11, 64, 8, 7, 7), _fresh(seed, 12, 256, 64, 5, 5)]
    if kind == "rstdp":
        return [_trained(seed, 11, 30, 6, 5, 5, share=0.5), _trained(seed, 12, 250, 30, 3, 3, share=0.5),
                _fresh(seed, 13, 200, 250, 5, 5)]
    return [_fresh(seed, 11, C1, 2, 5, 5), _fresh(seed, 12, C2, C1, 5, 5)]


def _layer(weights, pad, precision):
    cout, cin, kh, kw = weights.shape
    layer = sp.Conv(cin, cout, (kh, kw), pad=pad)
    layer.kernel.copy_(weights)
    layer.stdpconfig = [sp.STDPConfig(*RATES)]
    layer.precision = precision
    return layer


class State:
    pass


def prepare(case, seed):
    st = State()
    st.case, kind = case, case["kind"]
    if kind == "sweep":
        st.sweep = sweep.Sweep(nets=case["nets"], images=case["images"], seed=seed % 100003, path="search")
        st.start = [st.sweep.w1.clone(), st.sweep.w2.clone()]
        st.sweep.capture()
        return st
    if kind == "sparse":
        times = _events(case, seed)
        n, s, t = case["batch"], case["side"], case["time"]
        st.events = sp.SparseTensor(sp.scatter(times.reshape(n, -1), t).view(n, t, 2, s, s), 0.0)
    else:
        st.images = (_textures if kind == "textures" else _strokes)(case["batch"], case["side"], seed)
    if kind == "backprop":
        st.net = temporal.TemporalNet(time=case["time"], seed=seed, precision=case["precision"], size=case["side"])
        st.target = torch.randint(0, 10, (case["batch"],), generator=_gen(seed, 4), device="cuda")
        return st
    st.start = _weights(case, seed)
    if kind == "rstdp":
        st.net = rstdp.MozafariNetwork(precision=case["precision"])
        for layer, w in zip((st.net.conv1, st.net.conv2, st.net.conv3), st.start):
            layer.kernel.copy_(w)
        st.target = torch.randint(0, 10, (case["batch"],), generator=_gen(seed, 4), device="cuda")
        return st
    if kind == "textures":
        st.bank = sp.Gabor(5, [sp.GaborFilter(*f) for f in GABOR], pad=5)
        st.layers = [_layer(w, p, case["precision"]) for w, p in zip(st.start, (3, 2))]
    else:
        st.bank = sp.DoG(3, [sp.DoGFilter(*f) for f in DOG], pad=3)
        st.layers = [_layer(w, 2, case.get("precision")) for w in st.start]
    return st


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------


def _run_features(st):
    case = st.case
    codes = sp.code(st.bank(st.images), case["time"])
    _, _, maps = sp.conv_fire_wta(codes, st.layers[0], TH1, 0, 0, pool=2)
    _, _, out = sp.conv_fire_wta(maps, st.layers[1], TH2, 0, 0, pool=maps.shape[-1])
    return {"maps": maps, "features": out}


def _run_textures(st):
    codes = sp.code(st.bank(st.images), st.case["time"])
    _, _, maps = sp.conv_fire_wta(codes, st.layers[0], 20.0, 0, 0, pool=2)
    _, _, out = sp.conv_fire_wta(maps, st.layers[1], 12.0, 0, 0, pool=2)
    return {"maps": maps, "features": out}


def _run_train(st):
    case = st.case
    x = sp.code(st.bank(st.images), case["time"])
    out = {}
    for i, (theta, radius, count) in enumerate(((TH1, 3, 5), (TH2, 1, 8))[: case["layers"]]):
        layer = st.layers[i]
        layer.kernel.copy_(st.start[i])
        spikes, winners, pooled = sp.conv_fire_wta(x, layer, theta, radius, count, pool=2 if i == 0 else x.shape[-1])
        layer.stdp(x, winners, spikes)
        out[f"winners{i}"], out[f"weights{i}"], out[f"pooled{i}"] = winners.records, layer.kernel, pooled
        x = pooled
    return out


def _run_ops(st):
    x = sp.code(st.bank(st.images), st.case["time"])
    out = {}
    for i, (theta, radius, count) in enumerate(((TH1, 3, 5), (TH2, 1, 8))):
        layer = st.layers[i]
        layer.kernel.copy_(st.start[i])
        pot = sp.inhibit(sp.threshold(layer(x), theta))
        spikes = sp.fire(pot)
        winners = sp.convwta(pot, radius, count)
        layer.stdp(x, winners, spikes)
        pooled = sp.pool(spikes, 2 if i == 0 else x.shape[-1])
        out[f"winners{i}"], out[f"weights{i}"], out[f"pooled{i}"] = winners.records, layer.kernel, pooled
        out[f"potentials{i}"] = pot
        x = pooled
    return out


def _run_backprop(st):
    net = st.net
    t_out = net.forward(net.input_times(st.images))
    loss = net.loss(t_out, st.target)
    grads = torch.autograd.grad(loss, net.weights)
    return {"times": t_out.detach(), "loss": loss.detach(), "grads": list(grads)}


def _run_sparse(st):
    th = _sparse_thresholds(st.case)
    x, out = st.events, {}
    for i, (radius, count) in enumerate(((3, 5), (1, 8))):
        layer = st.layers[i]
        layer.kernel.copy_(st.start[i])
        y = sparse.inhibit(sparse.conv(x, layer.kernel, th[i], 1, 2))
        winners = sparse.convwta(y, radius, count)
        sparse.stdp(layer, x, winners)
        out[f"winners{i}"], out[f"weights{i}"] = winners.records, layer.kernel
        if i == 0:
            x = sparse.pool(y, 2)
            out["maps"] = sparse.gather(x)
        else:
            out["times"] = sparse.gather(y)
    return out


def _run_rstdp(st):
    net = st.net
    net.conv3.kernel.copy_(st.start[2])
    labels = net.train_layer3(net.transform(st.images), st.target)
    return {"labels": labels, "weights": net.conv3.kernel}


def _run_sweep(st):
    st.sweep.w1.copy_(st.start[0])
    st.sweep.w2.copy_(st.start[1])
    features = torch.cat(list(st.sweep.replay()))[st.sweep.order]  # of size after size, put into the order of the streams
    return {"features": features, "weights": [st.sweep.w1, st.sweep.w2]}


RUN = {"features": _run_features, "textures": _run_textures, "train": _run_train, "ops": _run_ops,
       "backprop": _run_backprop, "sparse": _run_sparse, "rstdp": _run_rstdp, "sweep": _run_sweep}


def run(state):
    return RUN[state.case["kind"]](state)


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------


def work(case):
    """Bytes: the images or events, the weights (read, and written where they learn), and what the calls hand back, each
    once.  FLOPs: every input neuron's weights added once to the potentials they reach (its spike lasts to the last step,
    so no step needs them again); a backward pass adds each of them twice more."""
    kind = case["kind"]
    if kind == "sweep":
        n, px = case["nets"] * case["images"], (400 + 784 + 1600 + 4096) / 4
        layers = [(2, C1, 25, px), (C1, C2, 25, px / 4)]
        out = n * 15 * (C1 * px * 1.25 + C2 * (px / 4 + 1))
        w = case["nets"] * sum(ci * co * k for ci, co, k, _ in layers)
        return {"bytes": 4 * n * px + out + 8 * w, "flops": 2 * n * sum(ci * co * k * p for ci, co, k, p in layers)}
    n, s = case["batch"], case["side"]
    t = case.get("time", 15)
    if kind == "textures":
        layers = [(8, 64, 49, s * s), (64, 256, 25, (s // 2) ** 2)]
        out = t * (64 * (s * s + (s // 2) ** 2) + 256 * ((s // 2) ** 2 + (s // 4) ** 2))
    elif kind == "rstdp":
        p2 = s // 2
        p3 = p2 // 3
        layers = [(6, 30, 25, s * s), (30, 250, 9, p2 * p2), (250, 200, 25, p3 * p3)]
        out = t * (30 * (5 * s * s + p2 * p2) + 250 * (5 * p2 * p2 + p3 * p3) + 200 * 5 * p3 * p3)
    elif kind == "backprop":
        p2, p3 = s // 2, s // 4
        layers = [(1, 32, 25, s * s), (32, 64, 9, p2 * p2), (64 * p3 * p3, 10, 1, 1)]
        out = 2 * 4 * (s * s + 32 * (s * s + p2 * p2) + 64 * (p2 * p2 + p3 * p3) + 10)
    else:
        p2 = s // 2
        layers = [(2, C1, 25, s * s), (C1, C2, 25, p2 * p2)][: case.get("layers", 2)]
        each = 5 if kind == "ops" else 1  # op by op the potentials (F32) come back too
        if kind == "sparse":
            out = C1 * p2 * p2 + C2 * p2 * p2
        else:
            out = t * C1 * (each * s * s + p2 * p2) + (t * C2 * (each * p2 * p2 + 1) if len(layers) == 2 else 0)
    w = sum(ci * co * k for ci, co, k, _ in layers)
    flops = 2 * n * sum(ci * co * k * p for ci, co, k, p in layers)
    learns = kind in ("train", "ops", "sparse", "rstdp", "backprop")
    image = 2 * s * s * case["density"] * 4 if kind == "sparse" else 4 * s * s
    if kind == "sparse":
        flops *= case["density"]
    return {"bytes": n * (image + out) + (8 if learns else 4) * w, "flops": flops * (3 if kind == "backprop" else 1)}


# ---------------------------------------------------------------------------
# the same in 64 bits, in plain torch and numpy
# ---------------------------------------------------------------------------


def _filter64(images, bank):
    kernels = []
    n = torch.arange(-3, 4, dtype=torch.float64)
    d2 = n[:, None] ** 2 + n[None, :] ** 2
    for std in [f[0] for f in bank] + [f[1] for f in bank]:
        k = torch.exp(-0.5 * d2 / std ** 2)
        kernels.append((k / k.sum()).float().double())
    mid = F.conv2d(images.double(), torch.stack(kernels)[:, None].cuda(), padding=3).float()
    return (mid[:, : len(bank)] - mid[:, len(bank):]).clamp_min(0)


def _code_times64(x, t):
    """Rank order, larger first, ties by index; the row's minima keep counting on from the others."""
    flat = x.flatten(1)
    order = flat.sort(dim=1, descending=True, stable=True).indices
    rank = torch.empty_like(order).scatter_(1, order, torch.arange(flat.shape[1], device="cuda").expand_as(order))
    above = (flat > flat.amin(1, keepdim=True)).sum(1, keepdim=True)
    scale = numpy.float32(numpy.float32(t) + numpy.float32(1e-5))
    scale = torch.tensor(scale, device="cuda") / above.float()
    return (rank.float() * scale).clamp_max(t).floor().view_as(x).to(torch.int64)


def _conv64(times, w, pad, t):
    """Potentials [n, t, z, h, w], summed in 64 bits, stored in 32."""
    n = times.shape[0]
    steps = torch.arange(t, device="cuda").view(1, t, 1, 1, 1)
    x = (times[:, None] <= steps).flatten(0, 1).double()
    v = F.conv2d(x, w.double(), padding=pad).float()
    return v.view(n, t, *v.shape[1:])


def _first(fired, t):
    """First step of cumulative spikes along dim 1, t where none."""
    return t - fired.sum(1)


def _pool64(times, p):
    return -F.max_pool2d(-times.double(), p).long()


def _inhibit64(v, theta):
    t = v.shape[1]
    v = torch.where(v > theta, v, torch.zeros_like(v))
    best, ch = v.max(2)
    win = ch.gather(1, (t - (best > 0).sum(1).clamp_min(1))[:, None])
    return v * (torch.arange(v.shape[2], device="cuda").view(1, 1, -1, 1, 1) == win[:, :, None])


def _winners64(v, radius, count):
    """[n, count, 3] (map, y, x), -1 where there is no further winner."""
    n, t, c, h, w = v.shape
    lo, hi = v.flatten(1).amin(1).view(n, 1, 1, 1), v.flatten(1).amax(1).view(n, 1, 1, 1)
    first = _first(v > 0, t)
    at = v.gather(1, first.clamp_max(t - 1)[:, None])[:, 0]
    key = torch.where(first < t, (t - 1 - first).float() + (at - lo) / ((hi - lo) * 2), torch.full_like(at, -1e30))
    ys, xs = torch.arange(h, device="cuda").view(1, 1, h, 1), torch.arange(w, device="cuda").view(1, 1, 1, w)
    out = []
    for _ in range(count):
        # the first of the largest
        top = key.flatten(1).amax(1, keepdim=True)
        idx = (key.flatten(1) == top).int().argmax(1)
        z, y, x = idx // (h * w), idx % (h * w) // w, idx % w
        alive = top[:, 0] > -1e29
        out.append(torch.where(alive[:, None], torch.stack([z, y, x], 1), -1))
        z, y, x = (q.view(n, 1, 1, 1) for q in (z, y, x))
        gone = ((ys - y).abs() <= radius) & ((xs - x).abs() <= radius)
        gone = gone | (torch.arange(c, device="cuda").view(1, c, 1, 1) == z)
        key = torch.where(gone, torch.full_like(key, -1e30), key)
    return torch.stack(out, 1)


def _stdp64(w, times, post, winners, pad, configs, choice=None, bound=(0.0, 1.0), stabilize=True):
    """Every winner in turn pulls its map's weights up where the input fired no later than it did, else down."""
    w = w.double().cpu().numpy().copy()
    pre = F.pad(times, (pad,) * 4, value=1 << 20).cpu().numpy()
    post, winners = post.cpu().numpy(), winners.cpu().numpy()
    k = w.shape[-1]
    lo, hi = bound
    for i in range(len(winners)):
        for z, y, x in winners[i]:
            if z < 0:
                break
            up, down = configs[0 if choice is None else int(choice[i])]
            m = w[z]
            rate = numpy.where(pre[i, :, y:y + k, x:x + k] <= post[i, z, y, x], up, down)
            w[z] = numpy.clip(m + rate * ((m - lo) * (hi - m) if stabilize else 1.0), lo, hi)
    return torch.from_numpy(w)


def _chunks(n, most=64):
    return [slice(a, min(n, a + most)) for a in range(0, n, most)]


def _layer64(times, w, theta, pad, t, radius, count, keep=False):
    first, wins, pots = [], [], []
    for s in _chunks(len(times)):
        v = _inhibit64(_conv64(times[s], w, pad, t), theta)
        first.append(_first(v > 0, t))
        wins.append(_winners64(v, radius, count))
        if keep:
            pots.append(v)
    return torch.cat(first), torch.cat(wins), torch.cat(pots) if keep else None


def _exact_train(case, seed, keep):
    t, out = case["time"], {}
    times = _code_times64(_filter64(_strokes(case["batch"], case["side"], seed), DOG), t)
    for i, (theta, radius, count) in enumerate(((TH1, 3, 5), (TH2, 1, 8))[: case.get("layers", 2)]):
        w = _weights(case, seed)[i]
        post, wins, pot = _layer64(times, w, theta, 2, t, radius, count, keep)
        out[f"winners{i}"], out[f"pooled{i}"] = None, None
        out[f"weights{i}"] = _stdp64(w, times, post, wins, 2, [RATES])
        if keep:
            out[f"potentials{i}"] = pot.double()
        times = _pool64(post, 2)
    return out


def _exact_sparse(case, seed):
    """Event lists: a position's first event inhibits the other maps there; winners in order of (step, map, pixel)."""
    t, th, out = case["time"], _sparse_thresholds(case), {"maps": None, "times": None}
    times = _events(case, seed).long()
    for i, (radius, count) in enumerate(((3, 5), (1, 8))):
        w = _weights(case, seed)[i]
        posts, wins = [], []
        for s in _chunks(len(times)):
            fired = _conv64(times[s], w, 2, t) > th[i]
            first = _first(fired, t)
            n, c, h, wd = first.shape
            best = first.amin(1, keepdim=True)
            ch = (first == best).int().argmax(1, keepdim=True)
            keep = (torch.arange(c, device="cuda").view(1, c, 1, 1) == ch) & (first < t)
            first = torch.where(keep, first, torch.full_like(first, t))
            posts.append(first)
            key = torch.where(keep, (t - first).float(), torch.zeros_like(first, dtype=torch.float32))
            # as potentials of a single step, earlier is larger; the first of the largest wins
            ranked = []
            ys, xs = torch.arange(h, device="cuda").view(1, 1, h, 1), torch.arange(wd, device="cuda").view(1, 1, 1, wd)
            for _ in range(count):
                top = key.flatten(1).amax(1, keepdim=True)
                idx = (key.flatten(1) == top).int().argmax(1)
                zyx = torch.stack([idx // (h * wd), idx % (h * wd) // wd, idx % wd], 1)
                ranked.append(torch.where(top > 0, zyx, -1))
                z, y, x = (q.view(n, 1, 1, 1) for q in zyx.unbind(1))
                gone = (((ys - y).abs() <= radius) & ((xs - x).abs() <= radius)) | (
                    torch.arange(c, device="cuda").view(1, c, 1, 1) == z)
                key = torch.where(gone, torch.zeros_like(key), key)
            wins.append(torch.stack(ranked, 1))
        post, win = torch.cat(posts), torch.cat(wins)
        out[f"winners{i}"] = None
        out[f"weights{i}"] = _stdp64(w, times, post, win, 2, [RATES])
        times = _pool64(post, 2)
    return out


def _exact_rstdp(case, seed):
    t = 15
    x = _filter64(_strokes(case["batch"], case["side"], seed), DOG6)
    times = _code_times64(torch.where(x > 0.02, x, torch.zeros_like(x)), t)
    w = _weights(case, seed)
    for i, (theta, pad, p) in enumerate(((15.0, 2, 2), (5.0, 1, 3))):
        times = torch.cat([_pool64(_first(_conv64(times[s], w[i], pad, t) > theta, t), p)
                           for s in _chunks(len(times), 16)])
    v = torch.cat([_conv64(times[s], w[2], 2, t)[:, -1] for s in _chunks(len(times), 16)])
    n, c, h, wd = v.shape
    lo, hi = torch.zeros_like(v.flatten(1)[:, :1]), v.flatten(1).amax(1, keepdim=True)
    key = torch.where(v.flatten(1) > 0, (v.flatten(1) - lo) / ((hi - lo) * 2), torch.full_like(v.flatten(1), -1))
    top = key.amax(1, keepdim=True)
    idx = (key == top).int().argmax(1)
    win = torch.where(top >= 0, torch.stack([idx // (h * wd), idx % (h * wd) // wd, idx % wd], 1), -1)[:, None]
    target = torch.randint(0, 10, (n,), generator=_gen(seed, 4), device="cuda")
    wrong = (win[:, 0, 0] // (c // 10)) != target
    post = torch.full((n, c, h, wd), t - 1)
    out = _stdp64(w[2], times, post, win, 2, [(0.004, -0.003), (-0.004, 0.0005)], wrong.tolist(), (0.2, 0.8), False)
    return {"labels": None, "weights": out}


def _exact_backprop(case, seed):
    t, n = case["time"], case["batch"]
    net = temporal.TemporalNet(time=t, seed=seed, size=case["side"])  # its seeded weights
    w = [x.detach().double() for x in net.weights]
    th = (0.5, 2.0, 40.0)
    x0 = _code_times64(_strokes(n, case["side"], seed), t)

    def conv(times, k, theta, pad):
        return torch.cat([_first(_conv64(times[s], k, pad, t) > theta, t) for s in _chunks(n, 16)])

    def pool(times):
        o, i = F.max_pool2d(-times.double(), 2, return_indices=True)
        return -o.long(), i

    a1 = conv(x0, w[0], th[0], 2)
    p1, i1 = pool(a1)
    a2 = conv(p1, w[1], th[1], 1)
    p2, i2 = pool(a2)
    flat = p2.reshape(n, -1, 1, 1)
    w3 = w[2].reshape(10, -1, 1, 1)
    out = conv(flat, w3, th[2], 0).reshape(n, 10)

    target = torch.randint(0, 10, (n,), generator=_gen(seed, 4), device="cuda")
    now = out.double()
    least = now.amin(1, keepdim=True)
    upper = least + 3.0
    want = torch.where((now < upper) & (least != t), upper.clamp_max(t), now)
    want.scatter_(1, target[:, None], least.clamp_min(0))
    g = (want - now) / t
    loss = (g ** 2).sum() * (0.5 * t)

    def back(tin, k, tout, go, pad, need_in):
        kh = k.shape[-1]
        oh, ow = tout.shape[2:]
        tp = F.pad(tin, (pad,) * 4, value=1 << 20)
        gk, gi = torch.zeros_like(k), torch.zeros(tp.shape, dtype=torch.float64, device="cuda")
        for s in _chunks(n, 4):
            for y in range(kh):
                for x in range(kh):
                    before = tp[s, None, :, y:y + oh, x:x + ow] < tout[s, :, None]
                    sel = before * go[s, :, None]
                    gk[:, :, y, x] -= sel.sum((0, 3, 4))
                    if need_in:
                        gi[s, :, y:y + oh, x:x + ow] += (sel * k[None, :, :, y, x, None, None]).sum(1)
        h, wd = tin.shape[2:]
        return gk, gi[:, :, pad:pad + h, pad:pad + wd]

    def unpool(go, index, like):
        return torch.zeros_like(like, dtype=torch.float64).flatten(2).scatter_(2, index.flatten(2), go.flatten(2)) \
            .view(like.shape)

    g3, gi = back(flat, w3, out.view(n, 10, 1, 1), -g.view(n, 10, 1, 1), 0, True)
    g2, gi = back(p1, w[1], a2, unpool(gi.reshape(p2.shape), i2, a2), 1, True)
    g1, _ = back(x0, w[0], a1, unpool(gi, i1, a1), 2, False)
    return {"times": now, "loss": loss, "grads": [g1, g2, g3.reshape(10, -1)]}


def exact(case, seed):
    kind = case["kind"]
    if kind in ("train", "ops"):
        return _exact_train(case, seed, kind == "ops")
    if kind == "sparse":
        return _exact_sparse(case, seed)
    if kind == "rstdp":
        return _exact_rstdp(case, seed)
    if kind == "backprop":
        return _exact_backprop(case, seed)
    return None  # features, textures: bytes only; sweep: its networks draw their own streams
