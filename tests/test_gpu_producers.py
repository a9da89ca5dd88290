"""Operand gathering of the tensor-core convolutions at its edges: 8- and
16-byte loads (channel groups), fewer K blocks than producer groups, last K
blocks of one half, strides, pads wider than the input, several channel parts
with ties between them; against FP64 sums."""

import numpy as np
import pytest
import torch

import spyker_b200 as spyker

pytestmark = pytest.mark.gpu

# n, cin, h, w, cout, k, stride, pad
SHAPES = [
    (1, 2, 1, 1, 3, 1, 1, 0),
    (3, 8, 5, 4, 17, 1, 1, 0),
    (2, 16, 9, 9, 40, 3, 2, 4),
    (5, 24, 7, 6, 130, 3, 1, 1),
    (2, 48, 6, 6, 250, 5, 1, 2),
    (40, 33, 12, 12, 33, 2, 3, 0),
]


@pytest.mark.parametrize("precision,eps", [("bf16x3", 2.0**-22), ("bf16x2", 2.0**-14)])
@pytest.mark.parametrize("shape", SHAPES)
def test_potentials(shape, precision, eps):
    n, cin, h, w, cout, k, stride, pad = shape
    g = torch.Generator().manual_seed(cin)
    x = (torch.rand((n, 1, cin, h, w), generator=g) < 0.4).to(torch.uint8)
    kern = torch.randn((cout, cin, k, k), generator=g)
    out = spyker.conv(x.cuda(), kern.cuda(), stride, pad, precision=precision).cpu().double()[:, 0]
    ref = torch.nn.functional.conv2d(x[:, 0].double(), kern.double(), stride=stride, padding=pad)
    mag = torch.nn.functional.conv2d(x[:, 0].double(), kern.double().abs(), stride=stride, padding=pad)
    # each weight's split and the FP32 accumulation of K products, relative to the sum of magnitudes
    assert bool(((out - ref).abs() <= mag * (eps + cin * k * k * 2.0**-23) + 1e-30).all())


@pytest.mark.parametrize("cin,cout,k", [(4, 40, 3), (16, 200, 3), (40, 300, 5), (24, 130, 1)])
def test_search_rounds_parts(port, cin, cout, k):
    rng = np.random.default_rng(cout)
    b, t, side = (300, 5, 24) if cin == 4 else (60, 5, 24)
    fst = rng.integers(0, t + 2, size=(b, cin, side, side))
    x = (fst[:, None] <= np.arange(t)[None, :, None, None, None]).astype(np.uint8)
    kern = (rng.integers(0, 2, size=(cout, cin, k, k)) * 0.5).astype(np.float32)
    kern[cout // 2:] = kern[:cout - cout // 2] * rng.choice([1, 1, 0.125], size=(cout - cout // 2, 1, 1, 1)).astype(np.float32)
    thr = float(cin * k * k) * 0.2
    conv = spyker.Conv(cin, cout, k, pad=k // 2)
    conv.kernel.copy_(torch.from_numpy(kern))
    conv.precision = "bf16x3"
    spk, wins = spyker.conv_fire_wta(torch.from_numpy(x).cuda(), conv, thr, 1, 4)
    assert spyker._lib.lib.spk_device_status(1) == 0
    take = 2
    inh = port.inhibit(port.threshold(port.conv(x[:take], kern, (1, 1), (k // 2,) * 4), thr))
    assert np.array_equal(spk[:take].cpu().numpy(), port.fire(inh))
    rec, cnt = port.convwta(inh, (1, 1), 4)
    for i in range(take):
        rec[i, cnt[i]:] = 0
    assert np.array_equal(wins.records[:take].cpu().numpy(), rec)
    assert int(spk[:, -1].sum()) > 0
