"""The first-crossing search's rounds (layers of more pixels than the walk takes)
against the oracle's pipeline, where their decisions are hardest: weights at the
bounds STDP drives them to, far below the largest of their channel and in between,
ties of a potential with the threshold and between channels (across channel parts
too), weights reached by training, and every pipeline schedule.  The results, bit
for bit, do not show which search ran; the number of launches does."""

import numpy as np
import pytest
import torch

import spyker_b200 as spyker
from tests.test_gpu_fused_search import check, cuda, cumulative, host, trained, weights  # noqa: F401

pytestmark = pytest.mark.gpu

LAYERS = [
    # b, t, cin, h, w, cout, k, pad, theta, radius, count
    (172, 15, 2, 28, 28, 30, 5, 2, 15.0, 3, 5),
    (125, 15, 30, 14, 14, 100, 5, 2, 10.0, 1, 8),
]
PARTS = (150, 6, 16, 10, 10, 256, 5, 2, 10.0, 1, 4)  # two parts of 128 channels


def rounds(port, x, w, *args, **kwargs):
    n = spyker._lib.lib.spk_launch_count()
    out = check(port, x, w, *args, **kwargs)
    assert spyker._lib.lib.spk_launch_count() - n > 12, "the layer took the walk"
    return out


@pytest.mark.parametrize("layer", LAYERS + [PARTS])
@pytest.mark.parametrize("kind", ["binary", "near_one", "tiny", "log_uniform", "halves"])
def test_saturated_weights(port, layer, kind):
    b, t, cin, h, wd, cout, k, pad, theta, radius, count = layer
    rng = np.random.default_rng(sum(map(ord, kind)) + cin)
    x = cumulative(rng, b, t, cin, h, wd)
    w = weights(kind, rng, (cout, cin, k, k))
    if cout == 256:
        w[200:] = w[:56]  # channels 200.. tie exactly with channels 0..55 (other part)
    # a threshold the potentials reach exactly (a half-integer near the median)
    th = float(np.round(np.median(port.conv(x[:8, -1:], w, (1, 1), (pad,) * 4)) * 2) / 2)
    assert rounds(port, x, w, max(th, 1.0), radius, count, pad)[0] > 0


@pytest.mark.parametrize("layer", LAYERS)
def test_channel_ties(port, layer):
    b, t, cin, h, wd, cout, k, pad, theta, radius, count = layer
    rng = np.random.default_rng(3)
    x = cumulative(rng, b, t, cin, h, wd)
    w = rng.uniform(0.3, 1.0, size=(cout, cin, k, k)).astype(np.float32)
    w[1::2] = w[0::2][: w[1::2].shape[0]]
    w[cout - 3] = w[2]
    assert rounds(port, x, w, theta, radius, count, pad)[0] > 0


def test_potentials_at_threshold(port):
    rng = np.random.default_rng(9)
    x = cumulative(rng, 172, 15, 2, 28, 28)
    w = np.ones((30, 2, 5, 5), np.float32)
    w[::3, 1] = 0.0
    for theta in (10.0, 22.0):
        rounds(port, x, w, theta, 3, 5, 2)


def test_trained_weights(port, trained):  # noqa: F811
    w1, w2, codes = trained
    spk1 = port.fire(port.inhibit(port.threshold(port.conv(codes, w1, (1, 1), (2,) * 4), 15.0)))
    assert rounds(port, np.concatenate([codes, codes[::-1]]), w1, 15.0, 3, 5, 2)[0] > 0
    maps = port.pool(spk1, (2, 2))
    assert rounds(port, np.concatenate([maps, maps[::-1]]), w2, 10.0, 1, 8, 2, pool=7)[0] > 0


@pytest.mark.parametrize("schedule", [(2, 1, 1), (3, 2, 1), (6, 1, 2)])
def test_schedules(port, schedule):
    b, t, cin, h, wd, cout, k, pad, theta, radius, count = LAYERS[1]
    rng = np.random.default_rng(8)
    x = cumulative(rng, b, t, cin, h, wd)
    w = rng.uniform(0.0, 1.0, size=(cout, cin, k, k)).astype(np.float32)
    spyker._lib.call("spk_set_conv_schedule", *schedule)
    try:
        assert rounds(port, x, w, 60.0, radius, count, pad)[0] > 0
    finally:
        spyker._lib.call("spk_set_conv_schedule", 0, 0, 0)


def test_walk_and_rounds_agree():
    """A layer of 256 channels in one call (rounds) and image by image (walk)."""
    g = torch.Generator("cuda").manual_seed(4)
    x = (torch.randint(0, 12, (100, 1, 12, 16, 16), generator=g, device="cuda")
         <= torch.arange(9, device="cuda").view(1, 9, 1, 1, 1)).to(torch.uint8)
    conv = spyker.Conv(12, 200, 5, pad=2)
    conv.kernel.copy_(torch.exp2(-20 * torch.rand(conv.kernel.shape, generator=g, device="cuda")))
    conv.precision = "bf16x3"
    count = spyker._lib.lib.spk_launch_count
    n = count()
    spk, wins, pooled = spyker.conv_fire_wta(x, conv, 8.0, 1, 5, pool=2)
    assert count() - n > 12
    for i in range(0, 100, 23):
        n = count()
        s, w, p = spyker.conv_fire_wta(x[i:i + 1], conv, 8.0, 1, 5, pool=2)
        assert count() - n < 12
        assert torch.equal(s, spk[i:i + 1]) and torch.equal(p, pooled[i:i + 1])
        assert torch.equal(w.records, wins.records[i:i + 1])
    assert int(spk[:, -1].sum()) > 0
