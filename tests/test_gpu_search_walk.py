"""The search by walking inputs in spike order (few output pixels) at the edges
of its ranges (inputs and channels per lane, strides, pads, T = 1 and 32, no
spikes, saturated and tiny weights, thresholds on exact sums, a zero threshold),
against the oracle's pipeline, and equal to the bisection rounds that larger
calls take."""

import numpy as np
import pytest
import torch

import spyker_b200 as spyker

pytestmark = pytest.mark.gpu

# b, t, cin, h, w, cout, k, stride, pad
LAYERS = [
    (1, 1, 1, 1, 1, 2, 1, 1, 0),
    (3, 32, 1, 9, 7, 30, 3, 1, 1),
    (2, 15, 2, 12, 12, 33, 5, 2, 2),  # two channels a lane
    (2, 8, 9, 7, 11, 64, 5, 1, 2),  # 50 groups of 8 inputs: two loads a lane
    (2, 15, 30, 10, 10, 100, 5, 1, 2),  # four loads, four channels
    (1, 12, 64, 6, 6, 129, 5, 1, 0),  # 200 groups: eight loads, eight channels a lane
    (1, 9, 64, 8, 8, 256, 5, 1, 2),
    (2, 7, 80, 5, 5, 20, 5, 1, 2),  # 250 groups
    (1, 7, 88, 5, 5, 20, 5, 1, 2),  # 275 groups: the rounds
]


def weights(kind, rng, shape):
    if kind == "fresh":
        return np.clip(rng.normal(0.8, 0.05, size=shape), 0, 1).astype(np.float32)
    if kind == "trained":  # most near the ends, far below the channel's grid
        return (1 / (1 + np.exp(-rng.normal(0, 6, size=shape)))).astype(np.float32)
    return (rng.integers(0, 3, size=shape) * 0.5).astype(np.float32)  # halves: ties, sums on the threshold


@pytest.mark.parametrize("kind", ["fresh", "trained", "halves"])
@pytest.mark.parametrize("layer", LAYERS)
def test_walk_equals_oracle(port, layer, kind):
    b, t, cin, h, w, cout, k, stride, pad = layer
    rng = np.random.default_rng(cin + cout + t)
    fst = rng.integers(0, t + 3, size=(b, cin, h, w))
    fst[0] = np.where(rng.random(fst[0].shape) < 0.8, t, fst[0])  # a sparse sample
    x = (fst[:, None] <= np.arange(t)[None, :, None, None, None]).astype(np.uint8)
    kern = weights(kind, rng, (cout, cin, k, k))
    pots = port.conv(x, kern, (stride, stride), (pad,) * 4)
    mid = float(np.round(np.median(pots[:, -1].max(1)) * 2) / 2)
    for thr in (0.0, mid, 1e9):
        layer_ = spyker.Conv(cin, cout, k, stride=stride, pad=pad)
        layer_.kernel.copy_(torch.from_numpy(kern))
        layer_.precision = "bf16x3"
        spk, wins = spyker.conv_fire_wta(torch.from_numpy(x).cuda(), layer_, thr, 1, 4)
        assert spyker._lib.lib.spk_device_status(1) == 0
        inh = port.inhibit(port.threshold(pots, thr))
        assert np.array_equal(spk.cpu().numpy(), port.fire(inh))
        rec, cnt = port.convwta(inh, (1, 1), 4)
        assert np.array_equal(wins.counts.cpu().numpy(), cnt)
        for i in range(b):
            rec[i, cnt[i]:] = 0
        assert np.array_equal(wins.records.cpu().numpy(), rec)  # zero past the count


def test_walk_equals_rounds():
    """The same images one by one (walk) and in one call above the walk's
    pixels (rounds): spikes, pooled spikes and winners."""
    rng = np.random.default_rng(6)
    b = 200
    fst = torch.from_numpy(rng.integers(0, 22, size=(b, 2, 28, 28)))
    x = (fst[:, None] <= torch.arange(15).view(1, 15, 1, 1, 1)).to(torch.uint8).cuda()
    conv = spyker.Conv(2, 30, 5, pad=2)
    conv.kernel.copy_(torch.from_numpy(weights("trained", rng, (30, 2, 5, 5))))
    conv.precision = "bf16x3"
    spk, wins, pooled = spyker.conv_fire_wta(x, conv, 9.0, 3, 5, pool=2)
    for i in range(0, b, 50):
        s, w, p = spyker.conv_fire_wta(x[i:i + 1], conv, 9.0, 3, 5, pool=2)
        assert torch.equal(s, spk[i:i + 1]) and torch.equal(p, pooled[i:i + 1])
        assert torch.equal(w.records, wins.records[i:i + 1]) and torch.equal(w.counts, wins.counts[i:i + 1])
    assert int(spk[:, -1].sum()) > 0
