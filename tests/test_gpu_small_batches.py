"""Few-sample forms of the fused layer's helpers against the oracle's pipeline:
a winner selection with a CTA per sample and with a warp per sample (few and
many samples, maps at the edges of their sizes, radii that leave the map, more
rounds than winners), and first-spike staging in runs of an image's pixels."""

import numpy as np
import pytest
import torch

import spyker_b200 as spyker

pytestmark = pytest.mark.gpu


# samples, side, radius, winners: a CTA per sample up to 8 per SM, a warp after
@pytest.mark.parametrize("b,side,radius,count", [(1, 1, 0, 3), (3, 16, 9, 4), (2, 17, 1, 6), (5, 32, 2, 5), (2, 33, 40, 3),
                                                 (1, 66, 3, 8), (1500, 6, 1, 3)])
def test_winners_of_few_and_many_samples(port, b, side, radius, count):
    rng = np.random.default_rng(b + side)
    fst = rng.integers(0, 9, size=(b, 2, side, side))
    x = (fst[:, None] <= np.arange(7)[None, :, None, None, None]).astype(np.uint8)
    kern = (rng.integers(0, 3, size=(6, 2, 3, 3)) * 0.25).astype(np.float32)  # quarters: equal keys
    conv = spyker.Conv(2, 6, 3, pad=1)
    conv.kernel.copy_(torch.from_numpy(kern))
    conv.precision = "bf16x3"
    _, wins = spyker.conv_fire_wta(torch.from_numpy(x).cuda(), conv, 1.0, radius, count)
    take = min(b, 40)
    inh = port.inhibit(port.threshold(port.conv(x[:take], kern, (1, 1), (1, 1, 1, 1)), 1.0))
    rec, cnt = port.convwta(inh, (radius, radius), count)
    for i in range(take):
        rec[i, cnt[i]:] = 0
    assert np.array_equal(wins.counts[:take].cpu().numpy(), cnt)
    assert np.array_equal(wins.records[:take].cpu().numpy(), rec)


# runs of 128 pixels: one, one and a bit, several, a last one of 4
@pytest.mark.parametrize("b,cin,h,w", [(1, 2, 8, 16), (2, 3, 4, 33), (1, 9, 20, 20), (3, 1, 26, 30), (1, 40, 18, 18)])
def test_staging_in_runs(port, b, cin, h, w):
    rng = np.random.default_rng(cin + h)
    fst = rng.integers(0, 14, size=(b, cin, h, w))
    x = (fst[:, None] <= np.arange(12)[None, :, None, None, None]).astype(np.uint8)
    kern = rng.random((8, cin, 3, 3)).astype(np.float32)
    pots = port.conv(x, kern, (1, 1), (1, 1, 1, 1))
    thr = float(np.median(pots[:, -1].max(1)))
    conv = spyker.Conv(cin, 8, 3, pad=1)
    conv.kernel.copy_(torch.from_numpy(kern))
    conv.precision = "bf16x3"
    spk, _ = spyker.conv_fire_wta(torch.from_numpy(x).cuda(), conv, thr, 1, 2)
    assert np.array_equal(spk.cpu().numpy(), port.fire(port.inhibit(port.threshold(pots, thr))))
