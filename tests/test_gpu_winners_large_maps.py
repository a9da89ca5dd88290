"""Winners of a fused layer on maps whose keys need more than the default shared
memory (above 6112 pixels, up to the layer's limit of 16384) against the oracle."""

import numpy as np
import pytest
import torch

import spyker_b200 as spyker

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("b,h,w", [(1, 78, 78), (2, 79, 79), (3, 96, 96), (1, 128, 128), (1, 1, 16384)])
def test_winners_of_large_maps(port, b, h, w):
    rng = np.random.default_rng(h)
    fst = rng.integers(0, 9, size=(b, 2, h, w))
    x = (fst[:, None] <= np.arange(7)[None, :, None, None, None]).astype(np.uint8)
    kern = (rng.integers(0, 3, size=(6, 2, 3, 3)) * 0.25).astype(np.float32)  # quarters: equal keys
    conv = spyker.Conv(2, 6, 3, pad=1)
    conv.kernel.copy_(torch.from_numpy(kern))
    conv.precision = "bf16x3"
    _, wins = spyker.conv_fire_wta(torch.from_numpy(x).cuda(), conv, 1.0, 2, 8)
    inh = port.inhibit(port.threshold(port.conv(x, kern, (1, 1), (1, 1, 1, 1)), 1.0))
    rec, cnt = port.convwta(inh, (2, 2), 8)
    for i in range(b):
        rec[i, cnt[i]:] = 0
    assert np.array_equal(wins.counts.cpu().numpy(), cnt)
    assert np.array_equal(wins.records.cpu().numpy(), rec)
