"""Winner selection with a warp per sample (more than 8 samples an SM) in its three
forms, of 8, 25 and 32 pixels a lane, at the edges of their sizes against the
oracle: radii that leave the map, more rounds than winners, equal keys."""

import numpy as np
import pytest
import torch

import spyker_b200 as spyker

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("h,w", [(16, 16), (1, 257), (17, 17), (28, 28), (25, 32), (27, 30), (32, 32)])
@pytest.mark.parametrize("radius,count", [(0, 40), (2, 5), (40, 3)])
def test_warp_forms(port, h, w, radius, count):
    rng = np.random.default_rng(h + radius)
    b, take = 8 * torch.cuda.get_device_properties(0).multi_processor_count + 10, 20
    fst = rng.integers(0, 9, size=(b, 2, h, w)).astype(np.uint8)
    x = (fst[:, None] <= np.arange(7)[None, :, None, None, None]).astype(np.uint8)
    kern = (rng.integers(0, 3, size=(6, 2, 3, 3)) * 0.25).astype(np.float32)  # quarters: equal keys
    conv = spyker.Conv(2, 6, 3, pad=1)
    conv.kernel.copy_(torch.from_numpy(kern))
    conv.precision = "bf16x3"
    _, wins = spyker.conv_fire_wta(torch.from_numpy(x).cuda(), conv, 1.0, radius, count)
    some = np.r_[0:take, b - take:b]
    inh = port.inhibit(port.threshold(port.conv(x[some], kern, (1, 1), (1, 1, 1, 1)), 1.0))
    rec, cnt = port.convwta(inh, (radius, radius), count)
    for i in range(len(some)):
        rec[i, cnt[i]:] = 0
    assert np.array_equal(wins.counts.cpu().numpy()[some], cnt)
    assert np.array_equal(wins.records.cpu().numpy()[some], rec)
