"""The search path's output writer: spikes and pooled spikes of shapes whose
planes, channel ranges and pooled cells do not fall on 16-byte boundaries,
from one sample (many CTAs each) to more samples than fill the chip, equal the
oracle's pipeline bit for bit."""

import numpy as np
import pytest
import torch

import spyker_b200 as spyker

pytestmark = pytest.mark.gpu

# b, t, cout, h, w, pool
SHAPES = [
    (1, 15, 30, 28, 28, 2),  # one sample: channel ranges, aligned runs
    (1, 15, 30, 28, 28, 28),  # global pool: cells run through the channels
    (3, 7, 10, 33, 33, 2),  # odd plane: chunks rebuilt at each step
    (5, 15, 17, 14, 14, 3),  # plane a multiple of 4 only; pooled 4 x 4
    (2, 5, 6, 3, 5, 2),  # plane below 16 pixels
    (2, 5, 40, 4, 4, 4),  # plane of 16 pixels, one cell a channel
    (2, 4, 33, 7, 9, 1),  # window 1: pooled equals spikes
    (900, 3, 5, 9, 7, 3),  # one CTA a sample
    (1, 3, 7, 131, 127, 2),  # above 16384 pixels, odd
    (2, 4, 20, 136, 136, 2),  # above 16384 pixels, aligned
    (1, 3, 3, 130, 128, 130),  # above 16384 pixels, window as tall as the map
]


@pytest.mark.parametrize("shape", SHAPES)
def test_writer_shapes(port, shape):
    b, t, cout, h, w, pool = shape
    rng = np.random.default_rng(sum(shape))
    fst = rng.integers(0, t + 3, size=(b, 2, h, w))
    x = (fst[:, None] <= np.arange(t)[None, :, None, None, None]).astype(np.uint8)
    k = rng.uniform(0.3, 1.0, size=(cout, 2, 3, 3)).astype(np.float32)
    conv = spyker.Conv(2, cout, 3, pad=1)
    conv.kernel.copy_(torch.from_numpy(k))
    conv.precision = "bf16x3"
    ph = min(pool, w)
    spk, _, pooled = spyker.conv_fire_wta(torch.from_numpy(x).cuda(), conv, 4.0, 0, 0, pool=(pool, ph))
    assert spyker._lib.lib.spk_device_status(1) == 0
    ref = port.fire(port.inhibit(port.threshold(port.conv(x, k, (1, 1), (1, 1, 1, 1)), 4.0)))
    assert np.array_equal(spk.cpu().numpy(), ref) and int(ref.sum()) > 0
    assert np.array_equal(pooled.cpu().numpy(), port.pool(ref, (pool, ph)))
