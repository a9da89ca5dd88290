"""First-spike layers either side of the line between the walk and the dense
kernel, and between the walk's forms (per-step sums, a warp per pixel with the
weights in shared memory or read through L1), against the FP64 restatement, on
weights whose sums are exact in every order."""

import numpy as np
import pytest
import torch

from oracle import temporal as tr
from spyker_b200 import temporal

pytestmark = pytest.mark.gpu

# b, c, side, z, k, time
LAYERS = [
    (1, 32, 14, 64, 3, 16),  # per-step sums, three CTAs an SM
    (1, 32, 14, 64, 3, 32),  # a warp per pixel, weights through L1
    (12, 32, 14, 64, 3, 4),
    (40, 32, 14, 64, 3, 8),  # dense
    (40, 32, 14, 64, 3, 17),  # walk (rows of 32 steps)
    (3, 128, 14, 16, 3, 16),  # dense: few pixels of many inputs
    (8, 64, 14, 64, 3, 65),
    (60, 1, 28, 32, 5, 4),  # dense
    (60, 1, 28, 32, 5, 8),  # walk, weights in shared memory
    (4, 8, 14, 128, 5, 9),
    (37, 40, 7, 10, 7, 64),  # fc: per-step sums
    (300, 16, 4, 10, 4, 64),
    (20, 40, 7, 10, 7, 65),  # fc: dense
]


@pytest.mark.parametrize("layer", LAYERS)
def test_either_side(layer):
    b, c, side, z, k, time = layer
    rng = np.random.default_rng(b + c + time)
    pad = 0 if k == side else k // 2
    t_in = rng.integers(0, time + time // 3 + 1, size=(b, c, side, side)).astype(np.float32)
    kern = (rng.integers(-1, 4, size=(z, c, k, k)) * 0.125).astype(np.float32)
    thr = 0.125 * round(0.3 * c * k * k)
    got = temporal.conv_forward(*(torch.from_numpy(a).cuda() for a in (t_in, kern)), thr, time, 1, pad)
    want = tr.conv_forward(t_in, kern, thr, time, (1, 1), (pad,) * 4)
    assert np.array_equal(got.cpu().numpy(), want)
    assert (want < time).any() and (want > 0).any()
