"""Input gradients of first-spike layers over the kernels' plans (one to eight sets
of sums, few and all channels a CTA, and the kernel that takes every position for
dense gradients of few maps) against the FP64 restatement."""

import numpy as np
import pytest
import torch

from oracle import temporal as tr
from spyker_b200 import temporal

pytestmark = pytest.mark.gpu

# b, c, side, z, k
LAYERS = [
    (1, 1, 28, 32, 5),  # eight sets, one channel
    (160, 1, 28, 9, 5),
    (37, 7, 14, 20, 3),  # four channels groups a CTA, the last one short
    (160, 7, 14, 20, 3),
    (4, 16, 32, 3, 3),  # every position
    (3, 40, 9, 33, 3),
    (2, 200, 4, 12, 3),
    (150, 300, 1, 10, 1),  # fc
    (5, 3, 13, 10, 11),  # four taps a lane
]


@pytest.mark.parametrize("zeros", [0.0, 0.7])
@pytest.mark.parametrize("layer", LAYERS)
def test_plans(layer, zeros):
    b, c, side, z, k = layer
    rng = np.random.default_rng(c + z)
    pad = k // 2
    t_in = rng.integers(0, 20, size=(b, c, side, side)).astype(np.float32)
    kern = rng.normal(size=(z, c, k, k)).astype(np.float32)
    t_out = rng.integers(0, 20, size=(b, z, side, side)).astype(np.float32)
    go = rng.normal(size=t_out.shape).astype(np.float32)
    go[rng.random(go.shape) < zeros] = 0.0
    def grad_in(lo):
        x, to, g = (torch.from_numpy(a[lo:].copy()).cuda() for a in (t_in, t_out, go))
        return temporal.conv_backward(x, torch.from_numpy(kern).cuda(), to, g, 1, pad, True, False)[0].cpu().numpy()

    # an FP32 chain of at most z * k * k terms of size |w g| (below 16 or so)
    close = dict(rtol=1e-5, atol=1e-6 * z * k * k + 1e-6)
    gi, take = grad_in(0), min(b, 6)
    want, _ = tr.conv_backward(t_in[:take], kern, t_out[:take], go[:take], (1, 1), (pad,) * 4)
    np.testing.assert_allclose(gi[:take], want, **close)
    if b > take:  # the last samples by themselves
        np.testing.assert_allclose(gi[-2:], grad_in(b - 2), **close)
