"""Input gradients of a first-spike layer whose weights hold infinities and NaN:
every (input before output) term is weight times gradient, the zero gradients
included (infinity times zero is NaN)."""

import numpy as np
import pytest
import torch

from spyker_b200 import temporal

pytestmark = pytest.mark.gpu

# b, c, h, w, z, k, pad
LAYERS = [
    (3, 2, 7, 6, 5, 3, 1),
    (2, 3, 20, 31, 9, 5, 2),  # positions in several blocks
    (200, 4, 4, 4, 3, 3, 1),  # one set of sums a CTA
    (2, 2, 9, 9, 3, 7, 3),  # two taps a lane
    (2, 40, 1, 1, 10, 1, 0),
]


@pytest.mark.parametrize("layer", LAYERS)
def test_weights_that_are_not_finite(layer):
    b, c, h, w, z, k, pad = layer
    rng = np.random.default_rng(c + z)
    t_in = rng.integers(0, 9, size=(b, c, h, w)).astype(np.float32)
    kern = rng.normal(size=(z, c, k, k)).astype(np.float32)
    odd = rng.random(kern.shape) < min(0.02, 2.0 / (k * k * z))
    odd.ravel()[rng.integers(odd.size)] = True
    kern = np.where(odd, rng.choice(np.array([np.inf, -np.inf, np.nan], np.float32), size=kern.shape), kern)
    oh, ow = h + 2 * pad - k + 1, w + 2 * pad - k + 1
    t_out = rng.integers(0, 9, size=(b, z, oh, ow)).astype(np.float32)
    go = rng.normal(size=t_out.shape).astype(np.float32)
    go[rng.random(go.shape) < 0.75] = 0.0
    want = np.zeros((b, c, h + 2 * pad, w + 2 * pad))
    padded = np.full(want.shape, np.inf)
    padded[:, :, pad:pad + h, pad:pad + w] = t_in
    with np.errstate(invalid="ignore"):
        for y in range(k):
            for x in range(k):
                before = padded[:, None, :, y:y + oh, x:x + ow] < t_out[:, :, None]
                term = kern[None, :, :, y, x, None, None].astype(np.float64) * go[:, :, None]
                want[:, :, y:y + oh, x:x + ow] += np.where(before, term, 0.0).sum(1)
    want = want[:, :, pad:pad + h, pad:pad + w]
    assert np.isnan(want).any() and np.isfinite(want).any()
    cuda = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()
    gi, _ = temporal.conv_backward(cuda(t_in), cuda(kern.astype(np.float32)), cuda(t_out), cuda(go), 1, pad)
    # an FP32 chain of at most z * k * k terms
    np.testing.assert_allclose(gi.cpu().numpy(), want, rtol=1e-5, atol=2e-7 * z * k * k + 1e-6, equal_nan=True)
