"""Inhibition bit for bit, signs of zeros included (NaN apart): few channels of
many columns (a thread per column) and either side of that line, and the strips'
forms."""

import numpy as np
import pytest
import torch

import spyker_b200 as spyker

pytestmark = pytest.mark.gpu

# b, t, c, h, w
SHAPES = [
    (64, 5, 1, 28, 28),
    (16, 15, 1, 28, 28),
    (64, 15, 2, 28, 28),
    (30, 15, 2, 28, 28),
    (64, 4, 4, 28, 28),
    (60, 4, 4, 28, 28),
    (130, 3, 8, 28, 28),
    (64, 40, 3, 28, 28),
    (200, 3, 2, 27, 26),  # pairs of columns
    (200, 3, 2, 27, 27),  # single ones
    (2, 800, 20, 4, 4),  # more steps than the strips hold
    (130, 2, 9, 28, 28),
    (3, 15, 30, 7, 9),
    (2, 16, 33, 5, 5),
    (3, 15, 100, 14, 14),
    (1, 3, 257, 4, 5),
    (1, 33, 9, 5, 5),
]


@pytest.mark.parametrize("shape", SHAPES)
def test_inhibit_bits(port, shape):
    rng = np.random.default_rng(sum(shape))
    v = (rng.integers(-3, 9, size=shape) * 0.5).astype(np.float32)  # ties, negative winners
    v[rng.random(shape) < 0.1] = -0.0
    for x in (np.nan, np.inf, -np.inf):
        v[rng.random(shape) < 0.002] = x
    for thr in (2.0, -100.0, 100.0):
        got = torch.from_numpy(v.copy()).cuda()
        spyker.inhibit(got, thr)
        with np.errstate(invalid="ignore"):
            want = port.inhibit(v, thr)
        out, nan = got.cpu().numpy(), np.isnan(want)
        assert np.array_equal(np.isnan(out), nan)
        assert np.array_equal(out.view(np.uint32)[~nan], want.view(np.uint32)[~nan])
