"""Inhibition and winner selection at the edges of their kernels' ranges
(channels and steps held in registers or not, strips cut by the last pixels,
the scan's vector and scalar forms, long and short samples) against the
oracle, bit for bit: ties between channels, NaN and infinite potentials,
negative ones, thresholds below and above everything."""

import numpy as np
import pytest
import torch

import spyker_b200 as spyker

pytestmark = pytest.mark.gpu

# b, t, c, h, w
SHAPES = [
    (1, 1, 1, 1, 1),
    (3, 15, 30, 7, 9),
    (2, 16, 32, 4, 8),
    (2, 16, 33, 5, 5),  # two lanes a column
    (2, 15, 52, 3, 11),
    (3, 15, 100, 14, 14),  # four lanes a column
    (2, 16, 105, 4, 4),
    (1, 9, 256, 6, 5),
    (1, 3, 257, 4, 5),  # strips read twice
    (2, 17, 32, 5, 7),  # a warp per step up to 32 steps
    (1, 32, 40, 6, 6),
    (1, 31, 128, 3, 5),
    (1, 33, 9, 5, 5),  # more steps than warps
    (1, 800, 3, 2, 3),  # no per-step table: a thread per pixel
    (2, 15, 60, 28, 28),  # keys in global memory
]


def potentials(shape, rng, special):
    v = rng.integers(-3, 9, size=shape).astype(np.float32) * 0.5  # ties
    v += (rng.random(shape) < 0.5) * rng.random(shape).astype(np.float32)
    if special:
        for x in (np.nan, np.inf, -np.inf):
            v[rng.random(shape) < 0.01] = x
    return v.astype(np.float32)


@pytest.mark.parametrize("special", [False, True])
@pytest.mark.parametrize("shape", SHAPES)
def test_inhibit_edges(port, shape, special):
    rng = np.random.default_rng(sum(shape))
    v = potentials(shape, rng, special)
    for thr in (2.0, -100.0, 100.0):
        got = torch.from_numpy(v).cuda()
        spyker.inhibit(got, thr)
        with np.errstate(invalid="ignore"):
            want = port.inhibit(v, thr)
        assert np.array_equal(got.cpu().numpy().view(np.uint32) & 0x7FFFFFFF, want.view(np.uint32) & 0x7FFFFFFF) or \
            np.array_equal(got.cpu().numpy(), want, equal_nan=True)


@pytest.mark.parametrize("shape", SHAPES)
def test_convwta_edges(port, shape):
    rng = np.random.default_rng(sum(shape) + 1)
    v = potentials(shape, rng, False)
    for thr, radius, count in ((2.0, 1, 8), (100.0, 2, 3), (-100.0, 0, 40)):
        win, cnt = port.convwta(v, (radius, radius), count, thr)
        got = spyker.convwta(torch.from_numpy(v).cuda(), radius, count, thr)
        rec, n = got.records.cpu().numpy(), got.counts.cpu().numpy()
        assert np.array_equal(n, cnt)
        for i in range(shape[0]):
            assert np.array_equal(rec[i, :n[i]], win[i, :n[i]])


def test_convwta_unaligned_input(port):
    """A view one value past an allocation: the scan's scalar form."""
    shape = (3, 15, 30, 28, 28)
    rng = np.random.default_rng(4)
    v = potentials(shape, rng, False)
    flat = torch.zeros(v.size + 1, device="cuda")
    flat[1:] = torch.from_numpy(v.ravel()).cuda()
    win, cnt = port.convwta(v, (3, 3), 5, 2.0)
    got = spyker.convwta(flat[1:].view(shape), 3, 5, 2.0)
    assert np.array_equal(got.counts.cpu().numpy(), cnt)
    assert np.array_equal(got.records.cpu().numpy(), win)
