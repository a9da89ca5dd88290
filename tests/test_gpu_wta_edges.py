"""Winner selection with infinite, NaN and equal potentials (keys that are
infinite or NaN, at position 0 and elsewhere), in the scan's form and in the form
of one CTA that reads the sample itself, and either side of the line between
them (short rows of many steps)."""

import numpy as np
import pytest
import torch

import spyker_b200 as spyker

pytestmark = pytest.mark.gpu

# b, t, c, h, w
SHAPES = [
    (3, 15, 30, 7, 9),  # 1890 positions
    (2, 1000, 1, 10, 10),  # one CTA
    (2, 100, 14, 10, 9),  # 1260 positions: one CTA
    (2, 100, 24, 10, 10),  # 2400 positions: one CTA
    (2, 100, 25, 10, 10),  # 2500: the scan
    (150, 15, 29, 10, 10),  # more samples than SMs: one CTA each
    (150, 15, 30, 10, 10),  # the scan
    (2, 64, 10, 5, 6),
    (3, 4, 5, 4, 5),
    (2, 15, 60, 28, 28),  # keys in global memory
]


def case(shape, rng, kind):
    v = np.cumsum(rng.random(shape).astype(np.float32), axis=1).astype(np.float32)
    if kind == "equal":  # no spread: every key is 0 / 0
        v[:] = 3.0
    elif kind == "infinite":  # an infinite spread: keys of infinity / infinity and finite / infinity
        v[rng.random(shape) < 0.02] = np.inf
        v[rng.random(shape) < 0.02] = -np.inf
    elif kind == "nan":
        v[rng.random(shape) < 0.03] = np.nan
    elif kind == "nan_first":  # NaN minimum and maximum
        v[:, 0, 0, 0, 0] = np.nan
    elif kind == "lowest":
        v[rng.random(shape) < 0.3] = -np.finfo(np.float32).max
    return v


@pytest.mark.parametrize("kind", ["plain", "equal", "infinite", "nan", "nan_first", "lowest"])
@pytest.mark.parametrize("shape", SHAPES)
def test_wta_special(port, shape, kind):
    v = case(shape, np.random.default_rng(sum(shape)), kind)
    for thr, radius, count in ((1.0, 1, 8), (-np.inf, 0, 30)):
        with np.errstate(all="ignore"):
            win, cnt = port.convwta(v, (radius, radius), count, thr)
        got = spyker.convwta(torch.from_numpy(v).cuda(), radius, count, thr)
        rec, n = got.records.cpu().numpy(), got.counts.cpu().numpy()
        assert np.array_equal(n, cnt)
        for i in range(shape[0]):
            assert np.array_equal(rec[i, :n[i]], win[i, :n[i]])
            assert not rec[i, n[i]:].any()
