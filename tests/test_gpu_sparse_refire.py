"""Event-list convolution with weights near FLT_MAX, which lift a parked neuron
over the threshold again: the lists equal the oracle's, less what a map lists
beyond its number of neurons, wherever in the map the repeats are."""

import numpy as np
import pytest
import torch

import spyker_b200 as spyker

pytestmark = pytest.mark.gpu

# u, t, c, h, w, cout, k, pad, rows of inputs that fire
SHAPES = [
    (2, 15, 2, 28, 28, 33, 5, 2, 6),  # seven bands of rows, the repeats in the first two
    (2, 15, 2, 28, 28, 33, 5, 2, 28),  # everywhere: maps with a surplus
    (2, 20, 4, 9, 33, 40, 3, 1, 9),
    (1, 12, 2, 60, 60, 3, 5, 2, 10),
    (1, 9, 3, 100, 40, 5, 3, 1, 30),  # more than 32 bands
    (3, 6, 3, 10, 10, 64, 5, 2, 10),  # one band
    (1, 12, 2, 60, 60, 13, 5, 2, 10),
    (1, 9, 3, 100, 40, 12, 3, 1, 30),  # more than 32 bands, a lane per map
]


def first_of_each_map(offsets, zyx, u, t, cout, ohw):
    """The lists without a (sample, map)'s events past its first ohw."""
    off, out = [0], []
    for i in range(u):
        seen = np.zeros(cout, np.int64)
        for step in range(t):
            ev = zyx[offsets[i * t + step]:offsets[i * t + step + 1]]
            for e in ev:
                if seen[e[0]] < ohw:
                    out.append(e)
                seen[e[0]] += 1
            off.append(len(out))
    return np.asarray(off, np.int64), np.asarray(out, np.uint8).reshape(-1, 3)


@pytest.mark.parametrize("value", [3.4e38, 2.0 ** 103, 2.0 ** 126])
@pytest.mark.parametrize("shape", SHAPES)
def test_repeated_events(port, shape, value):
    u, t, c, h, w, cout, k, pad, rows = shape
    rng = np.random.default_rng(sum(shape))
    fires = rng.random((u, c, h, w)) < 0.5
    fires[:, :, rows:] = False
    first = np.where(fires, rng.integers(0, t, size=(u, c, h, w)), t)
    dense = (first[:, None] <= np.arange(t)[None, :, None, None, None]).astype(np.uint8)
    ev = port.sparse_from_dense(dense)
    kern = rng.uniform(0.2, 1.0, size=(cout, c, k, k)).astype(np.float32)
    kern = np.where(rng.random(kern.shape) < 0.4, np.float32(value), kern).astype(np.float32)
    want, oshape = port.sparse_conv(ev, dense.shape, kern, 0.5, (pad,) * 4)
    ohw = oshape[3] * oshape[4]
    off, zyx = first_of_each_map(np.asarray(want[0]), np.asarray(want[1]).reshape(-1, 3), u, t, cout, ohw)
    st = spyker.SparseTensor.from_lists(ev[0], ev[1], dense.shape, torch.device("cuda"))
    got = spyker.sparse.conv(st, torch.from_numpy(kern).cuda(), 0.5, 1, (pad,) * 4)
    goff, gzyx = got.lists()
    assert np.array_equal(goff, off)
    assert np.array_equal(gzyx, zyx)
    if value > 1e38:
        assert len(zyx) > u * cout * ohw // 20
