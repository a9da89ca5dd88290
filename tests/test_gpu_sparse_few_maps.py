"""Event-list convolution either side of the line between a warp per map and a
lane per map (12 maps) against the oracle, lists in order."""

import numpy as np
import pytest
import torch

import spyker_b200 as spyker

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cout", [1, 11, 12, 13])
@pytest.mark.parametrize("u,c,h,w,k,pad", [(3, 2, 28, 28, 5, 2), (2, 3, 9, 14, 3, 1)])
def test_few_maps(port, u, c, h, w, k, pad, cout):
    rng = np.random.default_rng(cout + h)
    t = 9
    first = np.where(rng.random((u, c, h, w)) < 0.1, rng.integers(0, t, size=(u, c, h, w)), t)
    dense = (first[:, None] <= np.arange(t)[None, :, None, None, None]).astype(np.uint8)
    ev = port.sparse_from_dense(dense)
    kern = rng.uniform(0.2, 1.0, size=(cout, c, k, k)).astype(np.float32)
    want, oshape = port.sparse_conv(ev, dense.shape, kern, 0.9, (pad,) * 4)
    st = spyker.SparseTensor.from_lists(ev[0], ev[1], dense.shape, torch.device("cuda"))
    off, zyx = spyker.sparse.conv(st, torch.from_numpy(kern).cuda(), 0.9, 1, (pad,) * 4).lists()
    assert np.array_equal(off, np.asarray(want[0], np.int64))
    assert np.array_equal(zyx, np.asarray(want[1], np.uint8).reshape(-1, 3)) and len(zyx) > 0
