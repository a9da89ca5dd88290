"""3x3 pooling of U8 planes (a lane per output place) at its edges: one output,
32 outputs, just above (the staged kernel), odd planes, few and many planes,
unaligned inputs, right and bottom pads outside every window."""

import numpy as np
import pytest
import torch

import spyker_b200 as spyker

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,h,w,offset", [(1, 3, 3, 0), (5, 5, 4, 1), (7, 14, 14, 0), (3, 13, 26, 3), (2, 12, 25, 0),
                                          (4, 15, 21, 2), (9001, 6, 7, 0), (3, 99, 5, 1)])
def test_pool_three(n, h, w, offset):
    rng = np.random.default_rng(h * w + n)
    x = rng.integers(0, 256, size=(n, 1, 1, h, w)).astype(np.uint8)
    buf = torch.zeros(x.size + 4, dtype=torch.uint8, device="cuda")
    view = buf[offset:offset + x.size].view(x.shape)
    view.copy_(torch.from_numpy(x))
    oh, ow = h // 3, w // 3
    want = x[:, :, :, :oh * 3, :ow * 3].reshape(n, 1, 1, oh, 3, ow, 3).max(axis=(4, 6))
    assert np.array_equal(spyker.pool(view, 3).cpu().numpy(), want)
