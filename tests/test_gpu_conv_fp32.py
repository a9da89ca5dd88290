"""The FP32 convolution at the edges of its tiles: every potential is the FP32
chain over (channel, ky, kx), so it equals, bit for bit, the same chain run in
NumPy on inputs whose products are exact."""

import numpy as np
import pytest
import torch

import spyker_b200 as spyker

pytestmark = pytest.mark.gpu

# n, cin, h, w, cout, kernel, stride, pad
SHAPES = [
    (1, 1, 1, 1, 1, (1, 1), (1, 1), 0),
    (5, 2, 28, 28, 30, (5, 5), (1, 1), 2),  # 7 positions a thread, several images in a CTA's last tile
    (40, 5, 14, 14, 100, (5, 5), (1, 1), 2),  # images cut by tiles, 13 octets
    (130, 3, 4, 4, 9, (3, 3), (1, 1), 1),  # many images per CTA
    (300, 2, 1, 1, 17, (1, 1), (1, 1), 0),
    (3, 6, 9, 33, 24, (3, 3), (2, 1), 1),  # vertical stride, 8 positions a thread
    (2, 3, 11, 64, 8, (7, 7), (1, 1), 3),
    (2, 4, 12, 63, 41, (2, 7), (1, 1), (0, 3, 1, 2)),  # ragged pads, kernel taller than wide is not square
    (1, 2, 5, 600, 3, (3, 5), (1, 1), 2),  # rows longer than a CTA's positions
    (2, 3, 9, 9, 5, (4, 4), (1, 1), 1),  # the general kernel: width 4
    (2, 3, 9, 9, 5, (3, 3), (1, 2), 1),  # and a horizontal stride
]


def chain(x, k, stride, pad):
    n, cin, h, w = x.shape
    cout, _, kh, kw = k.shape
    top, left, bottom, right = (pad,) * 4 if isinstance(pad, int) else pad
    xp = np.pad(x.astype(np.float32), ((0, 0), (0, 0), (top, bottom), (left, right)))
    oh = (xp.shape[2] - kh) // stride[0] + 1
    ow = (xp.shape[3] - kw) // stride[1] + 1
    acc = np.zeros((n, cout, oh, ow), np.float32)
    for c in range(cin):
        for ky in range(kh):
            for kx in range(kw):
                win = xp[:, c, ky:ky + (oh - 1) * stride[0] + 1:stride[0], kx:kx + (ow - 1) * stride[1] + 1:stride[1]]
                acc += win[:, None] * k[None, :, c, ky, kx, None, None]
    return acc


@pytest.mark.parametrize("dtype", [np.uint8, np.float32])
@pytest.mark.parametrize("shape", SHAPES)
def test_fp32_chain(shape, dtype):
    n, cin, h, w, cout, kernel, stride, pad = shape
    rng = np.random.default_rng(n * 7 + cin * h + w)
    # spikes, or small integers; weights of 16 bits, so that products are exact
    x = rng.integers(0, 2 if dtype == np.uint8 else 9, size=(n, cin, h, w)).astype(dtype)
    k = (rng.integers(-(1 << 15), 1 << 15, size=(cout, cin, *kernel)) * 2.0 ** -17).astype(np.float32)
    k += (rng.integers(0, 4, size=k.shape) * 2.0 ** -19).astype(np.float32)
    got = spyker.conv(torch.from_numpy(x[:, None]).cuda(), torch.from_numpy(k).cuda(), stride, pad, precision="fp32")
    assert np.array_equal(got.cpu().numpy()[:, 0], chain(x, k, stride, pad))
