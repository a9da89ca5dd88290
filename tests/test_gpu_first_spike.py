"""The first-spike layer's walk and its gradients at the edges of their ranges,
against the NumPy FP64 restatement: one to 4096 inputs, 1 to 200 maps, equal
times, thresholds below zero and on exact sums, negative weights, layers above
the walk's sizes (the dense kernel), sparse and NaN-free zero gradients."""

import numpy as np
import pytest
import torch

from oracle import temporal as tr
from spyker_b200 import temporal

pytestmark = pytest.mark.gpu


def cuda(a):
    return torch.from_numpy(np.ascontiguousarray(a, dtype=np.float32)).cuda()


# b, c, h, w, z, kh, kw, stride, pad, time
LAYERS = [
    (1, 1, 1, 1, 1, 1, 1, (1, 1), (0, 0, 0, 0), 1),
    (3, 2, 7, 9, 33, 3, 5, (2, 1), (1, 2, 0, 1), 126),
    (2, 32, 6, 6, 64, 3, 3, (1, 1), (1, 1, 1, 1), 64),  # K = 288
    (2, 3, 9, 8, 65, 1, 1, (1, 1), (0, 0, 0, 0), 9),  # K = 3, four groups of maps
    (130, 1, 5, 5, 10, 5, 5, (1, 1), (2, 2, 2, 2), 16),
    (4, 4096, 1, 1, 10, 1, 1, (1, 1), (0, 0, 0, 0), 100),  # weights through L1
    (2, 4097, 1, 1, 3, 1, 1, (1, 1), (0, 0, 0, 0), 20),  # above the walk's inputs
    (2, 16, 4, 4, 160, 7, 7, (1, 1), (3, 3, 3, 3), 12),  # weights too many for the walk
]


@pytest.mark.parametrize("kind", ["positive", "signed", "halves"])
@pytest.mark.parametrize("layer", LAYERS)
def test_walk_times(layer, kind):
    b, c, h, w, z, kh, kw, stride, pad, time = layer
    rng = np.random.default_rng(c + z + time)
    t_in = rng.integers(0, time + 1, size=(b, c, h, w)).astype(np.float32)
    shape = (z, c, kh, kw)
    k = c * kh * kw
    if kind == "halves":  # sums land exactly on the threshold
        kern, thr = rng.integers(0, 3, size=shape) * 0.5, 0.25 * k // 0.5 * 0.5
    elif kind == "signed":
        kern, thr = rng.normal(0.02, 0.1, size=shape), 0.2
    else:
        kern, thr = rng.uniform(0.0, 0.1, size=shape), 0.02 * k
    kern = kern.astype(np.float32)
    for th in (thr, -0.5):
        got = temporal.conv_forward(cuda(t_in), cuda(kern), th, time, stride, pad)
        assert np.array_equal(got.cpu().numpy(), tr.conv_forward(t_in, kern, th, time, stride, pad))


def test_walk_repeats_and_odd_times():
    """Input times outside 0..T-1 never spike; the same call twice gives the
    same times."""
    rng = np.random.default_rng(2)
    t_in = rng.choice(np.array([-3.0, 0.0, 1.5, 2.0, 7.0, 8.0, 1e9, np.inf], np.float32), size=(3, 4, 6, 6))
    kern = rng.uniform(0, 0.3, size=(9, 4, 3, 3)).astype(np.float32)
    got = [temporal.conv_forward(cuda(t_in), cuda(kern), 1.0, 8, 1, 1).cpu().numpy() for _ in range(2)]
    assert np.array_equal(*got)
    clean = np.where((t_in >= 0) & (t_in < 8), np.floor(t_in), 8.0).astype(np.float32)
    assert np.array_equal(got[0], tr.conv_forward(clean, kern, 1.0, 8, (1, 1), (1, 1, 1, 1)))


GRADS = [
    # b, c, h, w, z, kh, kw, stride, pad, time
    (1, 1, 1, 1, 1, 1, 1, (1, 1), (0, 0, 0, 0), 4),
    (5, 3, 9, 7, 9, 3, 3, (1, 1), (1, 1, 1, 1), 12),
    (3, 2, 20, 31, 17, 5, 5, (2, 3), (2, 0, 1, 4), 20),  # positions in two blocks of 256
    (2, 33, 6, 5, 8, 3, 3, (1, 1), (0, 0, 0, 0), 16),
    (2, 2, 12, 12, 3, 7, 7, (1, 1), (3, 3, 3, 3), 16),  # taps over two passes of the lanes
    (1, 2, 13, 13, 3, 11, 11, (1, 1), (5, 5, 5, 5), 16),
    (1, 1, 20, 20, 2, 13, 13, (1, 1), (6, 6, 6, 6), 16),  # more taps than the input gradient's lanes take
    (40, 300, 1, 1, 11, 1, 1, (1, 1), (0, 0, 0, 0), 30),
]


@pytest.mark.parametrize("zeros", [0.0, 0.75, 1.0])
@pytest.mark.parametrize("layer", GRADS)
def test_gradients(layer, zeros):
    b, c, h, w, z, kh, kw, stride, pad, time = layer
    rng = np.random.default_rng(c * 3 + z)
    t_in = rng.integers(0, time + 1, size=(b, c, h, w)).astype(np.float32)
    kern = rng.normal(0.0, 0.3, size=(z, c, kh, kw)).astype(np.float32)
    oh = (h + pad[0] + pad[2] - kh) // stride[0] + 1
    ow = (w + pad[1] + pad[3] - kw) // stride[1] + 1
    t_out = rng.integers(0, time + 1, size=(b, z, oh, ow)).astype(np.float32)
    go = rng.normal(size=t_out.shape).astype(np.float32)
    go[rng.random(go.shape) < zeros] = 0.0
    gi, gk = temporal.conv_backward(cuda(t_in), cuda(kern), cuda(t_out), cuda(go), stride, pad)
    wi, wk = tr.conv_backward(t_in, kern, t_out, go, stride, pad)
    # the kernel gradient is an FP64 sum rounded once; the input gradient an
    # FP32 chain of at most z * kh * kw terms of size |w g|
    np.testing.assert_allclose(gk.cpu().numpy(), wk, rtol=1e-6, atol=1e-6)
    np.testing.assert_allclose(gi.cpu().numpy(), wi, rtol=1e-5, atol=2e-7 * z * kh * kw + 1e-6)


@pytest.mark.parametrize("shape", [((2, 2), (9, 11)), ((3, 2), (9, 8)), ((4, 4), (4, 4)), ((2, 3), (5, 5))])
def test_pool_backward_whole_windows(shape):
    k2, (h, w) = shape
    rng = np.random.default_rng(h)
    t = rng.integers(0, 5, size=(3, 5, h, w)).astype(np.float32)
    go = rng.normal(size=(3, 5, h // k2[0], w // k2[1])).astype(np.float32)
    gi = temporal.pool_backward(cuda(t), cuda(go), k2)
    assert np.array_equal(gi.cpu().numpy(), tr.pool_backward(t, go, k2, k2, (0, 0, 0, 0)).astype(np.float32))
