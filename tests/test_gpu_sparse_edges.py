"""Event-list kernels at the edges of their ranges (planes and cell maps in
shared memory or not, lanes of the last map group, kernel sizes with and without
the lane-per-map form, negative thresholds, weights that fire a neuron twice)
against the oracle, lists in order."""

import numpy as np
import pytest
import torch

import spyker_b200 as spyker

pytestmark = pytest.mark.gpu
DEV = "cuda"

# u, t, c, h, w, cout, k, pad
SHAPES = [
    (1, 1, 1, 1, 1, 1, 3, 1),
    (3, 15, 2, 28, 28, 30, 5, 2),
    (2, 7, 3, 14, 14, 100, 5, 2),
    (2, 40, 4, 9, 33, 33, 3, 1),
    (2, 5, 2, 31, 64, 32, 5, 2),  # rows of 64 neurons
    (2, 5, 2, 64, 20, 5, 3, 1),  # 64 rows
    (2, 5, 2, 20, 65, 5, 3, 1),  # longer rows: a warp per map
    (1, 4, 2, 60, 60, 3, 5, 2),  # a plane above shared memory
    (2, 6, 5, 12, 12, 9, 4, 1),  # 4 x 4 kernel
    (1, 3, 60, 40, 40, 4, 3, 1),  # more cells than a map in shared memory
    (2, 300, 2, 8, 8, 256, 3, 1),
    (2, 6, 3, 10, 10, 40, 5, 2),  # one band of rows
]


def lists(t):
    off, zyx = t.lists()
    return off, zyx


def check(got, want):
    off, zyx = lists(got)
    assert np.array_equal(off, np.asarray(want[0], np.int64))
    assert np.array_equal(zyx, np.asarray(want[1], np.uint8).reshape(-1, 3))


@pytest.mark.parametrize("shape", SHAPES)
def test_sparse_edges(port, shape):
    u, t, c, h, w, cout, k, pad = shape
    rng = np.random.default_rng(sum(shape))
    first = np.where(rng.random((u, c, h, w)) < 0.1, rng.integers(0, t, size=(u, c, h, w)), t)
    dense = (first[:, None] <= np.arange(t)[None, :, None, None, None]).astype(np.uint8)
    ev = port.sparse_from_dense(dense)
    shp = dense.shape
    st = spyker.SparseTensor.from_lists(ev[0], ev[1], shp, torch.device(DEV))
    assert np.array_equal(spyker.sparse.gather(st).cpu().numpy(), port.sparse_gather(ev, shp))
    p4 = (pad,) * 4
    # ordinary weights; some of them lift a parked neuron back over the threshold
    kern = rng.uniform(0.2, 1.0, size=(cout, c, k, k)).astype(np.float32)
    huge = np.where(rng.random(kern.shape) < 0.1, np.float32(3.4e38), kern).astype(np.float32)
    for weights, thr in ((kern, 0.9), (kern, 0.0), (kern, -0.1), (huge, 0.5)):
        if weights is huge and h * w > 100:  # (a band of rows drops its own surplus)
            continue
        want, oshape = port.sparse_conv(ev, shp, weights, thr, p4)
        if len(np.asarray(want[1]).reshape(-1, 3)) > u * cout * oshape[3] * oshape[4]:
            continue  # more events than neurons: the surplus is dropped
        over = False
        off, zyx = np.asarray(want[0]), np.asarray(want[1]).reshape(-1, 3)
        for i in range(u):
            n = np.bincount(zyx[off[i * t]:off[(i + 1) * t], 0], minlength=cout)
            over |= bool((n > oshape[3] * oshape[4]).any())
        if over:
            continue
        check(spyker.sparse.conv(st, torch.from_numpy(weights).to(DEV), thr, 1, p4), want)
    want, oshape = port.sparse_conv(ev, shp, kern, 0.9, p4)
    out = spyker.SparseTensor.from_lists(want[0], want[1], oshape, torch.device(DEV))
    inh = port.sparse_inhibit(want, oshape)
    check(spyker.sparse.inhibit(out), inh)
    if min(oshape[3:]) >= 2:
        check(spyker.sparse.pool(out, 2), port.sparse_pool(want, oshape, (2, 2))[0])
    win, cnt = port.sparse_convwta(inh, oshape, (1, 1), 4)
    layer = spyker.Conv(c, cout, k, pad=pad)
    layer.kernel.copy_(torch.from_numpy(kern))
    layer.stdpconfig = [spyker.STDPConfig(0.05, -0.04)]
    got = spyker.sparse.convwta(spyker.SparseTensor.from_lists(inh[0], inh[1], oshape, torch.device(DEV)), 1, 4)
    assert np.array_equal(got.counts.cpu().numpy(), cnt)
    layer.stdp(st, got)
    assert np.array_equal(layer.kernel.cpu().numpy(),
                          port.sparse_stdp(ev, shp, kern, [(0.05, -0.04, 1, 0, 1)], win, cnt, p4))


@pytest.mark.parametrize("config", [(0.3, -0.4, 1, 0.2, 0.8), (0.3, -0.4, 0, 0.1, 0.7), (0.1, -0.1, 0, 0.9, 0.1)])
def test_stdp_bounds(port, config):
    """Soft and hard bounds that F32 does not hold exactly, weights on and
    beyond them, and a lower bound above the upper one."""
    rng = np.random.default_rng(8)
    b, t, cin, h, w, cout, k = 40, 6, 3, 9, 9, 7, 3
    fst = rng.integers(0, t + 2, size=(b, cin, h, w))
    x = (fst[:, None] <= np.arange(t)[None, :, None, None, None]).astype(np.uint8)
    out = (rng.integers(0, t + 2, size=(b, 1, cout, h, w)) <= np.arange(t)[None, :, None, None, None]).astype(np.uint8)
    kern = rng.choice(np.array([0.2, 0.8, 0.1, 0.7, 0.5, -1.0, 2.0], np.float32), size=(cout, cin, k, k))
    win, cnt = port.convwta(out.astype(np.float32), (1, 1), 4)
    layer = spyker.Conv(cin, cout, k, pad=1)
    layer.kernel.copy_(torch.from_numpy(kern))
    layer.stdpconfig = [spyker.STDPConfig(config[0], config[1], bool(config[2]), config[3], config[4])]
    xo = torch.from_numpy(out).cuda()
    layer.stdp(torch.from_numpy(x).cuda(), spyker.convwta(xo.float(), 1, 4), xo)
    assert np.array_equal(layer.kernel.cpu().numpy(),
                          port.convstdp(x, kern, out, [config], win, cnt, (1, 1), (1, 1, 1, 1)))
