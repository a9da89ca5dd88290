"""The output writer off the search path (a negative weight, or input that is not
cumulative 0/1): it zero-fills spikes and pooled spikes for the dense kernel, in
every form the search path's shapes give it, and the results equal the oracle's
pipeline.  The last shape's pooled plane is larger than any table of first steps
in shared memory (163,840 cells), so the writer has no shared memory there."""

import numpy as np
import pytest
import torch

import spyker_b200 as spyker

pytestmark = pytest.mark.gpu

# b, t, cout, h, w, pool
SHAPES = [
    (1, 15, 30, 28, 28, 2),
    (3, 7, 10, 33, 33, 2),
    (2, 5, 6, 3, 5, 2),
    (900, 3, 5, 9, 7, 3),
    (1, 3, 7, 131, 127, 2),  # above 16384 pixels
    (2, 4, 20, 136, 136, 2),
    (1, 2, 3, 816, 824, 2),
]


@pytest.mark.parametrize("kind", ["negative", "noncumulative"])
@pytest.mark.parametrize("shape", SHAPES)
def test_writer_off_search(port, shape, kind):
    b, t, cout, h, w, pool = shape
    rng = np.random.default_rng(sum(shape))
    fst = rng.integers(0, t + 3, size=(b, 2, h, w))
    x = (fst[:, None] <= np.arange(t)[None, :, None, None, None]).astype(np.uint8)
    k = (rng.integers(1, 9, size=(cout, 2, 3, 3)) * 0.25).astype(np.float32)  # sums are exact in any order
    if kind == "negative":
        k[0, 0, 0, 0] = -0.25
    else:
        x[:, :, 0, 0, 0] = np.arange(t) % 2 == 0  # an input that stops firing
        x[-1, 0, 1, 1, 1] = 2  # and one above 1
    conv = spyker.Conv(2, cout, 3, pad=1)
    conv.kernel.copy_(torch.from_numpy(k))
    conv.precision = "bf16x3"
    ph = min(pool, w)
    spk, _, pooled = spyker.conv_fire_wta(torch.from_numpy(x).cuda(), conv, 9.0, 0, 0, pool=(pool, ph))
    assert spyker._lib.lib.spk_device_status(1) == 0
    ref = port.fire(port.inhibit(port.threshold(port.conv(x, k, (1, 1), (1, 1, 1, 1)), 9.0)))
    assert np.array_equal(spk.cpu().numpy(), ref) and int(ref.sum()) > 0
    assert np.array_equal(pooled.cpu().numpy(), port.pool(ref, (pool, ph)))
