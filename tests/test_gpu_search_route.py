"""Which search a fused layer takes (the walk is a few launches, the rounds are
some twenty): the walk only where its work, pixels x inputs x channels a lane, is
small; and equal results from both at either side of the line."""

import pytest
import torch

import spyker_b200 as spyker

pytestmark = pytest.mark.gpu

# b, t, cin, side, cout, k, walks
LAYERS = [
    (1, 15, 2, 28, 30, 5, True),
    (64, 15, 2, 28, 30, 5, True),
    (200, 15, 2, 28, 30, 5, False),
    (1, 15, 30, 14, 100, 5, True),
    (60, 15, 30, 14, 100, 5, False),
    (1, 15, 64, 48, 256, 5, False),  # one image of a texture's second layer
    (1, 15, 64, 128, 256, 5, False),
    (8, 15, 64, 32, 64, 3, True),
    (24, 15, 64, 32, 64, 3, False),
    (2, 4, 64, 14, 256, 5, False),  # few pixels: the latency of one
]


def layer_of(cin, cout, k, seed):
    g = torch.Generator("cuda").manual_seed(seed)
    conv = spyker.Conv(cin, cout, k, pad=k // 2)
    conv.kernel.copy_(torch.rand(conv.kernel.shape, generator=g, device="cuda"))
    conv.precision = "bf16x3"
    return conv


@pytest.mark.parametrize("layer", LAYERS)
def test_route(layer):
    b, t, cin, side, cout, k, walks = layer
    g = torch.Generator("cuda").manual_seed(cin)
    fst = torch.randint(0, t + 3, (b, 1, cin, side, side), generator=g, device="cuda")
    x = (fst <= torch.arange(t, device="cuda").view(1, t, 1, 1, 1)).to(torch.uint8)
    conv = layer_of(cin, cout, k, cout)
    count = spyker._lib.lib.spk_launch_count
    n = count()
    spk, wins = spyker.conv_fire_wta(x, conv, 0.15 * cin * k * k, 1, 4)
    assert spyker._lib.lib.spk_device_status(1) == 0
    assert (count() - n < 12) == walks
    if b > 1:  # a sample by itself
        one, w1 = spyker.conv_fire_wta(x[1:2], conv, 0.15 * cin * k * k, 1, 4)
        assert torch.equal(one, spk[1:2]) and torch.equal(w1.records, wins.records[1:2])
    assert int(spk[:, -1].sum()) > 0
