"""A fused layer whose spikes of one sample and step are 2^31 bytes or more
(256 maps of 2900 x 2900): each pixel has one input, and input i's weights are
largest in one channel, so the spikes are known without a pipeline."""

import pytest
import torch

import spyker_b200 as spyker

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("side", [2900, 2901])  # planes of whole 16-byte words, and odd ones
def test_step_of_two_gigabytes(side):
    cout, home = 256, (0, 131, 255)
    g = torch.Generator("cuda").manual_seed(side)
    which = torch.randint(0, 4, (side, side), generator=g, device="cuda")  # 3: no input
    x = torch.stack([which == i for i in range(3)]).to(torch.uint8)[None, None]
    conv = spyker.Conv(3, cout, 1)
    kern = torch.full((cout, 3, 1, 1), 0.25, device="cuda")
    for i, c in enumerate(home):
        kern[c, i] = 1.0
    conv.kernel.copy_(kern)
    conv.precision = "bf16x3"
    spk, _, pooled = spyker.conv_fire_wta(x, conv, 0.5, 0, 0, pool=side // 2)
    assert spyker._lib.lib.spk_device_status(1) == 0
    assert spk[0, 0].numel() >= 1 << 31
    half = side // 2
    for i, c in enumerate(home):
        assert torch.equal(spk[0, 0, c].bool(), which == i)
        cells = (which[:2 * half, :2 * half] == i).view(2, half, 2, half).permute(0, 2, 1, 3).flatten(2).any(2)
        assert torch.equal(pooled[0, 0, c].bool(), cells)
    for c in range(cout):  # nothing else
        if c not in home:
            assert not bool(spk[0, 0, c].any()) and not bool(pooled[0, 0, c].any())
