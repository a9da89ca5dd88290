"""Potentials of few input channels: their K is the reference's order without
padding, so that the tensor cores' FP32 sums take as few steps as the taps
need.  One output position of [Cin, k, k] inputs has the same K as a [Cin k, k]
receptive field of one channel: the two agree bit for bit."""

import pytest
import torch

import spyker_b200 as spyker
from spyker_b200 import _lib

SHAPES = [(2, 3), (2, 5), (3, 7), (4, 5), (6, 5), (7, 3), (7, 7)]


@pytest.mark.parametrize("cin,k", SHAPES)
@pytest.mark.parametrize("precision,terms", [(1, 2), (2, 3)])
def test_workspace_holds_the_weights_alone(cin, k, precision, terms):
    cout = 48
    blocks = -(-cin * k * k // 64)
    for n in (1, 3000):
        size = _lib.lib.spk_conv_workspace(n, cin, 28, 28, cout, k, k, precision)
        assert size == blocks * terms * cout * 128


@pytest.mark.gpu
@pytest.mark.parametrize("cin,k", SHAPES)
@pytest.mark.parametrize("precision", ["bf16x3", "bf16x2"])
def test_same_sums_as_one_channel(cin, k, precision):
    g = torch.Generator("cuda").manual_seed(cin * 10 + k)
    n, cout = 20000, 48
    x = (torch.rand((n, 1, cin, k, k), generator=g, device="cuda") < 0.5).to(torch.uint8)
    # as after training: most weights near 0 or 1
    side = torch.where(torch.rand((cout, cin, k, k), generator=g, device="cuda") < 0.4, 4.0, -4.0)
    w = torch.sigmoid(torch.randn((cout, cin, k, k), generator=g, device="cuda") * 3 + side)
    out = spyker.conv(x, w, precision=precision)
    one = spyker.conv(x.view(n, 1, 1, cin * k, k), w.view(cout, 1, cin * k, k), precision=precision)
    assert out.shape == (n, 1, cout, 1, 1)
    assert torch.equal(out, one)
