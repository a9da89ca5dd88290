"""Rank codes of row lengths around the sort kernels' limits, with many and with
no values tied at the minimum, equal the stable-order rank code."""

import numpy as np
import pytest
import torch

import spyker_b200 as spyker
from tests.test_gpu_ops import stable_code

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ties", [0.0, 0.7, 0.999])
@pytest.mark.parametrize("x", [257, 2048, 2049, 2178, 4096, 4097, 4704, 8191, 8192, 8193])
def test_rank_rows(x, ties):
    rng = np.random.default_rng(x)
    v = rng.random((3, 1, 1, x)).astype(np.float32)
    v[rng.random(v.shape) < ties] = 0.0
    v[0, 0, 0, :: 7] = 0.25  # ties away from the minimum
    v[0, 0, 0, 0] = 1.0
    got = spyker.code(torch.from_numpy(v).cuda(), 15).cpu().numpy()
    assert np.array_equal(got, stable_code(v, 15))
    u8 = (v * 255).astype(np.uint8)
    assert np.array_equal(spyker.code(torch.from_numpy(u8).cuda(), 9).cpu().numpy(), stable_code(u8.astype(np.float32), 9))
