"""Two host threads on streams of their own, calling the same kernels with large and
small shared memory in turn: no launch fails and every result is right (a kernel's
limit of dynamic shared memory is shared by all threads)."""

import threading

import pytest
import torch

import spyker_b200 as spyker
from spyker_b200 import sparse, temporal

pytestmark = pytest.mark.gpu
ROUNDS = 400


def event_lists(c, side):
    g = torch.Generator("cuda").manual_seed(c)
    when = torch.randint(0, 12, (2, c, side, side), generator=g, device="cuda").clamp(max=8).float()
    x = spyker.SparseTensor(spyker.scatter(when.reshape(2, -1), 8).view(2, 8, c, side, side), 0.0)
    return lambda: sparse.gather(x)


def first_steps(c, side, time):
    g = torch.Generator("cuda").manual_seed(c)
    t_in = torch.randint(0, time + 1, (40, c, side, side), generator=g, device="cuda").float()
    kern = torch.randint(0, 4, (33, c, 3, 3), generator=g, device="cuda").float()
    return lambda: temporal.conv_forward(t_in, kern, 1.5 * c, time, 1, 1)


def convolution(c, side):
    g = torch.Generator("cuda").manual_seed(c)
    x = (torch.rand((2, 3, c, side, side), generator=g, device="cuda") < 0.5).to(torch.uint8)
    conv = spyker.Conv(c, 9, 5, pad=2)
    conv.kernel.copy_(torch.rand(conv.kernel.shape, generator=g, device="cuda"))
    conv.precision = "fp32"
    return lambda: conv(x)


def winners(n):
    v = torch.randn((2, 4, n), generator=torch.Generator("cuda").manual_seed(n), device="cuda")
    return lambda: spyker.fcwta(v, 1, 2).records


@pytest.mark.parametrize("make", [
    lambda big: event_lists(30, 36) if big else event_lists(20, 25),
    lambda big: first_steps(200, 8, 60) if big else first_steps(60, 8, 60),
    lambda big: convolution(40, 60) if big else convolution(3, 12),
    lambda big: winners(40000) if big else winners(13000),
])
def test_two_threads(make):
    calls = [make(True), make(False)]
    want = [f().clone() for f in calls]
    torch.cuda.synchronize()
    errors = []

    def work(i):
        try:
            with torch.cuda.stream(torch.cuda.Stream()):
                for k in range(ROUNDS):
                    out = calls[i]()
                    if k % 50 == 0:
                        assert torch.equal(out, want[i])
                torch.cuda.current_stream().synchronize()
        except Exception as e:  # noqa: BLE001
            errors.append(repr(e))

    threads = [threading.Thread(target=work, args=(i,)) for i in (0, 1, 1)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors


def test_launches_back_to_back():
    """The same through the C ABI alone, so that the threads meet between a call's
    setting of the limit and its launch."""
    import numpy as np

    from spyker_b200._lib import lib, ptr

    sets, keep = [], []
    for c, side in ((30, 36), (20, 25), (17, 28), (25, 36)):
        g = torch.Generator("cuda").manual_seed(c)
        when = torch.randint(0, 12, (2, c, side, side), generator=g, device="cuda").clamp(max=8).float()
        x = spyker.SparseTensor(spyker.scatter(when.reshape(2, -1), 8).view(2, 8, c, side, side), 0.0)
        out, ws, st = torch.empty_like(when), torch.empty(1 << 22, dtype=torch.uint8, device="cuda"), torch.cuda.Stream()
        keep.append((x, when, out, ws, st))
        sets.append((ptr(x.offsets), ptr(x.events), 2, 8, c, side, side, ptr(out), sparse.type_code(torch.float32),
                     ptr(ws), ws.numel(), st.cuda_stream))
    torch.cuda.synchronize()
    failed = np.zeros(len(sets), int)

    def work(i):
        for _ in range(10000):
            failed[i] += lib.spk_sparse_gather(*sets[i]) != 0

    threads = [threading.Thread(target=work, args=(i,)) for i in range(len(sets))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    torch.cuda.synchronize()
    assert not failed.any(), failed
    for _, when, out, _, _ in keep:
        assert torch.equal(out, when)
