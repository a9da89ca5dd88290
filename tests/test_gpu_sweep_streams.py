"""The sweep's search path, whose calls run on streams of their own, on a current
stream that is not the default one: eager steps and the captured graph give what
they give on the default stream, with the allocator busy on both."""

import torch

import pytest

from spyker_b200 import sweep

pytestmark = pytest.mark.gpu


def state(s, feats):
    torch.cuda.synchronize()
    return [t.clone() for t in (s.w1, s.w2, *s.rec, *s.cnt, *feats)]


def test_other_current_stream():
    def make():
        return sweep.Sweep(nets=3, images=20, seed=5, path="search")

    ref = make()
    want = [state(ref, ref.step()) for _ in range(3)]
    side, noise = torch.cuda.Stream(), torch.cuda.Stream()
    other = make()
    torch.cuda.synchronize()
    for k in range(3):
        with torch.cuda.stream(side):
            torch.cuda._sleep(2_000_000)  # the step is enqueued while its stream is busy
            feats = other.step()
            # blocks that the step gave back, overwritten at once on the same stream
            junk = [torch.full((1 << 22,), 255, dtype=torch.uint8, device="cuda") for _ in range(16)]
        with torch.cuda.stream(noise):
            torch.ones(1 << 20, device="cuda").sum()
        side.synchronize()
        del junk
        assert all(torch.equal(a, b) for a, b in zip(state(other, feats), want[k]))
    graph = make()
    with torch.cuda.stream(side):
        graph.capture()
    first = [graph.w1.clone(), graph.w2.clone()]
    ref.w1.copy_(first[0])
    ref.w2.copy_(first[1])
    eager = state(ref, ref.step())
    torch.cuda.synchronize()
    with torch.cuda.stream(side):
        feats = graph.replay()
    assert all(torch.equal(a, b) for a, b in zip(state(graph, feats), eager))


def test_dense_path_has_no_lanes():
    assert sweep.Sweep(nets=2, images=8, seed=1, path="dense", tune=False).lanes == []
