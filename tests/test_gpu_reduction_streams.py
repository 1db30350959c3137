"""Reductions that overlap: on several streams with hundreds of calls queued on
each, on more streams than have scratch of their own, and in replays of a
captured graph beside calls outside it.

Tolerance: none.  A sum is formed in a fixed order, so each call must give the
bits that it gives alone."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def a4():
    import aces4_gb300

    aces4_gb300.build()
    aces4_gb300.device.init(0)
    return aces4_gb300


class _Work:
    """One block's amplitude update (its error norm) and (T)-energy-like sum, added to two numbers of its own."""

    SEGS = [6, 33, 41]

    def __init__(self, a4, seed):
        import torch

        self.a4, o, va, vb = a4, *self.SEGS
        self.ext, self.iv = [va, o, vb, o], [2, 1, 3, 1]
        n, norb = int(np.prod(self.ext)), sum(self.SEGS)
        rng = np.random.default_rng(seed)
        dev = lambda x: torch.tensor(x, device="cuda")
        self.e = dev(np.concatenate([rng.uniform(-2.0, -0.5, o), rng.uniform(0.2, 5.0, norb - o)]))
        self.x = [dev(rng.normal(0.0, 0.1, n)) for _ in range(4)]
        self.err, self.next = torch.zeros_like(self.x[0]), torch.zeros_like(self.x[0])
        self.norm, self.energy, self.n = dev(np.zeros(1)), dev(np.zeros(1)), norb

    def run(self, times, stream):
        d = self.a4.device
        for _ in range(times):
            d.update_t2(self.iv, self.ext, *self.x, self.err, self.next, [self.n], self.e, self.SEGS, self.norm, stream=stream)
            d.energy_contract(self.iv, self.ext, self.x[0], [self.n], self.e, self.SEGS, 0.5, self.energy, stream=stream)

    def take(self):
        out = self.norm.item(), self.energy.item()
        self.norm.zero_(), self.energy.zero_()
        return out


def _alone(works, times):
    import torch

    want = []
    for w in works:
        w.run(times, torch.cuda.current_stream())
        torch.cuda.synchronize()
        want.append(w.take())
    torch.cuda.synchronize()
    return want


def test_streams_with_many_calls_queued(a4):
    import torch

    works = [_Work(a4, q) for q in range(4)]
    want = _alone(works, 300)
    streams = [torch.cuda.Stream() for _ in works]
    torch.cuda.synchronize()
    for lag in range(3):  # the first stream is 100, 200, 300 calls ahead
        works[0].run(100 * (lag + 1), streams[0])
        for _ in range(300):
            for w, s in zip(works[1:], streams[1:]):
                w.run(1, s)
        works[0].run(300 - 100 * (lag + 1), streams[0])
        torch.cuda.synchronize()
        assert [w.take() for w in works] == want


def test_more_streams_than_slots(a4):
    import torch

    rt = torch.cuda.cudart()
    works = [_Work(a4, q) for q in range(8)]
    want = _alone(works, 1)
    handles = []
    for _ in range(320):
        h = ctypes.c_uint64(0)
        assert int(rt.cudaStreamCreate(ctypes.addressof(h))) == 0
        handles.append(h.value)
    torch.cuda.synchronize()
    for first in range(0, len(handles), len(works)):
        for w, h in zip(works, handles[first:]):
            w.run(1, torch.cuda.ExternalStream(h))
        torch.cuda.synchronize()
        assert [w.take() for w in works] == want, first
    for h in handles:
        assert int(rt.cudaStreamDestroy(h)) == 0


def test_replays_beside_calls(a4):
    import torch

    inside, outside = [_Work(a4, q) for q in range(2)], _Work(a4, 9)
    want_in = _alone(inside, 40)
    want_out = _alone([outside], 400)
    s, t = torch.cuda.Stream(), torch.cuda.Stream()
    for _ in range(2):  # the second graph after the first is gone
        graph = torch.cuda.CUDAGraph()
        torch.cuda.synchronize()
        with torch.cuda.graph(graph, stream=s):
            t.wait_stream(s)
            inside[0].run(40, s)
            inside[1].run(40, t)
            s.wait_stream(t)
        for w in inside:
            assert w.take() == (0.0, 0.0)
        torch.cuda.synchronize()
        for _ in range(3):
            outside.run(200, t)
            with torch.cuda.stream(s):
                graph.replay()
            outside.run(200, t)
            torch.cuda.synchronize()
            assert [w.take() for w in inside] == want_in
            assert outside.take() == want_out[0]
            torch.cuda.synchronize()
        del graph
