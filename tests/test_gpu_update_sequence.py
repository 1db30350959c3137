"""Amplitude updates in sequence: each call's launch may overlap the end of the
one before, so a call that reads what the one before wrote, the running norm
and replayed graphs (the first update behind a fill, the last before a copy)
have to give what the calls give one at a time with a synchronisation between.
Planes at the edges of the tiles (one and several passes, 8 and fewer a side).

Tolerance: none, the same kernels on the same values."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def a4():
    import aces4_gb300

    aces4_gb300.build()
    aces4_gb300.device.init(0)
    return aces4_gb300


@pytest.mark.parametrize("segs", [[5, 24, 24], [6, 33, 41], [3, 7, 9], [20, 48, 26], [2, 1, 100]])
def test_chained_updates(a4, segs):
    import torch

    o, va, vb = segs
    ext, pext, iv, piv = [va, o, vb, o], [vb, o, va, o], [2, 1, 3, 1], [3, 1, 2, 1]
    n = int(np.prod(ext))
    g = torch.Generator(device="cuda")
    g.manual_seed(n)
    rnd = lambda: torch.empty(n, dtype=torch.float64, device="cuda").normal_(0.0, 0.1, generator=g)
    norb = sum(segs)
    rng = np.random.default_rng(n)
    e = torch.tensor(np.concatenate([rng.uniform(-2.0, -0.5, o), rng.uniform(0.2, 5.0, norb - o)]), device="cuda")
    xn, xnp, old, oldp = rnd(), rnd(), rnd(), rnd()
    bufs = [[torch.zeros_like(xn) for _ in range(2)] for _ in range(3)]
    err, norm, out = torch.zeros_like(xn), torch.zeros(1, dtype=torch.float64, device="cuda"), torch.zeros_like(xn)
    st = torch.cuda.Stream()

    def steps(wait):
        norm.zero_()
        a, b = old, oldp
        for q in range(3):  # each step reads both blocks that the one before wrote
            na, nb = bufs[q]
            a4.device.update_t2(iv, ext, xn, xnp, a, b, err, na, [norb], e, segs, norm, stream=st)
            wait()
            a4.device.update_t2(piv, pext, xnp, xn, b, a, None, nb, [norb], e, segs, norm, stream=st)
            wait()
            a, b = na, nb
        out.copy_(a)

    state = lambda: [x.cpu().numpy().copy() for x in (err, norm, out, *(y for p in bufs for y in p))]
    torch.cuda.synchronize()
    with torch.cuda.stream(st):
        steps(torch.cuda.synchronize)
        torch.cuda.synchronize()
        want = state()
        for x in (err, out, *(y for p in bufs for y in p)):
            x.fill_(float("nan"))
        steps(lambda: None)
        torch.cuda.synchronize()
        for x, y in zip(state(), want):
            assert np.array_equal(x, y)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=st):
        steps(lambda: None)
    for _ in range(2):
        for x in (err, out, *(y for p in bufs for y in p)):
            x.fill_(float("nan"))
        torch.cuda.synchronize()
        graph.replay()
        torch.cuda.synchronize()
        for x, y in zip(state(), want):
            assert np.array_equal(x, y)
