"""Amplitude updates that write the blocks which the update before them read,
back and forth between two pairs of buffers, each launch overlapping the end of
the one before: no call may see an element from before the last write.  A plane
of one tile and planes of several, on few and on all SMs.

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


@pytest.mark.parametrize("segs", [[2, 9, 7], [5, 24, 24], [20, 33, 41]])
def test_back_and_forth(a4, segs):
    import torch

    o, va, vb = segs
    ext, pext, iv, piv = [va, o, vb, o], [vb, o, va, o], [2, 1, 3, 1], [3, 1, 2, 1]
    n, norb = int(np.prod(ext)), sum(segs)
    rng = np.random.default_rng(n)
    dev = lambda x: torch.tensor(x, device="cuda")
    e = dev(np.concatenate([rng.uniform(-2.0, -0.5, o), rng.uniform(0.2, 5.0, norb - o)]))
    xn, xnp = dev(rng.normal(0.0, 0.1, n)), dev(rng.normal(0.0, 0.1, n))
    first = [dev(rng.normal(0.0, 0.1, n)) for _ in range(2)]
    st = torch.cuda.Stream()

    def steps(wait):
        """T2new and T2old change places at every step, so that each value depends on all the steps before it."""
        x, y = [[b.clone() for b in first], [xn.clone(), xnp.clone()]]
        z = [torch.empty_like(xn), torch.empty_like(xn)]
        norm = torch.zeros(1, dtype=torch.float64, device="cuda")
        torch.cuda.synchronize()
        for _ in range(30):
            a4.device.update_t2(iv, ext, x[0], x[1], y[0], y[1], None, z[0], [norb], e, segs, norm, stream=st)
            wait()
            a4.device.update_t2(piv, pext, x[1], x[0], y[1], y[0], None, z[1], [norb], e, segs, norm, stream=st)
            wait()
            x, y, z = y, z, x
        torch.cuda.synchronize()
        return [t.cpu().numpy() for t in (*x, *y, norm)]

    want = steps(torch.cuda.synchronize)
    assert all(np.isfinite(w).all() for w in want)
    for _ in range(3):
        for got, w in zip(steps(lambda: None), want):
            np.testing.assert_array_equal(got, w)
