"""Transposing permutes with so many slices that a block takes 4, 8 or 16 of
them (the last block fewer), and denominators of any order whose last run of
four is short.

Tolerances: permutes, additions and quotients bit for bit; the energy is a sum
of n products in another order, within n 2^-52 of the sum of magnitudes."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def a4():
    import aces4_gb300

    aces4_gb300.build()
    aces4_gb300.device.init(0)
    return aces4_gb300


# one tile a slice: 152 SMs x 16 x (4, 8, 16) slices and a remainder
@pytest.mark.parametrize("mid", [(60, 41), (99, 99), (141, 142), (201, 199), (300, 211)])
def test_slices_of_a_block(a4, mid):
    import torch

    ext, labels = [2, *mid, 3], [4, 3, 2, 1]  # all four indices turned round
    n = int(np.prod(ext))
    rng = np.random.default_rng(n)
    x, l = rng.normal(size=n), rng.normal(size=n)
    want = x.reshape(ext, order="F").transpose(3, 2, 1, 0).ravel(order="F")
    tx, tl, out = torch.tensor(x, device="cuda"), torch.tensor(l, device="cuda"), torch.zeros(n, dtype=torch.float64, device="cuda")
    s = torch.cuda.current_stream()
    a4.device.permute(ext, [4, 3, 2, 1], tx, out, stream=s)
    assert np.array_equal(out.cpu().numpy(), want)
    a4.device.add_sub(True, labels, [1, 2, 3, 4], ext, out, tl, tx, stream=s)
    assert np.array_equal(out.cpu().numpy(), l - want)


@pytest.mark.parametrize("o,a,b", [(3, 5, 7), (3, 7, 9), (2, 5, 3), (1, 3, 1), (7, 33, 12)])
def test_runs_of_four(a4, o, a, b):
    import torch

    segs, norb = [o, a, b], o + a + b
    rng = np.random.default_rng(norb)
    e = np.concatenate([rng.uniform(-2.0, -0.5, o), rng.uniform(0.2, 5.0, a + b)])
    eo, ea, eb = e[:o], e[o:o + a], e[o + a:]
    dev, s = lambda x: torch.tensor(x, device="cuda"), torch.cuda.current_stream()
    # rank 2: e_i - e_a
    x = rng.normal(size=a * o)
    x[rng.random(x.size) < 0.2] = 0.0
    tx = dev(x)
    a4.device.energy_denominator([2, 1], [a, o], tx, [norb], dev(e), segs, stream=s)
    assert np.array_equal(tx.cpu().numpy(), x / (eo[None, :] - ea[:, None]).ravel(order="F"))
    # rank 4, stored as (b, j, a, i): positions a, i, b, j of the denominator are dimensions 2, 3, 0, 1
    w = rng.normal(size=b * o * a * o)
    w[rng.random(w.size) < 0.2] = 0.0
    eps = ((eo[None, None, None, :] + eo[None, :, None, None]) - ea[None, None, :, None]) - eb[:, None, None, None]
    terms = w * (w / eps.ravel(order="F"))
    esum = dev(np.zeros(1))
    a4.device.energy_contract([3, 1, 2, 1], [b, o, a, o], dev(w), [norb], dev(e), segs, 1.0, esum, den_order=[2, 3, 0, 1], stream=s)
    assert abs(esum.item() - terms.sum()) <= w.size * 2.0 ** -52 * np.abs(terms).sum()
