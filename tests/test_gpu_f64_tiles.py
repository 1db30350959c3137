"""Tiles of the plain FP64 contraction, one pair and a whole step: rows and
columns at the edges of the 8 x 8 tiles, columns that run as FMAs beside
them, k off the 16-wide steps and off the clusters' shares, each operand
orientation, fresh and added-to destinations.

Tolerance: none.  The operands are whole numbers of at most 8, so every sum
of up to 2^40 products is exact in any order."""
import numpy as np
import pytest

from oracle import oracle

pytestmark = pytest.mark.gpu

LABELS = {"nn": ([1, 2], [1, 3], [3, 2]), "tn": ([1, 2], [3, 1], [3, 2]), "nt": ([1, 2], [1, 3], [2, 3]),
          "tt_dt": ([2, 1], [3, 1], [2, 3])}
SIZES = [(1, 1, 1), (8, 8, 16), (7, 9, 17), (144, 25, 144), (64, 31, 33), (65, 32, 15), (72, 5, 2000), (33, 6, 129),
         (40, 39, 64), (257, 100, 48), (9, 300, 500), (600, 520, 70)]


@pytest.fixture(scope="module")
def a4():
    import aces4_gb300

    aces4_gb300.build()
    aces4_gb300.device.init(0)
    return aces4_gb300


def _whole(rng, ext):
    return rng.integers(-8, 9, int(np.prod(ext))).astype(np.float64)


def _matrix(x, ext, labels, order):
    """Operand (first index fastest) as a matrix over labels `order`."""
    t = x.reshape(ext, order="F")
    return t if labels == order else t.T


@pytest.mark.parametrize("orient", list(LABELS))
@pytest.mark.parametrize("m,n,k", SIZES)
@pytest.mark.parametrize("beta", [0, 1])
def test_pair(a4, orient, m, n, k, beta):
    import torch

    ld, ll, lr = LABELS[orient]
    size = {1: m, 2: n, 3: k}
    de, le, re = ([size[q] for q in w] for w in (ld, ll, lr))
    ptrn = oracle.get_contraction_ptrn(2, 2, 2, ld + ll + lr)[1]
    rng = np.random.default_rng(m * 7 + n * 3 + k)
    l, r, d = _whole(rng, le), _whole(rng, re), _whole(rng, de)
    want = _matrix(l, le, ll, [1, 3]) @ _matrix(r, re, lr, [3, 2])
    want = want if ld == [1, 2] else want.T
    want = want.ravel(order="F") + beta * d
    dt = torch.tensor(d, device="cuda")
    a4.device.contract(ptrn, torch.tensor(l, device="cuda"), le, torch.tensor(r, device="cuda"), re, dt, de, beta=beta,
                       stream=torch.cuda.current_stream())
    assert np.array_equal(dt.cpu().numpy(), want)


@pytest.mark.parametrize("ks", [[16], [5, 40, 17], [1, 1], [144] * 16, [33] * 7, [700, 3]])
@pytest.mark.parametrize("blocks", [[(144, 25)], [(40, 31), (9, 33), (64, 8)], [(100, 60)] * 40])
def test_step(a4, ks, blocks):
    import torch

    ptrn = oracle.get_contraction_ptrn(2, 2, 2, [1, 2, 1, 3, 3, 2])[1]
    rng = np.random.default_rng(len(ks) + len(blocks))
    trip, want, D = [], [], []
    for m, n in blocks:
        d = torch.full((m * n,), float("nan"), dtype=torch.float64, device="cuda")
        total = np.zeros((m, n))
        for k in ks:
            l, r = _whole(rng, [m, k]), _whole(rng, [k, n])
            trip.append((d, torch.tensor(l, device="cuda"), torch.tensor(r, device="cuda"), [m, n], [m, k], [k, n]))
            total += l.reshape((m, k), order="F") @ r.reshape((k, n), order="F")
        D.append(d)
        want.append(total.ravel(order="F"))
    b = a4.device.Batch(ptrn, 2, 2, 2, trip, precision=a4.device.PREC_FP64)
    st = torch.cuda.current_stream()
    b.run(stream=st)
    for d, w in zip(D, want):
        assert np.array_equal(d.cpu().numpy(), w)
    b.close()
