"""Row exponents of row-major left blocks: row counts around the thread
layouts (8, 16 and 32 row pairs) and the 64-row pieces, k around the 256-wide
pieces, odd row counts (8-byte loads), several blocks along k.  Each row holds
multiples of its own power of two up to 127 of them, the largest at one random
place: one slice is exact if, and only if, that place is found.

Tolerance: none (sums stay below 2^24 units)."""
import numpy as np
import pytest

from oracle import oracle

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def a4():
    import aces4_gb300

    aces4_gb300.build()
    aces4_gb300.device.init(0)
    return aces4_gb300


@pytest.mark.parametrize("m", [1, 2, 15, 16, 17, 32, 33, 64, 65, 66, 130, 200])
@pytest.mark.parametrize("ks", [[7], [255], [256], [257, 3], [600], [32, 31, 33]])
def test_row_maxima(a4, m, ks):
    import torch

    n = 24
    rng = np.random.default_rng(m + len(ks))
    ptrn = oracle.get_contraction_ptrn(2, 2, 2, [1, 2, 1, 3, 3, 2])[1]
    scale = 2.0 ** rng.integers(-40, 40, m)
    L = [np.outer(scale, np.ones(k)) * rng.integers(-9, 10, (m, k)) for k in ks]
    for i in range(m):
        q = int(rng.integers(len(ks)))
        L[q][i, int(rng.integers(ks[q]))] = scale[i] * 127 * rng.choice([-1, 1])
    R = [rng.integers(-9, 10, (k, n)).astype(np.float64) for k in ks]
    dev = lambda x: torch.tensor(x.ravel(order="F"), device="cuda")
    d = torch.full((m * n,), float("nan"), dtype=torch.float64, device="cuda")
    trip = [(d, dev(l), dev(r), [m, n], [m, k], [k, n]) for l, r, k in zip(L, R, ks)]
    b = a4.device.Batch(ptrn, 2, 2, 2, trip, precision=a4.device.PREC_OZAKI_BF16, slices=1)
    b.run(stream=torch.cuda.current_stream())
    want = sum(l @ r for l, r in zip(L, R))
    assert np.array_equal(d.cpu().numpy(), want.ravel(order="F"))
    b.close()
