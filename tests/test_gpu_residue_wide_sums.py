"""Seven slices over k ranges whose sums pass 2^127: fifteen moduli and a
five-word reconstruction.  Rows and columns on three scales (sums near 2^127,
below 2^96 and zero), both signs, stored and added.

Tolerance: none.  Whole numbers of at most 7, next to an element of 2^40 that
meets zeros, lie on the operands' 55-bit grids, and every sum is below 2^53."""
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


@pytest.mark.parametrize("k,beta", [(135000, 0), (150001, 1)])
def test_wide_sums(a4, k, beta):
    import torch

    m, n = 500, 490  # large enough that the products saved pay for the panels
    rng = np.random.default_rng(k)
    L, R = rng.integers(-7, 8, (m, k)).astype(np.float64), rng.integers(-7, 8, (k, n)).astype(np.float64)
    L[0::7] = np.abs(L[0::7])
    R[:, 0::5] = np.abs(R[:, 0::5])  # some sums near the largest
    L[1::7] = -np.abs(L[1::7])
    L[:, :2], R[:2, :] = 0, 0
    L[::2, 0] = 2.0 ** 40
    R[1, ::3] = -2.0 ** 40
    L[3, 2:] = 0
    d0 = rng.integers(-9, 10, (m, n)).astype(np.float64)
    ptrn = oracle.get_contraction_ptrn(2, 2, 2, [1, 2, 1, 3, 3, 2])[1]
    dev = lambda x: torch.tensor(x.ravel(order="F"), device="cuda")
    d = dev(d0)
    b = a4.device.Batch(ptrn, 2, 2, 2, [(d, dev(L), dev(R), [m, n], [m, k], [k, n])],
                        precision=a4.device.PREC_OZAKI_BF16, slices=7, beta=beta)
    assert b.products() == 15
    b.run(stream=torch.cuda.current_stream())
    want = L @ R + beta * d0
    assert np.array_equal(d.cpu().numpy(), want.ravel(order="F"))
    b.close()
