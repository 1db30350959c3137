"""Reconstruction from residues at both sizes of the integer: sums above 2^64
(rounded without a branch) and below (the general path: rows and columns whose
scale is set by one element that multiplies a zero), zeros, both signs, stored,
added and negated.

Tolerance: none.  Whole numbers of at most 7 next to an element of 2^30 lie on
the operands' fixed-point grids (39 bits), and every sum is below 2^53."""
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


@pytest.mark.parametrize("m,n", [(130, 70), (64, 9), (33, 128)])
@pytest.mark.parametrize("beta", [0, 1])
@pytest.mark.parametrize("negate", [False, True])
def test_small_and_large_sums(a4, m, n, beta, negate):
    import torch

    k = 1600
    rng = np.random.default_rng(m + n)
    L, R = rng.integers(-7, 8, (m, k)).astype(np.float64), rng.integers(-7, 8, (k, n)).astype(np.float64)
    L[:, 0], R[0, :], L[:, 1], R[1, :] = 0, 0, 0, 0
    L[::2, 0] = 2.0 ** 30   # every other row scaled by an element that meets zeros
    R[1, ::3] = -2.0 ** 30  # every third column as well
    L[3, 2:] = 0            # a row of zeros
    d0 = rng.integers(-9, 10, (m, n)).astype(np.float64)
    ptrn = oracle.get_contraction_ptrn(2, 2, 2, [1, 2, 1, 3, 3, 2])[1]
    dev = lambda x: torch.tensor(x.ravel(order="F"), device="cuda")
    d = dev(d0)
    b = a4.device.Batch(ptrn, 2, 2, 2, [(d, dev(L), dev(R), [m, n], [m, k], [k, n])],
                        precision=a4.device.PREC_OZAKI_BF16, slices=5, beta=beta, negate=int(negate))
    assert b.products() >= 10  # residues (digits: 5)
    b.run(stream=torch.cuda.current_stream())
    want = (-1 if negate else 1) * (L @ R) + beta * d0
    assert np.array_equal(d.cpu().numpy(), want.ravel(order="F"))
    b.close()
