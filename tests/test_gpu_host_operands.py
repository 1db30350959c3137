"""Drop-in contractions of host blocks on both sides of the size from which
their operands are copied to the device first (16384 elements), with a result
block that is an operand too.

Tolerance: none; the operands are whole numbers of at most 8, every sum is
exact."""
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


@pytest.mark.parametrize("n", [3, 90, 91, 200])  # 2 n^2 elements: 16200 and 16562 around the line
@pytest.mark.parametrize("alias", [None, "left", "right", "operands"])
def test_host_contraction(a4, n, alias):
    rng = np.random.default_rng(n)
    whole = lambda: rng.integers(-8, 9, n * n).astype(np.float64)
    l, r = whole(), whole()
    if alias == "operands":
        r = l
    want = (l.reshape((n, n), order="F") @ r.reshape((n, n), order="F")).ravel(order="F")
    d = l if alias == "left" else r if alias == "right" else np.full(n * n, np.nan)
    ptrn = oracle.get_contraction_ptrn(2, 2, 2, [1, 2, 1, 3, 3, 2])[1]
    assert a4.ref.tensor_block_contract(ptrn, l, [n, n], r, [n, n], d, [n, n]) == 0
    assert np.array_equal(d, want)
