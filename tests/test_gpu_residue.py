"""The residue form of the split-precision batch (5 or more slices, k ranges of
1536 and more): products modulo coprime numbers, reconstructed exactly.

Where an operand element is a fixed-point number of the slice count, the
result is the exactly rounded product sum, so integer data must come back bit
for bit: on every operand layout, at k lengths around the point where one more
modulus is needed, with every element at the largest magnitude, and through
every store path.  On other data the form keeps the digit form's operand
rounding and drops nothing, so its error stays below the digit form's (the
same step with a pinned variant).
"""
import numpy as np
import pytest
import torch

from oracle import oracle

pytestmark = pytest.mark.gpu

LADDER = ([1, 2, 3, 4], [1, 2, 5, 6], [5, 6, 3, 4])
RING = ([1, 3, 2, 4], [1, 7, 5, 3], [5, 2, 7, 4])


@pytest.fixture(scope="module")
def a4():
    import aces4_gb300

    aces4_gb300.build()
    aces4_gb300.device.init(0)
    return aces4_gb300


def _ptrn(labels):
    d, l, r = labels
    ierr, p = oracle.get_contraction_ptrn(len(d), len(l), len(r), d + l + r)
    assert ierr == 0
    return p


def _step(labels, de, le, re, pairs, fill, seed):
    """One destination block fed by `pairs` block pairs."""
    rng = np.random.default_rng(seed)
    ls = [fill(rng, int(np.prod(le))) for _ in range(pairs)]
    rs = [fill(rng, int(np.prod(re))) for _ in range(pairs)]
    want = sum(oracle.contract_blas(_ptrn(labels), ls[q], le, rs[q], re, de) for q in range(pairs))
    d = torch.full((int(np.prod(de)),), float("nan"), dtype=torch.float64, device="cuda")
    trip = [(d, torch.tensor(ls[q], device="cuda"), torch.tensor(rs[q], device="cuda"), de, le, re)
            for q in range(pairs)]
    return d, trip, want


def _integers(bits):
    return lambda rng, n: rng.integers(-(1 << bits), (1 << bits) + 1, n).astype(np.float64)


def _batch(a4, labels, trip, slices, products, **kw):
    n = [len(x) for x in labels]
    b = a4.device.Batch(_ptrn(labels), *n, trip, precision=a4.device.PREC_OZAKI_BF16, slices=slices, **kw)
    assert b.products() == products
    return b


# the sum's bound is K 4^(8 slices - 1): 10 moduli hold 5 slices up to K = 1629
# (25 k blocks of 64), 11 beyond; 12 hold 6 slices here, 14 hold 7
@pytest.mark.parametrize("slices,k,products", [(5, (40, 40), 10), (5, (40, 41), 11), (5, (73, 29), 11),
                                               (6, (40, 41), 12), (7, (41, 39), 14)])
@pytest.mark.parametrize("labels", [LADDER, RING])
def test_integers_exact_on_every_layout(a4, labels, slices, k, products):
    """|x| <= 2^17 and K below 2^12: every sum is below 2^53, FP64 is exact.
    Odd extents: partial tiles, k lengths that are no multiple of 8."""
    kc, kd = k
    if labels is LADDER:
        de, le, re = [7, 5, 3, 11], [7, 5, kc, kd], [kc, kd, 3, 11]
    else:
        de, le, re = [7, 3, 5, 11], [7, kc, kd, 3], [kd, 5, kc, 11]
    d, trip, want = _step(labels, de, le, re, 1, _integers(17), 3)
    b = _batch(a4, labels, trip, slices, products)
    b.run()
    a4.device.sync()
    np.testing.assert_array_equal(d.cpu().numpy(), want)


@pytest.mark.parametrize("slices,products", [(5, (10, 11)), (6, (12, 12))])
@pytest.mark.parametrize("kb", [25, 26])
def test_largest_magnitudes(a4, slices, products, kb):
    """Every element is +-(1 - 2^-53), the largest below its row scale, whose
    fixed-point value rounds up to +-2^(8 slices - 1): every partial sum and
    residue sum at its bound; the result is +-K exactly (the sign pattern of
    the columns)."""
    K, M, N = 64 * kb, 130, 70
    labels = ([1, 2], [1, 3], [3, 2])
    big = 1.0 - 2.0 ** -53
    l = torch.full((M * K,), big, dtype=torch.float64, device="cuda")
    sign = torch.where(torch.arange(N, device="cuda") % 3 == 1, -1.0, 1.0).to(torch.float64)
    r = (sign.view(N, 1) * big).expand(N, K).contiguous().view(-1)
    d = torch.full((M * N,), float("nan"), dtype=torch.float64, device="cuda")
    b = _batch(a4, labels, [(d, l, r, [M, N], [M, K], [K, N])], slices, products[kb - 25])
    b.run()
    a4.device.sync()
    assert torch.equal(d.view(N, M), (sign * K).view(N, 1).expand(N, M))


@pytest.mark.parametrize("slices,products,tol", [(5, 11, 1e-10), (6, 13, 1e-12), (7, 14, 1e-14)])
def test_error_below_the_digit_form(a4, slices, products, tol):
    """Operands over a wide range (1 % of the entries a thousand times larger):
    the same operand rounding as the digit form and no dropped term."""
    def fill(rng, n):
        x = rng.normal(0.0, 0.1, n)
        x[rng.random(n) < 0.01] *= 1e3
        return x

    de, le, re = [24, 20, 12, 13], [24, 20, 45, 44], [45, 44, 12, 13]
    d, trip, want = _step(LADDER, de, le, re, 4, fill, 9)
    b = _batch(a4, LADDER, trip, slices, products)
    b.run()
    bound = b.error_bound()
    err = np.linalg.norm(d.cpu().numpy() - want) / np.linalg.norm(want)
    digits = _batch(a4, LADDER, trip, slices, slices * (slices + 1) // 2, variant=3)
    digits.run()
    a4.device.sync()
    err_digits = np.linalg.norm(d.cpu().numpy() - want) / np.linalg.norm(want)
    # both against FP64 BLAS, itself within K 2^-53 of the exact sum
    assert err <= err_digits + 7920 * 2.0 ** -53, (err, err_digits)
    assert err <= tol and err <= bound


def test_store_modes_graph_hold_rebind_and_pipeline(a4):
    """Accumulate and negate, a graph replay, a held operand, another pair of
    blocks, the pipelined GEMM: integer data, so all are exact."""
    de, le, re = [30, 9, 6, 5], [30, 9, 40, 44], [40, 44, 6, 5]
    d, trip, want = _step(LADDER, de, le, re, 2, _integers(12), 4)
    d2, trip2, want2 = _step(LADDER, de, le, re, 2, _integers(12), 5)
    base = torch.randint(-1000, 1000, d.shape, device="cuda").to(torch.float64)
    d.copy_(base)
    b = _batch(a4, LADDER, trip, 5, 11, beta=1, negate=True)
    b.run_graph()
    b.run_graph()
    a4.device.sync()
    np.testing.assert_array_equal(d.cpu().numpy(), base.cpu().numpy() - 2 * want)
    b = _batch(a4, LADDER, trip, 5, 11)
    b.hold(1)
    b.run()
    a4.device.sync()
    np.testing.assert_array_equal(d.cpu().numpy(), want)
    b.hold(1, False)
    b.rebind(trip2)
    b.run_graph()
    a4.device.sync()
    np.testing.assert_array_equal(d2.cpu().numpy(), want2)
    p = _batch(a4, LADDER, trip, 5, 11, pipeline=3)
    d.fill_(float("nan"))
    p.run()
    a4.device.sync()
    np.testing.assert_array_equal(d.cpu().numpy(), want)


def test_columns_contiguous_destination(a4):
    """D unit-stride along the columns (stored through shared memory): the
    first destination has one column, so the operands keep their roles, and the
    second has 45."""
    labels = ([1, 2], [2, 3], [3, 1])
    d1, t1, w1 = _step(labels, [1, 70], [70, 1700], [1700, 1], 1, _integers(16), 6)
    d2, t2, w2 = _step(labels, [45, 70], [70, 1700], [1700, 45], 1, _integers(16), 7)
    b = _batch(a4, labels, t1 + t2, 5, 11)
    b.run()
    a4.device.sync()
    np.testing.assert_array_equal(d1.cpu().numpy(), w1)
    np.testing.assert_array_equal(d2.cpu().numpy(), w2)


@pytest.mark.parametrize("slices,products", [(5, 11), (7, 14)])
def test_non_finite_and_extreme_rows(a4, slices, products):
    """A NaN poisons its row, an infinity its column; zero rows, rows of
    subnormal size and rows near the largest double stay exact beside them."""
    labels = ([1, 2], [1, 3], [3, 2])
    M, N, K = 70, 20, 1700
    rng = np.random.default_rng(8)
    l = rng.integers(-500, 501, (K, M)).astype(np.float64)  # [k][m]: m fastest
    r = rng.integers(-500, 501, (N, K)).astype(np.float64)
    l[:, 3] = 0.0
    l[:, 4] *= 2.0 ** -1060   # exact subnormal multiples
    l[:, 5] *= 2.0 ** 1000
    l[7, 6] = np.nan
    r[2, 9] = np.inf
    with np.errstate(over="ignore", invalid="ignore"):
        want = np.zeros((N, M))
        for m in range(M):
            s = {4: 2.0 ** -1060, 5: 2.0 ** 1000}.get(m, 1.0)
            want[:, m] = (np.nan_to_num(r, posinf=0.0) @ (l[:, m] / s)) * s
    want[:, 6] = np.nan
    want[2, :] = np.nan
    d = torch.zeros(M * N, dtype=torch.float64, device="cuda")
    b = _batch(a4, labels, [(d, torch.tensor(l.ravel(), device="cuda"), torch.tensor(r.ravel(), device="cuda"),
                             [M, N], [M, K], [K, N])], slices, products)
    b.run()
    a4.device.sync()
    np.testing.assert_array_equal(d.view(N, M).cpu().numpy(), want)
