"""A right block that a destination skips (its left partner is a zero block)
must not reach that destination: neither its non-finite values nor its scale,
although other destinations of the same step multiply it.

Every destination is scaled by the blocks that it multiplies, so its result is
the same bit for bit whatever the skipped block holds; and it is within the
1e-10 (relative, Frobenius) that five slices give on operands of one scale."""
import numpy as np
import pytest
import torch

from oracle import oracle

pytestmark = pytest.mark.gpu

LABELS = ([1, 2], [1, 3], [3, 2])
ROWS, COLS, KS = [40, 129, 7], 70, [640, 576, 704, 640]  # whole 64s of k: overlapping sets cost nothing to join
SKIPPED = [2, 0, 3]  # the right block that destination m does not multiply
SPOILED = 2          # the one that is changed: skipped by the first destination only


@pytest.fixture(scope="module")
def a4():
    import aces4_gb300

    aces4_gb300.build()
    aces4_gb300.device.init(0)
    return aces4_gb300


def _step(seed):
    rng = np.random.default_rng(seed)
    r = [rng.normal(0.0, 0.1, k * COLS) for k in KS]
    l = [[rng.normal(0.0, 0.1, m * k) if q != SKIPPED[i] else None for q, k in enumerate(KS)] for i, m in enumerate(ROWS)]
    return l, r


def _run(a4, ptrn, l, r, **kw):
    tr = [torch.tensor(x, device="cuda") for x in r]
    outs, trip = [], []
    for i, m in enumerate(ROWS):
        d = torch.full((m * COLS,), float("nan"), dtype=torch.float64, device="cuda")
        outs.append(d)
        for q, k in enumerate(KS):
            tl = None if l[i][q] is None else torch.tensor(l[i][q], device="cuda")
            trip.append((d, tl, tr[q], [m, COLS], [m, k], [k, COLS]))
    b = a4.device.Batch(ptrn, 2, 2, 2, trip, precision=a4.device.PREC_OZAKI_BF16, **kw)
    b.run()
    a4.device.sync()
    return [d.cpu().numpy() for d in outs], b.products()


# digits at two slice counts, the same five slices with a pinned digit form, residues
FORMS = [(2, 0, 3), (4, 0, 10), (5, 3, 15), (5, 0, 11), (7, 0, 14)]


@pytest.mark.parametrize("slices,variant,products", FORMS)
@pytest.mark.parametrize("spoil", ["nan", "inf", "2^10", "2^20", "2^40"])
def test_skipped_block_does_not_reach_the_result(a4, slices, variant, products, spoil):
    ierr, ptrn = oracle.get_contraction_ptrn(2, 2, 2, sum(LABELS, []))
    assert ierr == 0
    l, r = _step(11)
    plain, n = _run(a4, ptrn, l, r, slices=slices, variant=variant)
    assert n == products
    if spoil in ("nan", "inf"):
        bad = float(spoil)
        r[SPOILED][[5, 64 * KS[SPOILED] + 9]] = bad  # columns 0 and 64
    else:
        r[SPOILED] = r[SPOILED] * 2.0 ** int(spoil[2:])
    spoiled, _ = _run(a4, ptrn, l, r, slices=slices, variant=variant)
    np.testing.assert_array_equal(spoiled[0], plain[0])
    want = sum(oracle.contract_blas(ptrn, l[0][q], [ROWS[0], KS[q]], r[q], [KS[q], COLS], [ROWS[0], COLS])
               for q in range(len(KS)) if q != SKIPPED[0])
    if slices >= 5:
        assert np.linalg.norm(spoiled[0] - want) <= 1e-10 * np.linalg.norm(want)
    if spoil in ("nan", "inf"):  # the destinations that multiply it: these columns and no other
        for i in (1, 2):
            cols = np.isnan(spoiled[i].reshape(COLS, ROWS[i])).any(axis=1)
            assert np.flatnonzero(cols).tolist() == [0, 64]
