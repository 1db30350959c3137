"""Right-operand panels shared by destinations whose zero blocks leave them with
different, overlapping sets of right blocks: ragged k lengths, gaps at the
start, the middle and the end, pairs in different orders.  Integer data, so
every form must return the exact sums."""
import numpy as np
import pytest
import torch

from oracle import oracle

pytestmark = pytest.mark.gpu

LABELS = ([1, 2], [1, 3], [3, 2])


@pytest.fixture(scope="module")
def a4():
    import aces4_gb300

    aces4_gb300.build()
    aces4_gb300.device.init(0)
    return aces4_gb300


@pytest.mark.parametrize("slices,variant,k", [(2, 1, [5, 17, 64, 33, 16, 70]), (2, 6, [5, 17, 64, 33, 16, 70]),
                                              (5, 0, [500, 333, 640, 417, 1001, 64])])
def test_overlapping_right_sets(a4, slices, variant, k):
    rng = np.random.default_rng(3)
    ierr, p = oracle.get_contraction_ptrn(2, 2, 2, sum(LABELS, []))
    assert ierr == 0
    ms, ns = [40, 129, 7], [31, 70]
    live = [[1, 2, 3, 5], [0, 1, 4, 5], [4, 3, 2, 0]]  # which k blocks destination row m has, in its own order
    r = {(q, n): rng.integers(-99, 100, k[q] * ns[n]).astype(np.float64) for q in range(len(k)) for n in range(len(ns))}
    tr = {key: torch.tensor(x, device="cuda") for key, x in r.items()}
    trip, want, outs = [], [], []
    for m, rows in enumerate(ms):
        ls = {q: rng.integers(-99, 100, rows * k[q]).astype(np.float64) for q in live[m]}
        tl = {q: torch.tensor(x, device="cuda") for q, x in ls.items()}
        order = live[m] + [q for q in range(len(k)) if q not in live[m]]
        for n, cols in enumerate(ns):
            d = torch.full((rows * cols,), float("nan"), dtype=torch.float64, device="cuda")
            trip += [(d, tl.get(q), tr[q, n], [rows, cols], [rows, k[q]], [k[q], cols]) for q in order]
            want.append(sum(oracle.contract_blas(p, ls[q], [rows, k[q]], r[q, n], [k[q], cols], [rows, cols])
                            for q in live[m]))
            outs.append(d)
    b = a4.device.Batch(p, 2, 2, 2, trip, precision=a4.device.PREC_OZAKI_BF16, slices=slices, variant=variant)
    b.run()
    a4.device.sync()
    for d, w in zip(outs, want):
        np.testing.assert_array_equal(d.cpu().numpy(), w)
