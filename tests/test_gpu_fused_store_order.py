"""Where a fused step's store form puts its results: destinations whose
fastest index is a row of the product or a column of it (the second is turned
in shared memory), at ragged tile edges (rows off 32 and 128, columns off 8,
16 and 64), into fresh blocks and into blocks that are added to.

Tolerance: 1e-10 of a block's Frobenius norm at 5 slices, the bound of the
other fused tests."""
import numpy as np
import pytest

from oracle import oracle

pytestmark = pytest.mark.gpu

ORDERS = {"rows": [1, 2, 3, 4], "cols": [3, 4, 1, 2], "mixed_cols": [3, 1, 2, 4], "mixed_rows": [1, 3, 2, 4],
          "cols_outer": [4, 2, 3, 1]}


@pytest.fixture(scope="module")
def a4():
    import aces4_gb300

    aces4_gb300.build()
    aces4_gb300.device.init(0)
    return aces4_gb300


@pytest.mark.parametrize("order", list(ORDERS))
@pytest.mark.parametrize("beta", [0, 1])
@pytest.mark.parametrize("ext", [(5, 7, 3, 3), (11, 13, 9, 8), (16, 8, 8, 8), (3, 1, 1, 1), (9, 15, 17, 5)])
@pytest.mark.parametrize("variant", [0, 7])
def test_store_order(a4, order, beta, ext, variant):
    import torch

    labels = ORDERS[order]
    size = {i + 1: e for i, e in enumerate(ext)}
    size[5], size[6] = 7, 5
    _, ptrn = oracle.get_contraction_ptrn(4, 4, 4, labels + [1, 2, 5, 6] + [5, 6, 3, 4])[:2]
    dext, lext, rext = ([size[q] for q in w] for w in (labels, [1, 2, 5, 6], [5, 6, 3, 4]))
    g = torch.Generator(device="cuda")
    g.manual_seed(sum(ext) + beta)
    new = lambda e: torch.empty(int(np.prod(e)), dtype=torch.float64, device="cuda").uniform_(-1.0, 1.0, generator=g)
    L, R, D = new(lext), new(rext), new(dext)
    want = oracle.contract_blas(ptrn, L.cpu().numpy(), lext, R.cpu().numpy(), rext, dext) + beta * D.cpu().numpy()
    if not beta:
        D.fill_(float("nan"))
    f = a4.device.Fused(4, 4, 4, [(ptrn, [(D, L, R, dext, lext, rext)], 1)], beta=beta, variant=variant)
    torch.cuda.synchronize()
    f.run()
    a4.device.sync()
    got = D.cpu().numpy()
    assert np.all(np.isfinite(got))
    assert np.linalg.norm(got - want) <= 1e-10 * np.linalg.norm(want)
    f.close()
