"""Residues against digits on the same step, each into a destination of its own:
operands over a wide range (1 % of the entries a thousand times larger), where
the residues round like the digits and drop no product, so that their error
stays below the digits'.

Tolerance: both are measured against an FP64 BLAS product, itself within
K 2^-53 of the exact sum."""
import numpy as np
import pytest

from oracle import oracle

pytestmark = pytest.mark.gpu

LABELS = ([1, 2], [1, 3], [3, 2])
M, N, KS = 200, 90, [900, 1100]


@pytest.fixture(scope="module")
def a4():
    import aces4_gb300

    aces4_gb300.build()
    aces4_gb300.device.init(0)
    return aces4_gb300


@pytest.mark.parametrize("slices,products", [(5, 11), (6, 12), (7, 14)])
def test_errors(a4, slices, products):
    import torch

    rng = np.random.default_rng(slices)

    def fill(n):
        x = rng.normal(0.0, 0.1, n)
        x[rng.random(n) < 0.01] *= 1e3
        return x

    ptrn = oracle.get_contraction_ptrn(2, 2, 2, sum(LABELS, []))[1]
    ls, rs = [fill(M * k) for k in KS], [fill(k * N) for k in KS]
    want = sum(oracle.contract_blas(ptrn, l, [M, k], r, [k, N], [M, N]) for l, r, k in zip(ls, rs, KS))
    tl, tr = [torch.tensor(x, device="cuda") for x in ls], [torch.tensor(x, device="cuda") for x in rs]

    def run(variant):
        d = torch.full((M * N,), float("nan"), dtype=torch.float64, device="cuda")
        b = a4.device.Batch(ptrn, 2, 2, 2, [(d, l, r, [M, N], [M, k], [k, N]) for l, r, k in zip(tl, tr, KS)],
                            precision=a4.device.PREC_OZAKI_BF16, slices=slices, variant=variant)
        b.run()
        a4.device.sync()
        x = d.cpu().numpy()
        return b.products(), x, np.linalg.norm(x - want) / np.linalg.norm(want)

    n_res, res, err = run(0)
    n_dig, dig, err_digits = run(3)
    assert (n_res, n_dig) == (products, slices * (slices + 1) // 2)
    assert np.isfinite(dig).all() and np.isfinite(res).all()
    assert slices == 7 or not np.array_equal(res, dig)
    assert err <= err_digits + sum(KS) * 2.0 ** -53
