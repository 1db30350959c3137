"""The energy array's rank and extents belong to a fused step's structure: a
rebind that brings another shape is refused (the blocks' offsets would be taken
from another layout), one that brings other values of the same shape is not."""
import numpy as np
import pytest

from tests import test_gpu_fused as fused

pytestmark = pytest.mark.gpu

a4 = fused.a4


def test_rebind_with_another_energy_shape_is_refused(a4):
    import torch

    o_segs, v_segs = [6], [9, 8]
    V1, V2, T, fock = fused._problem(o_segs, v_segs, 3)
    norb = sum(o_segs) + sum(v_segs)
    W, terms = fused._step(V1, V2, T, o_segs, v_segs, 0, 0)
    good = fused._energy_args(W, o_segs, v_segs, torch.tensor(fock, device="cuda"))
    step = a4.device.Fused(6, 4, 4, terms, energy=good)
    e0, e1 = (torch.zeros(1, dtype=torch.float64, device="cuda") for _ in range(2))
    torch.cuda.synchronize()
    step.run(e0)
    a4.device.sync()
    diagonal = np.diagonal(fock.reshape(norb, norb)).copy()
    wide = np.diag(np.concatenate([diagonal, np.ones(5)])).ravel(order="F").copy()
    # A4G_ERR_UNSUPPORTED: rank 6 takes the diagonal of a matrix only; A4G_ERR_ARG: another structure
    for ext1, e, code in (([norb], diagonal, 6), ([norb + 5, norb + 5], wide, 1),
                          ([norb, norb + 5], np.zeros(norb * (norb + 5)), 1)):
        other = dict(good, ext1=ext1, e_or_fock=torch.tensor(e, device="cuda"))
        with pytest.raises(a4.device.A4GError) as err:
            step.rebind(terms, energy=other)
        assert err.value.rc == code
    step.rebind(terms, energy=dict(good, e_or_fock=torch.tensor(fock, device="cuda")))
    step.run(e1)
    a4.device.sync()
    assert e1.item() == e0.item() != 0.0
