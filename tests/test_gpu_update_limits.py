"""Blocks beyond the amplitude update's range are refused before anything is
launched: more than 65535 (i,j) pairs."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def a4():
    import aces4_gb300

    aces4_gb300.build()
    aces4_gb300.device.init(0)
    return aces4_gb300


@pytest.mark.parametrize("o,refused", [(255, False), (256, True)])
def test_too_many_occupied_pairs(a4, o, refused):
    import torch

    segs, ext = [o, 1, 1], [1, o, 1, o]
    x = [torch.full((o * o,), 0.25, dtype=torch.float64, device="cuda") for _ in range(4)]
    nxt, norm = torch.zeros_like(x[0]), torch.zeros(1, dtype=torch.float64, device="cuda")
    e = torch.tensor(np.concatenate([np.full(o, -1.0), [1.0, 1.0]]), device="cuda")
    call = lambda: a4.device.update_t2([2, 1, 3, 1], ext, *x, None, nxt, [o + 2], e, segs, norm)
    torch.cuda.synchronize()
    if refused:
        with pytest.raises(a4.device.A4GError) as err:
            call()
        assert err.value.rc == 7  # A4G_ERR_RANGE
        a4.device.sync()
        assert norm.item() == 0.0 and not nxt.any()
    else:
        call()
        a4.device.sync()
        assert (nxt == -0.0625).all()  # (0.25 + 0.25) / 2 / (-4)
