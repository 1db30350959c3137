"""Amplitude update at both ends of the range: (0.5 t) / eps where t / eps is
subnormal, overflows although its half does not, or is not finite.

Tolerance: none, the reference's two operations in order, rounded each."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def a4():
    import aces4_gb300

    aces4_gb300.build()
    aces4_gb300.device.init(0)
    return aces4_gb300


def test_quotients_at_the_ends_of_the_range(a4):
    import torch

    o, v = 1, 6
    ext, segs, iv = [v, o, v, o], [o, v, v], [2, 1, 3, 1]
    n = v * v
    e = np.concatenate([[0.0], np.array([-1e-3, -1e-2, 0.25, 3.0, 7.0, 0.0]), np.array([-1e-3, 1e-2, 0.5, 2.0, 5.0, 0.0])])
    a, b = e[o:o + v], e[o + v:]
    eps = (((0.0 + 0.0) - a[:, None]) - b[None, :]).ravel(order="F")
    rng = np.random.default_rng(2)
    for scale in (1.6e308, 4e305, 2e304, 1e-305, 1e-307, 3e-308, 1e-310, 5e-324, 1.0):
        t = rng.uniform(0.5, 1.0, n) * scale * rng.choice([-1.0, 1.0], n)
        t1 = rng.normal(0.0, 1.0, n)
        with np.errstate(all="ignore"):
            want_err, want_next = -0.5 * (t1 - t / eps), (0.5 * t) / eps
        dev = lambda x: torch.tensor(x, device="cuda")
        zero, err, nxt = dev(np.zeros(n)), dev(np.zeros(n)), dev(np.zeros(n))
        torch.cuda.synchronize()
        a4.device.update_t2(iv, ext, dev(t), zero, dev(t1), zero, err, nxt, [13], dev(e), segs, None)
        a4.device.sync()
        np.testing.assert_array_equal(nxt.cpu().numpy(), want_next, err_msg=str(scale))
        np.testing.assert_array_equal(err.cpu().numpy(), want_err, err_msg=str(scale))
