"""Slice and insert over their forms: pairs and single elements (odd runs,
odd offsets, odd strides, blocks off 16 bytes), dims that join and unit dims,
CTA edges; and element-wise operations at the edges of a CTA's share.  Copies
and single operations: equal to numpy's bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

CASES = [  # block extents, slice extents, first element
    ([7], [3], [2]), ([8], [4], [2]), ([8], [4], [1]), ([1, 6], [1, 4], [0, 1]), ([6, 1, 4], [6, 1, 2], [0, 0, 1]),
    ([6, 5, 4], [4, 5, 4], [2, 0, 0]), ([6, 5, 4], [4, 5, 4], [1, 0, 0]), ([6, 5, 4], [6, 5, 2], [0, 0, 1]),
    ([5, 5, 4], [4, 5, 4], [0, 0, 0]), ([4, 3, 4], [4, 3, 4], [0, 0, 0]), ([5, 9, 6, 7], [1, 9, 1, 3], [4, 0, 5, 2]),
    ([12, 10, 6, 8], [8, 7, 5, 6], [2, 1, 0, 2]), ([3, 2, 3, 2, 3, 2], [2, 2, 1, 2, 3, 1], [1, 0, 2, 0, 0, 1]),
    ([40, 33, 2], [32, 32, 2], [8, 1, 0]), ([70000], [65537], [4000]), ([300, 301], [256, 300], [44, 1]),
]


@pytest.fixture(scope="module")
def a4():
    import aces4_gb300

    aces4_gb300.build()
    aces4_gb300.device.init(0)
    return aces4_gb300


@pytest.mark.parametrize("te,se,beg", CASES)
@pytest.mark.parametrize("shift", [0, 1])
def test_slice_insert(a4, te, se, beg, shift):
    import torch

    st = torch.cuda.current_stream()
    nt, ns = int(np.prod(te)), int(np.prod(se))
    t = torch.arange(nt + shift, dtype=torch.float64, device="cuda")[shift:]
    s = torch.full((ns + shift,), -1.0, dtype=torch.float64, device="cuda")[shift:]
    at = tuple(slice(b, b + n) for b, n in zip(beg, se))
    T = t.cpu().numpy().reshape(te, order="F")
    a4.device.slice_block(t, te, s, se, beg, stream=st)
    assert np.array_equal(s.cpu().numpy(), T[at].ravel(order="F"))
    u = torch.full((nt + shift,), 0.5, dtype=torch.float64, device="cuda")[shift:]
    a4.device.insert_block(u, te, s, se, beg, stream=st)
    U = np.full(te, 0.5, order="F")
    U[at] = T[at]
    assert np.array_equal(u.cpu().numpy(), U.ravel(order="F"))


@pytest.mark.parametrize("n", [1, 2, 3, 1023, 1024, 1025, 2049, 100001])
@pytest.mark.parametrize("shift", [0, 1])
def test_element_wise(a4, n, shift):
    import torch

    st = torch.cuda.current_stream()
    rng = np.random.default_rng(n)
    x, y = rng.normal(size=n), rng.normal(size=n)
    dev = lambda v: torch.cat([torch.zeros(shift, dtype=torch.float64), torch.from_numpy(v)]).cuda()[shift:]
    a, b = dev(x), dev(y)
    a4.device.add_scaled(a, b, 0.3, stream=st)
    assert np.array_equal(a.cpu().numpy(), x + y * 0.3)
    a4.device.scale_copy(a, b, -1.7, stream=st)
    assert np.array_equal(a.cpu().numpy(), y * -1.7)
    a4.device.fill(a, 2.5, stream=st)
    assert np.array_equal(a.cpu().numpy(), np.full(n, 2.5))
