"""Permutes and permuted add / subtract over their forms: runs along an index
that stays first (pairs, odd lengths, odd strides, blocks off 16 bytes), planes
at the edges of the 32- and 64-wide tiles, small planes, merged and unit dims.  Copies and single operations: equal to numpy's bit for bit."""
import itertools

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SHAPES = [(7, 5), (64, 65), (129, 3), (2, 300), (33, 20, 9), (48, 97, 5), (6, 4, 5, 8), (5, 3, 7, 4), (17, 64, 2, 66),
          (2, 2, 2, 500), (40, 12, 33, 10), (1, 6, 1, 9), (2, 3, 2, 4, 3), (70, 1, 130)]


@pytest.fixture(scope="module")
def a4():
    import aces4_gb300

    aces4_gb300.build()
    aces4_gb300.device.init(0)
    return aces4_gb300


@pytest.mark.parametrize("ext", SHAPES)
@pytest.mark.parametrize("shift", [0, 1])
def test_permute_add_sub(a4, ext, shift):
    import torch

    st = torch.cuda.current_stream()
    n = int(np.prod(ext))
    rng = np.random.default_rng(n)
    dev = lambda v: torch.cat([torch.zeros(shift, dtype=torch.float64), torch.from_numpy(v)]).cuda()[shift:]
    x, l = rng.normal(size=n), rng.normal(size=n)
    X, L, out = dev(x), dev(l), dev(np.zeros(n))
    perms = list(itertools.permutations(range(1, len(ext) + 1)))
    for o2n in perms if len(perms) <= 24 else perms[::7]:
        # index i of x is index o2n[i] of the result
        axes = [o2n.index(p + 1) for p in range(len(ext))]
        want = np.transpose(x.reshape(ext, order="F"), axes).ravel(order="F")
        out.fill_(float("nan"))
        a4.device.permute(ext, o2n, X, out, stream=st)
        assert np.array_equal(out.cpu().numpy(), want), o2n
        lab = list(range(1, len(ext) + 1))
        for sub in (False, True):
            out.fill_(float("nan"))
            a4.device.add_sub(sub, lab, list(o2n), ext, out, L, X, stream=st)
            assert np.array_equal(out.cpu().numpy(), l - want if sub else l + want), o2n
