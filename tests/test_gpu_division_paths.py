"""The interleaved exact division in its callers: blocks whose extents leave
part of a tile, of a group of elements or of a warp empty, and elements that
leave the integer path (zeros, subnormals, infinities), against the oracle's
sequence of the reference's operations, bit for bit (sums to the rounding of a
long FP64 sum).  The division itself tolerates a reciprocal seed one unit off
(host run of the same source)."""
import os
import shutil
import subprocess

import numpy as np
import pytest

from oracle import oracle

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.mark.parametrize("ulp", [-1, 1])
def test_division_with_the_seed_one_unit_off(tmp_path, ulp):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("nvcc not available")
    exe = tmp_path / "check"
    r = subprocess.run([nvcc, "-std=c++17", "-O2", "-x", "cu", f"-DA4G_RCP_ULP={ulp}", "-I",
                        os.path.join(ROOT, "aces4_gb300", "csrc"), "-o", str(exe),
                        os.path.join(ROOT, "tests", "exact_fp", "check.cu")], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([str(exe), "400000"], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and "mismatches 0" in r.stdout, r.stdout + r.stderr


@pytest.fixture(scope="module")
def a4():
    import aces4_gb300

    aces4_gb300.build()
    aces4_gb300.device.init(0)
    return aces4_gb300


def _odd_values(rng, n):
    """Ordinary amplitudes with a zero, a negative zero, subnormal and tiny values among them."""
    x = rng.standard_normal(n) * 0.1
    pick = rng.permutation(n)[:max(6, n // 50)]
    x[pick] = rng.choice([0.0, -0.0, 5e-324, -3e-310, 2e-308, 1e-300], pick.size)
    return x


def _energies(rng, segs):
    e = np.concatenate([rng.uniform(-2.0, -0.5, segs[0]), rng.uniform(0.2, 5.0, sum(segs[1:]))])
    return np.diag(e).ravel(order="F").copy(), len(e)


@pytest.mark.gpu
@pytest.mark.parametrize("segs", [[3, 48, 24], [2, 49, 25], [1, 1, 50], [4, 97, 23], [2, 7, 3]])
def test_update_tiles(a4, segs):
    import torch

    rng = np.random.default_rng(sum(segs))
    iv = [2, 1, 3, 1]
    ext = [segs[v - 1] for v in iv]
    n = int(np.prod(ext))
    xn, xnp, xo, xop = (_odd_values(rng, n) for _ in range(4))
    fock, norb = _energies(rng, segs)
    err, nxt, nrm = oracle.update_t2(iv, ext, xn, xnp, xo, xop, [norb, norb], fock, segs)
    d = lambda x: torch.tensor(x, device="cuda")
    e, t = (torch.full((n,), float("nan"), dtype=torch.float64, device="cuda") for _ in range(2))
    n2 = torch.zeros(1, dtype=torch.float64, device="cuda")
    a4.device.update_t2(iv, ext, d(xn), d(xnp), d(xo), d(xop), e, t, [norb, norb], d(fock), segs, n2)
    a4.device.sync()
    np.testing.assert_array_equal(e.cpu().numpy().view(np.int64), err.view(np.int64))
    np.testing.assert_array_equal(t.cpu().numpy().view(np.int64), nxt.view(np.int64))
    assert abs(float(n2.item()) - nrm) <= 1e-13 * nrm


@pytest.mark.gpu
@pytest.mark.parametrize("ext,iv,segs", [
    ([5, 7, 9, 3], [2, 1, 3, 4], [7, 5, 9, 3]),       # runs of 9: two groups of four and one element
    ([40, 21, 4, 2], [2, 1, 3, 4], [21, 40, 4, 2]),   # 840 positions: three CTAs of 288 threads
    ([3, 2, 4, 2, 5, 2], [2, 1, 3, 1, 4, 1], [2, 3, 4, 5]),
    ([20, 20, 2, 3, 7, 3], [2, 1, 3, 4, 5, 4], [20, 20, 2, 3, 7]),
])
def test_denominator_and_energy_groups(a4, ext, iv, segs):
    import torch

    rng = np.random.default_rng(len(ext) + ext[0])
    w = _odd_values(rng, int(np.prod(ext)))
    e = np.concatenate([rng.uniform(-2.0, -0.5, s) if k in (iv[1], iv[3]) else rng.uniform(0.2, 5.0, s)
                        for k, s in enumerate(segs, 1)])
    fock, norb = np.diag(e).ravel(order="F").copy(), len(e)
    want = w.copy()
    assert oracle.energy_denominator_rhf(iv, ext, want, [norb, norb], fock, segs) == 0
    d = torch.tensor(w, device="cuda")
    f = torch.tensor(fock, device="cuda")
    a4.device.energy_denominator(iv, ext, d, [norb, norb], f, segs)
    esum = torch.zeros(1, dtype=torch.float64, device="cuda")
    a4.device.energy_contract(iv, ext, torch.tensor(w, device="cuda"), [norb, norb], f, segs, 1.0, esum)
    a4.device.sync()
    np.testing.assert_array_equal(d.cpu().numpy().view(np.int64), want.view(np.int64))
    total = float(np.sum((w * want).astype(np.longdouble)))
    assert abs(float(esum.item()) - total) <= 1e-13 * np.sum(np.abs(w * want))
