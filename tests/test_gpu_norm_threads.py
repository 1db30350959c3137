"""Norms from several threads at once, on one stream and on the library's own:
each thread gets the norm of its own block, with the bits it gives alone."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def a4():
    import aces4_gb300

    aces4_gb300.build()
    aces4_gb300.device.init(0)
    return aces4_gb300


@pytest.mark.parametrize("own_stream", [True, False])
def test_norms_of_threads(a4, own_stream):
    import torch

    rng = np.random.default_rng(5)
    xs = [torch.tensor(rng.normal(0.0, 0.1 * (q + 1), 30000 + 17 * q), device="cuda") for q in range(12)]
    stream = torch.cuda.Stream() if own_stream else None
    torch.cuda.synchronize()
    want = [a4.device.norm2(x, stream) for x in xs]
    wrong, start = [], threading.Barrier(len(xs))

    def work(q):
        start.wait()
        for _ in range(400):
            got = a4.device.norm2(xs[q], stream)
            if got != want[q]:
                wrong.append((q, got, want[q]))

    threads = [threading.Thread(target=work, args=(q,)) for q in range(len(xs))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong, wrong[:3]
