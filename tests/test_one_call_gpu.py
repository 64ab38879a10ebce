"""The one-call operators keep their session between calls: results follow
the links and lattice of each call, whatever ran before, and from several
threads."""
import threading

import numpy as np
import pytest

from mrhs_qcu_gb300 import synthetic as S
from oracle import oracle as O
from tests.util import dev, rel

pytestmark = pytest.mark.gpu


def _call(torch, Q, L, seed, dagger):
    g, psi = S.random_gauge(L, 3, seed=seed), S.random_fermions(L, 3, 1, seed=seed + 1, parities=2)[0]
    dg, dp = dev(torch, g), dev(torch, psi)
    out = torch.zeros_like(dp)
    torch.cuda.synchronize()
    Q.fullDslashQcu(out.data_ptr(), dp.data_ptr(), dg.data_ptr(), L, dagger)
    torch.cuda.synchronize()
    got = out.cpu().numpy()
    want = np.stack([O.dslash(psi[None, 1 - p], g, L, p, dagger, False)[0] for p in (0, 1)])
    assert rel(got, want) < 1e-13, (L, seed, dagger)


def test_lattices_and_links_change_between_calls(cuda, qcu_lib):
    Q = qcu_lib
    Q.set_antiperiodic_t(False)
    for L, seed in (((4, 4, 4, 4), 1), ((4, 4, 4, 4), 5), ((6, 4, 2, 8), 9), ((4, 4, 4, 8), 13), ((4, 4, 4, 4), 17)):
        for dagger in (0, 1):
            _call(cuda, Q, L, seed, dagger)
    Q.initGridSize((4, 4, 4, 4), 3)  # frees what is kept
    _call(cuda, Q, (4, 4, 4, 4), 21, 0)


def test_threads(cuda, qcu_lib):
    Q = qcu_lib
    Q.set_antiperiodic_t(False)
    failed = []

    def work(k):
        try:
            for i in range(3):
                _call(cuda, Q, ((4, 4, 4, 4), (4, 2, 4, 6))[k % 2], 31 + 10 * k + i, i % 2)
        except Exception as e:  # reported by the main thread
            failed.append(e)

    threads = [threading.Thread(target=work, args=(k,)) for k in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failed, failed
