"""out = a D in + b out, the xpay field written over: the first call on a shape, which times kernels with the
caller's fields, applies the hop once all the same."""
import numpy as np
import pytest

from mrhs_qcu_gb300 import synthetic as S
from oracle import oracle as O
from tests.util import TOL, dev, rel

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec,n,nrhs", [(2, 3, 3), (1, 3, 10), (1, 6, 5), (0, 3, 6), (4, 4, 12), (5, 5, 20)])
def test_first_call(cuda, qcu_lib, monkeypatch, prec, n, nrhs):
    torch, Q = cuda, qcu_lib
    monkeypatch.delenv("QCU_DSLASH_CONFIG", raising=False)
    L, a, b = (4, 6, 2, 10), -0.25, 0.5  # no other test tunes this lattice
    g = S.random_gauge(L, n, seed=61)
    full = S.random_fermions(L, n, nrhs, seed=62, parities=2)
    Q.initGridSize(L, n)
    Q.set_antiperiodic_t(True)
    dg = dev(torch, g)
    Q.loadQcuGauge(dg.data_ptr())
    db, nb = Q.field_bytes(prec, nrhs)
    f = [torch.zeros(db, dtype=torch.uint8, device="cuda") for _ in range(2)]
    s = [torch.zeros(max(nb, 16), dtype=torch.uint8, device="cuda") for _ in range(2)]
    src = [dev(torch, p) for p in full]
    for p in (0, 1):
        Q.pack_fermions(f[p].data_ptr(), s[p].data_ptr(), [x.data_ptr() for x in src], Q.QCU_SRC_EO_FULL, p, prec)
    for dagger in (0, 1):  # the second call takes the tuned shape
        Q.dslash_xpay_mrhs(f[0].data_ptr(), s[0].data_ptr(), f[1].data_ptr(), s[1].data_ptr(), f[0].data_ptr(),
                           s[0].data_ptr(), nrhs, 0, dagger, prec, a, b)
    out = [torch.zeros((S.half_volume(L), 4, n), dtype=torch.complex128, device="cuda") for _ in range(nrhs)]
    Q.unpack_fermions([o.data_ptr() for o in out], f[0].data_ptr(), s[0].data_ptr(), Q.QCU_SRC_EO_HALF, 0, prec)
    Q.synchronize()
    got, want = np.stack([o.cpu().numpy() for o in out]), full[:, 0]
    for dagger in (0, 1):
        want = a * O.dslash(full[:, 1], g, L, 0, dagger, True) + b * want
    assert rel(got, want) < TOL[prec]
