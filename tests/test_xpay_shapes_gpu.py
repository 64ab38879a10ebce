"""out = a D in + b x over the kernel families (register scalar and packed, split fixed point, MMA): b = 1 and
b != 1, small sizes of every SU(N), and the packed SU(5) kernels."""
import os
import numpy as np
import pytest
from mrhs_qcu_gb300 import synthetic as S
from oracle import oracle as O
from tests.util import TOL, dev, rel

pytestmark = pytest.mark.gpu


def _xpay(torch, Q, full, g, L, prec, parity, dagger, a, b):
    nrhs, _, vh, _, n = full.shape
    Q.initGridSize(L, n)
    Q.set_antiperiodic_t(True)
    dg = dev(torch, g)
    Q.loadQcuGauge(dg.data_ptr())
    db, nb = Q.field_bytes(prec, nrhs)
    f = [torch.empty(db // 8 + 2, dtype=torch.float64, device="cuda") for _ in range(3)]
    s = [torch.empty(max(nb, 16) // 4, dtype=torch.float32, device="cuda") for _ in range(3)]
    nrm = (lambda i: s[i].data_ptr()) if nb else (lambda i: None)
    src = [dev(torch, full[r]) for r in range(nrhs)]
    ptrs = [x.data_ptr() for x in src]
    Q.pack_fermions(f[0].data_ptr(), nrm(0), ptrs, Q.QCU_SRC_EO_FULL, 1 - parity, prec)
    Q.pack_fermions(f[1].data_ptr(), nrm(1), ptrs, Q.QCU_SRC_EO_FULL, parity, prec)
    Q.dslash_xpay_mrhs(f[2].data_ptr(), nrm(2), f[0].data_ptr(), nrm(0), f[1].data_ptr(), nrm(1), nrhs, parity,
                       dagger, prec, a, b)
    outs = [torch.zeros((vh, 4, n), dtype=torch.complex128, device="cuda") for _ in range(nrhs)]
    Q.unpack_fermions([o.data_ptr() for o in outs], f[2].data_ptr(), nrm(2), Q.QCU_SRC_EO_HALF, parity, prec)
    Q.synchronize()
    return np.stack([o.cpu().numpy() for o in outs])


@pytest.mark.parametrize("prec", [2, 1, 4])
@pytest.mark.parametrize("n,L,nrhs", [(3, (4, 4, 2, 4), 12), (3, (6, 2, 4, 4), 1), (4, (4, 2, 4, 4), 4), (5, (4, 2, 2, 4), 2),
                                      (6, (4, 2, 2, 4), 4), (8, (2, 2, 2, 4), 8)])
@pytest.mark.parametrize("b", [1.0, -0.75])
def test_xpay_every_shape(cuda, qcu_lib, prec, n, L, nrhs, b):
    """Every compiled shape that takes the RHS count, pinned in turn."""
    g = S.random_gauge(L, n, seed=140)
    full = S.random_fermions(L, n, nrhs, seed=141, parities=2)
    parity, dagger, a = 1, 1, -0.0144
    want = a * O.dslash(np.ascontiguousarray(full[:, 0]), g, L, parity, dagger, True) + b * full[:, 1]
    ran = 0
    for R, minb, pk, st, rc, lt in qcu_lib.dslash_kernels(prec, n):
        if nrhs % R or st > 0 or lt or (st < 0 and st != -5) or (st == -5 and nrhs % 4):
            continue
        os.environ["QCU_DSLASH_CONFIG"] = "1,0,0,0,0,0,5" if st else "%d,64,%d,%d,0,0,0,%d,0" % (R, minb, pk, rc)
        try:
            got = _xpay(cuda, qcu_lib, full, g, L, prec, parity, dagger, a, b)
        finally:
            del os.environ["QCU_DSLASH_CONFIG"]
        assert rel(got, want) < TOL[prec], (R, minb, pk, st, rc)
        ran += 1
    assert ran


def test_packed_su5_is_the_scalar_kernel(cuda, qcu_lib):
    """SU(5) FP32: the packed kernels against the scalar ones of the same R, bit for bit."""
    L, nrhs = (4, 2, 4, 4), 6
    g = S.random_gauge(L, 5, seed=142)
    full = S.random_fermions(L, 5, nrhs, seed=143, parities=2)
    out = {}
    for R, minb, pk, st, rc, lt in qcu_lib.dslash_kernels(1, 5):
        if st or lt or rc or nrhs % R:
            continue
        os.environ["QCU_DSLASH_CONFIG"] = "%d,64,%d,%d,0" % (R, minb, pk)
        try:
            out[R, pk, minb] = _xpay(cuda, qcu_lib, full, g, L, 1, 0, 0, 1.0, 0.5)
        finally:
            del os.environ["QCU_DSLASH_CONFIG"]
    packed = [k for k in out if k[1]]
    assert packed
    for R, _, minb in packed:
        for k, other in out.items():
            if k[0] == R and not k[1]:
                assert np.array_equal(out[R, 1, minb], other)
