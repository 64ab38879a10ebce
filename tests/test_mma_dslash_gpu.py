"""Register-fragment MMA dslash (tensor-core variant 5; FP16 and BF16 fields):
against the FP64 oracle, across layouts, and the independence of the RHS."""
import os

import numpy as np
import pytest

from mrhs_qcu_gb300 import synthetic as S
from oracle import oracle as O

from tests.util import TOL, abi_dslash, dev, rel

pytestmark = pytest.mark.gpu
HALF, BF16, SITE = 0, 4, 5


@pytest.fixture
def pinned():
    os.environ["QCU_DSLASH_CONFIG"] = "1,0,0,0,0,0,5"
    yield
    del os.environ["QCU_DSLASH_CONFIG"]


# RHS counts that fill the 16- and 32-RHS tiles, leave them partly empty, end inside a second
# tile or take a short last chunk (rows of whole sectors or not); half volumes that are not a
# multiple of the sites per warp or per CTA
@pytest.mark.parametrize("n,nrhs,L", [(3, 4, (4, 4, 4, 4)), (3, 12, (6, 4, 2, 6)), (3, 16, (2, 2, 2, 2)),
                                      (3, 36, (4, 4, 4, 4)), (4, 8, (2, 6, 2, 2)), (4, 64, (4, 4, 2, 4)),
                                      (5, 12, (6, 2, 2, 2)), (5, 20, (4, 4, 2, 4)), (6, 16, (6, 4, 2, 2)),
                                      (6, 48, (4, 2, 4, 4)), (7, 4, (2, 2, 2, 2)), (7, 16, (4, 4, 2, 4)),
                                      (7, 40, (4, 2, 2, 4)), (8, 12, (4, 4, 2, 2)), (8, 64, (4, 2, 4, 4))])
def test_against_oracle(cuda, qcu_lib, pinned, n, nrhs, L):
    """Both parities and dagger flags, antiperiodic t, every storage form; the two BF16 layouts agree bit for bit."""
    Q = qcu_lib
    g = S.random_gauge(L, n, seed=700 + n)
    psi = S.random_fermions(L, n, nrhs, seed=701)
    for parity, dag in ((0, 0), (1, 1), (1, 0)):
        ref = O.dslash(psi, g, L, parity, dag, True)
        got = {}
        for prec in (HALF, BF16, SITE):
            got[prec] = abi_dslash(cuda, Q, psi, g, L, parity, dag, prec, antiperiodic_t=True)
            assert Q.last_dslash_shape()[3] == -5
            assert rel(got[prec], ref) < TOL[prec], (prec, parity, dag)
        assert np.array_equal(got[BF16], got[SITE])


@pytest.mark.parametrize("prec", [HALF, BF16])
@pytest.mark.parametrize("n,nrhs", [(3, 12), (4, 20), (6, 16), (8, 24)])
def test_xpay(cuda, qcu_lib, pinned, prec, n, nrhs):
    """out = a D in + b x on resident fields (FP16: with the scales of x)."""
    torch, Q = cuda, qcu_lib
    L, a, b = (4, 4, 4, 4), -0.0144, 1.25
    g = S.random_gauge(L, n, seed=710)
    full = S.random_fermions(L, n, nrhs, seed=711, parities=2)
    Q.initGridSize(L, n)
    Q.set_antiperiodic_t(True)
    dg = dev(torch, g)
    Q.loadQcuGauge(dg.data_ptr())
    db, nb = Q.field_bytes(prec, nrhs)
    f = [torch.empty(db, dtype=torch.uint8, device="cuda") for _ in range(3)]
    s = [torch.empty(max(nb, 16), dtype=torch.uint8, device="cuda") for _ in range(3)]
    src = [dev(torch, full[r]) for r in range(nrhs)]
    for p in (0, 1):
        Q.pack_fermions(f[p].data_ptr(), s[p].data_ptr(), [x.data_ptr() for x in src], Q.QCU_SRC_EO_FULL, p, prec)
    Q.dslash_xpay_mrhs(f[2].data_ptr(), s[2].data_ptr(), f[0].data_ptr(), s[0].data_ptr(), f[1].data_ptr(),
                       s[1].data_ptr(), nrhs, 1, 1, prec, a, b)
    assert Q.last_dslash_shape()[3] == -5
    out = [torch.zeros((S.half_volume(L), 4, n), dtype=torch.complex128, device="cuda") for _ in range(nrhs)]
    Q.unpack_fermions([o.data_ptr() for o in out], f[2].data_ptr(), s[2].data_ptr(), Q.QCU_SRC_EO_HALF, 1, prec)
    Q.synchronize()
    want = a * O.dslash(full[:, 0], g, L, 1, 1, True) + b * full[:, 1]
    assert rel(np.stack([o.cpu().numpy() for o in out]), want) < TOL[prec]


@pytest.mark.parametrize("n,nrhs", [(3, 12), (6, 20)])
def test_non_finite_rhs_stays_alone(cuda, qcu_lib, pinned, n, nrhs):
    """An infinite component in one RHS leaves every other RHS bit-identical."""
    torch, Q = cuda, qcu_lib
    L, bad = (4, 4, 4, 4), 5
    g = S.random_gauge(L, n, seed=720)
    psi = S.random_fermions(L, n, nrhs, seed=721)
    clean = abi_dslash(torch, Q, psi, g, L, 0, 0, BF16, antiperiodic_t=True)
    psi[bad, 3, 1, n - 1] = np.inf
    got = abi_dslash(torch, Q, psi, g, L, 0, 0, BF16, antiperiodic_t=True)
    others = [r for r in range(nrhs) if r != bad]
    assert np.array_equal(got[others], clean[others])
    assert not np.isfinite(got[bad]).all()


@pytest.mark.parametrize("inner", [HALF, BF16])
def test_masked_solve(cuda, qcu_lib, pinned, inner):
    """The kernel as the inner hop of a masked CG (RHS converge at different
    iterations, one source is zero): the oracle's FP64 true residual."""
    torch, Q = cuda, qcu_lib
    L, n, nr, kappa, tol = (4, 4, 4, 8), 3, 12, 0.11, 1e-8
    g = S.random_gauge(L, n, seed=730)
    b = S.random_fermions(L, n, nr, seed=731, parities=2)
    b[1] *= 1e-4
    b[2] = 0
    Q.initGridSize(L, n)
    Q.set_antiperiodic_t(True)
    dg = dev(torch, g)
    Q.loadQcuGauge(dg.data_ptr())
    db = [dev(torch, b[r]) for r in range(nr)]
    dx = [torch.zeros_like(x) for x in db]
    p = Q.solver_params(kappa=kappa, tol=tol, inner_precision=inner, max_iter=5000)
    Q.invert([x.data_ptr() for x in dx], [x.data_ptr() for x in db], p)
    assert float(dx[2].abs().max()) == 0.0
    for r in range(nr):
        assert p.converged[r], r
        if r != 2:
            assert O.true_residual(dx[r].cpu().numpy(), b[r], g, L, kappa, antiperiodic_t=True) < 2 * tol, r
