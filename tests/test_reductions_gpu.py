"""FP32 norms and inner products, whose products are added in groups of four: group and wave edges, RHS
counts whose blocks are odd multiples of a warp, sums beyond FP32's range, infinities and NaN."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _field(torch, h):
    h = np.ascontiguousarray(h, dtype=np.complex64)
    return torch.from_numpy(h).cuda()


def _norm(torch, Q, h):
    k, nrhs = h.shape
    x = _field(torch, h)
    out = torch.zeros(nrhs, dtype=torch.float64, device="cuda")
    Q.blas_mrhs(Q.BLAS_NORM2_FP32, k * nrhs, nrhs, x.data_ptr(), 1, out=out.data_ptr())
    Q.synchronize()
    return out.cpu().numpy()


def _dot(torch, Q, u, v):
    k, nrhs = u.shape
    x, y = _field(torch, u), _field(torch, v)
    out = torch.zeros(nrhs, dtype=torch.complex128, device="cuda")
    Q.blas_mrhs(Q.BLAS_CDOT, k * nrhs, nrhs, x.data_ptr(), 1, y.data_ptr(), 1, out=out.data_ptr())
    Q.synchronize()
    return out.cpu().numpy()


@pytest.mark.parametrize("nrhs,k", [(1, 1), (1, 5), (2, 31), (3, 1021), (7, 97), (31, 33), (62, 65), (256, 9),
                                    (12, 60001), (1, 700001)])
def test_sums(cuda, qcu_lib, nrhs, k):
    """A product is rounded twice in FP32 (2^-23 of |u| |v| at most); the sums add nothing that counts."""
    qcu_lib.initGridSize((4, 4, 4, 4), 3)
    rng = np.random.default_rng(k + nrhs)
    u, v = ((rng.standard_normal((k, nrhs)) + 1j * rng.standard_normal((k, nrhs))).astype(np.complex64)
            for _ in range(2))
    ud, vd = u.astype(complex), v.astype(complex)
    want = np.sum(np.abs(ud) ** 2, axis=0)
    assert np.all(np.abs(_norm(cuda, qcu_lib, u) - want) <= 2.0 ** -23 * want)
    size = np.sum(np.abs(ud) * np.abs(vd), axis=0)
    err = _dot(cuda, qcu_lib, u, v) - np.sum(ud.conj() * vd, axis=0)
    assert np.all(np.abs(err.real) <= 2.0 ** -22 * size) and np.all(np.abs(err.imag) <= 2.0 ** -22 * size)


@pytest.mark.parametrize("nrhs", [1, 12])
def test_beyond_fp32_range(cuda, qcu_lib, nrhs):
    """Products of 1.44e38: four of them leave FP32's range, the FP64 sum does not."""
    qcu_lib.initGridSize((4, 4, 4, 4), 3)
    u = np.full((1003, nrhs), 1.2e19, np.complex64)
    v = u.copy()
    v[::2] *= -1
    one = float(np.float32(np.float32(1.2e19) ** 2))
    np.testing.assert_allclose(_norm(cuda, qcu_lib, u), 1003 * one, rtol=1e-12)
    np.testing.assert_allclose(_dot(cuda, qcu_lib, u, v).real, -one, rtol=1e-9)


@pytest.mark.parametrize("bad", [np.inf, np.nan])
def test_not_finite(cuda, qcu_lib, bad):
    """One element of one RHS: that RHS's sums are not finite, the others are untouched."""
    qcu_lib.initGridSize((4, 4, 4, 4), 3)
    rng = np.random.default_rng(5)
    u = rng.standard_normal((501, 6)).astype(np.complex64)
    clean_n, clean_d = _norm(cuda, qcu_lib, u), _dot(cuda, qcu_lib, u, u)
    u[77, 4] = bad
    n, d = _norm(cuda, qcu_lib, u), _dot(cuda, qcu_lib, u, u)
    keep = np.arange(6) != 4
    assert not np.isfinite(n[4]) and not np.isfinite(d[4].real)
    assert np.array_equal(n[keep], clean_n[keep]) and np.array_equal(d[keep], clean_d[keep])
