"""The FP64 hop part by part: every real part of the result, however small beside its site's largest, is as
good as that of FP64 multiply-adds, whatever the spread of the links' and the spinors' parts; and the two
forms of the kernel agree to the bit."""
import os

import numpy as np
import pytest

from mrhs_qcu_gb300 import synthetic as S
from tests.test_fixed_point_hop_gpu import _extended, _gamma
from tests.util import abi_dslash

pytestmark = pytest.mark.gpu
L = (4, 4, 2, 6)


def _magnitude(psi, gauge, parity, dagger):
    """The sum of the magnitudes of the real products that make up each real part of the hop."""
    lx, ly, lz, lt = L
    hx, psi, gauge = lx // 2, psi.astype(np.clongdouble), gauge.astype(np.clongdouble)
    i = np.arange(psi.shape[1])
    y, z, t = i // hx % ly, i // (hx * ly) % lz, i // (hx * ly * lz)
    x = 2 * (i % hx) + ((y + z + t) & 1 ^ parity)
    re, im = np.zeros(psi.shape, np.longdouble), np.zeros(psi.shape, np.longdouble)
    f = -1 if dagger else 1
    for mu in range(4):
        for s in (1, -1):
            c = [x, y, z, t]
            c[mu] = (c[mu] + s) % L[mu]
            nb = ((c[3] * lz + c[2]) * ly + c[1]) * hx + c[0] // 2
            u = gauge[mu, parity] if s > 0 else np.swapaxes(gauge[mu, 1 - parity][nb], -1, -2)
            h = np.einsum("st,rvtc->rvsc", (np.eye(4) - s * f * _gamma(mu)).astype(np.clongdouble), psi[:, nb])
            h = h.astype(complex)  # the projected spinor is rounded to double
            sum_ = lambda a, b: np.einsum("vab,rvsb->rvsa", np.abs(a), np.abs(b).astype(np.longdouble))  # noqa: E731
            # the lower rows are the upper ones times +-1 or +-i, so the same products as here
            re += sum_(u.real, h.real) + sum_(u.imag, h.imag)
            im += sum_(u.real, h.imag) + sum_(u.imag, h.real)
    return re, im


def _links(kind, n, rng):
    g = S.random_gauge(L, n, seed=51)
    if kind.startswith("near"):  # exp of a small anti-Hermitian matrix, to first order; the rest is far below
        a = 10.0 ** -int(kind[4:]) * (rng.standard_normal(g.shape) + 1j * rng.standard_normal(g.shape))
        g = np.eye(n) + a - np.conj(np.swapaxes(a, -1, -2))
    elif kind == "unit":
        g = np.broadcast_to(np.eye(n, dtype=complex), g.shape).copy()
    elif kind == "wide":
        g = g * 2.0 ** rng.integers(-50, 1, g.shape)
    return g


def _spinors(kind, n, nrhs):
    psi = S.random_fermions(L, n, nrhs, seed=52)
    rng = np.random.default_rng(53)
    if kind == "colour":
        psi[..., 1:] = 0
    elif kind == "spin":
        psi[:, :, 1:] = 0
    elif kind == "point":
        for r in range(nrhs):
            keep = psi[r, 5 + r, r % 4, r % n]
            psi[r] = 0
            psi[r, 5 + r, r % 4, r % n] = keep
    elif kind == "falling":
        psi = psi * 2.0 ** (-9.0 * np.arange(n))
    elif kind == "wide":
        psi = psi * 2.0 ** rng.integers(-60, 1, psi.shape)
    elif kind == "real":
        psi = psi.real.astype(complex)
    return psi


def _both_forms(cuda, qcu_lib, psi, g, n, parity, dagger):
    out = []
    for cfg in ("1,64,1,0,0", "1,128,7,1,0") if n <= 4 else ("1,64,1,0,0", "1,128,2,0,0"):
        os.environ["QCU_DSLASH_CONFIG"] = cfg
        try:
            out.append(abi_dslash(cuda, qcu_lib, psi, g, L, parity, dagger, 2))
        finally:
            del os.environ["QCU_DSLASH_CONFIG"]
    assert np.array_equal(out[0], out[1])
    return out[0]


@pytest.mark.parametrize("n", [3, 4, 6, 8])
@pytest.mark.parametrize("links", ["haar", "near1", "near3", "near9", "unit", "wide"])
@pytest.mark.parametrize("spinors", ["full", "colour", "spin", "point", "falling", "wide", "real"])
def test_every_part(cuda, qcu_lib, n, links, spinors):
    """Bound: a real part is a chain of 2 n multiply-adds in each of eight hops, which are added up, after a
    rounded projection: 2 n + 9 roundings of at most the sum of the products' magnitudes."""
    rng = np.random.default_rng(50)
    g, psi = _links(links, n, rng), _spinors(spinors, n, 5)
    for parity, dagger in ((0, 0), (1, 1)):
        got = _both_forms(cuda, qcu_lib, psi, g, n, parity, dagger)
        want = _extended_periodic(psi, g, parity, dagger)
        re, im = _magnitude(psi, g, parity, dagger)
        tol = (2 * n + 9) * 2.0 ** -53
        assert np.all(np.abs(got.real - want.real) <= tol * re)
        assert np.all(np.abs(got.imag - want.imag) <= tol * im)


def _extended_periodic(psi, g, parity, dagger):
    """_extended has an antiperiodic t: the boundary links negated make it periodic.  Its projected spinor is
    not rounded to double; that is one of the bound's roundings."""
    lx, ly, lz, lt = L
    g = g.copy()
    g[3, :, (lt - 1) * lx // 2 * ly * lz:] *= -1
    return _extended(psi, g, L, parity, dagger)


@pytest.mark.parametrize("n", [3, 4, 5, 8])
@pytest.mark.parametrize("scale", [-1020, -1000, -966, -960, -940])
def test_zeros_in_tiny_spinors(cuda, qcu_lib, n, scale):
    """Zeros beside parts near the bottom of the exponent range, multiplied by large links."""
    rng = np.random.default_rng(54)
    g = S.random_gauge(L, n, seed=55) * 2.0 ** 80
    psi = S.random_fermions(L, n, 5, seed=56) * 2.0 ** scale
    psi.real[rng.random(psi.shape) < 0.5] = 0
    psi.imag[rng.random(psi.shape) < 0.5] = 0
    got = _both_forms(cuda, qcu_lib, psi, g, n, 1, 0)
    want = _extended_periodic(psi, g, 1, 0)
    # 2 n + 9 roundings of double, and those of the projection to a subnormal
    tol = (2 * n + 9) * 2.0 ** -53 + 2.0 ** (-1074 - scale)
    size = np.max(np.abs(want), axis=(2, 3), keepdims=True)
    assert np.all(np.abs(got - want) <= 8 * n * tol * size)


@pytest.mark.parametrize("n", [3, 4, 5, 6, 7, 8])
@pytest.mark.parametrize("top", [2.0 ** -53, 2.0 ** -29, 2.0 ** -28, 3 * 2.0 ** -30])
def test_largest_sums(cuda, qcu_lib, n, top):
    """Every part at the top of its binade and every product of one sign: the integer sums at their bounds.
    Spin 0 and 1 alone are not zero, so the projected rows are these parts themselves."""
    c = 1.0 - top
    g = np.full((4, 2, L[0] * L[1] * L[2] * L[3] // 2, n, n), complex(c, -c))
    g[:, 1] = np.conj(g[:, 1])  # the backward links, conjugated, agree with the forward ones at parity 0
    for sign in (1, -1):
        psi = np.zeros((2, g.shape[2], 4, n), complex)
        psi[:, :, :2] = sign * complex(c, c)
        got = _both_forms(cuda, qcu_lib, psi, g, n, 0, 0)
        want = _extended_periodic(psi, g, 0, 0)
        re, im = _magnitude(psi, g, 0, 0)
        tol = (2 * n + 9) * 2.0 ** -53
        assert np.all(np.abs(got.real - want.real) <= tol * re)
        assert np.all(np.abs(got.imag - want.imag) <= tol * im)
