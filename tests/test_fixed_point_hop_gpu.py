"""The FP64 hop, whose colour multiply runs in block fixed point: against extended
precision over block edges and RHS counts (links in shared memory or not), and where a site has to take
the FP64 multiply-adds instead (wide spans, subnormal and extreme scales, infinities, NaN)."""
import os
import numpy as np
import pytest
from mrhs_qcu_gb300 import synthetic as S
from oracle import oracle as O
from tests.util import abi_dslash, rel

pytestmark = pytest.mark.gpu


def _gamma(mu):
    g = np.zeros((4, 4), complex)
    for r in range(4):
        sign = {0: 1 if r < 2 else -1, 1: -1 if r in (0, 3) else 1, 2: 1 if r in (0, 3) else -1, 3: 1}[mu]
        g[r, 3 - r if mu < 2 else r ^ 2] = sign * (1j if mu in (0, 2) else 1)
    return g


def _extended(psi, gauge, L, parity, dagger):
    """The hop (antiperiodic in t) in numpy's long double."""
    lx, ly, lz, lt = L
    hx = lx // 2
    psi, gauge = psi.astype(np.clongdouble), gauge.astype(np.clongdouble)
    i = np.arange(psi.shape[1])
    y, z, t = i // hx % ly, i // (hx * ly) % lz, i // (hx * ly * lz)
    x = 2 * (i % hx) + ((y + z + t) & 1 ^ parity)
    out = np.zeros_like(psi)
    f = -1 if dagger else 1
    for mu in range(4):
        for s in (1, -1):
            c = [x, y, z, t]
            c[mu] = (c[mu] + s) % L[mu]
            nb = ((c[3] * lz + c[2]) * ly + c[1]) * hx + c[0] // 2
            u = gauge[mu, parity] if s > 0 else np.conj(np.swapaxes(gauge[mu, 1 - parity][nb], -1, -2))
            h = np.einsum("st,rvtc->rvsc", (np.eye(4) - s * f * _gamma(mu)).astype(np.clongdouble), psi[:, nb])
            h = np.einsum("vab,rvsb->rvsa", u, h)
            if mu == 3:
                h = h * np.where(t == (lt - 1 if s > 0 else 0), -1, 1)[None, :, None, None]
            out += h
    return out


@pytest.mark.parametrize("n", [3, 4])
@pytest.mark.parametrize("L,nrhs", [((4, 4, 4, 4), 1), ((6, 4, 2, 4), 3), ((4, 2, 6, 4), 4), ((10, 2, 2, 6), 5),
                                    ((4, 4, 4, 6), 12), ((4, 2, 2, 4), 64)])
def test_against_extended_precision(cuda, qcu_lib, n, L, nrhs):
    """Every block size: the error stays below that of FP64 multiply-adds.  Bound: the final rounding
    (2^-53 / sqrt(3) of a part, at most 0.7e-16 in L2) and the projection's (half of it) make about
    0.9e-16; 1.2e-16 leaves a third.  FP64 arithmetic has 1.45e-16 on such fields."""
    g = S.random_gauge(L, n, seed=31)
    psi = S.random_fermions(L, n, nrhs, seed=32)
    first = None
    for parity, dagger in ((0, 0), (1, 1)):
        want = _extended(psi, g, L, parity, dagger)
        for shape, block in enumerate((32, 64, 128, 256)):
            minb = (1, 2, 7, 1)[shape]
            os.environ["QCU_DSLASH_CONFIG"] = "1,%d,%d,0,0" % (block, minb)
            try:
                got = abi_dslash(cuda, qcu_lib, psi, g, L, parity, dagger, 2, antiperiodic_t=True)
            finally:
                del os.environ["QCU_DSLASH_CONFIG"]
            err = float(np.sqrt(np.sum(np.abs(got - want) ** 2) / np.sum(np.abs(want) ** 2)))
            assert err < 1.2e-16, (block, minb, err)
            first = got if shape == 0 else first
            assert np.array_equal(got, first)


@pytest.mark.parametrize("n", [5, 6, 7, 8])
@pytest.mark.parametrize("L,nrhs", [((2, 2, 2, 4), 1), ((6, 2, 2, 4), 5), ((4, 2, 4, 4), 16)])
def test_large_groups_against_extended_precision(cuda, qcu_lib, n, L, nrhs):
    """SU(5) to SU(8) (58-bit parts).  To the two roundings above come eight hops of a unit's rounding and
    of the left-out low x low products, 1.3 units of a sum of 2^53.7 at SU(8): 0.85e-16; together 1.2e-16.
    1.5e-16 is also less than FP64 multiply-adds have."""
    g = S.random_gauge(L, n, seed=37)
    psi = S.random_fermions(L, n, nrhs, seed=38)
    first = None
    for block, minb in ((32, 1), (128, 2), (256, 1)):
        want = _extended(psi, g, L, 1, 0)
        os.environ["QCU_DSLASH_CONFIG"] = "1,%d,%d,0,0" % (block, minb)
        try:
            got = abi_dslash(cuda, qcu_lib, psi, g, L, 1, 0, 2, antiperiodic_t=True)
        finally:
            del os.environ["QCU_DSLASH_CONFIG"]
        err = float(np.sqrt(np.sum(np.abs(got - want) ** 2) / np.sum(np.abs(want) ** 2)))
        assert err < 1.5e-16, (block, minb, err)
        first = got if first is None else first
        assert np.array_equal(got, first)


@pytest.mark.parametrize("n", [3, 4, 6, 8])
def test_exact_on_unit_links(cuda, qcu_lib, n):
    """Unit links and small integers: nothing is rounded."""
    L, nrhs = (4, 4, 4, 4), 5
    g = np.zeros((4, 2, 128, n, n), complex)
    g[..., range(n), range(n)] = 1
    rng = np.random.default_rng(3)
    psi = (rng.integers(-99, 99, (nrhs, 128, 4, n)) + 1j * rng.integers(-99, 99, (nrhs, 128, 4, n))).astype(complex)
    psi[rng.random(psi.shape) < 0.4] = 0
    psi[1, 5:] = 0
    psi[2] = 0
    for d in (0, 1):
        got = abi_dslash(cuda, qcu_lib, psi, g, L, d, d, 2)
        assert np.array_equal(got, O.dslash(psi, g, L, d, d))


@pytest.mark.parametrize("n", [3, 4, 7])
@pytest.mark.parametrize("case", ["wide", "sites", "tiny", "huge", "subnormal", "scaled links", "mixed links"])
def test_scales(cuda, qcu_lib, n, case):
    """Scales that leave the fixed-point range: relative to each site's norm the result is the oracle's
    to 16 times the rounding of double (sums of 2 * 8 N products)."""
    L, nrhs = (4, 4, 4, 6), 5
    rng = np.random.default_rng(7)
    g = S.random_gauge(L, n, seed=33)
    psi = S.random_fermions(L, n, nrhs, seed=34)
    tol = 16 * 2.0 ** -52
    if case == "wide":      # parts of one spinor over 2^-60 .. 1
        psi = psi * 2.0 ** rng.integers(-60, 1, psi.shape)
    elif case == "sites":   # neighbours over 2^-400 .. 2^400
        psi = psi * 2.0 ** rng.integers(-400, 401, psi.shape[:2])[..., None, None]
    elif case == "tiny":
        psi = psi * 1e-290
    elif case == "huge":
        psi = psi * 1e305
    elif case == "subnormal":
        psi = psi * 2.0 ** -1040
    elif case == "scaled links":
        g = g * 3e40
    else:                   # links over 2^-300 .. 2^300
        g = g * 2.0 ** rng.integers(-300, 301, g.shape[:3])[..., None, None]
    got = abi_dslash(cuda, qcu_lib, psi, g, L, 1, 0, 2)
    want = O.dslash(psi, g, L, 1, 0)
    scale = np.max(np.abs(want.view(float)), axis=(2, 3), keepdims=True)
    floor = 64 * 2.0 ** -1074 if case == "subnormal" else 0.0
    assert np.all(np.abs((got - want).view(float)) <= tol * scale * n + floor)


@pytest.mark.parametrize("bad", [np.inf, -np.inf, np.nan])
def test_not_finite(cuda, qcu_lib, bad):
    """An infinity or NaN in one part reaches the oracle's outputs and no other site's bits."""
    L, nrhs = (4, 4, 4, 4), 4
    g = S.random_gauge(L, 3, seed=35)
    psi = S.random_fermions(L, 3, nrhs, seed=36)
    clean = abi_dslash(cuda, qcu_lib, psi, g, L, 0, 0, 2)
    psi[2, 17, 3, 1] = complex(bad, 0.5)
    got = abi_dslash(cuda, qcu_lib, psi, g, L, 0, 0, 2)
    hit = ~np.isfinite(O.dslash(psi, g, L, 0, 0)).all(axis=(2, 3))
    assert np.array_equal(~np.isfinite(got).all(axis=(2, 3)), hit) and 0 < hit.sum() <= 8
    assert np.array_equal(got[~hit], clean[~hit])


@pytest.mark.parametrize("n,L,nrhs", [(3, (4, 4, 4, 4), 1), (3, (6, 4, 2, 4), 5), (3, (4, 2, 2, 6), 12), (4, (6, 2, 2, 4), 3),
                                      (4, (4, 4, 4, 4), 8)])
def test_eight_threads_a_site(cuda, qcu_lib, n, L, nrhs):
    """The split form is the other form bit for bit: every block size, sites that take FP64 among them, a
    partial last block."""
    g = S.random_gauge(L, n, seed=41)
    psi = S.random_fermions(L, n, nrhs, seed=42)
    psi[0, 1] *= 2.0 ** -45      # its neighbours span too much
    psi[nrhs - 1, 4, 2, 1] = np.inf
    psi[0, 6] = 0
    for parity, dagger in ((0, 0), (1, 1)):
        out = {}
        for pk, minb in ((0, 1), (1, 2), (1, 7)):
            for block in (32, 64, 128, 256):
                os.environ["QCU_DSLASH_CONFIG"] = "1,%d,%d,%d,0" % (block, minb, pk)
                try:
                    out[pk, minb, block] = abi_dslash(cuda, qcu_lib, psi, g, L, parity, dagger, 2, antiperiodic_t=True)
                    assert qcu_lib.last_dslash_shape()[2] == pk
                finally:
                    del os.environ["QCU_DSLASH_CONFIG"]
        base = out[0, 1, 32]
        want = O.dslash(psi, g, L, parity, dagger, True)
        ok = np.isfinite(want).all(axis=(2, 3))
        assert rel(base[ok], want[ok]) < 1e-15
        for got in out.values():
            assert np.array_equal(got, base, equal_nan=True)
