"""Tiled layout transforms: caller fields <-> resident MRHS fields against
numpy, at the edges of the tiles, with untouched (null) RHS, and the
conversions at the ends of the number ranges."""
import numpy as np
import pytest

from mrhs_qcu_gb300 import synthetic as S

pytestmark = pytest.mark.gpu
HALF, SINGLE, DOUBLE, BF16, SITE = 0, 1, 2, 4, 5


def _lex_sites(L, parity):
    """Lexicographic index of every half-site of one parity."""
    x, y, z, t = L
    s = np.arange(x * y * z * t // 2)
    xh, s = s % (x // 2), s // (x // 2)
    yy, s = s % y, s // y
    zz, tt = s % z, s // z
    return ((tt * z + zz) * y + yy) * x + 2 * xh + ((parity + yy + zz + tt) & 1)


def _session(Q, torch, L, n):
    Q.initGridSize(L, n)


def _round_bf16(v):
    """FP64 -> BF16 -> FP64, one rounding to nearest even (normal range)."""
    m, e = np.frexp(v)
    return np.ldexp(np.rint(np.ldexp(m, 8)), e - 8)


# RHS counts: one, odd, exactly one tile of RHS, a second chunk of one RHS; half volumes that leave a
# partial tile of sites, or are smaller than one
@pytest.mark.parametrize("n,nrhs,L", [(3, 1, (6, 4, 2, 6)), (3, 5, (4, 4, 4, 4)), (3, 12, (6, 2, 4, 2)),
                                      (4, 33, (4, 2, 4, 2)), (8, 32, (2, 2, 2, 2)), (8, 64, (4, 4, 2, 2))])
@pytest.mark.parametrize("mode", [0, 1, 2])
def test_pack_unpack(cuda, qcu_lib, n, nrhs, L, mode):
    torch, Q = cuda, qcu_lib
    _session(Q, torch, L, n)
    vh, nc, parity = S.half_volume(L), 4 * n, 1
    rng = np.random.default_rng(800 + nrhs)
    sites = {0: vh, 1: 2 * vh, 2: 2 * vh}[mode]
    src = rng.standard_normal((nrhs, sites, nc)) + 1j * rng.standard_normal((nrhs, sites, nc))
    index = {0: np.arange(vh), 1: vh + np.arange(vh), 2: _lex_sites(L, parity)}[mode]
    want = src[:, index]  # [nrhs][vh][nc]
    dsrc = [torch.from_numpy(src[r].copy()).cuda() for r in range(nrhs)]
    skip = nrhs // 2 if nrhs > 1 else -1  # this RHS is a null pointer: neither read nor written
    for prec, real in ((DOUBLE, np.float64), (SINGLE, np.float32), (HALF, np.float16), (BF16, None), (SITE, None)):
        if prec == SITE and nrhs % 4:
            continue
        db, nb = Q.field_bytes(prec, nrhs)
        field = torch.full((db,), 17, dtype=torch.uint8, device="cuda")
        norm = torch.full((max(nb, 4),), 17, dtype=torch.uint8, device="cuda")
        ptr = [0 if r == skip else d.data_ptr() for r, d in enumerate(dsrc)]
        Q.pack_fermions(field.data_ptr(), norm.data_ptr(), ptr, mode, parity, prec)
        out = [torch.full((sites, nc), 3.0 + 0j, dtype=torch.complex128, device="cuda") for _ in range(nrhs)]
        Q.unpack_fermions([0 if r == skip else o.data_ptr() for r, o in enumerate(out)], field.data_ptr(),
                          norm.data_ptr(), mode, parity, prec)
        Q.synchronize()
        got = np.stack([o.cpu().numpy() for o in out])
        keep = [r for r in range(nrhs) if r != skip]
        shape = (vh, nc, nrhs) if prec == SITE else (nc, vh, nrhs)
        order = (2, 0, 1) if prec == SITE else (2, 1, 0)
        back = got[:, index]
        untouched = np.setdiff1d(np.arange(sites), index)
        assert (got[:, untouched] == 3.0).all()
        if skip >= 0:
            assert (got[skip] == 3.0).all()
        if prec in (DOUBLE, SINGLE):
            raw = field.cpu().numpy().view(real).reshape(*shape, 2)
            comp = (raw[..., 0] + 1j * raw[..., 1].astype(np.float64)).transpose(order)
            ref = want.real.astype(real).astype(np.float64) + 1j * want.imag.astype(real).astype(np.float64)
            assert np.array_equal(comp[keep], ref[keep])
            assert np.array_equal(back[keep], ref[keep])
            if skip >= 0:
                assert (field.cpu().numpy().reshape(*shape, -1)[..., skip, :] == 17).all()
        elif prec in (BF16, SITE):
            ref = _round_bf16(want.real) + 1j * _round_bf16(want.imag)
            assert np.array_equal(back[keep], ref[keep])
        else:  # FP16 with the site's scale: half an ulp of 2^-11 of the largest component
            big = np.abs(want.view(np.float64).reshape(nrhs, vh, -1)).max(-1, keepdims=True)
            err = np.maximum(np.abs(back.real - want.real), np.abs(back.imag - want.imag))
            assert (err[keep] <= 2.0 ** -11 * 1.001 * big[keep]).all()


def test_conversions_at_the_ends_of_the_ranges(cuda, qcu_lib):
    """FP64 -> FP32 bit for bit as IEEE rounding to nearest even: halfway cases, the denormal range, overflow, zeros,
    infinities and NaN; FP32 -> FP64 exact."""
    torch, Q = cuda, qcu_lib
    L, n = (4, 2, 2, 2), 3
    _session(Q, torch, L, n)
    vh, nc = S.half_volume(L), 4 * n
    tiny, big = float(np.finfo(np.float32).tiny), float(np.finfo(np.float32).max)
    special = [0.0, -0.0, np.inf, -np.inf, np.nan, 1.0, -1.0, 1 + 2.0 ** -24, 1 + 3 * 2.0 ** -24, 1 + 2.0 ** -24 + 2.0 ** -50,
               2 - 2.0 ** -25, tiny, tiny * (1 - 2.0 ** -25), tiny / 2, 2.0 ** -149, 2.0 ** -150, 2.0 ** -151, 5e-324,
               big, big * (1 + 2.0 ** -26), big * (1 + 2.0 ** -25), big * (1 + 2.0 ** -24), 1e300, -1e300, -tiny / 3]
    rng = np.random.default_rng(810)
    v = rng.standard_normal(2 * vh * nc) * 10.0 ** rng.uniform(-46, 39, 2 * vh * nc)
    v[:len(special)] = special
    src = torch.from_numpy(v.view(np.complex128).reshape(vh, nc).copy()).cuda()
    field = torch.zeros((nc, vh, 2), dtype=torch.float32, device="cuda")
    Q.pack_fermions(field.data_ptr(), None, [src.data_ptr()], Q.QCU_SRC_EO_HALF, 0, SINGLE)
    back = torch.zeros_like(src)
    Q.unpack_fermions([back.data_ptr()], field.data_ptr(), None, Q.QCU_SRC_EO_HALF, 0, SINGLE)
    Q.synchronize()
    with np.errstate(over="ignore", under="ignore"):
        want = v.reshape(vh, nc, 2).astype(np.float32)
    got = field.cpu().numpy().transpose(1, 0, 2)
    assert np.array_equal(got, want, equal_nan=True)
    assert np.array_equal(np.signbit(got), np.signbit(want))
    assert np.array_equal(back.cpu().numpy().view(np.float64).reshape(vh, nc, 2), want.astype(np.float64), equal_nan=True)
