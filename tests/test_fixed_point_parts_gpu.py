"""The FP64 hop on fields whose parts lie far apart; the two forms of the kernel agree to the bit."""
import os

import numpy as np
import pytest

from mrhs_qcu_gb300 import synthetic as S
from tests.test_fixed_point_hop_gpu import _extended
from tests.util import abi_dslash

pytestmark = pytest.mark.gpu
L = (4, 4, 2, 6)


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
