"""FP32 norms and inner products of fields whose products are exact in FP32: only the summation rounds, and it
rounds as FP64 sums of the products do.  One thread's elements are not zero, so that errors do not average out."""
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _sums(torch, Q, u, v):
    x, y = (torch.from_numpy(a).cuda() for a in (u, v))
    norm = torch.zeros(1, dtype=torch.float64, device="cuda")
    dot = torch.zeros(1, dtype=torch.complex128, device="cuda")
    Q.blas_mrhs(Q.BLAS_NORM2_FP32, len(u), 1, x.data_ptr(), 1, out=norm.data_ptr())
    Q.blas_mrhs(Q.BLAS_CDOT, len(u), 1, x.data_ptr(), 1, y.data_ptr(), 1, out=dot.data_ptr())
    Q.synchronize()
    return norm.item(), dot.item().real


@pytest.mark.parametrize("count", [3, 4, 5, 8, 12, 15, 16, 17, 21, 26, 28, 33])
def test_summation(cuda, qcu_lib, count):
    """`count` elements of one thread (the grid is one wave of 1024 threads an SM): 12 significant bits, over 26
    binades.  At most count / 4 groups, as many additions of errors for every fourth, two at the end: count
    / 4 * 1.25 + 3 roundings of double, relative to the sum of the magnitudes."""
    torch, Q = cuda, qcu_lib
    Q.initGridSize((4, 4, 4, 4), 3)
    wave = 1024 * torch.cuda.get_device_properties(0).multi_processor_count
    tol = (math.ceil(count / 4) * 1.25 + 3) * 2.0 ** -53
    for seed in range(12):
        rng = np.random.default_rng(1000 * count + seed)

        def value():
            return (rng.integers(2048, 4096, count) * rng.choice([-1, 1], count) * 2.0 ** rng.integers(-26, 1, count))

        u, v = (np.zeros(wave * count, np.complex64) for _ in range(2))
        a, b = value(), value()
        u[::wave], v[::wave] = a, b
        norm, dot = _sums(torch, Q, u, v)
        assert abs(norm - math.fsum(a * a)) <= tol * math.fsum(a * a)
        assert abs(dot - math.fsum(a * b)) <= tol * math.fsum(abs(a * b))
