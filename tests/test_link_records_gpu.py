"""The link records that a 16-bit hop builds are those of the kernels that tuning can choose."""
import pytest

from mrhs_qcu_gb300 import synthetic as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", [4, 5])  # BF16, component- and site-major
def test_tuning_builds_one_form(cuda, qcu_lib, monkeypatch, prec):
    """SU(4) 16^3x32: records of 8 x 16 complex elements a site and parity (67 MB) for the register-fragment
    MMAs; the tcgen05 kernels' 2 KB (268 MB), which no tuned shape reads, are not built."""
    torch, Q = cuda, qcu_lib
    monkeypatch.delenv("QCU_DSLASH_CONFIG", raising=False)
    L, n, nrhs = (16, 16, 16, 32), 4, 4
    vh = S.half_volume(L)
    Q.initGridSize(L, n)
    gauge = torch.randn((4, 2, vh, n, n), dtype=torch.complex128, device="cuda")
    torch.cuda.synchronize()
    Q.loadQcuGauge(gauge.data_ptr())
    db, _ = Q.field_bytes(prec, nrhs)
    a, b = (torch.zeros(db, dtype=torch.uint8, device="cuda") for _ in range(2))
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    Q.dslash_mrhs(b.data_ptr(), None, a.data_ptr(), None, nrhs, 0, 0, prec)
    Q.synchronize()
    used = free - torch.cuda.mem_get_info()[0]
    links = 8 * n * n * vh * 4
    records = 2 * vh * 8 * n * n * 4
    assert used <= links + records + (64 << 20), used  # and what the driver takes for modules and events
    Q.initGridSize((4, 4, 4, 4), 3)
