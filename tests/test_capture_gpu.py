"""A hop captured into a CUDA graph on a session whose earlier hops took another kernel shape: it allocates and
builds nothing while the stream is captured, and replays to the oracle's result."""
import os

import numpy as np
import pytest

from mrhs_qcu_gb300 import synthetic as S
from oracle import oracle as O
from tests.util import TOL, dev, rel

pytestmark = pytest.mark.gpu
FP32, HALF, BF16, SITE = 1, 0, 4, 5


@pytest.mark.parametrize("prec,n,nrhs,before,captured", [
    (FP32, 3, 12, "2,64,2,0,0,0,0,0", "2,64,2,0,0,0,0,1"),  # full links, then two-row ones
    (BF16, 3, 12, "2,64,2,0,0,0,0,0", "2,64,2,0,0,0,0,1"),
    (HALF, 4, 16, "1,64,1,0,0,0,0,0", "1,0,0,0,0,0,5"),     # the register kernel, then register-fragment MMAs
    (BF16, 6, 16, "1,64,1,0,0,0,0,0", "1,0,0,0,0,0,5"),
    (BF16, 6, 16, "1,0,0,0,0,0,5", "1,0,0,0,0,0,4"),        # the two forms of link records
    (SITE, 4, 16, "1,0,0,0,0,0,5", "1,0,0,0,0,0,4"),
    (SITE, 4, 16, "1,0,0,0,0,0,4", "1,0,0,0,0,0,5"),
])
def test_other_shape_than_the_hops_before(cuda, qcu_lib, monkeypatch, prec, n, nrhs, before, captured):
    torch, Q = cuda, qcu_lib
    L = (4, 4, 4, 8)
    g, psi = S.random_gauge(L, n, seed=901), S.random_fermions(L, n, nrhs, seed=902)
    Q.initGridSize(L, n)
    Q.set_antiperiodic_t(True)
    dg, src = dev(torch, g), [dev(torch, p) for p in psi]
    Q.loadQcuGauge(dg.data_ptr())
    db, nb = Q.field_bytes(prec, nrhs)
    fin, out = (torch.zeros(db, dtype=torch.uint8, device="cuda") for _ in range(2))
    nin, nout = (torch.zeros(max(nb, 16), dtype=torch.uint8, device="cuda") for _ in range(2))
    Q.pack_fermions(fin.data_ptr(), nin.data_ptr(), [s.data_ptr() for s in src], Q.QCU_SRC_EO_HALF, 1, prec)

    def hop():
        Q.dslash_mrhs(out.data_ptr(), nout.data_ptr(), fin.data_ptr(), nin.data_ptr(), nrhs, 0, 0, prec)

    monkeypatch.setenv("QCU_DSLASH_CONFIG", before)
    hop()
    Q.synchronize()
    torch.cuda.synchronize()
    stream, graph = torch.cuda.Stream(), torch.cuda.CUDAGraph()
    monkeypatch.setenv("QCU_DSLASH_CONFIG", captured)
    Q.set_stream(stream.cuda_stream)
    try:
        with torch.cuda.graph(graph, stream=stream):
            hop()
        out.zero_()
        torch.cuda.synchronize()
        graph.replay()
        torch.cuda.synchronize()
    finally:
        Q.set_stream(None)
    res = [torch.zeros_like(s) for s in src]
    Q.unpack_fermions([r.data_ptr() for r in res], out.data_ptr(), nout.data_ptr(), Q.QCU_SRC_EO_HALF, 0, prec)
    Q.synchronize()
    got = np.stack([r.cpu().numpy() for r in res])
    assert rel(got, O.dslash(psi, g, L, 0, 0, True)) < TOL[prec]
