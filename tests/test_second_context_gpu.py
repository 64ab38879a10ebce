"""Kernels above 48 KB of shared memory in a second CUDA context of the process, as on a second device: the limit
that the first launch raises belongs to one context.  A process of its own, without torch."""
import json
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
RUNTIME = "/usr/local/cuda/lib64/libcudart.so"

CHILD = r"""
import ctypes, json, sys
sys.path.insert(0, sys.argv[1])
import numpy as np
import mrhs_qcu_gb300 as Q
from mrhs_qcu_gb300 import synthetic as S
from oracle import oracle as O
rt, cu = ctypes.CDLL(sys.argv[2]), ctypes.CDLL("libcuda.so.1")
prec, n, nrhs = (int(a) for a in sys.argv[3:6])
L = (4, 4, 4, 8)

def ok(e):
    assert e == 0, e

def up(a):
    a, p = np.ascontiguousarray(a, dtype=complex), ctypes.c_void_p()
    ok(rt.cudaMalloc(ctypes.byref(p), ctypes.c_size_t(a.nbytes)))
    ok(rt.cudaMemcpy(p, ctypes.c_void_p(a.ctypes.data), ctypes.c_size_t(a.nbytes), 1))
    return p

g, psi = S.random_gauge(L, n, seed=1), S.random_fermions(L, n, nrhs, seed=2)
want = O.dslash(psi, g, L, 0, 0, False)
errs = []

def work():
    Q.initGridSize(L, n)
    Q.set_antiperiodic_t(False)
    dg = up(g)
    Q.loadQcuGauge(dg.value)
    Q.getDslash(Q.DSLASH_WILSON, 0.0, n, nrhs, prec)
    ins, outs = [up(p) for p in psi], [up(0 * p) for p in psi]
    for i, o in zip(ins, outs):
        Q.pushBackFermions(o.value, i.value)
    Q.startDslash(0, 0)
    got = np.empty_like(psi)
    for r, o in enumerate(outs):
        ok(rt.cudaMemcpy(ctypes.c_void_p(got[r].ctypes.data), o, ctypes.c_size_t(got[r].nbytes), 2))
    errs.append([float(np.linalg.norm(got - want) / np.linalg.norm(want)), Q.last_dslash_shape()[3]])
    Q.initGridSize((2, 2, 2, 2), 3)  # the session's memory is freed in its own context

ok(rt.cudaFree(None))
work()
second, device = ctypes.c_void_p(), ctypes.c_int()
ok(cu.cuDeviceGet(ctypes.byref(device), 0))
ok(cu.cuCtxCreate_v2(ctypes.byref(second), 0, device))
work()
print(json.dumps(errs))
"""


@pytest.mark.parametrize("prec,n,nrhs", [(4, 6, 16), (0, 8, 32)])
def test_register_fragment_mma(cuda, qcu_lib, prec, n, nrhs):
    if not os.path.exists(RUNTIME):
        pytest.skip("no shared CUDA runtime")
    env = dict(os.environ, QCU_DSLASH_CONFIG="1,0,0,0,0,0,5", QCU_TUNE="0")
    r = subprocess.run([sys.executable, "-c", CHILD, ROOT, RUNTIME, str(prec), str(n), str(nrhs)], capture_output=True,
                       text=True, timeout=300, env=env)
    assert r.returncode == 0, r.stderr[-2000:]
    first, second = json.loads(r.stdout.strip().splitlines()[-1])
    assert first[1] == second[1] == -5
    assert first[0] < 5e-3 and second[0] < 5e-3
