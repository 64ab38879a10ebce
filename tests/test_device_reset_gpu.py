"""A program resets its device between one-call operators: the next call runs on the new context's memory, and
what the library held before is not freed where the program's own allocations now lie.  Each case is a process of
its own (it loads the shared CUDA runtime, not torch, and ends with the reset)."""
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
rt = ctypes.CDLL(sys.argv[2])

def ok(e):
    assert e == 0, e

def up(a):
    a, p = np.ascontiguousarray(a, dtype=complex), ctypes.c_void_p()
    ok(rt.cudaMalloc(ctypes.byref(p), ctypes.c_size_t(a.nbytes)))
    ok(rt.cudaMemcpy(p, ctypes.c_void_p(a.ctypes.data), ctypes.c_size_t(a.nbytes), 1))
    return p

def down(p, like):
    out = np.empty_like(like, dtype=complex)
    ok(rt.cudaMemcpy(ctypes.c_void_p(out.ctypes.data), p, ctypes.c_size_t(out.nbytes), 2))
    return out

errs = []
for k, L in enumerate([(4, 4, 4, 8), (4, 4, 4, 8), (6, 4, 4, 4), (6, 4, 4, 4)]):
    g, psi = S.random_gauge(L, 3, seed=k), S.random_fermions(L, 3, 1, seed=10 + k, parities=2)[0]
    # the program's allocations take the addresses that the library's had before the reset
    mine = [up(np.full(4096, j + 0.5)) for j in range(64)]
    if sys.argv[3] == "init" and k % 2:
        Q.initGridSize((4, 4, 4, 4), 3)  # drops what is kept
    dg, dp, do = up(g), up(psi), up(0 * psi)
    Q.fullDslashQcu(do.value, dp.value, dg.value, L, k % 2)
    got = down(do, psi)
    want = np.stack([O.dslash(psi[None, 1 - p], g, L, p, k % 2, False)[0] for p in (0, 1)])
    errs.append(float(np.linalg.norm(got - want) / np.linalg.norm(want)))
    for j, p in enumerate(mine):
        assert np.all(down(p, np.empty(4096)) == j + 0.5)
    for p in mine:
        ok(rt.cudaFree(p))
    if sys.argv[3] == "each" or k != 1:
        ok(rt.cudaDeviceReset())
print(json.dumps(errs))
"""


@pytest.mark.parametrize("case", ["each", "kept", "init"])
def test_reset_between_calls(cuda, qcu_lib, case):
    if not os.path.exists(RUNTIME):
        pytest.skip("no shared CUDA runtime")
    r = subprocess.run([sys.executable, "-c", CHILD, ROOT, RUNTIME, case], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]
    assert max(json.loads(r.stdout.strip().splitlines()[-1])) < 1e-13
