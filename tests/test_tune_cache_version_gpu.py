"""A tuning file of a build with other kernels is not used: its numbers may name kernels that were never timed
for them.  Each process is a fresh interpreter, so only the file carries the choice."""
import json
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
KEY = "4:4:16:256"  # BF16, SU(4), 16 RHS, Vh = 4*4*4*8/2

CHILD = r"""
import json, sys
sys.path.insert(0, sys.argv[1])
import torch
import mrhs_qcu_gb300 as Q
from mrhs_qcu_gb300 import synthetic as S
from tests.util import dev
L, n, nrhs = (4, 4, 4, 8), 4, 16
Q.initGridSize(L, n)
g = dev(torch, S.random_gauge(L, n, seed=1))
Q.loadQcuGauge(g.data_ptr())
print(json.dumps(list(Q.tune_dslash(nrhs, 4))))
"""


def _tuned(cache):
    env = dict(os.environ, QCU_TUNE_CACHE=str(cache))
    env.pop("QCU_DSLASH_CONFIG", None)
    r = subprocess.run([sys.executable, "-c", CHILD, ROOT], capture_output=True, text=True, env=env, timeout=600)
    assert r.returncode == 0, r.stderr[-2000:]
    return json.loads(r.stdout.strip().splitlines()[-1])


@pytest.mark.parametrize("first_line", ["", "kernels 1\n", "kernels 999\n", "junk\n"])
def test_other_set_is_not_used(cuda, tmp_path, first_line):
    cache = tmp_path / "tune.txt"
    cache.write_text(first_line + KEY + " 1 64 1 0 0 0 4 0 0\n")  # tensor-core variant 4, which tuning does not choose
    assert _tuned(cache)[4] != -4
    lines = cache.read_text().splitlines()
    assert lines[0].startswith("kernels ") and lines[0] != first_line.strip()
    assert sum(line.startswith(KEY + " ") for line in lines) == 1
    # this build's own file is used
    cache.write_text(lines[0] + "\n" + KEY + " 1 64 1 0 0 0 4 0 0\n")
    assert _tuned(cache)[4] == -4
