"""Which forms of a solve the workspace times before it chooses one (spmv::cg,
cg.cpp:11-83, and the mixed solver): the on-chip forms are taken unseen only where
they are far ahead.  Read from the library's debug lines, in a process of its own."""
import os
import subprocess
import sys
from pathlib import Path

import pytest

pytestmark = pytest.mark.gpu
ROOT = Path(__file__).resolve().parent.parent

SCRIPT = """
import sys
sys.path[:0] = [{root!r}, {root!r} + "/tests"]
import numpy as np
import spmv_b200 as S
from spmv_b200 import gen
from helpers import build
W = gen.workload({cfg!r}, {scale})
A = W.A
if {shuffled}:
    p = np.random.default_rng(0).permutation(A.nrows)
    G = A.scipy()[p][:, p].tocsr()
    G.sort_indices()
    A = gen.CSR(G.indptr.astype(np.int32), G.indices.astype(np.int32), G.data, A.nrows)
comm, cm, rm, M, D = build(A, 1)
M.set_kernel("staged", {width})
b = np.random.default_rng(1).standard_normal(A.nrows)
{solve}(comm, M, [b], 60, 1e-30)
print("form", M.cg_form({solver!r})[2])
"""


def run(solver, cfg, scale, width, shuffled=False):
    code = SCRIPT.format(root=str(ROOT), cfg=cfg, scale=scale, width=width, shuffled=shuffled,
                         solver=solver, solve={"cg": "S.cg", "mixed": "S.cg_mixed"}[solver])
    r = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, timeout=300,
                       env={**os.environ, "SPMV_B200_DEBUG": "1"})
    assert r.returncode == 0, r.stderr[-2000:]
    return r.stdout.split("form ")[-1].strip(), r.stderr


def test_cg_far_ahead_on_chip(cuda_device):
    form, log = run("cg", "c2", 64, 7)
    assert form == "tmem:m" and "cg form 1:tmem:m" in log and "cg form 2:smem" not in log


def test_cg_rows_in_random_order(cuda_device):
    form, log = run("cg", "c1", 1024, 5, shuffled=True)
    assert "cg form 1:tmem:m" in log and "cg form 2:smem:m" in log
    assert form != "tmem:m"

def test_mixed_with_narrow_windows(cuda_device):
    form, log = run("mixed", "c3", 64, 9)
    assert form == "tmem:m" and "cg_mixed form" not in log


def test_mixed_with_wide_windows(cuda_device):
    form, log = run("mixed", "c2", 112, 7)
    assert "cg_mixed form graph" in log and "cg_mixed form on chip" in log
