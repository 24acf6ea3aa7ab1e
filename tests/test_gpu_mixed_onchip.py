"""The on-chip form of the fused mixed-precision CG solve: p over the columns a
CTA gathers in shared memory, r, y and d in tensor memory, the matrix through
per-warp rings.  Against the graph form on the same matrix at the edges of its
shapes: 16- and 32-bit columns, slices of one and of several copies, ranks
that are empty or end inside a slice, fewer slices than CTAs, and windows that
do not fit in shared memory (their columns gathered from L2)."""
import os

import numpy as np
import pytest
import scipy.sparse as sp

import spmv_b200 as S
from spmv_b200 import gen
from helpers import build

pytestmark = pytest.mark.gpu

RTOL = 1e-10


def solve(monkeypatch, plan, A, b, P, max_its=20000, rtol=RTOL):
    monkeypatch.setenv("SPMV_B200_CG_MIXED_FUSED", plan)
    comm, cm, rm, M, D = build(A, P)
    M.set_kernel("staged", 8)
    bs = [b[D.ranges[q]:D.ranges[q + 1]].copy() for q in range(P)]
    x, info = S.cg_mixed(comm, M, bs, max_its, rtol)
    x2, info2 = S.cg_mixed(comm, M, bs, max_its, rtol)
    assert info2.iterations == info.iterations
    assert all(np.array_equal(u, v) for u, v in zip(x, x2))
    assert all(np.all(x[q][D.local_sizes[q]:] == 0.0) for q in range(P))
    return np.concatenate([x[q][:D.local_sizes[q]] for q in range(P)]), info, M


def check(monkeypatch, A, b, P):
    x0, i0, M0 = solve(monkeypatch, "0", A, b, P)
    x1, i1, M1 = solve(monkeypatch, "1:tmem:m", A, b, P)
    assert M0.cg_form("mixed") == ("graph", 0, None)
    assert M1.cg_form("mixed") == ("fused", 1, "tmem:m")
    assert i0.converged == 1 and i1.converged == 1 and i1.status == 0
    # The recurrences differ in FP32 rounding; the residuals do not.
    assert abs(i1.iterations - i0.iterations) <= max(5, i0.iterations // 5), (i0, i1)
    rel = np.linalg.norm(b - A.scipy() @ x1) / np.linalg.norm(b)
    assert rel < 1.5 * RTOL and abs(i1.relres - rel) <= 0.05 * rel + 1e-14
    assert np.linalg.norm(x1 - x0) <= 1e-6 * np.linalg.norm(x0)


@pytest.mark.parametrize("bits", ["16", "32"])
@pytest.mark.parametrize("cfg,scale,P", [("c2", 32, 8), ("c2", 31, 8), ("c2", 40, 3),
                                         ("c1", 65, 3), ("c1", 8, 1), ("c3", 24, 2)])
def test_onchip_matches_graph_form(monkeypatch, cuda_device, bits, cfg, scale, P):
    if bits == "32":
        monkeypatch.setenv("SPMV_B200_D16", "0")
    W = gen.workload(cfg, scale)
    check(monkeypatch, W.A, W.b, P)


@pytest.mark.parametrize("n,per_row,P", [(150_001, 3, 1), (150_001, 3, 5), (2_500, 10, 2)])
def test_onchip_windows(monkeypatch, cuda_device, n, per_row, P):
    # Columns anywhere: 150,001 rows of p do not fit in shared memory, 2,500 do,
    # and rows of about 20 entries are several copies each.
    rng = np.random.default_rng(n)
    i, j = rng.integers(0, n, (2, per_row * n))
    G = sp.csr_matrix((rng.uniform(-1.0, 1.0, i.size), (i, j)), shape=(n, n))
    G = (G + G.T).tocsr()
    G.setdiag(0.0)
    s = np.asarray(abs(G).sum(axis=1)).ravel()
    G = (G + sp.diags(1.05 * s + 0.1)).tocsr()
    G.sort_indices()
    A = gen.CSR(G.indptr.astype(np.int32), G.indices.astype(np.int32), G.data, n)
    check(monkeypatch, A, rng.standard_normal(n), P)


def test_onchip_caps_and_zero_sides(monkeypatch, cuda_device):
    W = gen.workload("c2", 24)
    x, info, M = solve(monkeypatch, "1:tmem:m", W.A, np.zeros(W.A.nrows), 2)
    assert info.iterations == 0 and info.converged == 1 and not x.any()
    x, info, M = solve(monkeypatch, "1:tmem:m", W.A, W.b, 2, max_its=5)
    assert info.iterations == 5 and info.converged == 0 and info.refinements >= 1
    rel = np.linalg.norm(W.b - W.A.scipy() @ x) / np.linalg.norm(W.b)
    assert abs(info.relres - rel) <= 1e-10
    x, info, M = solve(monkeypatch, "1:tmem:m", W.A, W.b, 2, max_its=0)
    assert info.iterations == 0 and not x.any()


def test_onchip_bounded_wait(monkeypatch, cuda_device):
    # A limit of 1 ns makes the waits run out on a healthy solve: an error, and
    # the next solve on the same matrix succeeds.
    monkeypatch.setenv("SPMV_B200_CG_MIXED_FUSED", "1:tmem:m")
    W = gen.workload("c2", 24)
    comm, cm, rm, M, D = build(W.A, 1)
    M.set_kernel("staged", 8)
    S.cg_mixed(comm, M, [W.b.copy()], 20000, RTOL)
    os.environ["SPMV_B200_WAIT_LIMIT_NS"] = "1"
    try:
        with pytest.raises(S.SpmvError, match="timed out"):
            S.cg_mixed(comm, M, [W.b.copy()], 20000, RTOL)
    finally:
        del os.environ["SPMV_B200_WAIT_LIMIT_NS"]
    _, info = S.cg_mixed(comm, M, [W.b.copy()], 20000, RTOL)
    assert M.cg_form("mixed") == ("fused", 1, "tmem:m") and info.converged == 1
