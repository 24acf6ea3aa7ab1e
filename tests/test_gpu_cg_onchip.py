"""The on-chip form of the fused CG solve (spmv::cg, cg.cpp:11-83): p in
shared memory, r, y (and x where it fits) in tensor memory, the matrix through
per-warp rings.  Against the graph form on the same product at the edges of
its shapes: every ring width, 16- and 32-bit columns,
slices wider than a slot, ranks that are empty or end inside a slice, fewer
slices than warps, and a size whose x stays in global memory."""
import numpy as np
import pytest

import spmv_b200 as S
from spmv_b200 import gen
from helpers import build

pytestmark = pytest.mark.gpu

PLANS = ["1:tmem:m"]


def solve(monkeypatch, plan, A, b, rtol, P, width=8, max_its=10000):
    monkeypatch.setenv("SPMV_B200_CG_FUSED", plan)
    comm, cm, rm, M, D = build(A, P)
    M.set_kernel("staged", width)
    bs = [b[D.ranges[q]:D.ranges[q + 1]].copy() for q in range(P)]
    x, k, info = S.cg(comm, M, bs, max_its, rtol, info=True)
    x2, k2 = S.cg(comm, M, bs, max_its, rtol)
    assert k2 == k and all(np.array_equal(u, v) for u, v in zip(x, x2))
    assert all(np.all(x[q][D.local_sizes[q]:] == 0.0) for q in range(P))
    return np.concatenate([x[q][:D.local_sizes[q]] for q in range(P)]), k, info, M


def check(monkeypatch, plan, A, b, rtol, P, width, max_its=10000):
    x0, k0, i0, M0 = solve(monkeypatch, "0", A, b, rtol, P, width, max_its)
    x1, k1, i1, M1 = solve(monkeypatch, plan, A, b, rtol, P, width, max_its)
    assert M1.cg_form() == ("fused", int(plan[0]), "tmem:m")
    assert i1.status == 0 and abs(k1 - k0) <= 2, (k0, k1)
    assert np.linalg.norm(x1 - x0) <= 1e-9 * np.linalg.norm(x0)
    rel = np.linalg.norm(b - A.scipy() @ x1) / np.linalg.norm(b)
    assert rel < 1.5 * rtol or k1 == max_its


@pytest.mark.parametrize("plan", PLANS)
@pytest.mark.parametrize("bits", ["16", "32"])
@pytest.mark.parametrize("cfg,scale,P,width", [("c2", 32, 8, 8), ("c2", 40, 3, 4),
                                               ("c2", 31, 8, 7), ("c1", 65, 3, 5),
                                               ("c3", 24, 2, 9), ("c1", 8, 1, 4)])
def test_onchip_matches_graph_form(monkeypatch, cuda_device, plan, bits, cfg, scale, P, width):
    if bits == "32":
        monkeypatch.setenv("SPMV_B200_D16", "0")
    W = gen.workload(cfg, scale)
    check(monkeypatch, plan, W.A, W.b, W.rtol, P, width)


@pytest.mark.parametrize("plan", PLANS)
def test_onchip_x_in_global_memory(monkeypatch, cuda_device, plan):
    # 128^3 rows: r and y take the tensor memory, x stays in global memory.
    W = gen.workload("c2")
    check(monkeypatch, plan, W.A, W.b, 1e-6, W.P, 7, 60)
    check(monkeypatch, plan, W.A, W.b, W.rtol, W.P, 7)


@pytest.mark.parametrize("plan", PLANS)
def test_onchip_with_an_empty_rank_and_unaligned_ranks(monkeypatch, cuda_device, plan):
    W = gen.workload("c1", 32)
    monkeypatch.setattr(gen, "owner_ranges", lambda P, n: np.array([0, 300, 300, n]))
    check(monkeypatch, plan, W.A, W.b, W.rtol, 3, 5)


@pytest.mark.parametrize("plan", PLANS)
def test_onchip_uneven_rows(monkeypatch, cuda_device, plan):
    # Rows of 13 to over 20 entries (several items per slice, masked ends), far
    # columns (32-bit), an identity row.
    A = gen.knn_laplacian(7001, 12, 3, 0, 1e-1)
    b = gen.normal(5, 1, A.nrows)
    check(monkeypatch, plan, A, b, 1e-9, 2, 4)
    check(monkeypatch, plan, A, b, 1e-9, 1, 7)


@pytest.mark.parametrize("plan", PLANS)
def test_onchip_caps_zero_and_breakdown(monkeypatch, cuda_device, plan):
    W = gen.workload("c2", 24)
    x, k, info, M = solve(monkeypatch, plan, W.A, W.b, W.rtol, 8, 7, 7)
    assert k == 7
    x0, k0, _, _ = solve(monkeypatch, "0", W.A, W.b, W.rtol, 8, 7, 7)
    assert np.linalg.norm(x - x0) <= 1e-12 * np.linalg.norm(x0)
    x, k, info, M = solve(monkeypatch, plan, W.A, 0.0 * W.b, W.rtol, 8, 7)
    assert k == 0 and np.all(x == 0.0)
    zero = gen.CSR(W.A.rowptr, W.A.cols, 0.0 * W.A.vals, W.A.ncols)
    with pytest.raises(S.SpmvError) as e:
        solve(monkeypatch, plan, zero, W.b, W.rtol, 2, 7)
    assert e.value.status == 5


def test_onchip_wait_limit_reports_an_error(monkeypatch, cuda_device):
    """Bounded grid waits at 1 ns: every CTA that waits gives up, frees its
    tensor memory and leaves; the next solve runs."""
    W = gen.workload("c2", 32)
    monkeypatch.setenv("SPMV_B200_CG_FUSED", "1:tmem:m")
    comm, cm, rm, M, D = build(W, 8)
    M.set_kernel("staged", 7)
    b = [W.b[D.ranges[q]:D.ranges[q + 1]].copy() for q in range(8)]
    monkeypatch.setenv("SPMV_B200_WAIT_LIMIT_NS", "1")
    with pytest.raises(S.SpmvError) as e:
        S.cg(comm, M, b, 10000, W.rtol)
    assert "timed out" in str(e.value)
    monkeypatch.delenv("SPMV_B200_WAIT_LIMIT_NS")
    x, k, info = S.cg(comm, M, b, 10000, W.rtol, info=True)
    xg = np.concatenate([x[q][:D.local_sizes[q]] for q in range(8)])
    assert info.status == 0
    assert np.linalg.norm(W.b - W.A.scipy() @ xg) < 1.5 * W.rtol * np.linalg.norm(W.b)
