"""SPMV_B200_CG_FUSED and SPMV_B200_CG_MIXED_FUSED set for a whole program: a plan of
the staged product is forced where the product is staged, and other matrices solve in
their graph form."""
import numpy as np
import pytest

import spmv_b200 as S
from spmv_b200 import gen
from helpers import build

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("solver,env,plans", [
    ("cg", "SPMV_B200_CG_FUSED", ["0", "1:smem", "2:smem", "3:global:m"]),
    ("mixed", "SPMV_B200_CG_MIXED_FUSED", ["0", "2:smem", "3:global"])])
def test_staged_plan_on_a_matrix_without_a_staged_product(monkeypatch, cuda_device, solver, env,
                                                          plans):
    # Rows of 80 entries: no slice of them fits a stage of the staged product.
    n = 3000
    rng = np.random.default_rng(0)
    cols = np.sort((np.arange(n)[:, None] + np.arange(-40, 40)[None, :]) % n, axis=1)
    vals = np.where(cols == np.arange(n)[:, None], 200.0, -1.0)
    A = gen.CSR(np.arange(0, 80 * n + 1, 80).astype(np.int32), cols.reshape(-1).astype(np.int32),
                vals.reshape(-1), n)
    b = rng.standard_normal(n)
    for plan in plans:
        monkeypatch.setenv(env, plan)
        comm, cm, rm, M, D = build(A, 1)
        if solver == "cg":
            x, k = S.cg(comm, M, [b], 1000, 1e-10)
        else:
            x, info = S.cg_mixed(comm, M, [b], 1000, 1e-10)
        assert M.cg_form(solver) == ("graph", 0, None)
        rel = np.linalg.norm(b - A.scipy() @ x[0][:n]) / np.linalg.norm(b)
        assert rel < 1.5e-10


@pytest.mark.parametrize("plan", ["0", "2:smem", "1:tmem:m"])
def test_mixed_breakdown_counts_its_iteration(monkeypatch, cuda_device, plan):
    monkeypatch.setenv("SPMV_B200_CG_MIXED_FUSED", plan)
    W = gen.workload("c2", 24)
    Z = gen.CSR(W.A.rowptr, W.A.cols, 0.0 * W.A.vals, W.A.ncols)
    comm, cm, rm, M, D = build(Z, 1)
    M.set_kernel("staged", 7)
    with pytest.raises(S.SpmvError, match="breakdown .* after 1 iterations"):
        S.cg_mixed(comm, M, [W.b.copy()], 100, 1e-8)
