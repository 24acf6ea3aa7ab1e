"""A solve kept for one matrix runs again after another matrix has planned a
smaller launch of the same kernel (spmv::cg, cg.cpp:11-83, and the mixed
solver): the kernel's shared-memory limit is not one matrix's."""
import numpy as np
import pytest

import spmv_b200 as S
from spmv_b200 import gen
from helpers import build

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("solver,env,plan", [
    ("cg", "SPMV_B200_CG_FUSED", "1:tmem:m"),
    ("cg", "SPMV_B200_CG_FUSED", "2:smem"),
    ("cg", "SPMV_B200_CG_FUSED", "2:smem:m"),
    ("mixed", "SPMV_B200_CG_MIXED_FUSED", "1:tmem:m"),
    ("mixed", "SPMV_B200_CG_MIXED_FUSED", "2:smem"),
])
def test_large_solve_after_a_small_matrix_was_planned(monkeypatch, cuda_device, solver, env, plan):
    monkeypatch.setenv(env, plan)

    def setup(scale):
        W = gen.workload("c2", scale)
        comm, cm, rm, M, D = build(W, 2)
        M.set_kernel("staged", 7)
        return comm, M, [W.b[D.ranges[q]:D.ranges[q + 1]].copy() for q in range(2)]

    fn = S.cg if solver == "cg" else S.cg_mixed
    large, small = setup(72), setup(24)
    x, k = fn(*large, 20000, 1e-10)
    fn(*small, 20000, 1e-10)
    x2, k2 = fn(*large, 20000, 1e-10)
    form = plan.split(":", 1)
    assert large[1].cg_form(solver) == small[1].cg_form(solver) == ("fused", int(form[0]), form[1])
    if solver == "mixed":
        k, k2 = k.iterations, k2.iterations
    assert k2 == k and all(np.array_equal(u, v) for u, v in zip(x, x2))
