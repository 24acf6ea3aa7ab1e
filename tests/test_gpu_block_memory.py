"""Device memory of block CG between solves: small workspaces stay with the
matrix, large ones (here five vectors of 226 MB) are given back."""
import numpy as np
import pytest
import torch

from spmv_b200 import core, gen
from helpers import build

pytestmark = pytest.mark.gpu


def test_block_cg_gives_large_vectors_back(cuda_device):
    W = gen.workload("c2", 96)
    comm, cm, rm, M, D = build(W, 2)

    def solve(k):
        b = [torch.ones((n, k), dtype=torch.float64, device="cuda") for n in D.local_sizes]
        x = [torch.empty((cm.vec_len(q), k), dtype=torch.float64, device="cuda")
             for q in range(2)]
        torch.cuda.synchronize()
        before = torch.cuda.mem_get_info()[0]
        core.cg_block(comm, M, b, 10, 1e-30, X=x)
        torch.cuda.synchronize()
        return x, before - torch.cuda.mem_get_info()[0]

    solve(1)
    n = sum(D.local_sizes)
    assert 5 * 8 * n * 32 > 1 << 30
    x, used = solve(32)
    assert used <= 32 << 20
    again, _ = solve(32)
    assert all(torch.equal(u, v) for u, v in zip(x, again))
    assert np.isfinite(x[0].cpu().numpy()).all()
