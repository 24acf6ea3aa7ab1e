"""The block product and block CG where a CTA takes several chunks of rows (block CG)
or the chunks are several rounds of the chip (the product): 56^3 rows over 3 ranks."""
import numpy as np
import pytest
import torch

import spmv_b200 as S
from spmv_b200 import gen
from spmv_b200.core import cg_block
from helpers import build

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k", [31, 32])
def test_block_cg_of_several_rounds(cuda_device, k):
    W = gen.workload("c2", 56)
    comm, cm, rm, M, D = build(W, 3)
    rng = np.random.default_rng(k)
    Bg = rng.uniform(-1, 1, (W.A.nrows, k))
    B = [torch.from_numpy(np.ascontiguousarray(Bg[D.ranges[q]:D.ranges[q + 1]])).cuda()
         for q in range(3)]
    X, info = cg_block(comm, M, B, 10000, 1e-8)
    Xg = np.concatenate([X[q][:D.local_sizes[q]].cpu().numpy() for q in range(3)])
    rel = np.linalg.norm(Bg - W.A.scipy() @ Xg, axis=0) / np.linalg.norm(Bg, axis=0)
    assert np.all(rel < 1.5e-8), rel
    for col in (0, k - 1):
        x, its = S.cg(comm, M, [b[:, col].contiguous() for b in B], 10000, 1e-8)
        assert abs(info[col].iterations - its) <= 2 and info[col].status == 0


@pytest.mark.parametrize("k", [1, 3, 16, 31])
def test_block_product_of_several_rounds(cuda_device, k):
    W = gen.workload("c2", 56)
    comm, cm, rm, M, D = build(W, 3)
    X = [np.random.default_rng(q).standard_normal((cm.vec_len(q), k)) for q in range(3)]
    Y = M.mult_block([torch.from_numpy(x).cuda() for x in X])
    Z = M.mult_block([torch.from_numpy(x).cuda() for x in X])
    for q in range(3):
        rp, ci, va = D.blocks[q]
        A = gen.CSR(rp, ci, va, cm.vec_len(q)).scipy()
        y = Y[q].cpu().numpy()
        # Rows of at most 7 products in storage order, as scipy sums them.
        bound = 7 * np.finfo(np.float64).eps * (abs(A) @ np.abs(X[q]))
        assert np.all(np.abs(y - A @ X[q]) <= bound)
        assert torch.equal(Y[q], Z[q])
