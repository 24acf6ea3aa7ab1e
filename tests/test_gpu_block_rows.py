"""The block product and block CG at the edges of their dispatch: every lane
group width and run length (right-hand sides 1 to 32, odd ones, vectors that
start off a 16-byte boundary), rows longer than one CTA's share, empty rows
and ranks without rows; block CG's cap, zero columns and breakdown."""
import numpy as np
import pytest
import torch

import oracle
import spmv_b200 as S
from spmv_b200 import gen
from spmv_b200.core import cg_block
from helpers import TOL_F32, TOL_F64, abs_mult, assert_spmv_close, build, random_csr

pytestmark = pytest.mark.gpu


def check_product(M, D, cm, k, dtype, shift=0):
    rng = np.random.default_rng(k)
    tdt = torch.float64 if dtype == np.float64 else torch.float32
    X, Xd = [], []
    for q in range(D.P):
        x = rng.standard_normal((cm.vec_len(q), k)).astype(dtype)
        buf = torch.empty(x.size + shift, dtype=tdt, device="cuda")
        d = buf[shift:].view(x.shape)
        d.copy_(torch.from_numpy(x))
        X.append(x)
        Xd.append(d)
    Y = M.mult_block(Xd)
    tol = TOL_F64 if dtype == np.float64 else TOL_F32
    for q in range(D.P):
        rp, ci, va = D.blocks[q]
        y = Y[q].cpu().numpy()
        for col in range(k):
            x = np.ascontiguousarray(X[q][:, col])
            assert_spmv_close(y[:, col], oracle.csr_mult(rp, ci, va, x),
                              abs_mult(D.blocks[q], x), tol)


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("k", [1, 2, 3, 4, 6, 7, 12, 16, 17, 20, 32])
def test_block_product_widths_and_long_rows(cuda_device, monkeypatch, k, dtype):
    # Row lengths around the batch of 8 and the CTA's 512; ranks of 1, 0 and
    # 2399 rows.
    rng = np.random.default_rng(11)
    A = random_csr(rng, 2400, 2400, density=0.004, long_rows=(0, 700, 701, 2399),
                   empty_frac=0.2)
    monkeypatch.setattr(gen, "owner_ranges", lambda P, n: np.array([0, 1, 1, n]))
    comm, cm, rm, M, D = build(A, 3, dtype=dtype)
    check_product(M, D, cm, k, dtype)
    check_product(M, D, cm, k, dtype, shift=1)


def test_block_product_row_lengths(cuda_device):
    # Every row length from 0 to 40 and around the CTA's share of 512.
    lens = list(range(41)) + [511, 512, 513, 520, 1024]
    rng = np.random.default_rng(4)
    n = 1500
    cols = [np.sort(rng.choice(n, size=m, replace=False)) for m in lens]
    rp = np.concatenate([[0], np.cumsum(lens)]).astype(np.int32)
    ci = np.concatenate(cols).astype(np.int32)
    va = rng.standard_normal(len(ci))
    comm = S.Comm(size=1, device=0)
    cm = S.L2GMap(comm, [n], [[]])
    rm = S.L2GMap(comm, [len(lens)], [[]])
    M = S.Matrix(comm, [(rp, ci, va)], cm, rm)
    for k in (1, 8, 32):
        X = rng.standard_normal((n, k))
        Y = M.mult_block([torch.from_numpy(X).cuda()])[0].cpu().numpy()
        for col in range(k):
            x = np.ascontiguousarray(X[:, col])
            assert_spmv_close(Y[:, col], oracle.csr_mult(rp, ci, va, x),
                              oracle.csr_mult(rp, ci, np.abs(va), np.abs(x)), TOL_F64)


@pytest.mark.parametrize("k", [1, 3, 5, 6, 12, 31])
def test_block_cg_widths(cuda_device, k):
    W = gen.workload("c2", 20)
    comm, cm, rm, M, D = build(W, 3)
    rng = np.random.default_rng(k)
    Bg = rng.uniform(-1, 1, (W.A.nrows, k))
    B = [np.ascontiguousarray(Bg[D.ranges[q]:D.ranges[q + 1]]) for q in range(3)]
    X, info = cg_block(comm, M, B, 10000, 1e-8)
    X2, info2 = cg_block(comm, M, B, 10000, 1e-8)
    for q in range(3):
        np.testing.assert_array_equal(X[q], X2[q])  # reproducible run to run
    Xg = np.concatenate([X[q][:D.local_sizes[q]] for q in range(3)])
    Sp = W.A.scipy()
    rel = np.linalg.norm(Bg - Sp @ Xg, axis=0) / np.linalg.norm(Bg, axis=0)
    assert np.all(rel < 1.5e-8), rel
    for col in range(k):
        x, its = S.cg(comm, M, [np.ascontiguousarray(b[:, col]) for b in B], 10000, 1e-8)
        assert abs(info[col].iterations - its) <= 2 and info[col].status == 0


def test_block_cg_cap_and_zero_columns(cuda_device):
    W = gen.workload("c2", 16)
    comm, cm, rm, M, D = build(W, 2)
    rng = np.random.default_rng(0)
    B = [rng.uniform(-1, 1, (n, 4)) for n in D.local_sizes]
    for b in B:
        b[:, 2] = 0.0
    X, info = cg_block(comm, M, B, 7, 1e-12)
    assert [i.iterations for i in info] == [7, 7, 0, 7]
    assert all(np.all(x[:, 2] == 0.0) for x in X)
    X, info = cg_block(comm, M, B, 0, 1e-12)
    assert [i.iterations for i in info] == [0, 0, 0, 0]
    assert all(np.all(x == 0.0) for x in X)
    Z = gen.CSR(W.A.rowptr, W.A.cols, 0.0 * W.A.vals, W.A.ncols)
    comm, cm, rm, M, D = build(Z, 2)
    with pytest.raises(S.SpmvError) as e:
        cg_block(comm, M, B, 10, 1e-12)
    assert e.value.status == 5
