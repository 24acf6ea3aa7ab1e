"""Batched solves with every unit in its own group of CTAs (onchip.cu):
sizes around the edges of slices, CTAs and groups, blocks of columns, both
precisions and index widths, against the lockstep kernel on the same batch and
the FP64 residual of the user's own matrix."""
import numpy as np
import pytest
import scipy.sparse as sp

import spmv_b200 as S
from spmv_b200.core import Batch

pytestmark = pytest.mark.gpu

RTOL = 1e-10


def _same(A):
    """Both kernels stop at a relative residual of at most RTOL confirmed in FP64, so each
    solution is within cond(A) RTOL of the exact one; cond by Gershgorin's circles."""
    d = A.diagonal()
    s = np.asarray(abs(A).sum(axis=1)).ravel() - d
    return 4 * RTOL * (d + s).max() / (d - s).min()


def _banded(n, half, seed):
    """SPD: `half` off-diagonals at random distances, dominated by its diagonal."""
    rng = np.random.default_rng(seed)
    offs = sorted(rng.choice(np.arange(1, max(2, min(n, 4 * half + 1))),
                             size=min(half, max(0, n - 1)), replace=False)) if n > 1 else []
    L = sp.diags([rng.uniform(0.1, 1.0, n - o) for o in offs], [int(o) for o in offs],
                 shape=(n, n)) if offs else sp.csr_matrix((n, n))
    A = (L + L.T).tocsr()
    return _dominant(A)


def _star(n, far, seed):
    """A few rows with `far` entries all over the system (wide slices, wide
    windows) on top of a band."""
    rng = np.random.default_rng(seed)
    A = _banded(n, 3, seed).tolil()
    for i in rng.choice(n, 3, replace=False):
        for j in rng.choice(n, far, replace=False):
            if i != j:
                A[i, j] = A[j, i] = 0.5
    return _dominant(A.tocsr())


def _random(n, per_row, seed):
    """Entries anywhere: no order makes it a band."""
    rng = np.random.default_rng(seed)
    i, j = rng.integers(0, n, (2, per_row * n))
    A = sp.csr_matrix((rng.uniform(0.1, 1.0, i.size), (i, j)), shape=(n, n))
    return _dominant((A + A.T).tocsr())


def _dominant(A):
    A = A.tolil()
    A.setdiag(0.0)
    A = A.tocsr()
    A.eliminate_zeros()
    s = np.asarray(abs(A).sum(axis=1)).ravel()
    A = (A + sp.diags(1.05 * s + 0.1)).tocsr()
    A.sort_indices()
    return A


BATCHES = {
    "tiny": ([("b", 1, 0), ("b", 2, 1), ("b", 31, 3), ("b", 32, 3), ("b", 33, 3)], None),
    "edges": ([("b", 640, 5), ("b", 641, 16), ("b", 639, 17), ("b", 1280, 8), ("b", 21000, 7)],
              (1, 1)),
    "block": ([("b", 3000, 6), ("b", 100, 6), ("b", 50001, 6)], (0, 32)),
    "wide": ([("s", 9000, 700), ("b", 500, 40)], (1, 3)),
    "idx32": ([("r", 70000, 4), ("b", 65, 2)], (1, 5)),
}


@pytest.mark.parametrize("precision", ["mixed", "fp64"])
@pytest.mark.parametrize("name", list(BATCHES))
def test_against_lockstep(cuda_device, name, precision):
    spec, block = BATCHES[name]
    kinds = {"b": _banded, "s": _star, "r": _random}
    mats = [kinds[k](n, w, 7 + i) for i, (k, n, w) in enumerate(spec)]
    comm = S.Comm(size=1, device=0)
    B = Batch(comm, [(A.indptr.astype(np.int32), A.indices.astype(np.int32), A.data)
                     for A in mats], block=block)
    assert B.stats()["index_bits"] == (32 if name == "idx32" else 16)
    rng = np.random.default_rng(3)
    bs = [rng.standard_normal(A.shape[0]) for A in mats]
    Bb = rng.standard_normal((mats[block[0]].shape[0], block[1])) if block else None
    run = lambda: B.solve([b.copy() for b in bs], 5000, RTOL,
                          block_b=None if Bb is None else Bb.copy(), precision=precision)
    first, again = run(), run()
    B.set_config(2, 256, 32, True, precision=precision)
    lock = run()

    def columns(r):
        out = list(zip(mats, r[0], bs, r[1]))
        if block:
            out += [(mats[block[0]], r[2][:, l], Bb[:, l], r[3][l]) for l in range(block[1])]
        return out

    for (A, x, b, i), (_, x2, _, _), (_, y, _, j) in zip(columns(first), columns(again),
                                                         columns(lock)):
        assert i.status == 0 and i.converged == 1 and j.converged == 1
        assert np.linalg.norm(b - A @ x) <= 1.5 * RTOL * np.linalg.norm(b)
        assert np.linalg.norm(x - y) <= _same(A) * np.linalg.norm(y)
        assert abs(i.iterations - j.iterations) <= max(3, j.iterations // 10)
        assert np.array_equal(x, x2)  # the same bits each time


@pytest.mark.parametrize("precision", ["mixed", "fp64"])
def test_caps_and_zero_sides(cuda_device, precision):
    mats = [_banded(n, 4, n) for n in (700, 4000, 90)]
    comm = S.Comm(size=1, device=0)
    B = Batch(comm, [(A.indptr.astype(np.int32), A.indices.astype(np.int32), A.data)
                     for A in mats], block=(2, 2))
    rng = np.random.default_rng(5)
    bs = [rng.standard_normal(700), np.zeros(4000), rng.standard_normal(90)]
    Bb = np.stack([np.zeros(90), rng.standard_normal(90)], axis=1).copy()
    x, info, X, binfo = B.solve(bs, 2, 1e-14, block_b=Bb, precision=precision)
    assert info[0].iterations == 2 and info[0].converged == 0 and info[0].refinements >= 1
    r = np.linalg.norm(bs[0] - mats[0] @ x[0]) / np.linalg.norm(bs[0])
    assert abs(info[0].relres - r) <= 1e-10
    assert info[1].iterations == 0 and info[1].converged == 1 and not x[1].any()
    assert binfo[0].converged == 1 and not X[:, 0].any() and binfo[1].iterations == 2
    x, info, X, binfo = B.solve(bs, 0, RTOL, block_b=Bb, precision=precision)
    assert all(i.iterations == 0 for i in info) and not x[0].any()
