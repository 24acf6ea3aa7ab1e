"""The block product's walk (one right-hand side per lane): every lane group width,
in both types, on matrices that are its own by the dispatch rule (rows of several
batches with single loads; narrow rows; one right-hand side), with ranks that are
empty, of one row, or end inside a tile."""
import numpy as np
import pytest

from spmv_b200 import gen
from helpers import build
from test_gpu_block_rows import check_product

pytestmark = pytest.mark.gpu


def rows_of(rng, n, lens):
    cols = [np.sort(rng.choice(n, size=m, replace=False)) for m in lens]
    rp = np.concatenate([[0], np.cumsum(lens)]).astype(np.int32)
    return gen.CSR(rp, np.concatenate(cols).astype(np.int32), rng.standard_normal(rp[-1]), n)


def matrix(rows):
    rng = np.random.default_rng(7)
    n = 2003
    if rows == "long":    # mean above 8, lengths over several batches, none above 512
        return rows_of(rng, n, np.concatenate([rng.integers(0, 60, n - 3), [511, 512, 100]]))
    if rows == "narrow":  # mean at most 4
        return rows_of(rng, n, rng.integers(0, 8, n))
    return rows_of(rng, n, rng.integers(3, 8, n))  # mean at most 6


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("rows", ["long", "narrow", "five"])
@pytest.mark.parametrize("k", [1, 2, 3, 5, 7, 9, 12, 15, 17, 24, 31, 32])
def test_block_product_walk(cuda_device, monkeypatch, k, rows, dtype):
    monkeypatch.setattr(gen, "owner_ranges", lambda P, n: np.array([0, 1, 1, 700, n]))
    A = matrix(rows)
    assert rows != "long" or len(A.cols) > 8 * A.nrows
    comm, cm, rm, M, D = build(A, 4, dtype=dtype)
    check_product(M, D, cm, k, dtype)
    check_product(M, D, cm, k, dtype, shift=1)
