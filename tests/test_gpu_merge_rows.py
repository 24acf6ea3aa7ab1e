"""The merge-path product's sums by thread, warp and CTA at their edges: rows
of 31 to 34 and 255 to 258 entries, rows that span tiles of 2048 items, tiles
that are one row, runs of empty rows longer than a tile, and ends that fall on
tile boundaries.  Bitwise the same on a second call."""
import numpy as np
import pytest
import torch

import oracle
import spmv_b200 as S
from helpers import TOL_F32, TOL_F64, assert_spmv_close

pytestmark = pytest.mark.gpu

SHAPES = {
    "edges": [31, 32, 33, 34, 0, 255, 256, 257, 258, 1] * 40,
    "spans": [5000, 0, 3, 2047, 2048, 2049, 1, 12000, 0, 0, 7] * 3,
    "empty": [0] * 5000 + [3] + [0] * 4096 + [700] + [0] * 2048,
    "one": [30000],
    "tile_ends": [2047, 2047, 1023, 1023, 2046, 0, 2047],
    "mixed": None,
}


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("shape", sorted(SHAPES))
def test_merge_row_lengths(cuda_device, shape, dtype):
    rng = np.random.default_rng(len(shape))
    lens = SHAPES[shape]
    if lens is None:
        lens = np.minimum((2.0 * rng.random(6000) ** -0.9).astype(int), 9000).tolist()
    n = 31000
    rp = np.concatenate([[0], np.cumsum(lens)]).astype(np.int32)
    ci = rng.integers(0, n, size=rp[-1]).astype(np.int32)
    va = rng.standard_normal(rp[-1]).astype(dtype)
    half = len(lens) // 2  # two ranks: the second's first tile starts mid-table
    cut = [0, half, len(lens)]
    comm = S.Comm(size=2, device=0)
    blocks = [((rp[a:b + 1] - rp[a]).astype(np.int32), ci[rp[a]:rp[b]], va[rp[a]:rp[b]])
              for a, b in zip(cut[:-1], cut[1:])]
    M = S.Matrix(comm, blocks, None, None, ncols=[n, n])
    M.set_kernel("merge")
    xs = [rng.standard_normal(n).astype(dtype) for _ in range(2)]
    xd = [torch.from_numpy(x).cuda() for x in xs]
    ys = [y.cpu().numpy() for y in M.mult(xd)]
    again = [y.cpu().numpy() for y in M.mult(xd)]
    # FP32: a pairwise-like sum of up to 30000 terms stays within 2e-5 of |A||x|
    # (30000 eps / 2 = 9e-4 would be the serial worst case; each partial sum here
    # has at most 2048 / 256 + 8 + 15 terms in sequence).
    tol = TOL_F64 if dtype == np.float64 else TOL_F32
    for q in range(2):
        assert np.array_equal(ys[q], again[q])
        a = (blocks[q][0], blocks[q][1], np.abs(blocks[q][2]))
        ref = oracle.csr_mult(*[v.astype(np.float64) if i == 2 else v
                                for i, v in enumerate(blocks[q])], xs[q].astype(np.float64))
        bound = oracle.csr_mult(a[0], a[1], a[2].astype(np.float64),
                                np.abs(xs[q]).astype(np.float64))
        assert_spmv_close(ys[q], ref, bound, tol)
