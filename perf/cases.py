"""Performance cases of spmv_b200: what a user's program has it do, called
through the public entry points, over the range of sizes, types and options
the library is used with.

A case is a dict of plain values; `prepare` builds what a program holds before
the call (matrices, maps, right-hand sides, all from the seed), `run` makes one
pass, `work` states the bytes and operations the pass cannot do without, and
`exact` gives the same outputs in 64 bits from plain torch.

Kinds:

  product    L2GMap.update + Matrix.mult on every rank (an explicit operator
             application, a residual, a time step)
  restrict   Matrix.transpmult + L2GMap.reverse_update (a restriction, an
             adjoint operator, an assembly of contributions)
  block      Matrix.mult_block: several vectors at once
  cg         cg: one symmetric positive definite solve
  mixed      cg_mixed: the same with FP32 inner iterations
  cgblock    cg_block: several right-hand sides of one matrix
  batch      Batch.solve: many small systems (and a block) in one call
  gradient   spd_solve forward and backward: gradients through a solve

Matrices: weighted stencils (5-, 7- and 27-point), the k-nearest-neighbour
graph of jittered points (an unstructured mesh's row lengths and numbering)
and rows with a power-law length (a network's adjacency).
"""
import math

import numpy as np
import torch

import spmv_b200 as S
from spmv_b200 import autograd, core

_TORCH = {"float64": torch.float64, "float32": torch.float32, "complex64": torch.complex64,
          "complex128": torch.complex128}
_ITEM = {"float64": 8, "float32": 4, "complex64": 8, "complex128": 16}


def listed():
    return [
        # A small operator split over four ranks (a coarse grid, an inner step
        # of a time loop): the cost of the two calls themselves.
        {"name": "product_small_2d", "kind": "product", "matrix": "grid5", "nx": 96, "ny": 90,
         "nz": 1, "ranks": 4, "dtype": "float64", "tuned": False},
        # The benchmark's operator: 7-point stencil on 128^3 over eight ranks.
        {"name": "product_3d", "kind": "product", "matrix": "grid7", "nx": 128, "ny": 128,
         "nz": 128, "ranks": 8, "dtype": "float64", "tuned": False},
        # Single precision 27-point stencil, product kernel autotuned once by
        # the program, odd extents.
        {"name": "product_27pt_f32", "kind": "product", "matrix": "grid27", "nx": 101,
         "ny": 95, "nz": 97, "ranks": 1, "dtype": "float32", "tuned": True},
        # An unstructured mesh: uneven rows, numbering with partial locality.
        {"name": "product_mesh", "kind": "product", "matrix": "mesh", "nx": 83, "ny": 79,
         "nz": 71, "ranks": 2, "dtype": "float64", "tuned": False},
        # A network: a few rows with thousands of entries, most with a few.
        {"name": "product_network", "kind": "product", "matrix": "network", "nx": 300007,
         "ny": 1, "nz": 1, "ranks": 1, "dtype": "float64", "tuned": False},
        # The transposed operator with its scatter-add, complex (a wave
        # problem's adjoint), ragged ranks.
        {"name": "restrict_complex", "kind": "restrict", "matrix": "grid7", "nx": 75,
         "ny": 71, "nz": 83, "ranks": 6, "dtype": "complex128", "tuned": False},
        # Sixteen vectors at once (subspace iteration, several load cases).
        {"name": "block_product", "kind": "block", "matrix": "grid7", "nx": 96, "ny": 96,
         "nz": 96, "ranks": 4, "dtype": "float64", "tuned": False, "rhs": 16},
        # The benchmark's solve: diffusion on 128^3 over eight ranks.
        {"name": "solve_3d", "kind": "cg", "matrix": "grid7", "nx": 128, "ny": 128, "nz": 128,
         "ranks": 8, "dtype": "float64", "tuned": False},
        # FP32 inner iterations on a 27-point graph Laplacian.
        {"name": "solve_mixed_27pt", "kind": "mixed", "matrix": "grid27", "nx": 96, "ny": 96,
         "nz": 96, "ranks": 1, "dtype": "float64", "tuned": False},
        # Eight right-hand sides of one matrix.
        {"name": "solve_block", "kind": "cgblock", "matrix": "grid7", "nx": 64, "ny": 64,
         "nz": 61, "ranks": 4, "dtype": "float64", "tuned": False, "rhs": 8},
        # Many small systems of uneven size with a 16-column block on one.
        {"name": "solve_batch", "kind": "batch", "systems": 24, "smallest": 2048,
         "largest": 24000, "rhs": 16, "precision": "mixed"},
        # Gradients of a loss through a solve on the 1024^2 grid graph.
        {"name": "gradient_2d", "kind": "gradient", "matrix": "grid5", "nx": 1024, "ny": 1024,
         "nz": 1, "ranks": 1, "dtype": "float64", "tuned": False},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["product", "product", "product", "restrict", "block", "cg", "cg",
                       "mixed", "cgblock", "batch", "gradient"])
    if kind == "batch":
        lo = _log(rng, 500, 4000)
        return {"kind": "batch", "systems": rng.randint(4, 24), "smallest": lo,
                "largest": _log(rng, lo, 24000), "rhs": rng.choice([0, 0, 5, 16, 32]),
                "precision": rng.choice(["mixed", "mixed", "fp64"])}
    c = {"kind": kind, "ranks": rng.choice([1, 1, 2, 4, 7, 8]), "dtype": "float64",
         "tuned": False}
    if kind in ("product", "restrict", "block"):
        c["matrix"] = rng.choice(["grid5", "grid7", "grid7", "grid27", "mesh", "network"])
    elif kind == "gradient":
        c["matrix"], c["ranks"] = "grid5", 1
    elif kind == "mixed":
        c["matrix"] = rng.choice(["grid7", "grid27", "grid27"])
    else:
        c["matrix"] = rng.choice(["grid5", "grid7", "grid7", "grid27", "mesh"])
    if kind in ("product", "restrict"):
        c["dtype"] = rng.choice(["float64", "float64", "float32", "complex128", "complex64"])
        c["tuned"] = kind == "product" and rng.random() < 0.3
    elif kind == "block":
        c["dtype"] = rng.choice(["float64", "float64", "float32"])
    if kind in ("block", "cgblock"):
        c["rhs"] = rng.choice([2, 3, 4, 8, 12, 16, 32])
    # Rows: from a few thousand up to the listed cases' largest, less where a
    # row or a vector has more to move.
    top = {"grid5": 1 << 20, "grid7": 1 << 21, "grid27": 900_000, "mesh": 460_000,
           "network": 300_000}[c["matrix"]]
    if kind in ("block", "cgblock"):
        top = min(top, (885_000 if kind == "block" else 250_000) * 8 // c["rhs"])
    rows = _log(rng, 4000, top)
    if c["matrix"] == "network":
        c["nx"], c["ny"], c["nz"] = rows, 1, 1
    elif c["matrix"] == "grid5":
        c["nx"] = max(8, int(math.sqrt(rows) * rng.uniform(0.7, 1.3)))
        c["ny"], c["nz"] = max(8, rows // c["nx"]), 1
    else:
        c["nx"] = max(6, int(rows ** (1 / 3) * rng.uniform(0.8, 1.2)))
        c["ny"] = max(6, int(rows ** (1 / 3) * rng.uniform(0.8, 1.2)))
        c["nz"] = max(6, rows // (c["nx"] * c["ny"]))
    return c


# --------------------------------------------------------------------------
# Inputs (on the GPU, from the seed alone).
# --------------------------------------------------------------------------
def _gen(seed, stream):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed) * 1000 + stream)
    return g


def _normal(seed, stream, shape, dtype=torch.float64):
    return torch.randn(shape, generator=_gen(seed, stream), device="cuda", dtype=dtype)


def _offsets(matrix):
    if matrix == "grid5":
        return [(0, -1, 0), (0, 0, -1), (0, 0, 0), (0, 0, 1), (0, 1, 0)]
    if matrix == "grid7":
        return [(-1, 0, 0), (0, -1, 0), (0, 0, -1), (0, 0, 0), (0, 0, 1), (0, 1, 0), (1, 0, 0)]
    r = (-1, 0, 1)
    return [(a, b, c) for a in r for b in r for c in r]


def _stencil(case, seed):
    """Weighted stencil: a coefficient per node, a coupling per edge (the mean
    of its nodes' coefficients), the diagonal the sum of the node's couplings
    plus a shift; the 7-point operator has fixed (Dirichlet) values outside,
    the others none and a shift that keeps them definite."""
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    n = nx * ny * nz
    coef = torch.exp(0.5 * _normal(seed, 1, n)).view(nz, ny, nx)
    fixed = case["matrix"] == "grid7"
    shift = {"grid5": 1e-3, "grid7": 0.0, "grid27": 1e-2}[case["matrix"]]
    iz = torch.arange(nz, device="cuda").view(nz, 1, 1)
    iy = torch.arange(ny, device="cuda").view(1, ny, 1)
    ix = torch.arange(nx, device="cuda").view(1, 1, nx)
    node = (iz * ny + iy) * nx + ix
    cols, vals, there, diag, at = [], [], [], torch.full_like(coef, shift), None
    for dz, dy, dx in _offsets(case["matrix"]):
        if dz == dy == dx == 0:
            at = len(cols)
            cols.append(node)
            vals.append(diag)
            there.append(torch.ones_like(node, dtype=torch.bool))
            continue
        ok = (((iz + dz >= 0) & (iz + dz < nz)) & ((iy + dy >= 0) & (iy + dy < ny))
              & ((ix + dx >= 0) & (ix + dx < nx)))
        w = 0.5 * (coef + torch.roll(coef, (-dz, -dy, -dx), (0, 1, 2)))
        w = torch.where(ok, w, coef if fixed else torch.zeros_like(coef))
        diag = diag + w
        cols.append(node + (dz * ny + dy) * nx + dx)
        vals.append(-w)
        there.append(ok)
    vals[at] = diag
    there = torch.stack([t.reshape(-1) for t in there], 1)
    cols = torch.stack([t.reshape(-1) for t in cols], 1)[there]
    vals = torch.stack([t.reshape(-1) for t in vals], 1)[there]
    rp = torch.zeros(n + 1, dtype=torch.int64, device="cuda")
    rp[1:] = torch.cumsum(there.sum(1), 0)
    return rp, cols, vals


def _mesh(n3, seed, window=4096, k=12, shift=1e-2):
    """Symmetric k-nearest-neighbour graph Laplacian of points jittered about
    an nx x ny x nz lattice, weights exp(-d^2) times the mean of a coefficient
    at the edge's points, numbered at random within windows of `window` points
    of the lattice order.  The points and their numbering follow from the
    extents (a given mesh), the coefficients from the seed."""
    nx, ny, nz = n3
    n = nx * ny * nz
    i = torch.arange(n, device="cuda")
    lat = torch.stack([i % nx, (i // nx) % ny, i // (nx * ny)], 1)
    pos = lat + 0.9 * torch.rand((n, 3), generator=_gen(0, 2), device="cuda",
                                 dtype=torch.float64)
    r = range(-2, 3)
    off = torch.tensor([(a, b, c) for c in r for b in r for a in r if (a, b, c) != (0, 0, 0)],
                       device="cuda")
    size = torch.tensor([nx, ny, nz], device="cuda")
    near = []
    for s in range(0, n, 65536):
        q = lat[s:s + 65536, None, :] + off[None]
        ok = ((q >= 0) & (q < size)).all(2)
        j = (q[..., 2] * ny + q[..., 1]) * nx + q[..., 0]
        j = torch.where(ok, j, 0)
        d = (pos[j] - pos[s:s + 65536, None, :]).square().sum(2)
        d = torch.where(ok, d, math.inf)
        near.append(torch.gather(j, 1, torch.topk(d, k, 1, largest=False)[1]))
    near = torch.cat(near)
    name = i // window + torch.rand(n, generator=_gen(0, 3), device="cuda",
                                    dtype=torch.float64)
    old = torch.argsort(name)                # new number -> lattice number
    new = torch.empty_like(old)
    new[old] = i
    a, b = new[i[:, None].expand(n, k).reshape(-1)], new[near.reshape(-1)]
    key = torch.unique(torch.cat([a * n + b, b * n + a, i * n + i]))
    rows, cols = key // n, key % n
    rp = torch.zeros(n + 1, dtype=torch.int64, device="cuda")
    rp[1:] = torch.cumsum(torch.bincount(rows, minlength=n), 0)
    coef = torch.exp(0.3 * _normal(seed, 1, n))
    w = torch.exp(-(pos[old[rows]] - pos[old[cols]]).square().sum(1))
    w = w * (0.5 * (coef[rows] + coef[cols]))
    w = torch.where(rows == cols, 0.0, w).cpu().numpy()
    # Row sums on the host, in order (every row has its diagonal entry).
    total = torch.from_numpy(np.add.reduceat(w, rp[:-1].cpu().numpy())).cuda()
    w = torch.from_numpy(w).cuda()
    return rp, cols, torch.where(rows == cols, total[rows] + shift, -w)


def _network(n, seed):
    """Rows with a power-law length (most a few entries, the longest n / 8),
    columns drawn towards the low numbers; the pattern follows from n, the
    values from the seed."""
    u = torch.rand(n, generator=_gen(0, 4), device="cuda", dtype=torch.float64)
    length = torch.clamp(4.0 * u ** -0.7, max=n / 8).to(torch.int64)
    rp = torch.zeros(n + 1, dtype=torch.int64, device="cuda")
    rp[1:] = torch.cumsum(length, 0)
    nnz = int(rp[-1])
    v = torch.rand(nnz, generator=_gen(0, 5), device="cuda", dtype=torch.float64)
    cols = torch.clamp((n * v ** 1.5).to(torch.int64), max=n - 1)
    return rp, cols, _normal(seed, 6, nnz)


def _matrix(case, seed):
    """Global CSR (int64 rowptr and columns, values in the case's type)."""
    if case["matrix"] == "mesh":
        rp, cols, vals = _mesh((case["nx"], case["ny"], case["nz"]), seed)
    elif case["matrix"] == "network":
        rp, cols, vals = _network(case["nx"], seed)
    else:
        rp, cols, vals = _stencil(case, seed)
    if case["dtype"].startswith("complex"):
        vals = torch.complex(vals, 0.3 * _normal(seed, 7, vals.numel()))
    return rp, cols, vals.to(_TORCH[case["dtype"]])


def _ranges(n, P):
    return [n * r // P for r in range(P + 1)]


def _split(case, rp, cols, vals):
    """Row blocks over the ranks: each rank's CSR with owned columns first and
    its ghosts after them, rows sorted by local column."""
    n = rp.numel() - 1
    R = _ranges(n, case["ranks"])
    sizes, ghosts, blocks = [], [], []
    for r0, r1 in zip(R[:-1], R[1:]):
        a, b = int(rp[r0]), int(rp[r1])
        c, v, m = cols[a:b], vals[a:b], r1 - r0
        lens = rp[r0 + 1:r1 + 1] - rp[r0:r1]
        out = (c < r0) | (c >= r1)
        g = torch.unique(c[out])
        loc = torch.where(out, m + torch.searchsorted(g, c), c - r0)
        if g.numel():
            row = torch.repeat_interleave(torch.arange(m, device="cuda"), lens)
            order = torch.argsort(row * (m + g.numel()) + loc, stable=True)
            loc, v = loc[order], v[order]
        sizes.append(m)
        ghosts.append(g.cpu().numpy())
        blocks.append(((rp[r0:r1 + 1] - rp[r0]).to(torch.int32).cpu().numpy(),
                       loc.to(torch.int32).cpu().numpy(), v.cpu().numpy()))
    return sizes, ghosts, blocks


def _vector(case, seed, n, k=None):
    dt = _TORCH[case["dtype"]]
    return _normal(seed, 8, (n,) if k is None else (n, k), dt)


def _systems(case):
    """Extents of the batch's systems: rows spread over [smallest, largest]."""
    ns, lo, hi = case["systems"], case["smallest"], case["largest"]
    out = []
    for s in range(ns):
        n = lo + (hi - lo) * ((s * 7) % ns) / max(1, ns - 1)
        side = max(6, int(n ** (1 / 3)))
        out.append((side, side, max(6, int(n) // (side * side))))
    return out


def prepare(case, seed):
    if case["kind"] == "batch":
        dims = _systems(case)
        mats = [_mesh(d, seed * 100 + s, window=1 << 30) for s, d in enumerate(dims)]
        comm = S.Comm(size=1, device=0)
        B = core.Batch(comm, [(rp.to(torch.int32).cpu().numpy(),
                               c.to(torch.int32).cpu().numpy(), v.cpu().numpy())
                              for rp, c, v in mats],
                       block=(0, case["rhs"]) if case["rhs"] else None)
        b = [_normal(seed, 20 + s, d[0] * d[1] * d[2]) for s, d in enumerate(dims)]
        n0 = dims[0][0] * dims[0][1] * dims[0][2]
        return {"case": case, "comm": comm, "batch": B, "b": b,
                "B": _normal(seed, 19, (n0, case["rhs"])) if case["rhs"] else None}
    rp, cols, vals = _matrix(case, seed)
    n = rp.numel() - 1
    if case["kind"] == "gradient":
        sys_ = autograd.SpdSystem(rp.to(torch.int32).cpu().numpy(),
                                  cols.to(torch.int32).cpu().numpy(), vals.cpu().numpy())
        return {"case": case, "system": sys_, "vals": vals.requires_grad_(True),
                "b": _normal(seed, 8, n).requires_grad_(True), "target": _normal(seed, 9, n)}
    sizes, ghosts, blocks = _split(case, rp, cols, vals)
    comm = S.Comm(size=case["ranks"], device=0)
    cmap = S.L2GMap(comm, sizes, ghosts)
    rmap = S.L2GMap(comm, sizes, [[] for _ in sizes])
    A = S.Matrix(comm, blocks, cmap, rmap)
    if case["tuned"]:
        A.autotune()
    st = {"case": case, "comm": comm, "cmap": cmap, "rmap": rmap, "A": A}
    x = _vector(case, seed, n, case.get("rhs"))
    R = _ranges(n, case["ranks"])
    own = [x[a:b] for a, b in zip(R[:-1], R[1:])]
    if case["kind"] == "product":
        # Owned entries, then room for the ghosts that update brings.
        st["x"] = [torch.cat([v, torch.zeros(len(g), dtype=v.dtype, device="cuda")])
                   for v, g in zip(own, ghosts)]
    elif case["kind"] == "block":
        st["x"] = [torch.cat([v, x[torch.from_numpy(g).cuda()]]) for v, g in zip(own, ghosts)]
    else:
        st["b"] = [v.contiguous() for v in own]
    return st


_RTOL = 1e-12
_MAX_ITS = 20000


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "product":
        state["cmap"].update(state["x"])
        return {"x": state["x"], "y": state["A"].mult(state["x"])}
    if kind == "restrict":
        y = state["A"].transpmult(state["b"])
        state["cmap"].reverse_update(y)
        return {"y": y}
    if kind == "block":
        return {"y": state["A"].mult_block(state["x"])}
    if kind == "cg":
        return {"x": S.cg(state["comm"], state["A"], state["b"], _MAX_ITS, _RTOL)[0]}
    if kind == "mixed":
        return {"x": S.cg_mixed(state["comm"], state["A"], state["b"], _MAX_ITS, _RTOL)[0]}
    if kind == "cgblock":
        return {"x": core.cg_block(state["comm"], state["A"], state["b"], _MAX_ITS, _RTOL)[0]}
    if kind == "batch":
        r = state["batch"].solve(state["b"], _MAX_ITS, _RTOL, block_b=state["B"],
                                 precision=case["precision"])
        return {"x": r[0], "X": r[2] if case["rhs"] else None}
    x = autograd.spd_solve(state["vals"], state["b"], state["system"])
    loss = 0.5 * (x - state["target"]).square().sum()
    gv, gb = torch.autograd.grad(loss, (state["vals"], state["b"]))
    return {"x": x.detach(), "dvals": gv, "db": gb}


# --------------------------------------------------------------------------
# Work.
# --------------------------------------------------------------------------
def _size(case):
    """(rows, nonzeros, ghosts) of the case, near enough."""
    nx, ny, nz, P = case["nx"], case["ny"], case["nz"], case["ranks"]
    n = nx * ny * nz
    if case["matrix"] == "network":
        return n, int(12.5 * n), min(n, int(0.9 * n)) * (P - 1)
    if case["matrix"] == "mesh":
        return n, int(16.3 * n), 4 * nx * ny * (P - 1)
    plane = nx if case["matrix"] == "grid5" else nx * ny
    if case["matrix"] == "grid27":
        return n, (3 * nx - 2) * (3 * ny - 2) * (3 * nz - 2), 2 * plane * (P - 1)
    m = 2 if case["matrix"] == "grid5" else 3
    nnz = (2 * m + 1) * n - 2 * sum(n // e for e in (nx, ny, nz)[:m])
    return n, nnz, 2 * plane * (P - 1)


def _iterations(case):
    """About how many iterations a solve of the case takes (conjugate
    gradients' bound from the condition number, which for the fixed 7-point
    operator grows with the extent and for the others with 1 / shift)."""
    if case.get("matrix") == "grid7":
        return int(8.0 * max(case["nx"], case["ny"], case["nz"]))
    if case.get("matrix") == "grid5":
        return int(min(1500, 5.0 * max(case["nx"], case["ny"])))
    if case.get("matrix") == "grid27":
        return int(min(1000, 9.0 * max(case["nx"], case["ny"], case["nz"])))
    return 350


def work(case):
    kind = case["kind"]
    if kind == "batch":
        n = [a * b * c for a, b, c in _systems(case)]
        rows, k = sum(n), case["rhs"]
        its, s = _iterations(case), 4 if case["precision"] == "mixed" else 8
        # Per iteration: the matrix (the block's system serves all its
        # columns) and nine passes over the vectors.
        nnz = 16.3 * (rows + (n[0] if k else 0))
        return {"bytes": its * (nnz * (s + 2) + 9 * s * (rows + k * n[0])),
                "flops": its * 2 * 16.3 * (rows + k * n[0])}
    n, nnz, g = _size(case)
    s, P = _ITEM[case["dtype"]], case["ranks"]
    fl = 8 if case["dtype"].startswith("complex") else 2
    product = nnz * (s + 4) + 4 * (n + P) + s * (2 * n + g)
    if kind == "product":
        return {"bytes": product + g * (2 * s + 4), "flops": fl * nnz}
    if kind == "restrict":
        return {"bytes": product + g * (3 * s + 4), "flops": fl * nnz}
    if kind == "block":
        k = case["rhs"]
        return {"bytes": nnz * (s + 4) + 4 * (n + P) + k * s * (2 * n + g), "flops": 2 * nnz * k}
    its = _iterations(case)
    if kind == "cg":
        return {"bytes": its * (product + 9 * n * s), "flops": its * (2 * nnz + 10 * n)}
    if kind == "mixed":
        return {"bytes": its * (nnz * 8 + 4 * (n + P) + 11 * n * 4),
                "flops": its * (2 * nnz + 10 * n)}
    if kind == "cgblock":
        k = case["rhs"]
        return {"bytes": its * (nnz * (s + 4) + 4 * (n + P) + 11 * k * n * s),
                "flops": its * k * (2 * nnz + 10 * n)}
    return {"bytes": 2 * its * (product + 9 * n * s) + nnz * (3 * s + 4),
            "flops": 2 * its * (2 * nnz + 10 * n) + 2 * nnz}


# --------------------------------------------------------------------------
# The same outputs in 64 bits from plain torch.
# --------------------------------------------------------------------------
def _rows(rp):
    n = rp.numel() - 1
    return torch.repeat_interleave(torch.arange(n, device="cuda"), rp[1:] - rp[:-1])


def _solve(rp, cols, vals, b, rtol=1e-14, its=40000):
    """Conjugate gradients in 64 bits for one or several right-hand sides,
    restarted once from the true residual."""
    n = rp.numel() - 1
    A = torch.sparse_csr_tensor(rp, cols, vals, (n, n))
    b2 = b if b.dim() == 2 else b[:, None]
    x = torch.zeros_like(b2)
    bb = b2.square().sum(0)
    for _ in range(2):
        r = b2 - A @ x
        p, rr = r.clone(), r.square().sum(0)
        for k in range(its):
            if k % 32 == 0 and bool((rr <= rtol * rtol * bb).all()):
                break
            y = A @ p
            alpha = rr / (p * y).sum(0).clamp_min(1e-300)
            x += alpha * p
            r -= alpha * y
            new = r.square().sum(0)
            p = r + (new / rr.clamp_min(1e-300)) * p
            rr = new
    return x if b.dim() == 2 else x[:, 0]


def exact(case, seed):
    kind = case["kind"]
    if kind == "batch":
        dims = _systems(case)
        mats = [_mesh(d, seed * 100 + s, window=1 << 30) for s, d in enumerate(dims)]
        x = [_solve(*m, _normal(seed, 20 + s, m[0].numel() - 1)) for s, m in enumerate(mats)]
        X = None
        if case["rhs"]:
            X = _solve(*mats[0], _normal(seed, 19, (mats[0][0].numel() - 1, case["rhs"])))
        return {"x": x, "X": X}
    rp, cols, vals = _matrix(case, seed)
    vals = vals.to(torch.complex128 if vals.is_complex() else torch.float64)
    n = rp.numel() - 1
    rows = _rows(rp)
    if kind == "gradient":
        b, target = _normal(seed, 8, n), _normal(seed, 9, n)
        x = _solve(rp, cols, vals, b)
        lam = _solve(rp, cols, vals, x - target)
        return {"x": x, "dvals": -lam[rows] * x[cols], "db": lam}
    x = _vector(case, seed, n, case.get("rhs")).to(vals.dtype)
    R = _ranges(n, case["ranks"])
    cut = list(zip(R[:-1], R[1:]))
    if kind == "product" or kind == "block":
        y = torch.zeros_like(x)
        for s in range(0, rows.numel(), 1 << 22):
            e = slice(s, s + (1 << 22))
            v = vals[e] if x.dim() == 1 else vals[e, None]
            y.index_add_(0, rows[e], v * x[cols[e]])
        out = {"y": [y[a:b] for a, b in cut]}
        if kind == "product":
            ghosts = _split_ghosts(rp, cols, cut)
            out["x"] = [torch.cat([x[a:b], x[g]]) for (a, b), g in zip(cut, ghosts)]
        return out
    if kind == "restrict":
        # Each rank's transposed block, then the ghosts added to their owners.
        out = []
        total = torch.zeros_like(x).index_add_(0, cols, vals * x[rows])
        ghosts = _split_ghosts(rp, cols, cut)
        for (a, b), g in zip(cut, ghosts):
            e = slice(int(rp[a]), int(rp[b]))
            mine = torch.zeros_like(x).index_add_(0, cols[e], vals[e] * x[rows[e]])
            out.append(torch.cat([total[a:b], mine[g]]))
        return {"y": out}
    x = _solve(rp, cols, vals, x)
    # Each rank's solution with its ghost entries zero.
    ghosts = _split_ghosts(rp, cols, cut)
    return {"x": [torch.cat([x[a:b], torch.zeros((len(g),) + tuple(x.shape[1:]),
                                                 dtype=x.dtype, device="cuda")])
                  for (a, b), g in zip(cut, ghosts)]}


def _split_ghosts(rp, cols, cut):
    out = []
    for a, b in cut:
        c = cols[int(rp[a]):int(rp[b])]
        out.append(torch.unique(c[(c < a) | (c >= b)]))
    return out
