"""Workloads for timing the framework through its public entry points.

Sizes follow the repository's own configurations: the 64 x 64 Laplacian, the
biharmonic smoothing system on a jittered tet cube of up to 70^3 vertices
(alpha = 1e-4, FSAI widths 8 and 48, growth steps 1 and 2, factors in float64,
float32 and bfloat16), the 3 x 3 block coupling on up to 64^3 nodes, many
right-hand sides in one batched solve, and the lifted first-order system under
GMRES.  Inputs are synthetic, made from a seed alone.

``listed()`` gives the cases, ``draw(rng)`` one more of the same ranges,
``prepare(case, seed)`` what a program holds before the call, ``run(state)``
one pass, ``work(case)`` the bytes and operations of a pass, and
``exact(case, seed)`` the result in plain 64-bit torch where it has one.
"""

from __future__ import annotations

import itertools
import math

import torch

import warp_preconditioners_gb300 as wp
from warp_preconditioners_gb300 import batched, linear, sparse
from warp_preconditioners_gb300.biharmonic import BiharmonicSystem

ALPHA = 1.0e-4
DEV = "cuda"


# ---------------------------------------------------------------------------
# Problems.

def _rng(seed):
    return torch.Generator().manual_seed(int(seed) * 7919 + 17)


def _uniform(shape, gen):
    return (torch.rand(shape, generator=gen, dtype=torch.float64) * 2.0 - 1.0).to(DEV)


def _csr(n, cols, vals, keep):
    """CSR from [n, k] candidate columns (ascending) and values, where keep."""
    off = torch.zeros(n + 1, dtype=torch.int64, device=cols.device)
    off[1:] = torch.cumsum(keep.sum(1), 0)
    return sparse.BsrMatrix(n, n, (1, 1), off.to(torch.int32), cols[keep].to(torch.int32),
                            vals[keep].contiguous())


def _grid_laplacian(side, dim):
    """5-point / 7-point Dirichlet Laplacian, unscaled (2 dim on the diagonal, -1 off it)."""
    n = side ** dim
    i = torch.arange(n, device=DEV)
    coord = [(i // side ** a) % side for a in range(dim)]
    cols, vals, keep = [], [], []
    for a in reversed(range(dim)):
        cols.append(i - side ** a)
        keep.append(coord[a] > 0)
        vals.append(-torch.ones(n, dtype=torch.float64, device=DEV))
    cols.append(i)
    keep.append(torch.ones(n, dtype=torch.bool, device=DEV))
    vals.append(torch.full((n,), 2.0 * dim, dtype=torch.float64, device=DEV))
    for a in range(dim):
        cols.append(i + side ** a)
        keep.append(coord[a] < side - 1)
        vals.append(-torch.ones(n, dtype=torch.float64, device=DEV))
    return _csr(n, torch.stack(cols, 1), torch.stack(vals, 1), torch.stack(keep, 1))


def _tet_cube(side, gen, jitter=0.2):
    """Vertices, P1 stiffness K and lumped mass of a cube of side^3 vertices,
    every hex split into six tets, interior vertices jittered."""
    h = 1.0 / (side - 1)
    g = torch.arange(side, dtype=torch.float64) * h
    z, y, x = torch.meshgrid(g, g, g, indexing="ij")
    verts = torch.stack([x, y, z], dim=-1)
    inner = slice(1, side - 1)
    m = max(side - 2, 0)
    verts[inner, inner, inner] += (torch.rand((m, m, m, 3), generator=gen, dtype=torch.float64)
                                   * 2.0 - 1.0) * (jitter * h)
    verts = verts.to(DEV)
    e = side - 1

    def at(t, p):  # the corner p = (dx, dy, dz) of every cell
        return t[p[2]:p[2] + e, p[1]:p[1] + e, p[0]:p[0] + e]

    offsets = [p for p in itertools.product((0, 1), repeat=3) if any(p)]
    st = {p: torch.zeros((side, side, side), dtype=torch.float64, device=DEV) for p in offsets}
    diag = torch.zeros((side, side, side), dtype=torch.float64, device=DEV)
    mass = torch.zeros_like(diag)
    for perm in itertools.permutations(range(3)):
        path, step = [(0, 0, 0)], [0, 0, 0]
        for axis in perm:
            step[axis] = 1
            path.append(tuple(step))
        p = [at(verts, q) for q in path]
        e1, e2, e3 = p[1] - p[0], p[2] - p[0], p[3] - p[0]
        c = [None, torch.linalg.cross(e2, e3), torch.linalg.cross(e3, e1),
             torch.linalg.cross(e1, e2)]
        det = (e1 * c[1]).sum(-1)
        vol = det.abs() / 6.0
        grad = [None] + [q / det[..., None] for q in c[1:]]
        grad[0] = -(grad[1] + grad[2] + grad[3])
        for a in range(4):
            at(mass, path[a]).add_(vol / 4.0)
            at(diag, path[a]).add_(vol * (grad[a] * grad[a]).sum(-1))
            for b in range(a + 1, 4):
                d = tuple(path[b][k] - path[a][k] for k in range(3))
                at(st[d], path[a]).add_(vol * (grad[a] * grad[b]).sum(-1))
    n = side ** 3
    i = torch.arange(n, device=DEV)
    lin = {p: p[0] + p[1] * side + p[2] * side * side for p in offsets}
    order = sorted(offsets, key=lambda p: lin[p])
    zc, yc, xc = i // (side * side), (i // side) % side, i % side
    tiny = 1e-13 * max([float(diag.abs().max())] + [float(s.abs().max()) for s in st.values()])
    cols, vals, keep = [], [], []
    for p in reversed(order):  # columns below the row
        ok = (xc >= p[0]) & (yc >= p[1]) & (zc >= p[2])
        v = st[p].reshape(-1)[(i - lin[p]).clamp(min=0)]
        cols.append(i - lin[p])
        vals.append(v)
        keep.append(ok & (v.abs() > tiny))
    cols.append(i)
    vals.append(diag.reshape(-1))
    keep.append(torch.ones(n, dtype=torch.bool, device=DEV))
    for p in order:
        ok = (xc + p[0] < side) & (yc + p[1] < side) & (zc + p[2] < side)
        v = st[p].reshape(-1)
        cols.append(i + lin[p])
        vals.append(v)
        keep.append(ok & (v.abs() > tiny))
    K = _csr(n, torch.stack(cols, 1), torch.stack(vals, 1), torch.stack(keep, 1))
    return verts.reshape(n, 3), K, mass.reshape(-1).contiguous()


def _biharmonic(side, gen):
    """(vertices, K, mass, Q = alpha M + K M^-1 K) of the smoothing system."""
    verts, K, mass = _tet_cube(side, gen)
    return verts, K, mass, sparse.spgemm(K, K, 1.0 / mass, ALPHA * mass)


def _smoothing_rhs(verts, mass, gen):
    a = 0.5 + torch.rand(3, generator=gen, dtype=torch.float64).to(DEV)
    x, y, z = verts[:, 0], verts[:, 1], verts[:, 2]
    return ALPHA * mass * (a[0] * torch.sin(3 * x) + a[1] * torch.cos(2 * y) * z + a[2] * x * z)


def _matrix(problem, side, gen):
    if problem == "tet":
        return _biharmonic(side, gen)[3]
    A = _grid_laplacian(side, 2 if problem == "lap2d" else 3)
    # A symmetric diagonal scaling of up to 10% makes seeds differ.
    s = 1.0 + 0.1 * _uniform((A.nrow,), gen)
    rows = torch.repeat_interleave(torch.arange(A.nrow, device=DEV),
                                   (A.offsets[1:] - A.offsets[:-1]).to(torch.int64))
    A.values = A.values * (s[rows] * s[A.columns.to(torch.int64)])
    return A


def _coupling(side, gen, kappa=1e-6):
    """K (x) C as 3 x 3 blocks: K the 7-point Laplacian, C a rotated diag(1, 1, kappa)."""
    K = _grid_laplacian(side, 3)
    q, r = torch.linalg.qr(torch.randn((3, 3), generator=gen, dtype=torch.float64))
    q = q * torch.sign(torch.diagonal(r))[None, :]
    C = (q @ torch.diag(torch.tensor([1.0, 1.0, kappa], dtype=torch.float64)) @ q.T)
    C = ((C + C.T) * 0.5).to(DEV)
    blocks = (K.values[:, None, None] * C[None, :, :]).contiguous()
    return sparse.BsrMatrix(K.nrow, K.ncol, (3, 3), K.offsets, K.columns, blocks), C


_STORE = {"f64": {}, "f32": {"factor_dtype": torch.float32},
          "bf16": {"factor_dtype": torch.bfloat16, "apply_dtype": torch.float32}}


def _fsai(A, case, **more):
    return wp.FSAI(A, max_row_size=case["width"], max_step_size=case.get("step", 1),
                   kap_tolerance=1.0e-3, **_STORE[case.get("store", "f64")], **more)


# ---------------------------------------------------------------------------
# Cases.

def listed():
    return [
        # Preconditioner of the small plain configuration, as a user's own loop
        # applies it: all launch latency.
        {"name": "apply-lap2d-64-w8", "kind": "apply", "problem": "lap2d", "side": 64, "width": 8,
         "step": 1, "store": "f64"},
        # The same on the smoothing system at its full size.
        {"name": "apply-tet-70-w8", "kind": "apply", "problem": "tet", "side": 70, "width": 8,
         "step": 1, "store": "f64"},
        # The wide factor in its low-precision storage, at a ragged size.
        {"name": "apply-tet-53-w48-bf16", "kind": "apply", "problem": "tet", "side": 53,
         "width": 48, "step": 2, "store": "bf16"},
        # The factored operator alpha M + K M^-1 K of the smoothing system.
        {"name": "operator-tet-70", "kind": "operator", "side": 70, "dtype": "f64", "free": "all"},
        # Preconditioner setup of the smoothing system, and of its wide option.
        {"name": "setup-tet-70-w8", "kind": "setup", "problem": "tet", "side": 70, "width": 8,
         "step": 1, "store": "f64"},
        {"name": "setup-tet-45-w48", "kind": "setup", "problem": "tet", "side": 45, "width": 48,
         "step": 2, "store": "f64"},
        # New values on the same mesh: the factor refitted in place.
        {"name": "update-tet-57-w8", "kind": "update", "side": 57, "width": 8, "step": 1},
        # The small plain configuration whole: setup and solve of a new system.
        {"name": "solve-lap2d-64-w8", "kind": "solve", "problem": "lap2d", "side": 64, "width": 8,
         "step": 1},
        # One smoothing solve at full size, the headline's unit.
        {"name": "cg-tet-70-w8", "kind": "cg", "side": 70, "width": 8, "step": 1},
        # Block coupling: block ILU(0) with three sweeps, setup and solve.
        {"name": "blockilu-64", "kind": "blockilu", "side": 64},
        # Many right-hand sides of one system in one batched solve.
        {"name": "batched-tet-33-k32", "kind": "batched", "side": 33, "width": 8, "step": 1,
         "k": 32},
        # The lifted nonsymmetric system: two GMRES(31) cycles.
        {"name": "gmres-tet-40", "kind": "gmres", "side": 40, "width": 8, "steps": 62},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["apply", "apply", "operator", "setup", "setup", "update", "solve", "cg",
                       "blockilu", "batched", "batched", "gmres"])
    width, step = rng.choice([(4, 1), (8, 1), (8, 1), (8, 2), (16, 1), (48, 1), (48, 2)])
    if kind in ("apply", "setup"):
        problem = rng.choice(["lap2d", "lap3d", "tet", "tet"])
        top = {"lap2d": 500, "lap3d": 63, "tet": 70 if width <= 16 or kind == "apply" else 45}
        return {"kind": kind, "problem": problem, "side": _log(rng, 8, top[problem]),
                "width": width, "step": step, "store": rng.choice(["f64", "f64", "f32", "bf16"])}
    if kind == "operator":
        return {"kind": kind, "side": _log(rng, 6, 70), "dtype": rng.choice(["f64", "f64", "f32"]),
                "free": rng.choice(["all", "interior"])}
    if kind == "update":
        return {"kind": kind, "side": _log(rng, 8, 70 if width <= 16 else 45), "width": width,
                "step": step}
    if kind == "solve":
        problem = rng.choice(["lap2d", "lap3d"])
        return {"kind": kind, "problem": problem,
                "side": _log(rng, 8, 200 if problem == "lap2d" else 63), "width": min(width, 16),
                "step": step}
    if kind == "cg":
        return {"kind": kind, "side": _log(rng, 10, 60), "width": width, "step": step}
    if kind == "blockilu":
        return {"kind": kind, "side": _log(rng, 6, 64)}
    if kind == "batched":
        return {"kind": kind, "side": _log(rng, 8, 32), "width": min(width, 16), "step": step,
                "k": rng.choice([1, 2, 3, 4, 5, 7, 8, 12, 16, 19, 31, 32])}
    return {"kind": kind, "side": _log(rng, 6, 40), "width": min(width, 16),
            "steps": rng.randint(5, 62)}


def prepare(case, seed):
    kind, side, gen = case["kind"], case["side"], _rng(seed)
    s = {"kind": kind, "case": case}
    if kind == "apply":
        A = _matrix(case["problem"], side, gen)
        s["op"] = _fsai(A, case)
        s["x"] = _uniform((A.nrow,), gen)
        s["z"] = torch.empty_like(s["x"])
    elif kind == "operator":
        K, mass, free, x = _operator_inputs(case, gen)
        s["op"] = wp.SquaredLaplacianOperator(K, mass, free, mass_weight=ALPHA)
        s["x"] = x
        s["z"] = torch.empty_like(x)
    elif kind == "setup":
        s["A"] = _matrix(case["problem"], side, gen)
        s["out"] = _buffers(case, s["A"].nrow)
    elif kind == "update":
        _, K, mass, Q = _biharmonic(side, gen)
        # The same topology with other values: the mass term doubled.
        rows = torch.repeat_interleave(torch.arange(Q.nrow, device=DEV),
                                       (Q.offsets[1:] - Q.offsets[:-1]).to(torch.int64))
        more = torch.where(rows == Q.columns, ALPHA * mass[rows], torch.zeros_like(Q.values))
        s["A"] = sparse.BsrMatrix(Q.nrow, Q.ncol, (1, 1), Q.offsets, Q.columns, Q.values + more)
        s["op"] = _fsai(Q, case, reuse_pattern=True)
        s["out"] = _buffers(case, Q.nrow)
    elif kind == "solve":
        s["A"] = _matrix(case["problem"], side, gen)
        s["b"] = _uniform((s["A"].nrow,), gen)
        s["x"] = torch.empty_like(s["b"])
    elif kind == "cg":
        verts, K, mass, Q = _biharmonic(side, gen)
        free = torch.arange(K.nrow, dtype=torch.int32, device=DEV)
        s["A"] = wp.SquaredLaplacianOperator(K, mass, free, mass_weight=ALPHA)
        s["M"] = _fsai(Q, case)
        s["b"] = _smoothing_rhs(verts, mass, gen)
        s["x"] = torch.empty_like(s["b"])
    elif kind == "blockilu":
        s["A"], _ = _coupling(side, gen)
        s["b"] = _uniform((3 * s["A"].nrow,), gen)
        s["x"] = torch.empty_like(s["b"])
    elif kind == "batched":
        _, K, mass, Q = _biharmonic(side, gen)
        s["op"] = batched.BatchedSolver(K, mass, ALPHA, _fsai(Q, case))
        s["b"] = mass[:, None] * _uniform((K.nrow, case["k"]), gen)
        s["x"] = torch.empty_like(s["b"])
    else:
        _, K, mass = _tet_cube(side, gen)
        tau = 1.0 / ALPHA
        system = BiharmonicSystem(K, mass, tau)
        s["A"] = linear.aslinearoperator(system.matrix)
        s["M"] = system.preconditioner(max_row_size=case["width"])
        s["b"] = system.rhs(mass * _uniform((K.nrow,), gen)).reshape(-1).contiguous()
        s["x"] = torch.empty_like(s["b"])
    return s


def _operator_inputs(case, gen):
    side = case["side"]
    _, K, mass = _tet_cube(side, gen)
    n = K.nrow
    i = torch.arange(n, device=DEV)
    if case["free"] == "interior":
        inside = torch.ones(n, dtype=torch.bool, device=DEV)
        for a in range(3):
            c = (i // side ** a) % side
            inside &= (c > 0) & (c < side - 1)
        i = i[inside]
    x = _uniform((i.numel(),), gen)
    if case["dtype"] == "f32":
        K = sparse.bsr_copy(K, scalar_type=torch.float32)
        mass, x = mass.float(), x.float()
    return K, mass, i.to(torch.int32), x


def _kept(s, name, t):
    """A factor's array in the buffer that a program keeps for it: the number
    of entries depends on the values, the buffer has room for full rows."""
    s["out"][name][:t.numel()].copy_(t.reshape(-1))
    return s["out"][name]


def _buffers(case, n):
    size, val = n * case["width"], {"f64": torch.float64, "f32": torch.float32,
                                    "bf16": torch.bfloat16}[case.get("store", "f64")]
    return {name: torch.zeros(size, dtype=torch.int32 if "columns" in name else val, device=DEV)
            for name in ("columns", "values", "t_columns", "t_values")}


def run(s):
    kind, case = s["kind"], s["case"]
    if kind in ("apply", "operator"):
        s["op"].matvec(s["x"], s["z"], s["z"], 1.0, 0.0)
        return s["z"]
    if kind == "setup":
        M = _fsai(s["A"], case)
        return {"offsets": M.G.offsets, "columns": _kept(s, "columns", M.G.columns),
                "values": _kept(s, "values", M.G.values), "t_offsets": M.GT.offsets,
                "t_columns": _kept(s, "t_columns", M.GT.columns),
                "t_values": _kept(s, "t_values", M.GT.values), "scale": M.scale,
                "truncated": M.truncated_rows}
    if kind == "update":
        M = s["op"].update(s["A"])
        return {"values": _kept(s, "values", M.G.values),
                "t_values": _kept(s, "t_values", M.GT.values)}
    if kind == "gmres":
        s["x"].zero_()
        linear.gmres(s["A"], s["b"], s["x"], tol=1e-14, restart=31, maxiter=case["steps"],
                     M=s["M"], check_every=0)
        return s["x"]
    s["x"].zero_()
    if kind == "batched":
        s["op"].solve(s["b"], s["x"], tol=1e-8)
        return s["x"]
    if kind == "solve":
        M = _fsai(s["A"], case)
    elif kind == "blockilu":
        M = wp.BlockILU0(s["A"], factor_sweeps=3, solve_sweeps=3)
    else:
        M = s["M"]
    # The solution alone: the count and the recursive residual at which a long
    # solve stops move with the rounding of any sum on the way.
    linear.cg(s["A"], s["b"], s["x"], tol=1e-8, M=M, check_every=0)
    return s["x"]


# ---------------------------------------------------------------------------
# Work of a pass.

def _size(case):
    """(rows, entries of the operator A, entries of the matrix FSAI is built on)."""
    side, problem = case["side"], case.get("problem", "tet")
    if problem == "lap2d":
        return side ** 2, 5 * side ** 2 - 4 * side, 5 * side ** 2 - 4 * side
    if problem == "lap3d":
        return side ** 3, 7 * side ** 3 - 6 * side ** 2, 7 * side ** 3 - 6 * side ** 2
    m = side - 1
    k = side ** 3 + 2 * (3 * side * side * m + 3 * side * m * m + m ** 3)
    return side ** 3, k, 62 * side ** 3


def _factor_row(case):
    """Entries of a row of G: the width, or what the energy test keeps of it."""
    top = {"tet": {8: 8.0, 16: 14.0, 48: 25.4 if case.get("step", 1) == 1 else 37.0}}
    row = top.get(case.get("problem", "tet"), {}).get(case["width"], float(case["width"]))
    return min(row, 12.0) if case.get("problem", "tet") != "tet" else row


def work(case):
    kind = case["kind"]
    if kind == "blockilu":
        n = case["side"] ** 3
        nb = 7 * n
        its = 9.0 + 1.45 * case["side"]
        # The product, three lower and three upper sweeps, and the vectors.
        apply = nb * 9 * 2 + 3 * nb * 9 * 2
        return {"bytes": its * (2 * nb * 76 + 9 * 3 * n * 8) + nb * 76 * 2,
                "flops": its * apply + 3 * nb * 27 * 2 * 3}
    n, nnz, nnz_q = _size(case)
    if kind == "operator":
        v = 8 if case["dtype"] == "f64" else 4
        return {"bytes": nnz * (v + 4) + 4 * n + 3 * n * v, "flops": 4 * nnz + 3 * n}
    g = n * _factor_row(case)
    val = {"f64": 8, "f32": 4, "bf16": 2}[case.get("store", "f64")]
    if kind == "apply":
        return {"bytes": 2 * g * (val + 4) + 8 * n + 2 * n * 8, "flops": 4 * g}
    setup = {"bytes": nnz_q * 12 + 4 * n + 2 * g * (val + 4) + 16 * n,
             "flops": n * 11768.0 * (_factor_row(case) / 8.0) ** 2.8}
    if kind == "setup":
        return setup
    if kind == "update":
        row = _factor_row(case)
        return {"bytes": nnz_q * 12 + 4 * n + 4 * g * 12 + 16 * n,
                "flops": n * (row ** 3 / 3.0 + 2 * row ** 2)}
    iteration = {"bytes": nnz * 12 + 2 * g * 12 + 12 * n + 9 * n * 8, "flops": 4 * g + 12 * n}
    if kind == "solve":
        its = 8.0 + case["side"] if case["problem"] == "lap2d" else 12.0 + 1.35 * case["side"]
        return {"bytes": setup["bytes"] + its * iteration["bytes"],
                "flops": setup["flops"] + its * (iteration["flops"] + 2 * nnz)}
    if kind == "cg":
        its = 6950.0 * (case["side"] / 70.0) ** 2 * (8.0 / _factor_row(case)) ** 0.55
        return {"bytes": its * iteration["bytes"], "flops": its * (iteration["flops"] + 4 * nnz)}
    if kind == "batched":
        its = 6950.0 * (case["side"] / 70.0) ** 2 * (8.0 / _factor_row(case)) ** 0.55
        k = case["k"]
        return {"bytes": its * (nnz * 12 + 2 * g * 12 + 12 * n + 9 * n * 8 * k),
                "flops": its * k * (iteration["flops"] + 4 * nnz)}
    steps = case["steps"]  # the lifted operator, both factors, and two passes over the basis
    basis = min(steps, 31) / 2.0
    return {"bytes": steps * (nnz * 36 + 2 * g * 12 + 2 * basis * 2 * n * 8),
            "flops": steps * (4 * nnz + 8 * g + 8 * basis * 2 * n)}


# ---------------------------------------------------------------------------
# Results in 64 bits.

def _product(off, col, val, x):
    m = torch.sparse_csr_tensor(off.to(torch.int64), col.to(torch.int64), val.double(),
                                size=(off.numel() - 1, x.numel()))
    return m @ x.double()


def _poisson(side, dim, b):
    """The grid Laplacian's inverse by its sine eigenvectors; b: [side^dim, m]."""
    k = torch.arange(1, side + 1, dtype=torch.float64, device=DEV)
    S = math.sqrt(2.0 / (side + 1)) * torch.sin(math.pi / (side + 1) * k[:, None] * k[None, :])
    lam = 2.0 - 2.0 * torch.cos(math.pi / (side + 1) * k)
    t = b.reshape([side] * dim + [-1])
    total = torch.zeros([side] * dim, dtype=torch.float64, device=DEV)
    for a in range(dim):
        t = torch.movedim(torch.tensordot(S, t, dims=([1], [a])), 0, a)
        total = total + lam.reshape([-1 if q == a else 1 for q in range(dim)])
    t = t / total[..., None]
    for a in range(dim):
        t = torch.movedim(torch.tensordot(S, t, dims=([1], [a])), 0, a)
    return t.reshape(side ** dim, -1)


def exact(case, seed):
    kind, side, gen = case["kind"], case["side"], _rng(seed)
    if kind == "operator":
        K, mass, free, x = _operator_inputs(case, gen)
        full = torch.zeros(K.nrow, dtype=torch.float64, device=DEV)
        i = free.to(torch.int64)
        full[i] = x.double()
        t = _product(K.offsets, K.columns, K.values, full) / mass.double()
        z = _product(K.offsets, K.columns, K.values, t) + ALPHA * mass.double() * full
        return z[i]
    if kind == "solve":
        dim = 2 if case["problem"] == "lap2d" else 3
        n = side ** dim
        s = 1.0 + 0.1 * _uniform((n,), gen)  # as _matrix draws it
        b = _uniform((n,), gen)
        return _poisson(side, dim, (b / s)[:, None])[:, 0] / s
    if kind == "blockilu":
        _, C = _coupling(side, gen)
        b = _uniform((3 * side ** 3,), gen).reshape(-1, 3)
        return torch.linalg.solve(C, _poisson(side, 3, b).T).T.reshape(-1)
    # The adaptive factors have no closed form, and the smoothing systems no
    # direct solution at these sizes in reasonable time.
    return None
