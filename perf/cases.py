"""Performance cases of the SPAI + BiCGSTAB path, through its public entry points.

A case is a dict of plain values; ``prepare`` makes what a program holds before
the call (the matrix in CSC form, a right-hand side of a known solution, its
context), ``run`` is the call.  Every right-hand side is b = A x_true with
x_true ~ N(0, 1), so the exact answer of a solve is x_true itself.

Kinds:

* ``solve``    SPAI build + BiCGSTAB on device arrays (``Context.solve_d``)
* ``solve_h``  the same from pinned host buffers (``Context.solve_h_into``)
* ``build``    the preconditioner alone, with its column residuals (``build_d``)
* ``adjoint``  A^T x = b with a preconditioner in hand (``bicgstab_transpose_d``)
* ``grad``     forward and backward through ``spai_solve`` (torch.autograd)
* ``batch``    independent systems x right-hand sides (``batch_solve_d``)
* ``csr``      A's arrays by rows (``csc_to_csr_d``)

Matrices: ``2d`` / ``3d`` upwind convection-diffusion on an m^dim grid,
``varcoef`` variable-coefficient 2D diffusion, ``circuit`` the seeded
circuit-like matrix with hub rows and columns, ``mesh`` a 9-point mesh with a
quarter of its edges missing and unsymmetric values (columns of up to 9
entries, as a finite-element mesh has).

The stopping tolerance is 1e-8 where the iteration is insensitive to rounding,
tighter where it is not (large 2D grids, variable coefficients), so that the
answer, and not the path to it, is what comes back.
"""
import math

import numpy as np
import torch

from dcu_b200 import native as N
from dcu_b200 import workloads as W
from dcu_b200.api import Context
from dcu_b200.autograd import spai_solve

FORMS = {"fp64": N.PREC_FP64, "mixed_fp32": N.PREC_MIXED_FP32, "mixed_bf16": N.PREC_MIXED_BF16,
         "m_fp32": N.PREC_M_FP32, "m_bf16": N.PREC_M_BF16}
MAXITER = 3000


def listed():
    return [
        # the smallest whole solve: every launch and host round trip shows (64 x 64 grid, Pe 10)
        {"name": "solve_2d_64", "kind": "solve", "matrix": "2d", "m": 64, "pe": 10.0, "form": "fp64", "tol": 1e-8},
        # a circuit matrix of the size of the reference's own fixture: hub rows and columns of 200-400 entries
        {"name": "solve_circuit_4510", "kind": "solve", "matrix": "circuit", "n": 4510, "form": "fp64", "tol": 1e-10},
        # an ordinary 2D grid in the plain form, as one step of a time integration solves it
        {"name": "solve_2d_256", "kind": "solve", "matrix": "2d", "m": 256, "pe": 20.0, "form": "fp64", "tol": 1e-12},
        # an unstructured mesh: columns of up to 9 entries, odd size, an FP32 preconditioner
        {"name": "solve_mesh_193", "kind": "solve", "matrix": "mesh", "m": 193, "form": "m_fp32", "tol": 1e-10},
        # the large 3D problem in the plain form
        {"name": "solve_3d_128", "kind": "solve", "matrix": "3d", "m": 128, "pe": 20.0, "form": "fp64", "tol": 1e-8},
        # and in the mixed form that the benchmark reports
        {"name": "solve_3d_128_m_bf16", "kind": "solve", "matrix": "3d", "m": 128, "pe": 20.0, "form": "m_bf16",
         "tol": 1e-8},
        # a caller with host data: upload, solve, download; odd size
        {"name": "solve_h_3d_61", "kind": "solve_h", "matrix": "3d", "m": 61, "pe": 20.0, "form": "mixed_bf16",
         "tol": 1e-8},
        # the preconditioner alone on the mesh, plain form, dynamic schedule
        {"name": "build_mesh_300", "kind": "build", "matrix": "mesh", "m": 300, "form": "fp64", "schedule": 1},
        # the backward pass of a 512 x 512 problem whose forward pass left M behind
        {"name": "adjoint_2d_512", "kind": "adjoint", "matrix": "2d", "m": 512, "pe": 20.0, "form": "fp64",
         "tol": 1e-12},
        # one differentiable solve with random coefficients, forward and backward
        {"name": "grad_varcoef_96", "kind": "grad", "matrix": "varcoef", "m": 96, "form": "fp64", "tol": 1e-13},
        # a batch: 512 systems of 1e3..5e4 unknowns, 8 right-hand sides each
        {"name": "batch_512x8", "kind": "batch", "count": 512, "nrhs": 8, "n_lo": 1000, "n_hi": 50000,
         "tol": 1e-12},
        # a caller that keeps rows for its own products: the conversion alone
        {"name": "csr_mesh_500", "kind": "csr", "matrix": "mesh", "m": 500},
    ]


def draw(rng):
    def logint(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["solve", "solve", "solve", "solve_h", "build", "adjoint", "grad", "batch", "csr"])
    pe = round(rng.uniform(5.0, 50.0), 3)
    if kind == "batch":
        return {"kind": kind, "count": logint(4, 256), "nrhs": rng.choice([1, 2, 4, 8]), "n_lo": 300,
                "n_hi": logint(2000, 50000), "tol": 1e-12}
    if kind == "grad":
        return {"kind": kind, "matrix": "varcoef", "m": logint(24, 110), "form": "fp64", "tol": 1e-13}
    if kind == "adjoint":
        return {"kind": kind, "matrix": "2d", "m": logint(32, 512), "pe": pe, "form": "fp64", "tol": 1e-12}
    if kind == "csr":
        matrix = rng.choice(["mesh", "circuit"])
        return {"kind": kind, "matrix": matrix, **({"m": logint(24, 700)} if matrix == "mesh" else {"n": logint(1500, 6000)})}
    matrix = rng.choice(["2d", "3d", "mesh", "circuit"] if kind == "solve" else ["2d", "3d", "mesh"])
    case = {"kind": kind, "matrix": matrix}
    if matrix == "circuit":
        case["n"] = logint(1500, 6000)
    else:
        case["m"] = logint(24, 512) if matrix == "2d" else logint(10, 128) if matrix == "3d" else logint(24, 360)
        if kind == "solve_h":
            case["m"] = min(case["m"], 72 if matrix == "3d" else 400)
        if matrix != "mesh":
            case["pe"] = pe
    if kind == "build":
        # (an FP32 least-squares build shows through the solves that use it)
        case["form"], case["schedule"] = "fp64", rng.choice([0, 1])
        return case
    # FP32 vectors serve the well-conditioned 3D grids and the mesh
    case["form"] = rng.choice(["fp64", "fp64", "m_fp32", "m_bf16"] +
                              (["mixed_fp32", "mixed_bf16"] if matrix in ("3d", "mesh") else []))
    case["tol"] = {"2d": 1e-12, "3d": 1e-10, "mesh": 1e-10, "circuit": 1e-10}[matrix]
    return case


# ------------------------------------------------------------------ matrices
def _grid_csc(dim, m, pe):
    """(ptr, idx, val) of the upwind convection-diffusion matrix, on the GPU."""
    n = m ** dim
    c = torch.arange(n, device="cuda")
    x = c % m
    steps = [m ** k for k in range(dim - 1, 0, -1)]  # slowest axis first
    rows, vals = [], []

    def put(ok, row, val):
        rows.append(torch.where(ok, row, torch.full_like(row, -1)))
        vals.append(torch.full((n,), val, dtype=torch.float64, device="cuda"))

    for st in steps:
        put((c // st) % m >= 1, c - st, -1.0)
    put(x >= 1, c - 1, -1.0)
    put(x >= 0, c, 2.0 * dim + pe)
    put(x <= m - 2, c + 1, -(1.0 + pe))
    for st in reversed(steps):
        put((c // st) % m <= m - 2, c + st, -1.0)
    rows, vals = torch.stack(rows, 1), torch.stack(vals, 1)
    keep = rows >= 0
    ptr = torch.zeros(n + 1, dtype=torch.int64, device="cuda")
    ptr[1:] = keep.sum(1).cumsum(0)
    return ptr.int(), rows[keep].int(), vals[keep]


def _grid_apply(dim, m, pe, X, transpose=False):
    """A X (or A^T X) of that matrix for X of shape (n, R), every row summed in one fixed order."""
    g = X.reshape([m] * dim + [X.shape[1]])
    y = (2.0 * dim + pe) * g
    up, down = (1.0 + pe, 1.0) if not transpose else (1.0, 1.0 + pe)
    for ax in range(dim):
        a, b = (up, down) if ax == dim - 1 else (1.0, 1.0)
        y.narrow(ax, 1, m - 1).sub_(a * g.narrow(ax, 0, m - 1))
        y.narrow(ax, 0, m - 1).sub_(b * g.narrow(ax, 1, m - 1))
    return y.reshape(X.shape)


def _mesh(m, seed):
    """CSC of an m x m mesh with edges to the 8 neighbours, a quarter of them missing (structurally
    symmetric), unsymmetric values, a_ii = 1.1 x the row's sum of magnitudes."""
    rng = np.random.default_rng(m)  # the mesh by its size, the values by the seed
    n = m * m
    c = np.arange(n)
    x, y = c % m, c // m
    rr, cc = [], []
    for dx, dy in ((1, 0), (-1, 1), (0, 1), (1, 1)):
        ok = (x + dx >= 0) & (x + dx < m) & (y + dy < m) & (rng.random(n) < 0.75)
        a = c[ok]
        b = a + dy * m + dx
        rr += [a, b]
        cc += [b, a]
    R, C = np.concatenate(rr), np.concatenate(cc)
    V = -np.random.default_rng(seed).uniform(0.2, 1.0, len(R))
    diag = 1.1 * np.bincount(R, weights=-V, minlength=n) + 0.1
    R, C, V = np.concatenate([R, c]), np.concatenate([C, c]), np.concatenate([V, diag])
    order = np.argsort(C * n + R)
    ptr = np.concatenate([[0], np.cumsum(np.bincount(C, minlength=n))])
    return W.CSC(n, ptr.astype(np.int32), R[order].astype(np.int32), V[order])


def _host_matrix(case, seed):
    kind = case["matrix"]
    if kind == "mesh":
        return _mesh(case["m"], seed)
    if kind == "circuit":
        return W.circuit_like(n=case["n"], seed=seed, target_nnz=int(case["n"] * 4.7))
    return W.varcoef2d(case["m"], seed=seed, corr=max(4.0, case["m"] / 16))


def _apply(A, x, transpose=False):
    """A x (or A^T x) on the host, in storage order."""
    cols = np.repeat(np.arange(A.n), np.diff(A.ptr))
    r, c = (cols, A.idx) if transpose else (A.idx, cols)
    return np.bincount(r, weights=A.val * x[c], minlength=A.n)


def _normal(seed, *shape):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return torch.randn(*shape, generator=g, device="cuda", dtype=torch.float64)


def _problem(case, seed):
    """(ptr, idx, val, apply) on the GPU; apply(x, transpose) forms A x or A^T x."""
    if case["matrix"] in ("2d", "3d"):
        dim, m, pe = (2 if case["matrix"] == "2d" else 3), case["m"], case["pe"]
        ptr, idx, val = _grid_csc(dim, m, pe)
        return ptr, idx, val, lambda x, transpose=False: _grid_apply(dim, m, pe, x[:, None], transpose)[:, 0].contiguous()
    A = _host_matrix(case, seed)
    dev = [torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in (A.ptr, A.idx, A.val)]
    return (*dev, lambda x, transpose=False: torch.from_numpy(_apply(A, x.cpu().numpy(), transpose)).cuda())


def _batch_shapes(case, seed):
    """(dim, m, Pe) of every system: n log-uniform, half 2D and half 3D (by the batch's size), Pe in
    [0, 50] (by the seed)."""
    rng = np.random.default_rng(case["count"])
    ns = np.exp(rng.uniform(math.log(case["n_lo"]), math.log(case["n_hi"]), case["count"]))
    return [(2, int(round(v ** 0.5)), float(p)) if d else (3, int(round(v ** (1 / 3))), float(p))
            for v, d, p in zip(ns, rng.uniform(size=len(ns)) < 0.5,
                                np.random.default_rng(seed).uniform(0.0, 50.0, len(ns)))]


# ------------------------------------------------------------------ the cases
def prepare(case, seed):
    kind = case["kind"]
    # the caller's own stream: the context orders its work after it and before what follows on it
    stream = torch.cuda.Stream()
    ctx = Context(0)
    ctx.set_stream(stream.cuda_stream)
    s = {"kind": kind, "ctx": ctx, "stream": stream}
    if kind == "batch":
        parts, offs, nnz = [], [0], 0
        shapes = _batch_shapes(case, seed)
        for dim, m, pe in shapes:
            ptr, idx, val = _grid_csc(dim, m, pe)
            parts.append((ptr[:-1] + nnz, idx + offs[-1], val))
            offs.append(offs[-1] + m ** dim)
            nnz += val.numel()
        X = _normal(seed, offs[-1], case["nrhs"])
        s["B"] = torch.cat([_grid_apply(d, m, pe, X[a:b]) for (d, m, pe), a, b in zip(shapes, offs, offs[1:])])
        s["off"] = torch.tensor(offs, dtype=torch.int32, device="cuda")
        s["ptr"] = torch.cat([p[0] for p in parts] + [torch.tensor([nnz], dtype=torch.int32, device="cuda")])
        s["idx"], s["val"] = torch.cat([p[1] for p in parts]), torch.cat([p[2] for p in parts])
        s["n"], s["nnz"] = offs[-1], nnz
        s["opt"] = {"tol": case["tol"], "maxiter": MAXITER}
        torch.cuda.synchronize()
        return s
    ptr, idx, val, apply = _problem(case, seed)
    n, nnz = ptr.numel() - 1, val.numel()
    s.update(n=n, nnz=nnz, ptr=ptr, idx=idx, val=val)
    if kind in ("solve", "solve_h", "adjoint", "grad"):
        s["opt"] = {"precision": FORMS[case["form"]], "tol": case["tol"], "maxiter": MAXITER}
        s["b"] = apply(_normal(seed, n), kind == "adjoint")
    if kind == "solve_h":
        pin = {k: s.pop(k).cpu().pin_memory() for k in ("ptr", "idx", "val", "b")}
        pin["x"] = torch.zeros(n, dtype=torch.float64).pin_memory()
        s["pin"], s["host"] = pin, {k: v.numpy() for k, v in pin.items()}
    elif kind == "build":
        s["opt"] = {"precision": FORMS[case["form"]], "schedule": case["schedule"]}
    elif kind == "adjoint":
        s["mval"] = torch.zeros_like(val)
        torch.cuda.synchronize()
        ctx.build_d(n, nnz, ptr, idx, val, s["mval"], precision=FORMS[case["form"]])
    elif kind == "grad":
        # the incoming gradient of x: g = A^T lambda, so that dL/db = lambda
        s["g"] = apply(_normal(seed + 1, n), True)
        s["val"], s["b"] = val.requires_grad_(True), s["b"].requires_grad_(True)
    torch.cuda.synchronize()
    return s


def run(s):
    kind, ctx = s["kind"], s["ctx"]
    with torch.cuda.stream(s["stream"]):
        if kind == "solve":
            x = torch.zeros_like(s["b"])
            ctx.solve_d(s["n"], s["nnz"], s["ptr"], s["idx"], s["val"], s["b"], x, **s["opt"])
            return x
        if kind == "solve_h":
            h = s["host"]
            h["x"][:] = 0.0
            ctx.solve_h_into(s["n"], s["nnz"], h["ptr"], h["idx"], h["val"], h["b"], h["x"], **s["opt"])
            return h["x"]
        if kind == "build":
            mval = torch.empty_like(s["val"])
            colres = torch.empty(s["n"], dtype=torch.float64, device="cuda")
            ctx.build_d(s["n"], s["nnz"], s["ptr"], s["idx"], s["val"], mval, colres, **s["opt"])
            return {"m": mval, "colres": colres}
        if kind == "adjoint":
            x = torch.zeros_like(s["b"])
            ctx.bicgstab_transpose_d(s["n"], s["nnz"], s["ptr"], s["idx"], s["val"], s["mval"], s["b"], x, **s["opt"])
            return x
        if kind == "grad":
            x = spai_solve(s["val"], s["b"], s["ptr"], s["idx"], ctx, **s["opt"])
            dval, db = torch.autograd.grad(x, (s["val"], s["b"]), grad_outputs=s["g"])
            return {"x": x.detach(), "dval": dval, "db": db}
        if kind == "batch":
            X = torch.zeros_like(s["B"])
            ctx.batch_solve_d(s["off"], s["n"], s["nnz"], s["ptr"], s["idx"], s["val"], s["B"], X, **s["opt"])
            return X
        rptr = torch.empty_like(s["ptr"])
        ridx, rval = torch.empty_like(s["idx"]), torch.empty_like(s["val"])
        ctx.csc_to_csr_d(s["n"], s["nnz"], s["ptr"], s["idx"], s["val"], rptr, ridx, rval)
        return {"rptr": rptr, "ridx": ridx, "rval": rval}


# ------------------------------------------------------------------ size of the work
def _size(case):
    """(n, nnz, entries per column, iterations), the last an estimate by grid size and tolerance."""
    if case["kind"] == "batch":
        # the mean of a log-uniform size
        lo, hi = case["n_lo"], case["n_hi"]
        n = case["count"] * (hi - lo) / math.log(hi / lo)
        return n, 5.9 * n, 6, 60
    if case["matrix"] == "circuit":
        return case["n"], 4.7 * case["n"], 5, 140
    m = case["m"]
    if case["matrix"] == "3d":
        return m ** 3, 7 * m ** 3 - 6 * m * m, 7, 10 + m // 2
    if case["matrix"] == "mesh":
        return m * m, 7 * m * m, 7, 30
    return m * m, 5 * m * m - 4 * m, 5, (30 + 2 * m // 3 if case["matrix"] == "2d" else 2 * m)


def work(case):
    n, z, w, iters = _size(case)
    kind, rhs = case["kind"], case.get("nrhs", 1)
    matrix = 12 * z + 4 * n
    rows = w * w / 2  # |I| of a column of w entries
    build = 2 * rows * w * w * n
    # two products with A, two with M, ten vector updates and five dot products an iteration
    solve = iters * rhs * (8 * z + 30 * n)
    if kind == "csr":
        return {"bytes": 2 * matrix, "flops": 0}
    if kind == "build":
        return {"bytes": matrix + 8 * z + 8 * n, "flops": build}
    if kind == "adjoint":
        return {"bytes": matrix + 8 * z + 16 * n, "flops": solve}
    if kind == "grad":
        return {"bytes": matrix + 8 * z + 32 * n, "flops": build + 2 * solve + 2 * z}
    return {"bytes": matrix + 16 * n * rhs, "flops": build + solve}


# ------------------------------------------------------------------ the answers in 64 bits
def _exact_build(ptr, idx, val):
    """M's values and the column residuals: every column's least-squares problem by its normal equations
    in 64 bits, one step of refinement, columns padded to the widest."""
    n = ptr.numel() - 1
    ptr = ptr.long()
    w = int((ptr[1:] - ptr[:-1]).max())
    e = ptr[:-1, None] + torch.arange(w, device="cuda")
    ok = e < ptr[1:, None]
    e = torch.where(ok, e, torch.zeros_like(e))
    rows = torch.where(ok, idx.long()[e], torch.full_like(e, -1))   # [n, w]
    vals = torch.where(ok, val[e], torch.zeros_like(val[e]))
    m, res = torch.zeros_like(val), torch.zeros(n, dtype=torch.float64, device="cuda")
    for c0 in range(0, n, 8192):
        J = rows[c0:c0 + 8192]                                       # [c, w], -1 where absent
        have = J >= 0
        Jc = J.clamp(min=0)
        # entry (j, p): row R and value V of the p-th entry of column J_j; R = -1 where absent
        R = torch.where(have[:, :, None], rows[Jc], torch.full_like(rows[Jc], -1)).flatten(1)
        V = torch.where(have[:, :, None], vals[Jc], torch.zeros_like(vals[Jc])).flatten(1)
        c, ww = R.shape
        # dense rows: one for every entry whose row has not occurred before, so that each row of I is there once
        same = (R[:, :, None] == R[:, None, :]) & (R >= 0)[:, :, None]
        first = ~torch.tril(same, -1).any(2) & (R >= 0)
        D = (same * V[:, None, :]).reshape(c, ww, w, w).sum(3) * first[:, :, None]
        rhs = ((R == torch.arange(c0, c0 + c, device="cuda")[:, None]) & first).double()
        G = D.transpose(1, 2) @ D + torch.diag_embed((~have).double())
        L = torch.linalg.cholesky(G)
        x = torch.cholesky_solve(D.transpose(1, 2) @ rhs[:, :, None], L)
        x = x + torch.cholesky_solve(D.transpose(1, 2) @ (rhs[:, :, None] - D @ x), L)
        res[c0:c0 + c] = torch.linalg.vector_norm(rhs - (D @ x)[:, :, 0], dim=1)
        m[e[c0:c0 + c][have]] = x[:, :, 0][have]
    return {"m": m, "colres": res}


def exact(case, seed):
    kind = case["kind"]
    if kind == "csr":
        A = _host_matrix(case, seed)
        by_row = np.argsort(A.idx, kind="stable")
        return {"rptr": None, "ridx": None, "rval": A.val[by_row]}
    if kind == "batch":
        return _normal(seed, sum(m ** d for d, m, _ in _batch_shapes(case, seed)), case["nrhs"])
    if kind == "build":
        return _exact_build(*_problem(case, seed)[:3])
    if kind == "grad":
        A = _host_matrix(case, seed)
        x, lam = _normal(seed, A.n), _normal(seed + 1, A.n)
        cols = torch.from_numpy(np.repeat(np.arange(A.n), np.diff(A.ptr))).cuda()
        return {"x": x, "dval": -lam[torch.from_numpy(A.idx).cuda().long()] * x[cols], "db": lam}
    n = case["n"] if case["matrix"] == "circuit" else case["m"] ** (3 if case["matrix"] == "3d" else 2)
    x = _normal(seed, n)
    return x.cpu().numpy() if kind == "solve_h" else x
