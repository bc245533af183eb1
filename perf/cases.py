"""Cases that time the framework's main path through its public entry points.

Every case is one call that a program using the solvers makes with its operator, solver and
vectors resident on the GPU: a Krylov or multigrid solve (``apply``), the same with the operator
changed before it (``solve`` = ``update`` + ``apply``), a box-constrained solve, a differentiable
solve with its backward pass, a matrix product.  Problems are those of ``utopia_gb300.problems``
and of ``bench.py`` (Poisson and lognormal diffusion grids, obstacle problems, random graphs),
built on the GPU from a seed.
"""

from __future__ import annotations

import ctypes as C
import functools
import math

import numpy as np
import torch

import utopia_gb300 as U
from utopia_gb300 import problems as P
from utopia_gb300.autograd import DifferentiableGraphSolver, GraphSolve

DTYPES = {"f64": U.F64, "f32": U.F32, "bf16": U.BF16}


def listed():
    return [
        # the smallest Krylov solve of the tests: launches and latency count, not bytes
        {"name": "cg_jacobi_2d_48", "kind": "cg", "nx": 48, "ny": 48},
        # the plain Jacobi-preconditioned CG workload of the benchmark
        {"name": "cg_jacobi_2d_256", "kind": "cg", "nx": 256, "ny": 256},
        # a small, ragged box re-solved with new coefficients each time (update + solve), FP32 levels
        {"name": "mg_solve_f32_48x40x32", "kind": "mgsolve", "nx": 48, "ny": 40, "nz": 32, "levels": 4,
         "op": "lognormal", "smoother": "jacobi", "precision": "f32"},
        # FP64 multigrid-preconditioned CG with Chebyshev smoothing on a resident hierarchy
        {"name": "mg_apply_cheb_f64_128", "kind": "mg", "nx": 128, "ny": 128, "nz": 128, "levels": 4,
         "op": "poisson", "smoother": "chebyshev", "precision": "f64"},
        # the same program when its operator changed: hierarchy set-up, coarse factorisation, solve
        {"name": "mg_solve_cheb_f64_128", "kind": "mgsolve", "nx": 128, "ny": 128, "nz": 128, "levels": 4,
         "op": "poisson", "smoother": "chebyshev", "precision": "f64"},
        # the benchmark's headline: variable coefficients, mixed precision, and its plain FP64 form
        {"name": "mg_apply_bf16_192", "kind": "mg", "nx": 192, "ny": 192, "nz": 192, "levels": 5,
         "op": "lognormal", "smoother": "jacobi", "precision": "bf16"},
        {"name": "mg_apply_f64_192", "kind": "mg", "nx": 192, "ny": 192, "nz": 192, "levels": 5,
         "op": "lognormal", "smoother": "jacobi", "precision": "f64"},
        # a learning step through the solver: forward solve, adjoint solve, edge gradients
        {"name": "adjoint_bf16_128", "kind": "adjoint", "N": 128, "levels": 4, "precision": "bf16", "theta": "f32"},
        # algebraic multigrid on an odd box: aggregation set-up and solve from an operator alone
        {"name": "amg_solve_f64_95x89x97", "kind": "amg", "nx": 95, "ny": 89, "nz": 97, "precision": "f64"},
        # contact problems: MPRGP to convergence, and the monotone multigrid
        {"name": "mprgp_256", "kind": "mprgp", "nx": 256, "ny": 256},
        {"name": "mmg_512", "kind": "mmg", "nx": 512, "ny": 512, "levels": 6},
        # one product of an unstructured operator with an odd number of rows
        {"name": "spmv_graph_f64_300007", "kind": "spmv", "n": 300007, "degree": 4, "precision": "f64"},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _box(rng, lo, hi):
    """Grid sizes m 2^(levels-1) per dimension, ragged, between lo and hi, at most 4096 coarse nodes."""
    while True:
        levels = rng.randint(3, 5)
        f = 1 << (levels - 1)
        d = [max(3, round(_log_int(rng, lo, hi) / f)) * f for _ in range(3)]
        coarse = math.prod(v // f for v in d)
        if max(d) <= hi and min(d) >= lo // 2 and max(d) <= 3 * min(d) and 27 <= coarse <= 4096:
            return {"nx": d[0], "ny": d[1], "nz": d[2], "levels": levels}


def draw(rng):
    kind = rng.choice(["cg", "cg", "mg", "mg", "mg", "mgsolve", "mgsolve", "adjoint", "amg", "mprgp", "mmg", "spmv"])
    if kind == "cg":
        return {"kind": kind, "nx": _log_int(rng, 24, 320), "ny": _log_int(rng, 24, 320)}
    if kind in ("mg", "mgsolve"):
        return {"kind": kind, **_box(rng, 24, 192 if kind == "mg" else 128),
                "op": rng.choice(["poisson", "lognormal"]), "smoother": rng.choice(["jacobi", "chebyshev"]),
                "precision": rng.choice(["f64", "f32", "bf16"])}
    if kind == "adjoint":
        levels = rng.randint(3, 4)
        f = 1 << (levels - 1)
        N = min(16, max(4, round(_log_int(rng, 24, 128) / f))) * f
        return {"kind": kind, "N": N, "levels": levels, "precision": rng.choice(["f64", "f32", "bf16"]),
                "theta": rng.choice(["f32", "f64"])}
    if kind == "amg":
        return {"kind": kind, "nx": _log_int(rng, 24, 96), "ny": _log_int(rng, 24, 96), "nz": _log_int(rng, 24, 96),
                "precision": rng.choice(["f64", "bf16"])}
    if kind == "mprgp":
        return {"kind": kind, "nx": _log_int(rng, 32, 256), "ny": _log_int(rng, 32, 256)}
    if kind == "mmg":
        levels = rng.randint(4, 6)
        f = 1 << (levels - 1)
        d = [min(512 // f, max(8, round(_log_int(rng, 64, 512) / f))) * f for _ in range(2)]
        return {"kind": kind, "nx": d[0], "ny": d[1], "levels": levels}
    return {"kind": kind, "n": _log_int(rng, 2000, 600000) | 1, "degree": rng.randint(2, 6),
            "precision": rng.choice(["f64", "f32", "bf16"])}


# --------------------------------------------------------------------------------------
# operators and vectors on the GPU
# --------------------------------------------------------------------------------------
RTOL = 1e-8
_F64 = dict(dtype=torch.float64, device="cuda")


@functools.lru_cache(maxsize=None)
def _ctx():
    return U.Context(0)


def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _uniform(g, n, lo, hi):
    return torch.rand(n, generator=g, **_F64) * (hi - lo) + lo


def _dims(case):
    return [case["nx"], case["ny"]] + ([case["nz"]] if "nz" in case else [])


def _compress(cols, vals, valid):
    """An (n, k) table of entries with ascending columns -> (rowptr, colidx, values)."""
    rp = torch.zeros(cols.shape[0] + 1, dtype=torch.int64, device="cuda")
    torch.cumsum(valid.sum(1), 0, out=rp[1:])
    return rp.int(), cols[valid].int(), vals[valid]


def _stencil(dims, diag, faces):
    """5- or 7-point operator, x fastest: faces[d] couples a node to the next one along d (any value on
    the last layer), diag is the node's own entry."""
    n = math.prod(dims)
    idx = torch.arange(n, device="cuda")
    strides = [math.prod(dims[:d]) for d in range(len(dims))]
    low, up = [], []
    for d, s in enumerate(strides):
        pos = (idx // s) % dims[d]
        prev = torch.zeros_like(faces[d])
        prev[s:] = faces[d][:-s]
        low.append((idx - s, -prev, pos > 0))
        up.append((idx + s, -faces[d], pos < dims[d] - 1))
    ent = low[::-1] + [(idx, diag, torch.ones_like(idx, dtype=torch.bool))] + up
    return _compress(*[torch.stack([e[k] for e in ent], 1) for k in range(3)])


def _poisson(dims):
    n = math.prod(dims)
    one = torch.ones(n, **_F64)
    return _stencil(dims, 2.0 * len(dims) * one, [one] * len(dims))


def _lognormal(dims, g, corr=8.0):
    """-div(k grad u), k = exp of a unit Gaussian field with the given correlation length (cells)."""
    shape = dims[::-1]
    f = torch.fft.rfftn(torch.randn(shape, generator=g, **_F64))
    for ax, m in enumerate(shape):
        w = torch.fft.rfftfreq(m, **_F64) if ax == len(shape) - 1 else torch.fft.fftfreq(m, **_F64)
        f *= torch.exp(-2.0 * (math.pi * corr * w) ** 2).reshape([-1 if a == ax else 1 for a in range(len(shape))])
    k = torch.fft.irfftn(f, s=shape)
    k = ((k - k.mean()) / k.std()).reshape(-1)
    idx = torch.arange(k.numel(), device="cuda")
    diag, faces = torch.zeros_like(k), []
    for d, m in enumerate(dims):
        s = math.prod(dims[:d])
        pos = (idx // s) % m
        nxt = torch.zeros_like(k)
        nxt[:-s] = k[s:]
        face = torch.where(pos < m - 1, torch.exp(0.5 * (k + nxt)), torch.zeros_like(k))
        prev = torch.zeros_like(k)
        prev[s:] = face[:-s]
        diag += face + prev + torch.exp(k) * ((pos == 0).double() + (pos == m - 1).double())
        faces.append(face)
    return _stencil(dims, diag, faces)


def _interpolation(dims):
    """(Bi/tri)linear interpolation from the grid of half the size (problems.interpolation_2d/3d)."""
    n = math.prod(dims)
    idx = torch.arange(n, device="cuda")
    cols = torch.zeros(n, 1, dtype=torch.int64, device="cuda")
    vals = torch.ones(n, 1, **_F64)
    ok = torch.ones(n, 1, dtype=torch.bool, device="cuda")
    for d in range(len(dims) - 1, -1, -1):
        f = (idx // math.prod(dims[:d])) % dims[d]
        odd = f % 2 == 1
        c1 = torch.stack([torch.where(odd, f // 2, f // 2 - 1), f // 2], 1)
        v1 = torch.where(odd, 1.0, 0.5).double()[:, None].expand(n, 2)
        k1 = torch.stack([odd | (f >= 2), ~odd], 1)
        cols = (cols[:, :, None] * (dims[d] // 2) + c1[:, None, :]).reshape(n, -1)
        vals = (vals[:, :, None] * v1[:, None, :]).reshape(n, -1)
        ok = (ok[:, :, None] & k1[:, None, :]).reshape(n, -1)
    return _compress(cols, vals, ok)


def _graph(n, degree, g):
    """Weighted graph Laplacian of a random graph plus a small shift (problems.random_spd_graph)."""
    i = torch.arange(n, device="cuda").repeat_interleave(degree)
    j = torch.randint(0, n, (n * degree,), generator=g, device="cuda")
    w = _uniform(g, n * degree, 0.1, 2.0)
    i, j, w = i[i != j], j[i != j], w[i != j]
    d = torch.full((n,), 1e-3, **_F64).index_add_(0, i, w).index_add_(0, j, w)
    k = torch.arange(n, device="cuda")
    idx = torch.stack([torch.cat([i, j, k]), torch.cat([j, i, k])])
    m = torch.sparse_coo_tensor(idx, torch.cat([-w, -w, d]), (n, n)).coalesce()
    rp = torch.zeros(n + 1, dtype=torch.int64, device="cuda")
    torch.cumsum(torch.bincount(m.indices()[0], minlength=n), 0, out=rp[1:])
    return rp.int(), m.indices()[1].int(), m.values()


def _obstacle(dims, g):
    """Lower bound of problems.obstacle_qp: eight Gaussian bumps over the unit square, minus 0.2."""
    c, w = torch.rand(8, 2, generator=g, **_F64), torch.rand(8, generator=g, **_F64) * 0.08 + 0.02
    px, py = [(torch.arange(m, **_F64) + 1) / (m + 1) for m in dims]
    lb = torch.zeros(dims[1], dims[0], **_F64)
    for k in range(8):
        lb += torch.exp(-((px[None, :] - c[k, 0]) ** 2 + (py[:, None] - c[k, 1]) ** 2) / (2 * w[k] ** 2))
    return (0.3 * lb - 0.2).reshape(-1)


def _problem(case, seed):
    """(CSR on the GPU, right-hand side [, lower bound]) of a case that is not a graph solve."""
    g = _gen(seed)
    if case["kind"] == "spmv":
        csr = _graph(case["n"], case["degree"], g)
        return csr, _uniform(g, case["n"], -1, 1)
    dims = _dims(case)
    n = math.prod(dims)
    if case["kind"] in ("mprgp", "mmg"):
        return _poisson(dims), torch.full((n,), -20.0 / ((dims[0] + 1) * (dims[1] + 1)), **_F64), _obstacle(dims, g)
    csr = _lognormal(dims, g) if case.get("op", "poisson" if case["kind"] == "cg" else "lognormal") == "lognormal" \
        else _poisson(dims)
    return csr, _uniform(g, n, -1, 1)


def _matrix(csr, ncols=None):
    ctx, (rp, ci, v) = _ctx(), csr
    torch.cuda.synchronize()
    h = C.c_void_p()
    n = rp.numel() - 1
    ctx.check(ctx.lib.ugpu_csr_create_device(ctx.h, n, ncols or n, v.numel(), *[C.c_void_p(t.data_ptr())
                                                                                for t in (rp, ci, v)], C.byref(h)))
    return U.SparseMatrix(ctx, _handle=h)


def _transfers(case):
    """Interpolations ordered coarse -> fine."""
    ops, dims = [], _dims(case)
    for _ in range(case["levels"] - 1):
        ops.append(_matrix(_interpolation(dims), math.prod(dims) >> len(dims)))
        dims = [m // 2 for m in dims]
    return ops[::-1]


def _wrap(t):
    return U.Vector.wrap_device(_ctx(), t.data_ptr(), t.numel(), U.F64 if t.dtype == torch.float64 else U.F32)


@functools.lru_cache(maxsize=2)
def _edge_graph(N):
    return P.EdgeGraph(N)


# --------------------------------------------------------------------------------------
# the cases
# --------------------------------------------------------------------------------------
def prepare(case, seed):
    kind, ctx = case["kind"], _ctx()
    if kind == "adjoint":
        G, (theta, b, gx) = _edge_graph(case["N"]), _adjoint_inputs(case, seed)
        Ps = _transfers({**case, "nx": case["N"], "ny": case["N"], "nz": case["N"]})
        solver = DifferentiableGraphSolver(ctx, G, Ps, precision=DTYPES[case["precision"]], rtol=RTOL)
        return {"kind": kind, "solver": solver, "theta": theta.requires_grad_(), "b": b.requires_grad_(), "gx": gx}
    csr, b, *lb = _problem(case, seed)
    A = _matrix(csr)
    s = {"kind": kind, "A": A, "b": b, "x": torch.zeros_like(b)}
    if kind == "spmv":
        if case["precision"] != "f64":
            s["A"] = A.cast(DTYPES[case["precision"]])
            s["b"], s["x"] = b.float(), torch.zeros_like(b).float()
    elif kind in ("mprgp", "mmg"):
        h2 = 1.0 / ((case["nx"] + 1) * (case["ny"] + 1))
        if kind == "mprgp":
            s["ub"] = torch.full_like(b, np.finfo(np.float64).max)
            s["solver"] = U.MPRGP(ctx, atol=1e-8 * h2, rtol=1e-30, max_it=400000)
            s["solver"].set_box_constraints(_wrap(lb[0]), _wrap(s["ub"]))
            s["solver"].update(A)
        else:
            s["solver"] = U.MonotoneMultigrid(ctx, max_it=500, atol=1e-8 * h2, stol=1e-12)
            s["solver"].set_transfer_operators(_transfers(case))
            s["solver"].set_box_constraints(_wrap(lb[0]), None)
        s["lb"] = lb[0]
    else:
        s["prec"] = _preconditioner(case)
        mixed = case.get("precision", "f64") != "f64"
        s["solver"] = U.ConjugateGradient(ctx, atol=RTOL * b.norm().item(), flexible=1 if mixed else 0, max_it=5000)
        s["solver"].set_preconditioner(s["prec"])
        if kind in ("cg", "mg"):  # a resident operator and hierarchy, solved with again and again
            s["solver"].update(A)
    torch.cuda.synchronize()
    s["vb"], s["vx"] = _wrap(s["b"]), _wrap(s["x"])
    return s


def _preconditioner(case):
    ctx = _ctx()
    if case["kind"] == "cg":
        return U.InvDiagPreconditioner(ctx)
    if case["kind"] == "amg":
        return U.AlgebraicMultigrid(ctx, smoother="jacobi", omega=0.8, pre_smoothing_steps=2, post_smoothing_steps=2,
                                    n_levels=0, max_coarse_rows=4096, precision=DTYPES[case["precision"]])
    kw = (dict(pre_smoothing_steps=3, post_smoothing_steps=3) if case["smoother"] == "chebyshev" else
          dict(omega=0.8, pre_smoothing_steps=2, post_smoothing_steps=2))
    mg = U.Multigrid(ctx, smoother=case["smoother"], precision=DTYPES[case["precision"]], **kw)
    mg.set_transfer_operators(_transfers(case))
    return mg


def _adjoint_inputs(case, seed):
    N, g = case["N"], _gen(seed)
    E = 3 * N * N * (N - 1)
    theta = torch.randn(E, generator=g, **_F64) * 0.5
    b = _uniform(g, N ** 3, -0.01, 0.01)
    b[(N // 2 * N + N // 2) * N + N // 2] += 1.0
    return (theta if case["theta"] == "f64" else theta.float()), b, torch.randn(N ** 3, generator=g, **_F64)


def run(s):
    kind = s["kind"]
    if kind == "adjoint":
        x = GraphSolve.apply(s["theta"], s["b"], s["solver"])
        return (x.detach(), *torch.autograd.grad(x, (s["theta"], s["b"]), s["gx"]))
    if kind == "spmv":
        s["A"].apply(s["vb"], s["vx"])
        return s["x"]
    s["vx"].set(0.0)
    if kind in ("cg", "mg", "mprgp"):
        s["solver"].apply(s["vb"], s["vx"])
    else:
        s["solver"].solve(s["A"], s["vb"], s["vx"])
    return s["x"]


def work(case):
    """Inputs read once and outputs written once; the products of a usual number of iterations."""
    kind = case["kind"]
    size = {"f64": 8, "f32": 4, "bf16": 2}
    if kind == "spmv":
        n, s = case["n"], size[case["precision"]]
        nnz, v = n * (2 * case["degree"] + 1), 8 if s == 8 else 4
        return {"bytes": nnz * (s + 4) + 4 * (n + 1) + 2 * n * v, "flops": 2 * nnz}
    if kind == "adjoint":
        n, E = case["N"] ** 3, 3 * case["N"] ** 2 * (case["N"] - 1)
        t = size[case["theta"]]
        return {"bytes": E * (8 + 2 * t) + 8 * 4 * n + 4 * (2 * E + n), "flops": 2 * 9 * 10 * 2 * (2 * E + n)}
    dims = _dims(case)
    n = math.prod(dims)
    nnz = n * (1 + 2 * len(dims))
    its = {"cg": 3 * max(dims), "mg": 9 * 8, "mgsolve": 9 * 8, "amg": 50 * 7, "mprgp": 20 * max(dims), "mmg": 50 * 12}
    vectors = 3 if kind in ("mprgp", "mmg") else 2
    return {"bytes": 12 * nnz + 4 * (n + 1) + 8 * vectors * n, "flops": its[kind] * 2 * (nnz + 5 * n)}


# --------------------------------------------------------------------------------------
# the same answers in 64 bits from plain torch
# --------------------------------------------------------------------------------------
def _pcg(mul, diag, b, rtol=1e-10, max_it=30000):
    x, r = torch.zeros_like(b), b.clone()
    z = r / diag
    p, rz, stop = z.clone(), torch.dot(r, z), rtol * b.norm().item()
    for k in range(max_it):
        q = mul(p)
        a = rz / torch.dot(p, q)
        x += a * p
        r -= a * q
        if k % 25 == 24 and not r.norm().item() > stop:
            break
        z = r / diag
        old, rz = rz, torch.dot(r, z)
        p = z + (rz / old) * p
    return x


def _spd_solve(mul, diag, b):
    x = _pcg(mul, diag, b)
    for _ in range(2):  # residuals in 64 bits bring the error down to the rounding of the product
        x = x + _pcg(mul, diag, b - mul(x), 1e-6)
    return x


def _csr_mul(csr):
    n = csr[0].numel() - 1
    m = torch.sparse_csr_tensor(csr[0].long(), csr[1].long(), csr[2], (n, n))
    rows = torch.repeat_interleave(torch.arange(n, device="cuda"), (csr[0][1:] - csr[0][:-1]).long())
    diag = torch.zeros(n, **_F64)
    diag[rows[rows == csr[1]]] = csr[2][rows == csr[1]]
    return (lambda x: m @ x), diag


def _obstacle_exact(mul, diag, b, lb):
    """Primal-dual active set: the minimiser of 1/2 x'Ax - b'x over x >= lb."""
    x, active = lb.clone(), torch.ones_like(lb, dtype=torch.bool)
    for _ in range(150):
        lam = torch.where(active, mul(x) - b, torch.zeros_like(b))
        new = lam + diag * (lb - x) > 0
        if torch.equal(new, active) and _:
            return x
        active, free = new, (~new).double()
        base = torch.where(active, lb, torch.zeros_like(lb))
        rhs = free * (b - mul(base))
        x = base + free * _spd_solve(lambda v: free * mul(free * v) + (1 - free) * diag * v, diag, rhs)
    return None


def exact(case, seed):
    kind = case["kind"]
    if kind == "adjoint":
        N = case["N"]
        theta, b, gx = _adjoint_inputs(case, seed)
        k = torch.exp(theta.double())
        kx, ky, kz = [t.reshape(s) for t, s in zip(k.split(N * N * (N - 1)), ((N, N, N - 1), (N, N - 1, N), (N - 1, N, N)))]

        def diffs(v):
            v = v.reshape(N, N, N)
            return v[:, :, :-1] - v[:, :, 1:], v[:, :-1] - v[:, 1:], v[:-1] - v[1:]

        pos = torch.arange(N, device="cuda")
        edge = ((pos == 0).double() + (pos == N - 1).double())
        bnd = edge[:, None, None] + edge[None, :, None] + edge[None, None, :]

        def spread(fx, fy, fz, sign):
            y = torch.zeros(N, N, N, **_F64)
            y[:, :, :-1] += fx
            y[:, :, 1:] += sign * fx
            y[:, :-1] += fy
            y[:, 1:] += sign * fy
            y[:-1] += fz
            y[1:] += sign * fz
            return y

        def mul(v):
            dx, dy, dz = diffs(v)
            return (spread(kx * dx, ky * dy, kz * dz, -1.0) + bnd * v.reshape(N, N, N)).reshape(-1)

        diag = (spread(kx, ky, kz, 1.0) + bnd).reshape(-1)
        x, lam = _spd_solve(mul, diag, b), _spd_solve(mul, diag, gx)
        grad = -k * torch.cat([(p * q).reshape(-1) for p, q in zip(diffs(lam), diffs(x))])
        return x, grad, lam
    csr, b, *lb = _problem(case, seed)
    if kind == "spmv":
        rp, ci, v = csr
        if case["precision"] != "f64":
            v = (v.float() if case["precision"] == "f32" else v.bfloat16()).double()
            b = b.float().double()
        return _csr_mul((rp, ci, v))[0](b)
    mul, diag = _csr_mul(csr)
    return _obstacle_exact(mul, diag, b, lb[0]) if lb else _spd_solve(mul, diag, b)
