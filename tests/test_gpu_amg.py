"""AlgebraicMultigrid (greedy agglomeration + Galerkin hierarchy) through the C ABI against the
oracle: identical aggregates on every level, identical coarse-operator structure, and AMG-
preconditioned CG with the oracle's iteration count and solution."""
import numpy as np
import pytest

import utopia_gb300 as U
from utopia_gb300 import problems as P

pytestmark = pytest.mark.gpu

CASES = {
    "laplace1d_dirichlet": (lambda: P.laplacian_1d_dirichlet(100), dict(n_levels=6)),
    "lognormal24": (lambda: P.lognormal_diffusion_3d(24, 5)[0], dict(n_levels=0, max_coarse_rows=2000)),
    "random_graph": (lambda: P.random_spd_graph(20000, 4, 1), dict(n_levels=0, max_coarse_rows=2000)),
}


@pytest.mark.parametrize("name", list(CASES))
def test_amg_hierarchy_matches_oracle(ctx, oracle, name):
    make, kw = CASES[name]
    A = make()
    Am = oracle.Matrix(A)
    Ps, parents = oracle.amg_hierarchy(Am, **kw)
    amg = U.AlgebraicMultigrid(ctx, smoother="chebyshev", **kw)
    M = U.SparseMatrix(ctx, A)
    amg.update(M)
    assert amg.n_levels() == len(Ps) + 1
    for l, ref in enumerate(parents):
        got, nc = amg.parent(l)
        np.testing.assert_array_equal(got, ref)
        assert nc == Ps[len(Ps) - 1 - l].ncols
    omg = oracle.Multigrid(Am, Ps, smoother="chebyshev")
    for l in range(amg.n_levels()):
        G = amg.level_matrix(l)
        rp, ci, v = G.csr()
        orp, oci, ov = omg.level_matrix(l).arrays()
        np.testing.assert_array_equal(rp, orp)
        np.testing.assert_array_equal(ci, oci)
        np.testing.assert_allclose(v, ov, rtol=1e-12, atol=1e-12 * np.abs(ov).max())


@pytest.mark.parametrize("option", ["fix_semidefinite_operators", "keep_galerkin_structure"])
@pytest.mark.parametrize("name", ["lognormal24", "random_graph"])
def test_amg_galerkin_options(ctx, oracle, name, option):
    """A small operator (diagonals below 1e-12 on some levels and rows): with fixed semidefinite levels every coarser
    product is that of the fixed one, as in the oracle; a kept structure changes nothing."""
    make, kw = CASES[name]
    A = make()
    i = np.repeat(np.arange(A.nrows), np.diff(A.rowptr))
    scale = 1e-13 / np.median(A.values[i == A.colidx])
    A = P.CSR(A.nrows, A.ncols, A.rowptr, A.colidx, A.values * scale)
    kw = dict(kw, n_levels=4)
    fix = option == "fix_semidefinite_operators"
    Am = oracle.Matrix(A)
    Ps, _ = oracle.amg_hierarchy(Am, **kw)
    amg = U.AlgebraicMultigrid(ctx, smoother="jacobi", **{option: 1}, **kw)
    M = U.SparseMatrix(ctx, A)
    omg = oracle.Multigrid(Am, Ps, smoother="jacobi", fix_semidefinite=fix)
    for _ in range(2):
        amg.update(M)
        for l in range(amg.n_levels()):
            rp, ci, v = amg.level_matrix(l).csr()
            orp, oci, ov = omg.level_matrix(l).arrays()
            np.testing.assert_array_equal(rp, orp)
            np.testing.assert_array_equal(ci, oci)
            np.testing.assert_allclose(v, ov, rtol=1e-12, atol=1e-12 * np.abs(ov).max())


def test_reference_amg_1d_case(ctx, oracle):
    """utopia/tests/utopia_AMGTest.cpp:36-110 (1D Laplacian, 100 dofs, identity boundary rows,
    b = 2 with 0 on the boundary, 6 levels, atol 1e-6, ||r||_1 < 1e-5), with Chebyshev3level
    smoothing and the hierarchy as the CG preconditioner (the reference smooths with ILU)."""
    A = P.laplacian_1d_dirichlet(100)
    b = np.full(100, 2.0)
    b[0] = b[-1] = 0.0
    amg = U.AlgebraicMultigrid(ctx, smoother="chebyshev", n_levels=6, pre_smoothing_steps=3,
                               post_smoothing_steps=3)
    cg = U.ConjugateGradient(ctx, atol=1e-6, max_it=100)
    cg.set_preconditioner(amg)
    x = U.Vector(ctx, n=100)
    cg.solve(U.SparseMatrix(ctx, A), U.Vector(ctx, b), x)
    st = cg.solution_status()
    assert st["converged"] and np.abs(b - A.matvec(x.numpy())).sum() < 1e-5
    Am = oracle.Matrix(A)
    Ps, _ = oracle.amg_hierarchy(Am, n_levels=6)
    _, ost = oracle.cg_solve(Am, b, precond="mg", mg=oracle.Multigrid(Am, Ps, smoother="chebyshev"), atol=1e-6,
                             max_it=100)
    assert abs(st["iterates"] - ost["iterates"]) <= 1


@pytest.mark.parametrize("name", ["lognormal24", "random_graph"])
def test_amg_pcg_matches_oracle(ctx, oracle, name):
    make, kw = CASES[name]
    A = make()
    b = np.random.default_rng(0).uniform(-1, 1, A.nrows)
    atol = 1e-10 * np.linalg.norm(b)
    amg = U.AlgebraicMultigrid(ctx, smoother="chebyshev", pre_smoothing_steps=2, post_smoothing_steps=2, **kw)
    cg = U.ConjugateGradient(ctx, atol=atol, max_it=500)
    cg.set_preconditioner(amg)
    x = U.Vector(ctx, n=A.nrows)
    cg.solve(U.SparseMatrix(ctx, A), U.Vector(ctx, b), x)
    st = cg.solution_status()
    Am = oracle.Matrix(A)
    Ps, _ = oracle.amg_hierarchy(Am, **kw)
    omg = oracle.Multigrid(Am, Ps, smoother="chebyshev", pre=2, post=2)
    xr, ost = oracle.cg_solve(Am, b, precond="mg", mg=omg, atol=atol, max_it=500)
    assert st["converged"] and ost["converged"]
    assert abs(st["iterates"] - ost["iterates"]) <= 1
    xg = x.numpy()
    assert np.linalg.norm(b - A.matvec(xg)) <= atol * 1.0001
    assert np.linalg.norm(xg - xr) <= 1e-8 * np.linalg.norm(xr)


def _stencil(nx, ny, nz, offsets, seed):
    """A symmetric pattern with independent values of very different size in both directions, ordered by index."""
    import scipy.sparse as sp

    rng = np.random.default_rng(seed)
    n = nx * ny * nz
    i = np.arange(n)
    x, y, z = i % nx, i // nx % ny, i // (nx * ny)
    r, c = [i], [i]
    for dx, dy, dz in offsets:
        ok = ((x + dx >= 0) & (x + dx < nx) & (y + dy >= 0) & (y + dy < ny) & (z + dz >= 0) & (z + dz < nz))
        r.append(i[ok])
        c.append((i + dx + nx * (dy + ny * dz))[ok])
    r, c = np.concatenate(r), np.concatenate(c)
    A = sp.csr_matrix((rng.lognormal(0, 1.5, r.size) * rng.choice([-1.0, 1.0], r.size), (r, c)), shape=(n, n))
    A.sort_indices()
    return A


_BOX = [(a, b, c) for a in (-1, 0, 1) for b in (-1, 0, 1) for c in (-1, 0, 1) if (a, b, c) != (0, 0, 0)]
_STAR = [o for o in _BOX if sum(map(abs, o)) == 1]
_WIDE = [(a, b, 0) for a in range(-3, 4) for b in range(-3, 4) if (a, b) != (0, 0)]
AGGREGATE_FORMS = {
    "star": (lambda: _stencil(27, 26, 25, _STAR, 1), {}),
    "star_bmax1": (lambda: _stencil(27, 26, 25, _STAR, 2), dict(bmax=1, weight=0.9)),
    "box": (lambda: _stencil(27, 26, 25, _BOX, 3), dict(bmax=9)),
    "wide": (lambda: _stencil(135, 131, 1, _WIDE, 4), dict(weight=0.6)),
    "wide_rows_of_a_strip": (lambda: _stencil(9000, 2, 1, _WIDE, 5), {}),
    "few_rows_at_a_time": (lambda: _stencil(18000, 1, 1, [(-1, 0, 0), (1, 0, 0)], 6), {}),
    "threshold": (lambda: _stencil(128, 128, 1, [o for o in _BOX if o[2] == 0], 7), {}),
}


@pytest.mark.parametrize("excluded", [False, True])
@pytest.mark.parametrize("additive", [0, 1])
@pytest.mark.parametrize("name", list(AGGREGATE_FORMS))
def test_aggregates_of_large_levels(ctx, oracle, name, additive, excluded):
    """The aggregation in dependency order is the sequential one: every row's aggregate, over stencils that take
    one, four and eight lanes a row, rows with only a diagonal (their columns stay in other rows) and chains."""
    make, kw = AGGREGATE_FORMS[name]
    A = make()
    if excluded:  # every 11th row keeps its diagonal only
        import scipy.sparse as sp

        keep = np.repeat(np.arange(A.shape[0]), np.diff(A.indptr))
        ok = (keep % 11 != 3) | (A.indices == keep)
        A = sp.csr_matrix((A.data[ok], (keep[ok], A.indices[ok])), shape=A.shape)
        A.sort_indices()
    Ac = P.CSR.from_scipy(A)
    okw = dict(kw, use_additive_correction=additive)
    ref, Pm = oracle.agglomerate(oracle.Matrix(Ac), **okw)
    amg = U.AlgebraicMultigrid(ctx, smoother="jacobi", n_levels=2, **okw)
    try:
        amg.update(U.SparseMatrix(ctx, Ac))
    except U.UgpuError as e:  # the values make no definite operator; the aggregates are there before its factor
        assert "coarse operator is not symmetric positive definite" in str(e)
    got, nc = amg.parent(0)
    assert nc == Pm.ncols
    np.testing.assert_array_equal(got, ref)


def test_aggregates_of_a_long_row(ctx, oracle):
    """One row of an arrow matrix touches every other one: the sequential aggregation takes it."""
    import scipy.sparse as sp

    rng = np.random.default_rng(2)
    n = 20001
    A = sp.diags([rng.uniform(-1, 0, n - 1), rng.uniform(5, 9, n), rng.uniform(-1, 0, n - 1)], [-1, 0, 1]).tolil()
    A[0, 1:] = rng.uniform(-1, 0, n - 1)
    A[1:, 0] = rng.uniform(-1, 0, n - 1).reshape(-1, 1)
    A[0, 0] = 5.0 * n
    Ac = P.CSR.from_scipy(A.tocsr())
    ref, Pm = oracle.agglomerate(oracle.Matrix(Ac))
    amg = U.AlgebraicMultigrid(ctx, smoother="jacobi", n_levels=2)
    try:
        amg.update(U.SparseMatrix(ctx, Ac))
    except U.UgpuError as e:
        assert "coarse operator" in str(e) or "coarse solver" in str(e)
    got, nc = amg.parent(0)
    assert nc == Pm.ncols
    np.testing.assert_array_equal(got, ref)
