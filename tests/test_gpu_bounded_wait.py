"""Failure detection without a GPU fault: the shared-memory staged SpMV waits for its bulk copies
with a bounded mbarrier wait.  Through a test-only entry point the product runs with a short
limit (about a millisecond) and one stage's copies are never issued, so that wait runs out: the
kernel must record the context's error flag, let its other copies land and return; the next
synchronising call must report the error (and clear it), and the context must stay usable."""
import ctypes as C

import numpy as np
import pytest

import utopia_gb300 as U
from utopia_gb300 import problems as P

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [U.F32, U.BF16])
def test_staged_wait_runs_out_and_the_context_stays_usable(ctx, dtype):
    A = P.lognormal_diffusion_3d(48, 2)[0]
    M = U.SparseMatrix(ctx, A).cast(dtype)
    assert M.sell_interleaved()
    xh = np.random.default_rng(3).standard_normal(A.ncols).astype(np.float32)
    x = U.Vector(ctx, xh, dtype=U.F32)
    y = U.Vector(ctx, n=A.nrows, dtype=U.F32)
    lib = ctx.lib
    launched = C.c_int(0)
    rc = lib.ugpu_test_staged_wait_timeout(M.h, x.h, y.h, 2_000_000, C.byref(launched))
    assert rc == 0, lib.ugpu_last_error(ctx.h)
    assert launched.value == 1  # the operator ran through the staged kernel
    rc = lib.ugpu_synchronize(ctx.h)
    assert rc < 0
    assert b"timed out" in lib.ugpu_last_error(ctx.h)
    assert lib.ugpu_synchronize(ctx.h) == 0  # the flag was cleared
    # the context still works: an ordinary product through the same kernel is correct
    M.apply(x, y)
    ctx.synchronize()
    vals = M.csr()[2]
    ref = P.CSR(A.nrows, A.ncols, A.rowptr, A.colidx, vals).matvec(xh.astype(np.float64))
    np.testing.assert_allclose(y.numpy(), ref, rtol=2e-5, atol=2e-5 * np.abs(ref).max())


def _times_out_once(ctx, rc, message):
    lib = ctx.lib
    assert rc == 0, lib.ugpu_last_error(ctx.h)
    assert lib.ugpu_synchronize(ctx.h) < 0
    assert message in lib.ugpu_last_error(ctx.h)
    assert lib.ugpu_synchronize(ctx.h) == 0  # the flag was cleared


def test_product_wait_runs_out_and_the_context_stays_usable(ctx):
    """The split products of the dense factorisation: the tensor memory is given back and the next ones are right."""
    _times_out_once(ctx, ctx.lib.ugpu_test_product_wait_timeout(ctx.h, 2_000_000), b"dense product timed out")
    A, b = P.poisson2d_cg(32, 0)  # 1024 rows
    x = U.Vector(ctx, n=A.nrows)
    U.CholeskySolver(ctx).solve(U.SparseMatrix(ctx, A), U.Vector(ctx, b), x)
    assert np.linalg.norm(b - A.matvec(x.numpy())) <= 1e-12 * np.linalg.norm(b)


@pytest.mark.parametrize("cluster", [0, 1])
def test_exchange_wait_runs_out_and_the_context_stays_usable(ctx, cluster):
    _times_out_once(ctx, ctx.lib.ugpu_test_exchange_wait_timeout(ctx.h, cluster, 2_000_000), b"timed out waiting for its other")
    A, b = P.poisson2d_cg(48 if cluster else 100, 0)
    atol = 1e-8 * np.linalg.norm(b)
    s = U.ConjugateGradient(ctx, atol=atol)
    x = U.Vector(ctx, n=A.nrows)
    assert s.solve(U.SparseMatrix(ctx, A), U.Vector(ctx, b), x)
    assert np.linalg.norm(b - A.matvec(x.numpy())) <= atol * 1.001


def test_full_device_gives_the_pool_back(ctx):
    """A vector that finds no memory gets what finished set-ups left in the pool."""
    import torch

    A, Ps, _ = P.poisson3d_mg(64, 3, seed=1)
    mg = U.Multigrid(ctx, smoother="jacobi")
    mg.set_transfer_operators(Ps)
    mg.update(U.SparseMatrix(ctx, A))
    del mg
    ctx.synchronize()
    before = torch.cuda.mem_get_info()[0]
    assert ctx.lib.ugpu_test_fail_allocation() == 0
    v = np.random.default_rng(0).standard_normal(1000)
    x = U.Vector(ctx, v)
    np.testing.assert_array_equal(x.numpy(), v)
    assert torch.cuda.mem_get_info()[0] > before + (8 << 20)  # the hierarchy's 262,144 x 7 entries alone are 22 MB
