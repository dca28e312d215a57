"""The resident CG of compliance columns and of a caller's matrix (gbfem_res.cu), by the residuals of what it
returns.

Tolerance: the solves stop at |r| < tol |b| by their recursive residual, which drifts from b - A x by a few
iterations' roundings (100 x 2^-53 x cond(A) <= 1e-14 x 5e3): 2 tol at tol = 1e-10."""

import numpy as np
import pytest
import scipy.sparse as sp

from opensurgsim_gb300 import _lib, mesh

pytestmark = pytest.mark.gpu
TOL = 1e-10


def _residuals(A, X, B):
    return np.linalg.norm(B - A @ X, axis=0) / np.linalg.norm(B, axis=0)


# One share a column and many, whole and partial chunks, columns in one wave and in several launches.
@pytest.mark.parametrize("dims", [(1, 1, 1), (1, 3, 3), (7, 7, 7), (10, 11, 12), (20, 21, 31)])
@pytest.mark.parametrize("columns", [1, 5, 40, 700])
def test_compliance_columns_solve_the_system(gpu_lib, dims, columns):
    from opensurgsim_gb300.body import Body

    s = mesh.scene_cube(*dims, seed=3)
    if columns * s.mesh.num_nodes > 1e6:
        columns = 90
    kw = dict(rayleigh_mass=0.01, rayleigh_stiffness=0.001, gravity=(0, 0, -9.81), cg_tolerance=TOL)
    rng = np.random.default_rng(7)
    X = {}
    for precision in (_lib.PRECISION_FP64, _lib.PRECISION_MIXED):
        b = Body(s.mesh, precision=precision, **kw)
        v = np.random.default_rng(5).normal(0, 0.05, b.n)
        v[s.mesh.bc_dofs] = 0.0
        b.set_state(None, v)
        keep = _lib.STEP_KEEP_SYSTEM if precision == _lib.PRECISION_FP64 else 0
        assert b.step(1e-3, 1, keep) == _lib.GBFEM_OK
        if precision == _lib.PRECISION_FP64:
            B = rng.normal(size=(b.n, columns))
            colptr, rowidx = b.pattern()
            lower = sp.tril(sp.csc_matrix((b.system()["S"], rowidx, colptr), shape=(b.n, b.n)), format="csr")
            S = lower + sp.tril(lower, -1).T
            W = np.where(np.isin(np.arange(b.n), s.mesh.bc_dofs)[:, None], 0.0, B)
        X[precision], st, _ = b.apply_compliance(B)
        assert st == _lib.GBFEM_OK
        b.close()
    x = X[_lib.PRECISION_FP64]
    assert _residuals(S, x, W).max() <= 2 * TOL
    # The mixed form's system is assembled in FP32: its columns to the 1e-5 of the single-mesh tests.
    assert np.linalg.norm(X[_lib.PRECISION_MIXED] - x) <= 1e-5 * np.linalg.norm(x)


def _grid(*dims):
    n = int(np.prod(dims))
    A = sp.diags([2.0 + np.arange(n) % 7], [0], format="lil")
    ids = np.arange(n).reshape(dims)
    for axis in range(len(dims)):
        i, j = np.delete(ids, -1, axis).ravel(), np.delete(ids, 0, axis).ravel()
        A[i, j] = A[j, i] = -0.3
    return A.tocsc()


def _arrow(n):
    A = sp.diags([4.0 + np.arange(n) % 5], [0], format="lil")
    A[n // 2, :] = A[:, n // 2] = 1e-3
    A[n // 2, n // 2] = 50.0
    return A.tocsc()


def _random(n, k):
    rng = np.random.default_rng(n)
    R = sp.random(n, n, density=k / n, random_state=rng, format="csc")
    R = (R + R.T) * 0.5
    return (R + sp.diags([np.asarray(abs(R).sum(axis=1)).ravel() + 1.0], [0])).tocsc()


# A row-per-warp product (32 rows), one chunk and a row more, a share and several, rows of one very long one (not
# resident), rows that couple to everywhere, more rows than shares hold (not resident).
@pytest.mark.parametrize("matrix", [lambda: _grid(32), lambda: _grid(33), lambda: _grid(8, 17), lambda: _grid(13, 17, 19),
                                    lambda: _arrow(3000), lambda: _random(5000, 12), lambda: _random(40000, 8)])
def test_caller_matrix(gpu_lib, matrix):
    from opensurgsim_gb300.body import CgSolver

    A = matrix()
    A.sort_indices()
    n = A.shape[0]
    cg = CgSolver(A.indptr, A.indices, A.data)
    cg.set_tolerance(TOL)
    for seed in range(2):
        b = np.random.default_rng(seed).normal(size=n)
        x, it, res, st = cg.solve(b)
        assert st == _lib.GBFEM_OK and 0 < it < 200 and res < TOL
        assert _residuals(A, x[:, None], b[:, None])[0] <= 2 * TOL
    assert np.array_equal(cg.solve(b)[0], x)
    cg.set_max_iterations(2)
    _, it, res, st = cg.solve(b)
    assert st == _lib.GBFEM_CG_MAXITER and it == 2 and res > TOL
    x, it, res, st = cg.solve(np.zeros(n))
    assert st == _lib.GBFEM_OK and it == 0 and not x.any()
    b[n // 3] = np.nan
    _, it, _, st = cg.solve(b)
    assert st == _lib.GBFEM_CG_MAXITER and it == 0
    cg.close()
