"""The resident solves (gbfem_res.cu) at the ends of the number range, where the solves before them worked too."""

import numpy as np
import pytest
import scipy.sparse as sp

from opensurgsim_gb300 import _lib

pytestmark = pytest.mark.gpu


# Matrix entries of 1e4 put r.z below 1e-308 while |r|^2 is still above the threshold's floor of 2.2e-308.
@pytest.mark.parametrize("scale", [1.0, 1e4])
@pytest.mark.parametrize("exponent", [-140, -148, -150, -152])
def test_tiny_right_hand_sides(gpu_lib, scale, exponent):
    """A solve ends at |r|^2 < max(tol^2 |b|^2, 2.2e-308); the residual formed here adds the roundings of b - A x,
    1e-15 |b| at most (five of them a row, cond(A) < 10)."""
    from opensurgsim_gb300.body import CgSolver

    n = 300
    A = sp.diags([np.full(n - 1, -scale), np.full(n, 2.5 * scale), np.full(n - 1, -scale)], [-1, 0, 1], format="csc")
    cg = CgSolver(A.indptr, A.indices, A.data)
    cg.set_tolerance(1e-10)
    b = np.random.default_rng(1).normal(size=n)
    x, it, _, st = cg.solve(b * 10.0 ** exponent)
    cg.close()
    assert st == _lib.GBFEM_OK and 0 < it < 100
    r = np.linalg.norm(b - A @ (x * 10.0 ** -exponent))
    assert r <= max(1e-10 * np.linalg.norm(b), np.sqrt(2.3e-308) * 10.0 ** -exponent) + 1e-14 * np.linalg.norm(b)
