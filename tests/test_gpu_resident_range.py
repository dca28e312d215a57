"""The resident solves (gbfem_res.cu) at the ends of the number range, where the solves before them worked too."""

import numpy as np
import pytest
import scipy.sparse as sp

from opensurgsim_gb300 import _lib, mesh

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


@pytest.mark.parametrize("dims", [(3, 3, 4), (10, 10, 10), (11, 12, 30)])  # a cluster and more CTAs
@pytest.mark.parametrize("exponent", [-90, -60, 60, 100, 110])
def test_units_of_the_matrix(gpu_lib, dims, exponent):
    """Density and Young's modulus times 2^k scale the mixed form's system by 2^k and leave its solution and
    iterations. Both solves leave |b - S x| <= tol |b|, cond(S) below 5e3: 2 tol cond(S) of the velocities."""
    from opensurgsim_gb300.body import Body

    out = []
    for k in (0, exponent):
        s = mesh.scene_cube(*dims, seed=3, young=1e5 * 2.0 ** k, density=1000.0 * 2.0 ** k)
        b = Body(s.mesh, gravity=(0, 0, -9.81), rayleigh_mass=0.01, rayleigh_stiffness=0.001, cg_tolerance=1e-10,
                 precision=_lib.PRECISION_MIXED)
        assert b.step(1e-3) == _lib.GBFEM_OK
        out.append((b.stats()["cg_iterations"], b.state()[1]))
        b.close()
    assert out[0][0] == out[1][0]
    assert np.linalg.norm(out[0][1] - out[1][1]) <= 2e-10 * 5e3 * np.linalg.norm(out[0][1])
