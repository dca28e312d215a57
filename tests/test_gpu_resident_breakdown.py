"""What resident solves (gbfem_res.cu) report when they break down: as the launch-per-iteration and the persistent
solves do."""

import numpy as np
import pytest

from opensurgsim_gb300 import _lib, mesh
from opensurgsim_gb300.mesh import TetMesh

pytestmark = pytest.mark.gpu


def _light(**kw):
    """A body whose 1 / diag(S) is about 1e4."""
    from opensurgsim_gb300.body import Body

    return Body(mesh.scene_cube(3, 3, 4, seed=3, young=1.0, density=1e-3).mesh, cg_tolerance=1e-10, **kw)


@pytest.mark.parametrize("flags", [0, _lib.STEP_TIME_KERNELS])  # resident and not
def test_residual_of_a_step_that_overflows(gpu_lib, flags):
    b = _light(gravity=(0, 0, -1e160))
    assert b.step(1e-3, 1, flags) == _lib.GBFEM_NONFINITE
    q = b.stats()
    b.close()
    assert np.isnan(q["cg_relative_residual"]) and q["cg_max_iterations_hit"] == 1 and q["refinement_sweeps"] == 0


@pytest.mark.parametrize("flags", [0, _lib.STEP_TIME_KERNELS])
@pytest.mark.parametrize("value,residual", [(np.nan, 0.0), (np.inf, 0.0), (1e200, np.nan)])
def test_residual_of_a_step_without_a_norm(gpu_lib, flags, value, residual):
    """|b|^2 is not a number, where the residual is given as 0, or infinite, where it is infinity over infinity."""
    b = _light()
    v = np.zeros(b.n)
    v[-1] = value
    b.set_state(None, v)
    b.step(1e-3, 1, flags)
    q = b.stats()
    b.close()
    assert np.array_equal(q["cg_relative_residual"], residual, equal_nan=True) and q["cg_iterations"] == 0


def test_iterations_of_columns_that_overflow(gpu_lib):
    """r.z of the middle column is infinite: its first iteration gives NaN and is counted."""
    b = _light(gravity=(0, 0, -9.81))
    assert b.step(1e-3) == _lib.GBFEM_OK
    B = np.random.default_rng(2).normal(size=(b.n, 3))
    _, st, others = b.apply_compliance(B[:, ::2])
    assert st == _lib.GBFEM_OK
    B[:, 1] *= 1e151
    X, st, it = b.apply_compliance(B)
    assert st == _lib.GBFEM_CG_MAXITER and it == others + 1
    assert np.isnan(X[:, 1]).any() and np.isfinite(X[:, ::2]).all()
    B[:, 1] *= 1e10  # |b|^2 is infinite: no iteration
    _, st, it = b.apply_compliance(B)
    assert st == _lib.GBFEM_CG_MAXITER and it == others
    b.close()


def test_iterations_of_a_mixed_solve_that_breaks_down(gpu_lib):
    """One free node whose 3x3 block is 2^40 times ones (the damping; the element's own part rounds away) and the
    right-hand side 2^40 (1, 0, 0). In exact FP32: alpha = 1, r = (0, -1, -1), w.u = 4 = beta r.u / alpha, so the
    second alpha is 2 / 0. The iteration that would have used it is not counted."""
    from opensurgsim_gb300.body import Body

    nodes = 0.01 * np.array([[0, 0, 0], [1, 0, 0], [0, 1, 0], [0, 0, 1.0]])
    m = TetMesh(nodes, np.array([[0, 1, 2, 3]]), np.array([1e3]), np.array([0.4]), np.array([1000.0]),
                np.arange(3, 12), (1, 1, 1), 0.01)
    b = Body(m, gravity_enabled=False, cg_tolerance=1e-10, precision=_lib.PRECISION_MIXED)
    b.set_tuning(64, 4, 2, _lib.CG_ONE_PHASE)
    b.add_external_force(0, [1.0, 0, 0, 0], [2.0 ** 40, 0, 0], damping=2.0 ** 40 * np.ones((3, 3)))
    b.step(1e-3)
    q = b.stats()
    b.close()
    assert q["cg_max_iterations_hit"] == 1 and q["cg_iterations"] == 0
