"""What resident solves (gbfem_res.cu) report when they break down: as the launch-per-iteration and the persistent
solves do."""

import numpy as np
import pytest

from opensurgsim_gb300 import _lib, mesh

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
