"""The FP64 step's element kernel on both sides of its split over rows of the grid, against the general element
kernel (which exporting the system selects).

Tolerance: the elements agree to FP64 rounding (test_element_fp64.py); both solves leave |b - S x| <= 1e-12 |b|, cond(S)
below 5e3: 1e-8 of the velocity change."""

import numpy as np
import pytest

from opensurgsim_gb300 import _lib, mesh

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims", [(1, 1, 1), (4, 5, 3), (8, 10, 10), (9, 10, 9)])  # 5, 300, 4,000, 4,050 elements
@pytest.mark.parametrize("lumping", [False, True])
def test_step_with_and_without_the_system_export(gpu_lib, dims, lumping):
    from opensurgsim_gb300.body import Body

    s = mesh.scene_cube(*dims, seed=6)
    out = []
    for flags in (0, _lib.STEP_KEEP_SYSTEM):
        b = Body(s.mesh, rayleigh_mass=0.01, rayleigh_stiffness=0.001, gravity=(0, 0, -9.81), cg_tolerance=1e-12,
                 precision=_lib.PRECISION_FP64, mass_lumping=lumping)
        v = np.random.default_rng(2).normal(0, 0.05, b.n)
        v[s.mesh.bc_dofs] = 0.0
        b.set_state(None, v)
        assert b.step(1e-3, 1, flags) == _lib.GBFEM_OK
        out.append(b.state()[1] - v)
        b.close()
    assert np.linalg.norm(out[0] - out[1]) <= 1e-8 * np.linalg.norm(out[1])
