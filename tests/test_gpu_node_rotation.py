"""Compliance warping's node rotations (the running spherical averages of gbfem_kernels.cu) on both sides of the
slerp weights' series (1 - cos of the half angle between rotations at 0.01: 16 degrees between elements), through
the warped compliance columns against the oracle's."""

import numpy as np
import pytest

from opensurgsim_gb300 import _lib, mesh

pytestmark = pytest.mark.gpu


# Twists over the length of a bar of 4 cells: 0, 0.2 (elements a few degrees apart), 1.1 (about 16 degrees), 3 radians.
@pytest.mark.parametrize("twist", [0.0, 0.2, 1.1, 3.0])
def test_warped_columns_over_twists(gpu_lib, twist):
    from opensurgsim_gb300.body import Body
    from oracle import oracle as O

    s = mesh.scene_cube(2, 2, 4, seed=3, young=3e5)
    kw = dict(rayleigh_mass=0.01, rayleigh_stiffness=0.001, gravity=(0, 0, -9.81), cg_tolerance=1e-12)
    b, o = Body(s.mesh, **kw), O.OracleModel(s.mesh, **kw)
    X = s.mesh.nodes
    z = (X[:, 2] - X[:, 2].min()) / np.ptp(X[:, 2])
    c = X.mean(axis=0)
    ca, sa = np.cos(twist * z), np.sin(twist * z)
    x = X.copy()
    x[:, 0] = c[0] + ca * (X[:, 0] - c[0]) - sa * (X[:, 1] - c[1])
    x[:, 1] = c[1] + sa * (X[:, 0] - c[0]) + ca * (X[:, 1] - c[1])
    for m in (b, o):
        m.set_state(x.ravel(), np.zeros(b.n))
    assert b.step(1e-3) == _lib.GBFEM_OK and o.step(1e-3) == 0
    B = np.random.default_rng(0).normal(size=(b.n, 3))
    got, st, _ = b.apply_compliance(B, warping=True)
    want, ost, _ = o.apply_compliance(B, warping=True)
    assert st == _lib.GBFEM_OK and ost == 0
    assert np.linalg.norm(got - want) <= 1e-8 * np.linalg.norm(want)  # as the other compliance tests
