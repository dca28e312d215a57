"""The resident CG (gbfem_res.cu) against the solves it stands beside: FP64 against the launch-per-iteration
CG (which GBFEM_STEP_TIME_KERNELS selects), the mixed form against the two-phase persistent solve, at the
sizes where shares, chunks and halos begin and end.

Tolerance: both solutions x of one system have |b - S x| <= tol |b|, so they differ by at most
2 tol cond(S) |x|. These systems (S close to M / dt + dt K, cubes of 1 cm, E = 1e5) have cond(S) below 5e3
after the Jacobi scaling's units are uniform; with tol = 1e-12 that is 1e-8 of the velocity change."""

import numpy as np
import pytest

from opensurgsim_gb300 import _lib, mesh

pytestmark = pytest.mark.gpu
KW = dict(rayleigh_mass=0.01, rayleigh_stiffness=0.001, gravity=(0, 0, -9.81), cg_tolerance=1e-12)
BOUND = 1e-8


def _step(scene, two, **kw):
    """One step from a moving state: the velocity change and the CG iterations, resident or (two) not."""
    from opensurgsim_gb300.body import Body

    b = Body(scene.mesh, **{**KW, **kw})
    v = np.random.default_rng(5).normal(0, 0.05, b.n)
    v[scene.mesh.bc_dofs] = 0.0
    b.set_state(None, v)
    flags = 0
    if two and kw["precision"] == _lib.PRECISION_MIXED:
        b.set_tuning(64, 4, 2, _lib.CG_TWO_PHASE)
    elif two:
        flags = _lib.STEP_TIME_KERNELS
    assert b.step(1e-3, 1, flags) == _lib.GBFEM_OK
    launches = b.stats()["kernel_launches"]
    it = b.stats()["cg_iterations"]
    dv = b.state()[1] - v
    b.close()
    return dv, it, launches


# Nodes: 8 (a quarter of a chunk), 32 (one chunk exactly), 36, 64, then several shares: the small ones along a
# curve or in node order, the compact ones (four chunks and more), and shares that keep only part of their matrix.
@pytest.mark.parametrize("dims", [(1, 1, 1), (1, 3, 3), (2, 2, 3), (3, 3, 3), (7, 7, 7), (10, 11, 12), (17, 19, 23),
                                  (30, 31, 44)])
@pytest.mark.parametrize("precision", [_lib.PRECISION_FP64, _lib.PRECISION_MIXED])
def test_resident_solve_equals_the_others(gpu_lib, dims, precision):
    s = mesh.scene_cube(*dims, seed=3)
    a, ia, la = _step(s, False, precision=precision)
    b, ib, lb = _step(s, True, precision=precision)
    assert np.linalg.norm(a - b) <= BOUND * np.linalg.norm(b)
    if precision == _lib.PRECISION_FP64:  # the same recurrences (the mixed schedules run different ones)
        assert abs(ia - ib) <= max(4, 0.1 * ib), (ia, ib)
        assert la < 10 < lb  # one launch a solve


@pytest.mark.parametrize("element_type,lumping", [(_lib.ELEMENT_LINEAR_TET, False), (_lib.ELEMENT_HEXAHEDRON, False),
                                                  (_lib.ELEMENT_COROTATIONAL_TET, True)])
@pytest.mark.parametrize("precision", [_lib.PRECISION_FP64, _lib.PRECISION_MIXED])
def test_resident_solve_of_the_other_systems(gpu_lib, element_type, lumping, precision):
    hexes = element_type == _lib.ELEMENT_HEXAHEDRON
    s = mesh.scene_hex_cube(6, 7, 9, seed=4, jitter=0.1) if hexes else mesh.scene_cube(6, 7, 9, seed=4)
    kw = dict(precision=precision, element_type=element_type, mass_lumping=lumping)
    a, b = _step(s, False, **kw)[0], _step(s, True, **kw)[0]
    assert np.linalg.norm(a - b) <= BOUND * np.linalg.norm(b)


def test_vectors_in_global_memory(gpu_lib):
    """150,000 nodes: shares whose search direction and solution stay in global memory."""
    s = mesh.scene_cube(44, 45, 72, seed=2)
    a, b = (_step(s, two, precision=_lib.PRECISION_MIXED)[0] for two in (False, True))
    assert np.linalg.norm(a - b) <= BOUND * np.linalg.norm(b)


def test_more_shares_than_sms(gpu_lib):
    """A batch whose systems outnumber the SMs several times over, in both forms: the same bits run to run,
    every mesh as in a handle of its own."""
    from opensurgsim_gb300.body import Body

    scenes = [mesh.scene_cube(2 + k % 9, 3, 2 + k % 4, seed=k, young=1e4 * (1 + k % 50)) for k in range(500)]
    for precision in (_lib.PRECISION_FP64, _lib.PRECISION_MIXED):
        runs = []
        for _ in range(2):
            b = Body([s.mesh for s in scenes], precision=precision, **KW)
            assert b.step(1e-3, 2) == _lib.GBFEM_OK
            assert b.segment_stats()["converged"].all()
            runs.append(b.state()[1])
            offsets = b.node_offsets.copy()
            b.close()
        assert np.array_equal(*runs)
        for k in (0, 123, 499):
            one = Body(scenes[k].mesh, precision=precision, **KW)
            assert one.step(1e-3, 2) == _lib.GBFEM_OK
            v = runs[0][3 * offsets[k]:3 * offsets[k + 1]]
            assert np.linalg.norm(v - one.state()[1]) <= BOUND * np.linalg.norm(v)
            one.close()
