"""The solves that stand beside the resident CG, on systems whose shares do not fit an SM: a hub node that couples to
more rows than a share's shared memory holds. FP64 single bodies run the launch-per-iteration CG, FP64 batches and the
mixed form's one-phase schedule the persistent solve, compliance columns go eight at a time (those of batches always do).

Tolerance: a solve leaves |b - S x| <= tol |b| by its recursive or refreshed residual, which drifts from the true one by
a few iterations' roundings: 2 tol, measured with the system exported in FP64."""

import numpy as np
import pytest
import scipy.sparse as sp

from opensurgsim_gb300 import _lib, mesh
from opensurgsim_gb300.mesh import TetMesh

pytestmark = pytest.mark.gpu
TOL = 1e-10
KW = dict(rayleigh_mass=0.01, rayleigh_stiffness=0.001, gravity=(0, 0, -9.81), cg_tolerance=TOL)


def _hub(m=72):
    """A dome of m x m nodes, two tetrahedra a square, all of them with the centre (node 0); one edge is fixed."""
    a, b = np.meshgrid(np.linspace(-1, 1, m), np.linspace(-1, 1, m), indexing="ij")
    p = np.stack([a, b, np.full_like(a, 1.0)], -1).reshape(-1, 3)
    nodes = np.vstack([np.zeros(3), 0.05 * p / np.linalg.norm(p, axis=1)[:, None]])
    i, j = np.meshgrid(np.arange(m - 1), np.arange(m - 1), indexing="ij")
    k = (1 + i * m + j).ravel()
    tets = np.vstack([np.stack([0 * k, k, k + m, k + m + 1], 1), np.stack([0 * k, k, k + m + 1, k + 1], 1)])
    x = nodes[tets]
    assert (np.linalg.det(x[:, 1:] - x[:, :1]) > 0).all()
    E = len(tets)
    return TetMesh(nodes, tets, np.full(E, 1e3), np.full(E, 0.4), np.full(E, 1000.0), np.arange(3, 3 * (1 + m)), (), 0.0)


def _moving(m, precision, **kw):
    from opensurgsim_gb300.body import Body

    b = Body(m, precision=precision, **{**KW, **kw})
    meshes = m if isinstance(m, list) else [m]
    v = np.concatenate([np.random.default_rng(k).normal(0, 0.05, 3 * len(q.nodes)) for k, q in enumerate(meshes)])
    n0 = 0
    for q in meshes:
        v[3 * n0 + np.asarray(q.bc_dofs)] = 0.0
        n0 += len(q.nodes)
    b.set_state(None, v)
    return b, v


def _resident(b):
    return _lib.load().gbfem_set_solve_fault(b.handle, _lib.SOLVE_FAULT_SHARE, 1000) == _lib.GBFEM_OK and \
        _lib.load().gbfem_set_solve_fault(b.handle, _lib.SOLVE_FAULT_NONE, 0) == _lib.GBFEM_OK


def _system(m, v):
    """S and the right-hand side of the first step from velocities v."""
    b, _ = _moving(m, _lib.PRECISION_FP64)
    b.set_state(None, v)
    assert b.step(1e-3, 1, _lib.STEP_KEEP_SYSTEM) == _lib.GBFEM_OK
    colptr, rowidx = b.pattern()
    q = b.system()
    b.close()
    lower = sp.tril(sp.csc_matrix((q["S"], rowidx, colptr), shape=(v.size, v.size)), format="csr")
    return lower + sp.tril(lower, -1).T, q["rhs"]


@pytest.fixture(scope="module")
def hub():
    return _hub()


def test_fp64_batch(gpu_lib, hub):
    cube = mesh.scene_cube(9, 10, 11, seed=3).mesh
    b, v = _moving([hub, cube], _lib.PRECISION_FP64)
    x0 = b.state()[0]
    assert not _resident(b)
    assert b.step(1e-3) == _lib.GBFEM_OK and b.segment_stats()["converged"].all()
    dv = b.state()[1] - v
    n = 3 * len(hub.nodes)
    for part, m in ((slice(0, n), hub), (slice(n, None), cube)):
        S, rhs = _system(m, v[part])
        assert np.linalg.norm(rhs - S @ dv[part]) <= 2 * TOL * np.linalg.norm(rhs)
        one, _ = _moving(m, _lib.PRECISION_FP64)
        one.set_state(None, v[part])
        assert one.step(1e-3) == _lib.GBFEM_OK
        assert np.linalg.norm(rhs - S @ (one.state()[1] - v[part])) <= 2 * TOL * np.linalg.norm(rhs)
        assert _resident(one) == (m is cube)
        one.close()
    # The same in a graph.
    b.set_state(x0, v)
    assert b.step(1e-3, 1, _lib.STEP_GRAPH) == _lib.GBFEM_OK
    assert np.array_equal(b.state()[1] - v, dv)
    b.close()


def test_one_phase_schedule(gpu_lib, hub):
    """Against the two-phase schedule, by the difference's residual on the FP64 system (the FP32 one is within 1e-6)."""
    dv = []
    for schedule in (_lib.CG_ONE_PHASE, _lib.CG_TWO_PHASE):
        b, v = _moving(hub, _lib.PRECISION_MIXED)
        assert not _resident(b) and b.tuning()[3] == _lib.CG_ONE_PHASE
        b.set_tuning(64, 4, 2, schedule)
        assert b.step(1e-3) == _lib.GBFEM_OK
        dv.append(b.state()[1] - v)
        b.close()
    S, rhs = _system(hub, v)
    assert np.linalg.norm(S @ (dv[0] - dv[1])) <= 2.1 * TOL * np.linalg.norm(rhs)


@pytest.mark.parametrize("columns", [1, 11])
def test_compliance_of_a_body(gpu_lib, hub, columns):
    X = []
    for precision in (_lib.PRECISION_FP64, _lib.PRECISION_MIXED):
        b, v = _moving(hub, precision)
        B = np.random.default_rng(7).normal(size=(b.n, columns))
        assert b.step(1e-3) == _lib.GBFEM_OK
        x, st, it = b.apply_compliance(B)
        assert st == _lib.GBFEM_OK and it > columns and not _resident(b)
        X.append(x)
        b.close()
    S, _ = _system(hub, v)
    W = np.where(np.isin(np.arange(v.size), hub.bc_dofs)[:, None], 0.0, B)
    assert (np.linalg.norm(W - S @ X[0], axis=0) <= 2 * TOL * np.linalg.norm(W, axis=0)).all()
    # The mixed form's system is assembled in FP32.
    assert np.linalg.norm(X[1] - X[0]) <= 1e-5 * np.linalg.norm(X[0])


@pytest.mark.parametrize("warping", [False, True])
def test_compliance_of_a_batch(gpu_lib, warping):
    """Eight columns at a time over all meshes, against every mesh's own (resident) columns: |b - S x| <= tol |b| of the
    whole column in one and of the mesh's in the other, cond(S) below 5e3 for these cubes."""
    meshes = [mesh.scene_cube(3, 4, 5, seed=1).mesh, mesh.scene_cube(6, 5, 4, seed=2).mesh]
    b, v = _moving(meshes, _lib.PRECISION_FP64, cg_tolerance=1e-12)
    assert b.step(1e-3, 3) == _lib.GBFEM_OK
    B = np.random.default_rng(7).normal(size=(b.n, 11))
    X, st, _ = b.apply_compliance(B, warping=warping)
    assert st == _lib.GBFEM_OK
    off = 3 * b.node_offsets
    b.close()
    for k, m in enumerate(meshes):
        part = slice(off[k], off[k + 1])
        one, _ = _moving(m, _lib.PRECISION_FP64, cg_tolerance=1e-12)
        one.set_state(None, v[part])
        assert one.step(1e-3, 3) == _lib.GBFEM_OK
        x, st, _ = one.apply_compliance(B[part], warping=warping)
        assert st == _lib.GBFEM_OK
        assert np.linalg.norm(X[part] - x) <= 2e-8 * np.linalg.norm(X)
        one.close()


def test_statistics_say_which_solve_runs(gpu_lib, hub):
    cube = mesh.scene_cube(4, 4, 4).mesh
    for m, precision, schedule, resident in ((hub, _lib.PRECISION_FP64, None, 0), (hub, _lib.PRECISION_MIXED, None, 0),
                                             (cube, _lib.PRECISION_FP64, None, 1), (cube, _lib.PRECISION_MIXED, None, 1),
                                             (cube, _lib.PRECISION_MIXED, _lib.CG_TWO_PHASE, 0),
                                             ([hub, cube], _lib.PRECISION_FP64, None, 0), ([cube] * 3, _lib.PRECISION_FP64, None, 1)):
        b, _ = _moving(m, precision)
        if schedule is not None:
            b.set_tuning(64, 4, 2, schedule)
        assert b.step(1e-3) == _lib.GBFEM_OK and b.stats()["resident"] == resident
        b.close()
