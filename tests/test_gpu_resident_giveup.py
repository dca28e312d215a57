"""Waits of the resident solves (gbfem_res.cu) that run out, without a GPU fault: gbfem_set_solve_fault leaves a share
of a system out of the launch, so words that the others wait for are never sent. Every wait has a limit, after which
the solve reports an error; the tests check the status, the time it took and that the same handle then solves
as one that never failed (the exchange buffers' tags have moved on)."""

import time

import numpy as np
import pytest

from opensurgsim_gb300 import _lib, mesh

pytestmark = pytest.mark.gpu
KW = dict(rayleigh_mass=0.01, rayleigh_stiffness=0.001, gravity=(0, 0, -9.81), cg_tolerance=1e-10)
WAIT = 20_000_000


def _body(kind, precision, seed=3):
    from opensurgsim_gb300.body import Body

    if kind == "batch":  # several shares a mesh, FP64: more shares than SMs
        meshes = [mesh.scene_cube(14 + k, 15, 16, seed=k).mesh for k in range(12)]
    else:
        meshes = mesh.scene_cube(*kind, seed=seed).mesh
    return Body(meshes, precision=precision, **KW)


def _fault(b, fault, wait=WAIT):
    return _lib.load().gbfem_set_solve_fault(b.handle, fault, wait)


def _fails(b, f):
    t = time.perf_counter()
    with pytest.raises(_lib.GbfemError) as e:
        f()
    assert e.value.status == _lib.GBFEM_CUDA_ERROR and "timed out" in str(e.value)
    return time.perf_counter() - t


# Shares as one cluster (FP64 80 and mixed 1,331 nodes), over many CTAs, and a batch.
@pytest.mark.parametrize("kind,precision", [((3, 3, 4), _lib.PRECISION_FP64), ((10, 10, 10), _lib.PRECISION_MIXED),
                                            ((10, 10, 10), _lib.PRECISION_FP64), ((20, 20, 40), _lib.PRECISION_MIXED),
                                            ("batch", _lib.PRECISION_FP64), ("batch", _lib.PRECISION_MIXED)])
@pytest.mark.parametrize("fault", [_lib.SOLVE_FAULT_SHARE, _lib.SOLVE_FAULT_ROWS])
def test_a_missing_share_ends_the_solve(gpu_lib, kind, precision, fault):
    fresh = _body(kind, precision)
    assert fresh.step(1e-3, 2) == _lib.GBFEM_OK
    b = _body(kind, precision)
    for _ in range(2):
        assert _fault(b, fault) == _lib.GBFEM_OK
        x, v = b.state()
        seconds = _fails(b, lambda: b.step(1e-3))
        assert 1e-9 * WAIT <= seconds < 1e-9 * WAIT + 0.5
        assert all(np.array_equal(p, q) for p, q in zip((x, v), b.state()))
        # One failure a call, also of calls of another kind.
        assert _fault(b, _lib.SOLVE_FAULT_NONE) == _lib.GBFEM_OK
        assert b.step(1e-3) == _lib.GBFEM_OK
    assert all(np.array_equal(p, q) for p, q in zip(fresh.state(), b.state()))
    fresh.close()
    b.close()


@pytest.mark.parametrize("kind", [(10, 10, 10), (20, 20, 40), "batch"])
def test_graphs(gpu_lib, kind):
    b = _body(kind, _lib.PRECISION_MIXED)
    x, v = b.state()
    assert b.step(1e-3, 3, _lib.STEP_GRAPH) == _lib.GBFEM_OK
    want = b.state()
    b.set_state(x, v)
    assert _fault(b, _lib.SOLVE_FAULT_SHARE) == _lib.GBFEM_OK
    _fails(b, lambda: b.step(1e-3, 3, _lib.STEP_GRAPH))
    assert _fault(b, _lib.SOLVE_FAULT_NONE) == _lib.GBFEM_OK
    for flags in (0, _lib.STEP_GRAPH):
        b.set_state(x, v)
        assert b.step(1e-3, 3, flags) == _lib.GBFEM_OK
        assert all(np.array_equal(p, q) for p, q in zip(want, b.state()))
    b.close()


def test_arguments(gpu_lib):
    b = _body((10, 10, 10), _lib.PRECISION_MIXED)
    assert _fault(b, 3) == _fault(b, -1) == _fault(b, 1, 100) == _fault(b, 1, 2_000_000_000) == _lib.GBFEM_INVALID_ARG
    b.set_tuning(64, 4, 2, _lib.CG_TWO_PHASE)
    assert _fault(b, 1) == _lib.GBFEM_INVALID_ARG
    b.close()
    one = _body((1, 1, 1), _lib.PRECISION_FP64)
    assert _fault(one, 1) == _lib.GBFEM_INVALID_ARG and _fault(one, 0) == _lib.GBFEM_OK
    one.close()
