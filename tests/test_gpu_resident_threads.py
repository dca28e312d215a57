"""Resident solves of several handles from several threads at once (clusters, cooperative launches of part and all
of the chip, batches, compliance columns): the bits of the same work done alone."""

import threading

import numpy as np
import pytest

from opensurgsim_gb300 import _lib, mesh

pytestmark = pytest.mark.gpu
KW = dict(rayleigh_mass=0.01, rayleigh_stiffness=0.001, gravity=(0, 0, -9.81), cg_tolerance=1e-10)


def _bodies():
    from opensurgsim_gb300.body import Body

    batch = [s.mesh for s in mesh.scenes_batch(count=8, lo=300, hi=2000, seed=3)]
    return [Body(m, precision=p, **KW) for m, p in
            ((mesh.scene_cube(3, 3, 4).mesh, _lib.PRECISION_FP64), (mesh.scene_cube(10, 10, 10).mesh, _lib.PRECISION_FP64),
             (mesh.scene_cube(9, 9, 9).mesh, _lib.PRECISION_MIXED), (mesh.scene_cube(20, 20, 30).mesh, _lib.PRECISION_MIXED),
             (batch, _lib.PRECISION_FP64), (batch, _lib.PRECISION_MIXED))]


def _work(k, body, out):
    rng = np.random.default_rng(k)
    body.set_state(None, rng.normal(0, 0.02, body.n))
    if any(body.step(1e-3, 1) != _lib.GBFEM_OK for _ in range(20)):
        return
    columns = body.apply_compliance(rng.normal(size=(body.n, 5)))[0] if k < 4 else None
    out[k] = (*body.state(), columns)


def test_handles_in_threads_equal_handles_alone(gpu_lib):
    alone, together = {}, {}
    for k, b in enumerate(_bodies()):
        _work(k, b, alone)
        b.close()
    bodies = _bodies()
    threads = [threading.Thread(target=_work, args=(k, b, together)) for k, b in enumerate(bodies)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for b in bodies:
        b.close()
    assert sorted(alone) == sorted(together) == list(range(6))
    for k in alone:
        for a, b in zip(alone[k], together[k]):
            assert (a is None and b is None) or np.array_equal(a, b), k
