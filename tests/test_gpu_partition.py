"""The two-phase CG's split of a system over CTAs (gbfem_pcg.cu) where the search for a CTA's first chunk
cuts the chunk range into pieces of a multiple of 32 entries."""

import numpy as np
import pytest

from opensurgsim_gb300 import _lib, mesh

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims", [(24, 24, 104), (24, 27, 140)])  # 2,051 and 3,085 chunks
def test_partition_search_over_a_multiple_of_32_chunks(gpu_lib, dims):
    from opensurgsim_gb300.body import Body

    s = mesh.scene_cube(*dims, seed=1)
    out = []
    for schedule in (_lib.CG_TWO_PHASE, _lib.CG_ONE_PHASE):
        b = Body(s.mesh, rayleigh_mass=0.01, rayleigh_stiffness=0.001, gravity=(0, 0, -9.81), cg_tolerance=1e-10,
                 precision=_lib.PRECISION_MIXED)
        b.set_tuning(64, 4, 2, schedule)
        assert b.step(1e-3, 1) == _lib.GBFEM_OK
        out.append(b.state()[1])
        b.close()
    # |b - S x| <= 1e-10 |b| for both, cond(S) below 5e3 (a step of 1 ms): 1e-6 of the velocity.
    assert np.linalg.norm(out[0] - out[1]) <= 1e-6 * np.linalg.norm(out[1])
