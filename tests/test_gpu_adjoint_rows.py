"""The element adjoint's split of its passes over rows of the grid (gbfem_adjoint.cu), at element counts on both
sides of its rules: the FP32 and FP64 forms split differently, and their gradients agree as on small meshes."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


# 2,000 elements (ten rows), 2,520 (four), 102,060 (one row in FP32, four in FP64).
@pytest.mark.parametrize("dims", [(5, 8, 10), (7, 8, 9), (27, 27, 28)])
def test_gradients_agree_across_the_forms(gpu_lib, dims):
    from opensurgsim_gb300 import _lib, mesh
    from opensurgsim_gb300.autograd import rollout
    from opensurgsim_gb300.body import Body

    scene = mesh.scene_cube(*dims, seed=1)
    rng = np.random.default_rng(4)
    grads = []
    for precision in (_lib.PRECISION_FP64, _lib.PRECISION_MIXED):
        body = Body.from_scene(scene, precision=precision, cg_tolerance=1e-12)
        if not grads:
            v = rng.normal(0, 0.01, body.n)
            v[scene.mesh.bc_dofs] = 0.0
            w = rng.normal(0, 1, body.n)
        theta = torch.tensor(np.log(scene.mesh.young), dtype=torch.float64, device="cuda:0", requires_grad=True)
        x0, v0 = (torch.tensor(a, dtype=torch.float64, device="cuda:0", requires_grad=True)
                  for a in (scene.mesh.nodes.ravel(), v))
        xT, _ = rollout(body, theta, x0, v0, scene.dt, 1)
        (torch.tensor(w, device="cuda:0") * xT).sum().backward()
        grads.append([t.grad.cpu().numpy() for t in (theta, x0, v0)])
        body.close()
    for fp64, mixed in zip(*grads):
        assert np.linalg.norm(mixed - fp64) <= 1e-4 * np.linalg.norm(fp64)
