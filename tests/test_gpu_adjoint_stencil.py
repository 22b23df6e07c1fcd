"""The wide QEF adjoint where its stencil (the 32 samples around a cell) is clamped:
surfaces cut by the chunk's faces, chunks of a few samples, lists of any length.
Its gradient against the FP32 adjoint, a separate code path, within that path's
own bar (1e-2 relative L2: 1/s^2 times the ~1e-6 FP32 error of small kept
eigenvalues); double-float against FP64 within 2e-5."""
import numpy as np
import pytest
import torch

from binarymeshfitting_gb300 import _lib as L
from binarymeshfitting_gb300.fitting import FitPlan

pytestmark = pytest.mark.gpu


def _grids(n, dim, seed):
    g = np.arange(dim, dtype=np.float64)
    X, Y, Z = np.meshgrid(g, g, g, indexing="ij")
    rng = np.random.default_rng(seed)
    out = []
    for _ in range(n):
        c = rng.uniform(0.0, dim - 1.0, 3)  # anywhere: most spheres leave the chunk
        r = rng.uniform(0.35, 0.75) * dim
        out.append(np.sqrt((X - c[0]) ** 2 + (Y - c[1]) ** 2 + (Z - c[2]) ** 2) - r
                   + 0.35 * np.sin(0.9 * X + rng.uniform(0, 6)) * np.sin(0.8 * Y) * np.sin(1.1 * Z + 1.0))
    return np.concatenate([d.reshape(-1) for d in out]).astype(np.float32)


@pytest.mark.parametrize("n,dim", [(64, 3), (40, 5), (7, 9), (3, 17), (2, 33), (12, 33)])
def test_stencil_at_chunk_faces(ctx, n, dim):
    dens = torch.from_numpy(_grids(n, dim, 100 + dim)).cuda()
    grads, gp = {}, None
    for adjoint in ("f32", "df", "f64"):
        plan = FitPlan(ctx, n, dim, L.PLACE_QEF, 0, vcap=n * dim ** 3 * 2, adjoint=adjoint)
        plan.forward(dens)
        assert plan.n_verts > 0
        if gp is None:
            gp = torch.randn((plan.n_verts, 3), generator=torch.Generator(device="cuda").manual_seed(dim), device="cuda")
        grads[adjoint] = plan.backward(gp).double().cpu().numpy()
        plan.close()
    ref = np.linalg.norm(grads["f64"])
    assert np.isfinite(ref) and ref > 0
    assert np.linalg.norm(grads["df"] - grads["f64"]) <= 2e-5 * ref
    assert np.linalg.norm(grads["f32"] - grads["f64"]) <= 1e-2 * ref
