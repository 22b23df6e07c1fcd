"""The adjoint sweeps' three forms (whole mesh in one launch, step by step, chunk by
chunk), after each of the forward's, against a plan of the one chunk, whose
gradient the oracle tests pin.  The sweeps' values are the same in every form;
the placement adjoint adds a sample's at most 64 contributions by atomics in
any order, 64 * 2^-24 = 4e-6 of their magnitudes, so a chunk's gradient agrees
within 2e-5 (relative L2)."""
import numpy as np
import pytest
import torch

from binarymeshfitting_gb300 import _lib as L
from binarymeshfitting_gb300.fitting import FitPlan

pytestmark = pytest.mark.gpu


def _grids(n, dim, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    g = torch.arange(dim, dtype=torch.float32, device="cuda")
    out = []
    for _ in range(n):
        c = torch.rand(3, generator=gen, device="cuda") * (dim - 1)  # surfaces cut by the faces too
        r = (g[:, None, None] - c[0]) ** 2 + (g[None, :, None] - c[1]) ** 2 + (g[None, None, :] - c[2]) ** 2
        out.append((r.sqrt() - 0.45 * dim + 0.3 * torch.sin(1.3 * g)[None, None, :]).reshape(-1))
    return torch.cat(out)


@pytest.mark.parametrize("n,dim", [(3, 33), (150, 17), (36, 65), (70, 49), (260, 25), (256, 9), (300, 12), (165, 30)])
@pytest.mark.parametrize("iters", [1, 4])
def test_forms_match_single_chunk(ctx, n, dim, iters):
    dens = _grids(n, dim, 7 * n + dim)
    plan = FitPlan(ctx, n, dim, L.PLACE_MASSPOINT, iters, vcap=n * dim * dim * 6)
    plan.forward(dens)
    info = plan.info.cpu().numpy().reshape(n, 6)
    gen = torch.Generator(device="cuda").manual_seed(dim)
    gp = torch.randn((plan.n_verts, 3), generator=gen, device="cuda")
    short = plan.n_verts - 5  # the others count as zero
    whole = plan.backward(gp[:short]).reshape(n, -1)
    one = FitPlan(ctx, 1, dim, L.PLACE_MASSPOINT, iters, vcap=dim * dim * 6)
    for c in (0, 1, n // 2, n - 1):
        one.forward(dens.reshape(n, -1)[c].contiguous())
        v0, nv = int(info[c, 0]), int(info[c, 1])
        assert one.n_verts == nv > 0
        g = gp[v0:v0 + nv].clone()
        if v0 + nv > short:
            g[short - v0 - nv:] = 0.0
        want = one.backward(g).double().reshape(-1)
        err = torch.linalg.norm(whole[c].double() - want) / torch.linalg.norm(want)
        assert float(err) <= 2e-5, (c, float(err))
    plan.close()
    one.close()
