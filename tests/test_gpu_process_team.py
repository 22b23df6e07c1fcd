"""Smoothing of a caller's mesh in one launch: against the structured adjacency of
the same extracted mesh, and, with lists and indices that an extraction does not
give, against the step-by-step form, which a mesh padded with unused vertices
past the one-launch size takes.  Bit for bit, for lists that fit their valences
(of a longer one any entries are kept, in either form)."""
import numpy as np
import pytest
import torch

from binarymeshfitting_gb300 import _lib as L
from binarymeshfitting_gb300 import workloads
from binarymeshfitting_gb300.engine import ChunkMesh

pytestmark = pytest.mark.gpu

PAD = 200001


@pytest.mark.parametrize("dim", [3, 9, 33, 70, 129])
@pytest.mark.parametrize("mode,iters,boundary,normals", [(L.MODE_R, 4, False, True), (L.MODE_R, 1, True, False),
                                                         (L.MODE_Q, 5, True, True), (L.MODE_Q, 2, False, False)])
def test_extracted_mesh(ctx, dim, mode, iters, boundary, normals):
    scale = 128.0 / (dim - 1)
    desc, field = L.ChunkDesc.make((10.0, 5.0, 20.0), scale, dim), workloads.terrain_field()
    want = ctx.extract_chunk(desc, field, mode=mode, iters=iters, process_boundary=boundary, smooth_normals=normals)
    got = ctx.extract_chunk(desc, field, mode=mode)
    assert got.n_verts == want.n_verts > 0
    if normals:
        got.nrm = torch.zeros_like(got.pos)
    ctx.process(got, iters, boundary, normals)
    torch.cuda.synchronize()
    assert torch.equal(got.pos.contiguous().view(torch.int32), want.pos.contiguous().view(torch.int32))
    if normals:
        assert torch.equal(torch.nan_to_num(got.nrm), torch.nan_to_num(want.nrm))


def _mesh(nv, prims, N, seed, pad, wrong):
    rng = np.random.default_rng(seed)
    n = max(nv, PAD) if pad else nv
    idx = rng.integers(0, nv, (prims, N))
    m = min(prims // 3, 300)
    idx[:m, 0] = rng.integers(0, 3, m)  # a few vertices with long lists
    val = np.bincount(idx.reshape(-1), minlength=n)
    assert val.max() <= 255  # (of a longer list any 255 entries are kept, in either form)
    if wrong:  # indices outside the mesh: some valences are larger than their lists
        idx[rng.integers(0, prims, 5), 1] = 0x7FFFFFF0
    pos = np.zeros((n, 3), np.float32)
    pos[:nv] = rng.normal(size=(nv, 3))
    bnd = np.zeros(n, np.uint8)
    bnd[:nv] = rng.random(nv) < 0.2
    t = lambda a: torch.from_numpy(a).cuda()
    return ChunkMesh(pos=t(pos), nrm=torch.zeros((n, 3), device="cuda"), boundary=t(bnd),
                     valence=t(np.minimum(val, 255).astype(np.uint8)), idx=t(idx.astype(np.int32).reshape(-1)),
                     prim_size=N, contains_mesh=True)


@pytest.mark.parametrize("nv,prims,N", [(7, 3, 3), (40, 90, 3), (300, 700, 4), (2000, 5000, 3), (70000, 130000, 3)])
@pytest.mark.parametrize("wrong", [False, True])
def test_any_mesh(ctx, nv, prims, N, wrong):
    out = []
    for pad in (False, True):
        m = _mesh(nv, prims, N, nv + prims, pad, wrong)
        ctx.process(m, 3, False, True)
        torch.cuda.synchronize()
        out.append((m.pos[:nv].clone(), m.nrm[:nv].clone()))
    for a, b in zip(*out):
        assert torch.equal(torch.nan_to_num(a, nan=7.0), torch.nan_to_num(b, nan=7.0))
