"""The 2D heightmap's column fill (each column's first inside line by search, words
from ballots in between) against the full fill of every sample: word and line
ends, planes of one word and of many lines, columns all inside or all outside,
steep columns, and a negative scale, whose columns turn the other way."""
import pytest
import torch

from binarymeshfitting_gb300 import _lib as L
from binarymeshfitting_gb300 import workloads
from binarymeshfitting_gb300.engine import Batch

pytestmark = pytest.mark.gpu

DIMS = [2, 3, 31, 32, 33, 64, 65, 97, 130, 200]


@pytest.mark.parametrize("g,height", [(0.25, 75.0), (0.25, 4000.0), (-0.25, 75.0), (0.25, 0.0)])
def test_column_fill_matches_full(ctx, g, height):
    p = list(workloads.TERRAIN_2D_PARAMS)
    p[0], p[1] = g, height
    descs = []
    for i, d in enumerate(DIMS * 3):
        scale = (0.5, 4.0, 16.0)[i // len(DIMS)]
        descs.append(L.ChunkDesc.make((77.0 * i, (0.0, -0.5, -1.0)[i % 3] * (d - 1) * scale + 3.0, 41.0 * i), scale, d))
    b = Batch(ctx, descs, workloads.terrain2d_field(p), mode=L.MODE_R, iters=0)
    b.allocate(1 << 22, 1 << 24)
    b.set_tuning(fill_band=0)
    nv, ni = b.run(use_graph=False)
    assert nv > 1000
    pos, idx, info = b.bufs["pos"][:nv].clone(), b.bufs["idx"][:ni].clone(), b.bufs["info"].clone()
    b.bufs["pos"].zero_()
    b.set_tuning(fill_band=1)
    assert b.run(use_graph=False) == (nv, ni)
    assert torch.equal(b.bufs["info"], info)
    assert torch.equal(b.bufs["idx"][:ni], idx)
    assert torch.equal(b.bufs["pos"][:nv].view(torch.int32), pos.view(torch.int32))
    b.close()
