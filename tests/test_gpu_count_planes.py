"""The counts of a batch of many planes (a warp per plane, quiet words left out)
against the same chunks one by one (a block per plane): line and word ends,
full and empty neighbours, single-word lines, chunks without a surface."""
import pytest
import torch

from binarymeshfitting_gb300 import _lib as L
from binarymeshfitting_gb300 import workloads
from binarymeshfitting_gb300.engine import Batch

pytestmark = pytest.mark.gpu

DIMS = [2, 3, 31, 32, 33, 63, 64, 65, 95, 97, 129, 160]


@pytest.mark.parametrize("mode,placement", [(L.MODE_R, L.PLACE_CENTER), (L.MODE_Q, L.PLACE_CENTER),
                                            (L.MODE_Q, L.PLACE_QEF)])
def test_planes_match_single_chunks(ctx, mode, placement):
    field = workloads.terrain_field()
    descs = []
    for i, d in enumerate(DIMS * 4):
        scale = (0.25, 1.0, 3.0, 8.0)[i // len(DIMS)] * max(1.0, 16.0 / (d - 1))
        y = 64.0 - (0.5 if i % 5 else 1.4) * (d - 1) * scale  # every fifth mostly off the surface
        descs.append(L.ChunkDesc.make((100.0 + 57.0 * i, y, 900.0 - 31.0 * i), scale, d))
    descs += [L.ChunkDesc.make((0.0, 600.0, 0.0), 1.0, 33), L.ChunkDesc.make((0.0, -600.0, 0.0), 1.0, 65)]
    assert sum(d.dim for d in descs) >= 2048
    b = Batch(ctx, descs, field, mode=mode, placement=placement)
    b.allocate(1 << 21, 1 << 23)
    nv, ni = b.run(use_graph=False)
    assert nv > 50000
    for i, d in enumerate(descs):
        m = ctx.extract_chunk(d, field, mode=mode, placement=placement)
        got = b.chunk_mesh(i)
        assert (got["pos"].shape[0], got["idx"].shape[0]) == (m.n_verts, m.n_idx)
        if m.n_verts:
            assert torch.equal(got["idx"], m.idx)
            assert torch.equal(got["pos"].contiguous().view(torch.int32), m.pos.contiguous().view(torch.int32))
    b.close()
