"""Mode Q updates through the band fill: the densities the mesh reads are exact
whatever the arena held before, at word edges, chunk faces, few samples and
one to nine octaves; bit for bit the mesh of a full fill."""
import pytest
import torch

from binarymeshfitting_gb300 import _lib as L
from binarymeshfitting_gb300 import workloads
from binarymeshfitting_gb300.engine import Batch

pytestmark = pytest.mark.gpu

DIMS = [2, 3, 31, 32, 33, 34, 64, 65, 66, 97]


def _descs(shift):
    out = []
    for i, d in enumerate(DIMS * 2):
        scale = (0.5, 2.0, 8.0)[(i + i // len(DIMS)) % 3] * max(1.0, 16.0 / (d - 1))
        out.append(L.ChunkDesc.make((300.0 + 91.0 * i + shift, 64.0 - 0.5 * (d - 1) * scale, 700.0 - 37.0 * i), scale, d))
    return out


def _mesh(b):
    nv, ni = b.run(use_graph=False)
    return {k: b.bufs[k][:n].clone() for k, n in (("pos", nv), ("idx", ni), ("boundary", nv))} | {
        "info": b.bufs["info"].clone()}


@pytest.mark.parametrize("octaves", [1, 5, 9])
@pytest.mark.parametrize("placement", [L.PLACE_CENTER, L.PLACE_MASSPOINT, L.PLACE_QEF])
def test_band_matches_full(ctx, placement, octaves):
    p = list(workloads.TERRAIN_PARAMS)
    p[5] = octaves
    b = Batch(ctx, _descs(0.0), L.Field.make(L.FIELD_TERRAIN_FBM, p), mode=L.MODE_Q, placement=placement)
    b.allocate(400000, 1600000)
    b.set_tuning(fill_mode=0)  # every density exact
    full = _mesh(b)
    assert full["pos"].shape[0] > 10000
    b.set_descs(_descs(5000.0))  # leaves other densities in the arena
    other = _mesh(b)
    assert other["pos"].shape != full["pos"].shape
    b.set_descs(_descs(0.0))
    for mode in (1, 2):
        for run in (4, 8, 16):
            b.set_tuning(fill_mode=mode, fill_run=run)
            got = _mesh(b)
            for k, r in full.items():
                assert torch.equal(got[k].view(torch.uint8), r.view(torch.uint8)), (k, mode, run)
    b.run(use_graph=True)
    b.run(use_graph=True)
    assert torch.equal(b.bufs["pos"][:full["pos"].shape[0]].view(torch.int32), full["pos"].view(torch.int32))
    b.close()
