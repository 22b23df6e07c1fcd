"""The smoothing sweeps in each of their forms (one launch per step, one
cooperative launch, chunk by chunk with clusters) against the oracle, on walls
along the axes: there a vertex's new normal can have y == 0 exactly, and it
keeps its older one, from sweeps whose normals are not computed."""
import numpy as np
import pytest

from binarymeshfitting_gb300 import _lib as L
from binarymeshfitting_gb300.engine import Batch
from oracle import cpu

pytestmark = pytest.mark.gpu

# (chunks, dim, dim of every 50th chunk): a few columns (one cooperative launch),
# more than that in few chunks (launches), in many chunks (chunk by chunk, the
# large ones by clusters)
FORMS = {"team": (3, 33, 33), "launches": (100, 41, 41), "chunks": (330, 24, 65)}
# the 2D heightmap at a height where y is below its rounding: walls along y
FIELDS = {"walls": (L.FIELD_TERRAIN_2D, (0.25, 1e9, 13, 0.87, 0.585, 0.488, 5, 3)), "cuboid": (L.FIELD_CUBOID, (96.0,)),
          "sphere": (L.FIELD_SPHERE, (48.0,))}


def _chunks(n, dim, big, field, seed):
    rng = np.random.default_rng(seed)
    rows = np.zeros((n, 5), np.float32)
    for i in range(n):
        d = big if i % 50 == 0 else dim
        if field == "walls":
            rows[i] = (rng.uniform(500, 3000), -10.0, rng.uniform(500, 3000), 64.0, d)
        else:  # the field's centre inside the chunk, on a sample or off it
            c = rng.integers(d // 3, 2 * d // 3, 3) + (0.0 if i % 2 else 0.25)
            rows[i] = (-c[0], -c[1], -c[2], 1.0, d)
    return [L.ChunkDesc.make(r[:3], r[3], int(r[4])) for r in rows], rows


def _kept_older(kind, params, row):
    """Vertices of a chunk whose normal after three sweeps is the one of the second."""
    dim = int(row[4])
    d = cpu.fill_field(kind, list(params), dim, row[:3], float(row[3]))
    m = cpu.extract_r(dim, d, cpu.cell_masks(dim, cpu.label_grid(dim, d)[0]))
    a, b = (cpu.process(3, m["pos"].copy(), m["boundary"], m["valence"], m["idx"], k, False, True)[1] for k in (2, 3))
    return int(((a == b).all(1) & (b != 0).any(1)).sum())


@pytest.mark.parametrize("form", list(FORMS))
@pytest.mark.parametrize("field", list(FIELDS))
@pytest.mark.parametrize("mode,iters,normals,boundary", [
    (L.MODE_R, 1, True, False), (L.MODE_R, 2, True, False), (L.MODE_R, 3, True, True), (L.MODE_R, 4, True, False),
    (L.MODE_R, 5, True, False), (L.MODE_R, 14, True, False), (L.MODE_R, 4, False, False), (L.MODE_Q, 3, True, False),
    (L.MODE_Q, 4, True, True)])
def test_sweep_forms_match_oracle(ctx, form, field, mode, iters, normals, boundary):
    n, dim, big = FORMS[form]
    descs, rows = _chunks(n, dim, big, field, seed=3 + n)
    kind, params = FIELDS[field]
    b = Batch(ctx, descs, L.Field.make(kind, params), mode=mode, placement=L.PLACE_MASSPOINT, iters=iters,
              process_boundary=boundary, smooth_normals=normals)
    cap = int(30 * (rows[:, 4] ** 2).sum()) + 4096
    bufs = b.allocate(cap, 6 * cap, normals=normals)
    b.run(use_graph=True)
    counts, want = cpu.extract_batch_digest(rows, kind, list(params), mode, L.PLACE_MASSPOINT, iters, boundary, normals)
    info = bufs["info"].cpu().numpy()
    pos, idx = bufs["pos"].cpu().numpy(), bufs["idx"].cpu().numpy().view(np.uint32)
    nrm, bnd = bufs["nrm"].cpu().numpy() if normals else None, bufs["boundary"].cpu().numpy()
    assert np.array_equal(info[:, 1], counts[:, 1]) and info[:, 1].sum() > 0 and (info[:, 5] == 0).all()
    for i, (vo, vc, io, ic, _, _) in enumerate(info):
        got = cpu.chunk_digests(pos[vo:vo + vc], idx[io:io + ic], bnd[vo:vo + vc],
                                nrm[vo:vo + vc] if normals else None)
        k = 4 if normals else 3
        assert tuple(got)[:k] == tuple(want[i])[:k], (i, rows[i])
    if field == "walls":
        assert sum(_kept_older(kind, params, r) for r in rows[:3]) > 0  # the case the test is for
    b.close()
