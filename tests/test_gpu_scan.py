"""The word and plane scans (k_count's running sums, k_chunk_scan) at the sizes
where they can go wrong: dims around the word and CTA-step edges, more chunks
than one scan CTA takes, both plane-CTA widths, and replays of one plan."""
import numpy as np
import pytest

from binarymeshfitting_gb300 import _lib as L
from binarymeshfitting_gb300 import workloads
from binarymeshfitting_gb300.engine import Batch
from oracle import cpu

pytestmark = pytest.mark.gpu

# one chunk; one scan CTA exactly full; two scan CTAs; enough planes for the 64-thread count CTAs
CASES = [((64,), 1), ((2, 31, 32, 33), 32), ((2, 3, 33, 64, 65), 70), ((17, 33, 5), 150)]


@pytest.mark.parametrize("dims,n", CASES)
@pytest.mark.parametrize("mode", [L.MODE_R, L.MODE_Q])
def test_scans_match_oracle(ctx, dims, n, mode):
    descs, rows = workloads.lod_update(n=n, seed=11 + n)
    for i, (d, r) in enumerate(zip(descs, rows)):
        d.dim = dims[i % len(dims)]
        r[4] = d.dim
        d.origin[1] = r[1] = 64.0 - 0.5 * (d.dim - 1) * r[3]
    b = Batch(ctx, descs, workloads.terrain_field(), mode=mode, placement=L.PLACE_MASSPOINT, iters=2,
              smooth_normals=True)
    cap = int(8 * (rows[:, 4] ** 2).sum()) + 4096
    bufs = b.allocate(cap, 6 * cap, normals=True)
    counts, want = cpu.extract_batch_digest(rows[:, :5].astype(np.float32), L.FIELD_TERRAIN_FBM,
                                            list(workloads.TERRAIN_PARAMS), mode, L.PLACE_MASSPOINT, 2, False, True)
    for _ in range(2):
        b.run(use_graph=True)
        info = bufs["info"].cpu().numpy()
        pos, nrm = bufs["pos"].cpu().numpy(), bufs["nrm"].cpu().numpy()
        idx, bnd = bufs["idx"].cpu().numpy().view(np.uint32), bufs["boundary"].cpu().numpy()
        assert (info[:, 5] == 0).all() and np.array_equal(info[:, 1], counts[:, 1]) and info[:, 1].sum() > 0
        assert np.array_equal(info[:, 0], np.cumsum(info[:, 1]) - info[:, 1])
        assert np.array_equal(info[:, 2], np.cumsum(info[:, 3]) - info[:, 3])
        for i, (vo, vc, io, ic, _, _) in enumerate(info):
            got = cpu.chunk_digests(pos[vo:vo + vc], idx[io:io + ic], bnd[vo:vo + vc], nrm[vo:vo + vc])
            assert tuple(got) == tuple(want[i]), (i, rows[i])
    b.close()
