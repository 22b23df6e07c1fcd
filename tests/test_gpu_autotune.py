"""The autotuner's times: each is that of the stage it stands for."""
import pytest
import torch

from binarymeshfitting_gb300 import _lib as L
from binarymeshfitting_gb300 import workloads
from binarymeshfitting_gb300.engine import Batch

pytestmark = pytest.mark.gpu


def _plan(ctx, n, mode, place=L.PLACE_CENTER):
    descs, rows = workloads.lod_update(n=n, seed=21)
    b = Batch(ctx, descs, workloads.terrain_field(), mode=mode, placement=place, iters=4, smooth_normals=True)
    cap = int(2.4 * (rows[:, 4] ** 2).sum()) + 65536
    b.allocate(cap, 6 * cap, normals=True)
    return b


# the least of a stage's times, so that a pause of the machine between the events does not count
def _stage(b, k):
    return min(b.profile()[k] for _ in range(5))


@pytest.mark.parametrize("n", [20, 200, 400])  # one cooperative launch, one launch per step, chunk by chunk
@pytest.mark.parametrize("mode", [L.MODE_R, L.MODE_Q])
def test_sweep_candidates_are_timed(ctx, n, mode):
    b = _plan(ctx, n, mode)
    want = b.run()
    mesh = b.bufs["pos"][:want[0]].clone()
    block = b.tuning()["sweep_block"]
    chosen, ms = b.autotune(reps=3)
    sweeps = _stage(b, 5)
    assert len(ms) == 10 and all(0.5 * sweeps < t < 10.0 * sweeps for t in ms[7:]), (ms, sweeps)
    assert chosen["sweep_block"] == block or n == 200  # only one launch per step has a choice
    assert b.run() == want and torch.equal(b.bufs["pos"][:want[0]], mesh)
    b.close()


@pytest.mark.parametrize("mode,place", [(L.MODE_R, L.PLACE_CENTER), (L.MODE_Q, L.PLACE_QEF),
                                        (L.MODE_Q, L.PLACE_MASSPOINT), (L.MODE_Q, L.PLACE_CENTER)])
def test_fill_candidates_are_timed_whole(ctx, mode, place):
    """A band fill with what it leaves to the pass behind the count (Mode Q's QEF
    placement: about half as much again), a full fill by itself."""
    b = _plan(ctx, 400, mode, place)
    want = b.run()
    mesh = b.bufs["pos"][:want[0]].clone()
    _, ms = b.autotune(reps=5)
    for (fm, fr), t in zip([(0, 8), (1, 4), (1, 8), (1, 16), (2, 4), (2, 8), (2, 16)], ms):
        b.set_tuning(fill_mode=fm, fill_run=fr)
        fill = _stage(b, 0)
        assert 0.85 * fill < t < 1.5 * fill, (fm, fr, t, fill)
    assert b.run() == want and torch.equal(b.bufs["pos"][:want[0]], mesh)
    b.close()
