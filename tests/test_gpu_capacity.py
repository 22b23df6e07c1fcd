"""Output arenas that are too small, in the forms of the sweeps that a large
update takes: BMF_ERR_CAPACITY, nothing written past the arena, and the mesh of a
plan that always had the room once the arena has grown."""
import numpy as np
import pytest
import torch

from binarymeshfitting_gb300 import _lib as L
from binarymeshfitting_gb300 import workloads
from binarymeshfitting_gb300.engine import Batch
from binarymeshfitting_gb300.fitting import FitPlan

pytestmark = pytest.mark.gpu

GUARD = 4096
# (chunks, dim): one cooperative launch, one launch per step, and chunk by chunk
FORMS = {"team": (40, 33), "launches": (100, 41), "chunks": (330, 24)}


def _plan(ctx, form, mode, place=L.PLACE_MASSPOINT, iters=4):
    n, dim = FORMS[form]
    rng = np.random.default_rng(n + mode)
    descs = [L.ChunkDesc.make((rng.uniform(200, 3800), 64.0 - 2.0 * (dim - 1), rng.uniform(200, 3800)), 4.0, dim)
             for _ in range(n)]
    return Batch(ctx, descs, workloads.terrain_field(), mode=mode, placement=place, iters=iters, smooth_normals=True)


def _arena(b, vcap, icap):
    """An arena of exactly this capacity, and a check of the guards behind it."""
    dev = torch.device("cuda", 0)
    pos, nrm = (torch.full((vcap + GUARD, 3), -7.0, device=dev) for _ in range(2))
    bnd = torch.full((vcap + GUARD,), 9, dtype=torch.uint8, device=dev)
    idx = torch.full((icap + GUARD,), -1, dtype=torch.int32, device=dev)
    info = torch.zeros((b.n, 6), dtype=torch.int64, device=dev)
    b.bufs = dict(pos=pos, nrm=nrm, boundary=bnd, idx=idx, info=info)
    b.out = L.BatchOut(pos.data_ptr(), nrm.data_ptr(), bnd.data_ptr(), idx.data_ptr(), vcap, icap, info.data_ptr(), 0, 0)

    def intact():
        return bool((pos[vcap:] == -7.0).all() and (nrm[vcap:] == -7.0).all() and (bnd[vcap:] == 9).all() and
                    (idx[icap:] == -1).all())
    return intact


def _mesh(b, nv, ni):
    return [b.bufs[k][:n].clone() for k, n in (("pos", nv), ("nrm", nv), ("boundary", nv), ("idx", ni))]


def _equal(a, b):
    return all(torch.equal(x.view(torch.uint8), y.view(torch.uint8)) for x, y in zip(a, b))


@pytest.fixture(scope="module")
def whole(ctx):
    """(totals, mesh, chunk table) of a plan with room, per form and mode."""
    out = {}

    def get(form, mode, place=L.PLACE_MASSPOINT):
        if (form, mode, place) not in out:
            b = _plan(ctx, form, mode, place)
            cap = 12 * b.n * FORMS[form][1] ** 2
            b.allocate(cap, 6 * cap, normals=True)
            nv, ni = b.run()
            assert nv > 4 * b.n and (b.bufs["info"][:, 5] == 0).all()
            out[form, mode, place] = (nv, ni), _mesh(b, nv, ni), b.bufs["info"].cpu().numpy()
            b.close()
        return out[form, mode, place]
    return get


def _short(ctx, form, mode, vcap, icap, totals, want):
    """A plan whose arena is too small at first."""
    nv, ni = totals
    b = _plan(ctx, form, mode)
    intact = _arena(b, vcap, icap)
    for graph in (False, True):
        with pytest.raises(L.BmfError) as e:
            b.run(use_graph=graph)
        torch.cuda.synchronize()
        assert e.value.status == L.ERR_CAPACITY and (b.out.n_verts, b.out.n_idx) == (nv, ni) and intact()
    b.allocate(nv, ni, normals=True)
    assert b.run() == (nv, ni) and _equal(_mesh(b, nv, ni), want)
    b.close()


@pytest.mark.parametrize("form", list(FORMS))
@pytest.mark.parametrize("mode", [L.MODE_R, L.MODE_Q])
@pytest.mark.parametrize("share", [0.0, 0.4, 0.999])
def test_too_few_vertices(ctx, whole, form, mode, share):
    totals, want, _ = whole(form, mode)
    _short(ctx, form, mode, max(1, int(share * totals[0])), 6 * totals[0], totals, want)


@pytest.mark.parametrize("form", list(FORMS))
@pytest.mark.parametrize("mode", [L.MODE_R, L.MODE_Q])
@pytest.mark.parametrize("share", [0.0, 0.4, 0.999])
def test_too_few_indices(ctx, whole, form, mode, share):
    totals, want, _ = whole(form, mode)
    _short(ctx, form, mode, totals[0], max(1, int(share * totals[1])), totals, want)


def test_fit_chunk_sweeps_with_too_few_vertices(ctx):
    n, dim = 80, 48  # forward chunk by chunk
    dens, _ = workloads.fit_batch(n, dim=dim, seed=5, device=ctx.device)
    plan = FitPlan(ctx, n, dim, placement=L.PLACE_MASSPOINT, iters=3)
    want = [t.clone() for t in plan.forward(dens)]
    nv, ni = plan.n_verts, plan.n_idx
    for vcap in (1, nv // 3):
        small = FitPlan(ctx, n, dim, placement=L.PLACE_MASSPOINT, iters=3, vcap=vcap, icap=ni)
        small.pos = torch.full((vcap + GUARD, 3), -7.0, device=ctx.device)
        small.idx = torch.full((ni + GUARD,), -1, dtype=torch.int32, device=ctx.device)
        with pytest.raises(L.BmfError) as e:
            small.forward(dens)
        torch.cuda.synchronize()
        assert e.value.status == L.ERR_CAPACITY and (small.pos[vcap:] == -7.0).all() and (small.idx[ni:] == -1).all()
        small.close()
    assert _equal(plan.forward(dens), want)
    plan.close()


@pytest.mark.parametrize("mode", [L.MODE_R, L.MODE_Q])
def test_indices_may_be_rewritten_behind_the_extraction(ctx, whole, mode):
    """Consumers behind bmf_batch_wait_extraction own the indices: the sweeps that
    still run do not read them."""
    (nv, ni), want, _ = whole("chunks", mode)
    b = _plan(ctx, "chunks", mode)
    b.allocate(nv, ni, normals=True)
    side = torch.cuda.Stream()
    for graph in (False, True, True):
        b.run(use_graph=graph, sync=False)
        b.wait_extraction(side)
        with torch.cuda.stream(side):
            got = b.bufs["idx"].clone()
            b.bufs["idx"].zero_()
        torch.cuda.synchronize()
        assert torch.equal(got, want[3]) and _equal(_mesh(b, nv, ni)[:3], want[:3])
    b.close()


@pytest.mark.parametrize("form", list(FORMS))
@pytest.mark.parametrize("mode,place", [(L.MODE_R, L.PLACE_MASSPOINT), (L.MODE_Q, L.PLACE_QEF),
                                        (L.MODE_Q, L.PLACE_MASSPOINT)])
@pytest.mark.parametrize("share", [0.05, 0.15])
def test_chunks_that_fit_are_whole(ctx, whole, form, mode, place, share):
    """Far too small an arena (fewer entries than busy words): the chunks whose status
    is 0 are complete, and every vertex of the arena has a cell to be placed in."""
    (nv, ni), want, wtab = whole(form, mode, place)
    b = _plan(ctx, form, mode, place)
    intact = _arena(b, int(share * nv), int(share * ni))
    for graph in (False, True):
        with pytest.raises(L.BmfError) as e:
            b.run(use_graph=graph)
        torch.cuda.synchronize()
        assert e.value.status == L.ERR_CAPACITY and (b.out.n_verts, b.out.n_idx) == (nv, ni) and intact()
        tab = b.bufs["info"].cpu().numpy()
        fit = np.flatnonzero((tab[:, 5] == 0) & (tab[:, 1] > 0))
        assert len(fit) > 0 and np.array_equal(tab[:, :5], wtab[:, :5])
        for i in fit:
            vo, vc, io, ic = tab[i, :4]
            got = [b.bufs[k][vo:vo + vc] for k in ("pos", "nrm", "boundary")] + [b.bufs["idx"][io:io + ic]]
            assert _equal(got, [t[vo:vo + vc] for t in want[:3]] + [want[3][io:io + ic]]), i
    b.close()


@pytest.mark.parametrize("n,dim", [(1, 33), (200, 33)])
@pytest.mark.parametrize("adjoint", ["f32", "df"])
def test_fit_step_in_a_small_arena_stays_inside(ctx, n, dim, adjoint):
    """A whole fitting step without a host sync, on vertices that partly have no room."""
    dens, sph = workloads.fit_batch(n, dim=dim, seed=9, device=ctx.device)
    plan = FitPlan(ctx, n, dim, iters=2, adjoint=adjoint, vcap=40 * n, icap=40 * n)
    loss, grad_pos = torch.zeros(1, device=ctx.device), torch.zeros((plan.vcap, 3), device=ctx.device)
    grad = torch.full((dens.numel() + 2 * GUARD,), -7.0, device=ctx.device)
    plan.step_grad(dens, sph, loss, grad_pos, grad[GUARD:-GUARD])
    torch.cuda.synchronize()
    assert (grad[:GUARD] == -7.0).all() and (grad[-GUARD:] == -7.0).all()
    with pytest.raises(L.BmfError) as e:
        plan.forward(dens)
    assert e.value.status == L.ERR_CAPACITY
    plan.close()


@pytest.mark.parametrize("form", list(FORMS))
@pytest.mark.parametrize("mode", [L.MODE_R, L.MODE_Q])
@pytest.mark.parametrize("between", ["run", "profile"])
def test_a_graph_does_not_outlive_its_scratch(ctx, whole, form, mode, between):
    """A graph captured for one arena, replayed after a direct run on a larger one."""
    (nv, ni), want, _ = whole(form, mode)
    b = _plan(ctx, form, mode)
    b.allocate(nv, ni, normals=True)
    small = b.out, b.bufs
    assert b.run() == (nv, ni)
    b.allocate(2 * nv, 2 * ni, normals=True)
    if between == "run":
        assert b.run(use_graph=False) == (nv, ni) and _equal(_mesh(b, nv, ni), want)
    else:
        b.profile()
    b.out, b.bufs = small
    b.bufs["pos"].zero_()
    assert b.run() == (nv, ni) and _equal(_mesh(b, nv, ni), want)
    b.close()


@pytest.mark.parametrize("form", list(FORMS))
def test_first_chunks_are_exact_when_the_fixup_list_overflows(ctx, whole, form):
    """Room for the first chunks' vertices only: far fewer entries than the band fill
    leaves ends to make exact."""
    _, want, wtab = whole(form, L.MODE_R)
    k = int(np.flatnonzero(wtab[:, 1] > 0)[1])  # the second chunk with a mesh is the last that fits
    vcap, icap = int(wtab[k, 0] + wtab[k, 1]), int(wtab[k, 2] + wtab[k, 3])
    b = _plan(ctx, form, L.MODE_R)
    assert b.tuning()["fill_band"] == 1
    intact = _arena(b, vcap, icap)
    with pytest.raises(L.BmfError) as e:
        b.run()
    torch.cuda.synchronize()
    assert e.value.status == L.ERR_CAPACITY and intact() and (b.bufs["info"][:k + 1, 5] == 0).all()
    got = [b.bufs["pos"][:vcap], b.bufs["nrm"][:vcap], b.bufs["boundary"][:vcap], b.bufs["idx"][:icap]]
    assert _equal(got, [want[0][:vcap], want[1][:vcap], want[2][:vcap], want[3][:icap]])
    b.close()
