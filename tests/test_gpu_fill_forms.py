"""Density and words of the per-chunk fills at the sizes where their forms can
go wrong: word and run edges, the block / line kernel border of the terrain
fill, planes split among CTAs, few and many octaves; against the oracle, bit
for bit."""
import numpy as np
import pytest
import torch

from binarymeshfitting_gb300 import _lib as L
from binarymeshfitting_gb300 import workloads
from oracle import cpu

pytestmark = pytest.mark.gpu

TERRAIN = [(31, 5), (32, 5), (33, 1), (63, 5), (65, 9), (100, 5), (160, 3), (161, 3), (2, 5), (3, 32)]


def _check(ctx, kind, params, dim, origin, scale):
    desc, field = L.ChunkDesc.make(origin, scale, dim), L.Field.make(kind, params)
    dens, words, cm = ctx.sample_label(desc, field)
    want = cpu.fill_field(kind, list(params), dim, origin, scale)
    w, c = cpu.label_grid(dim, want)
    np.testing.assert_array_equal(dens.cpu().numpy().view(np.uint32), want.reshape(-1).view(np.uint32))
    np.testing.assert_array_equal(words.cpu().numpy().view(np.uint32), w.reshape(-1))
    assert cm == bool(c)
    # the words alone, and the same grid as a caller's
    np.testing.assert_array_equal(ctx.sample_label(desc, field, want_density=False)[1].cpu().numpy().view(np.uint32),
                                  w.reshape(-1))
    gw, gc = ctx.label_grid(dim, torch.from_numpy(want.reshape(-1)).to(ctx.device))
    np.testing.assert_array_equal(gw.cpu().numpy().view(np.uint32), w.reshape(-1))
    assert gc == bool(c)


@pytest.mark.parametrize("dim,octaves", TERRAIN)
def test_terrain_fill(ctx, dim, octaves):
    p = list(workloads.TERRAIN_PARAMS)
    p[5] = octaves
    scale = max(1.0, 96.0 / (dim - 1))
    _check(ctx, L.FIELD_TERRAIN_FBM, p, dim, (1234.5, 64.0 - 0.5 * (dim - 1) * scale, 777.25), scale)


@pytest.mark.parametrize("kind,params", [(L.FIELD_SPHERE_WAVE, workloads.SPHERE_WAVE_PARAMS),
                                         (L.FIELD_TERRAIN_2D, workloads.TERRAIN_2D_PARAMS), (L.FIELD_CUBOID, (96.0,)),
                                         (L.FIELD_TORUS_Z, (80.0,)), (L.FIELD_PLANE_Y, ()), (L.FIELD_SPHERE, (90.0,))])
@pytest.mark.parametrize("dim", [2, 31, 32, 33, 65, 100, 129, 140])
def test_plane_fill(ctx, kind, params, dim):
    half = 0.5 * (dim - 1)
    if kind == L.FIELD_SPHERE_WAVE:
        _check(ctx, kind, params, dim, (0.25, -3.0, 1.5), 64.0 / max(dim - 1, 32))
    elif kind == L.FIELD_TERRAIN_2D:
        _check(ctx, kind, params, dim, (500.0, -8.0 * half, 900.0), 8.0)
    else:
        _check(ctx, kind, params, dim, (-half, -half + 0.25, -half), 1.0)
