"""Performance cases of the chunk-extraction library: the calls a program makes
through its public entry points (the C ABI of include/bmf.h and the Python
layers engine, reference_api and fitting), from one small chunk to a whole
mixed-LOD world update and a batched fitting step.  Meshes are returned in the
fixed-capacity buffers that such a program keeps (zero past the counts).

Kinds of case:
  chunk   bmf_extract_chunk into the caller's buffers: one chunk from a field
          (a player edits one chunk, a tool previews one), with or without
          smoothing
  grid    bmf_label_grid -> bmf_polygonize -> bmf_process -> bmf_format on the
          caller's own density grid (a scan, a simulation)
  queue   reference_api.ChunkGenerator.process_queue: the reference's entry
          point, a queue of octree nodes at one resolution, gathered into the
          program's upload buffers
  update  Batch.set_descs + Batch.run: a streaming world's mixed-LOD update on
          a kept plan
  fit     FitPlan.step_grad: one step of fitting learnable density grids
          (forward, loss, adjoint)
"""
import ctypes
import math

import numpy as np
import torch

from binarymeshfitting_gb300 import _lib as L
from binarymeshfitting_gb300 import reference_api as R
from binarymeshfitting_gb300 import workloads
from binarymeshfitting_gb300.engine import Batch
from binarymeshfitting_gb300.fitting import FitPlan

PLACE = {"center": L.PLACE_CENTER, "mass": L.PLACE_MASSPOINT, "qef": L.PLACE_QEF}
MODE = {"R": L.MODE_R, "Q": L.MODE_Q}


def listed():
    return [
        # one world chunk, extracted and smoothed: the smallest call, all latency
        dict(name="chunk33_r", kind="chunk", field="terrain", dim=33, mode="R", place="center", iters=4),
        # the analytic sphere-wave chunk, quads at the cell centres, no smoothing
        dict(name="chunk65_wave_q", kind="chunk", field="wave", dim=65, mode="Q", place="center", iters=0),
        # the single terrain chunk of the benchmark: 4 sweeps, smoothed normals
        dict(name="chunk129_r", kind="chunk", field="terrain", dim=129, mode="R", place="center", iters=4),
        # the same chunk with hermite-QEF placement
        dict(name="chunk129_qef", kind="chunk", field="terrain", dim=129, mode="Q", place="qef", iters=4),
        # a caller's grid of an odd size through the stage calls, to the draw layout
        dict(name="grid100_r", kind="grid", dim=100, mode="R", place="center", iters=2),
        # a queue of nodes at the reference's chunk resolution on its default sampler
        dict(name="queue64", kind="queue", field="terrain2d", n=64, dim=32, iters=2),
        # a small streaming update (a camera step): fewer chunks than the GPU has SMs
        dict(name="update96_r", kind="update", field="terrain", n=96, mode="R", place="center", iters=4),
        # a mid-size update on the 2D heightmap, the reference's default world
        dict(name="update1024_2d_r", kind="update", field="terrain2d", n=1024, mode="R", place="center", iters=4),
        # a mid-size update as quads with hermite-QEF placement
        dict(name="update512_qef", kind="update", field="terrain", n=512, mode="Q", place="qef", iters=4),
        # the benchmark's whole mixed-LOD update
        dict(name="update4096_r", kind="update", field="terrain", n=4096, mode="R", place="center", iters=4),
        # fitting one grid: the smallest differentiable call
        dict(name="fit1_65", kind="fit", n=1, dim=65, iters=8),
        # the batched fitting step of the benchmark
        dict(name="fit512_65", kind="fit", n=512, dim=65, iters=8),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["chunk", "chunk", "grid", "queue", "update", "update", "fit"])
    mode = rng.choice(["R", "R", "Q"])
    place = rng.choice(["center", "mass", "qef"]) if mode == "Q" else "center"
    if kind == "chunk":
        return dict(kind=kind, field=rng.choice(["terrain", "terrain2d", "wave"]), dim=_log_int(rng, 17, 150), mode=mode,
                    place=place, iters=rng.choice([0, 1, 2, 4, 8]))
    if kind == "grid":
        return dict(kind=kind, dim=_log_int(rng, 20, 160), mode=mode, place=place, iters=rng.choice([0, 1, 2, 4, 6]))
    if kind == "queue":
        return dict(kind=kind, field=rng.choice(["terrain", "terrain2d"]), n=_log_int(rng, 8, 512),
                    dim=rng.choice([32, 33, 48]), iters=rng.choice([0, 2, 4]))
    if kind == "update":
        return dict(kind=kind, field=rng.choice(["terrain", "terrain2d"]), n=_log_int(rng, 16, 3000 if mode == "R" else 800),
                    mode=mode, place=place, iters=rng.choice([0, 2, 4, 5]))
    return dict(kind=kind, n=_log_int(rng, 1, 400), dim=rng.choice([33, 48, 65]), iters=rng.choice([0, 4, 8]))


# --------------------------------------------------------------------------
# inputs
# --------------------------------------------------------------------------
def _field(name, rng, dim):
    """(field, origin, scale) of one chunk that the field's surface crosses: the
    scale is the smallest LOD cell whose chunk spans the surface's band."""
    x, z = rng.uniform(200.0, 3800.0, 2)
    if name == "wave":  # the sphere-wave field scaled to the chunk: radius 20 at 65 samples
        half = 0.5 * (dim - 1)
        c = half + rng.uniform(-0.5, 0.5, 3)
        return L.Field.make(L.FIELD_SPHERE_WAVE, (c[0], c[1], c[2], 0.625 * half, 1.5, 0.3)), (0.0, 0.0, 0.0), 1.0
    band, mid = (96.0, 64.0) if name == "terrain" else (512.0, 0.0)
    scale = 2.0 ** max(0, math.ceil(math.log2(band / (dim - 1))))
    half = 0.5 * (dim - 1) * scale
    field = workloads.terrain_field() if name == "terrain" else workloads.terrain2d_field()
    return field, (x, mid - half + rng.uniform(-0.1, 0.1) * half, z), scale


def _grid(dim, seed, device):
    """A noisy blob in a caller's grid: a sphere with a bump and N(0, 0.1) noise."""
    gen = torch.Generator(device=device)
    gen.manual_seed(seed)
    g = torch.arange(dim, dtype=torch.float32, device=device)
    off = 2.0 * torch.rand(3, generator=gen, device=device) - 1.0 + (dim - 1) / 2.0
    x, y, z = (g - off[0])[:, None, None], (g - off[1])[None, :, None], (g - off[2])[None, None, :]
    d = (x * x + y * y + z * z).sqrt() - dim * 0.31
    d = d + 1.5 * torch.sin(0.3 * x) * torch.sin(0.3 * y) * torch.sin(0.3 * z)
    return (d + 0.1 * torch.randn(d.shape, generator=gen, device=device)).reshape(-1).contiguous()


def _tier_rows(n, field, seed):
    descs, rows = workloads.lod_update(n, seed=seed)
    if field == "terrain2d":  # its band lies around y = 0, the layout's around y = 64 and above
        for d in descs:
            d.origin[1] -= 128.0
    return descs, rows


def _mesh(ctx, verts, indices, normals):
    """Zeroed device buffers of one mesh and the bmf_mesh that names them."""
    z = dict(device=ctx.device)
    b = dict(pos=torch.zeros((verts, 3), **z), nrm=torch.zeros((verts, 3), **z) if normals else None,
             boundary=torch.zeros(verts, dtype=torch.uint8, **z), valence=torch.zeros(verts, dtype=torch.uint8, **z),
             idx=torch.zeros(indices, dtype=torch.int32, **z))
    m = L.Mesh(b["pos"].data_ptr(), b["nrm"].data_ptr() if normals else None, b["boundary"].data_ptr(),
               b["valence"].data_ptr(), b["idx"].data_ptr(), verts, indices, 0, 0, 0, 0)
    return m, b


def prepare(case, seed):
    kind = case["kind"]
    rng = np.random.default_rng(seed)
    ctx = R.context()
    s = dict(case=case, ctx=ctx)
    if kind in ("chunk", "grid"):
        # the buffers a program keeps: room for 4 vertices per column of the chunk
        verts = 4 * case["dim"] ** 2 + 4096
        s["mesh"], s["out"] = _mesh(ctx, verts, 6 * verts, case["iters"] > 0)
    if kind == "chunk":
        s["field"], org, scale = _field(case["field"], rng, case["dim"])
        s["desc"] = L.ChunkDesc.make(org, scale, case["dim"])
        s["opts"] = L.ExtractOpts(MODE[case["mode"]], PLACE[case["place"]], case["iters"], 0, int(case["iters"] > 0), 0)
    elif kind == "grid":
        s["density"] = _grid(case["dim"], seed, ctx.device)
        s["words"] = torch.zeros(case["dim"] ** 2 * ((case["dim"] + 31) // 32), dtype=torch.int32, device=ctx.device)
        s["cap"] = 6 * verts if case["mode"] == "Q" else verts
        s["draw"] = [torch.zeros((s["cap"], 3), device=ctx.device) for _ in range(3)]
    elif kind == "queue":
        props = R.WorldProperties(max_level=7, process_iters=case["iters"], smooth_normals=case["iters"] > 0)
        field = workloads.terrain_field() if case["field"] == "terrain" else workloads.terrain2d_field()
        s["gen"] = R.ChunkGenerator(props, R.Sampler(field), dim=case["dim"])
        mid = 64.0 if case["field"] == "terrain" else 0.0
        s["nodes"] = []
        for _ in range(case["n"]):
            level = int(rng.integers(4, 8))
            size = 32.0 * 2 ** (7 - level)
            x, z = (math.floor(v / size) * size for v in rng.uniform(200.0, 3800.0, 2))
            y = math.floor((mid + rng.normal(0.0, 24.0)) / size) * size
            s["nodes"].append(R.WorldOctreeNode(pos=(x, y, z), size=size, level=level))
        v = case["n"] * case["dim"] ** 2 * 4
        s["out"] = _mesh(ctx, v, 6 * v, case["iters"] > 0)[1]
        del s["out"]["valence"]  # a queue's meshes carry none
    elif kind == "update":
        s["descs"], rows = _tier_rows(case["n"], case["field"], seed)
        field = workloads.terrain_field() if case["field"] == "terrain" else workloads.terrain2d_field()
        s["batch"] = Batch(ctx, s["descs"], field, mode=MODE[case["mode"]], placement=PLACE[case["place"]],
                           iters=case["iters"], smooth_normals=case["iters"] > 0)
        # the arena a program keeps: room for 2.4 vertices per column of every
        # chunk of the tiers, whatever their order
        v = int(2.4 * float((rows[:, 4] ** 2).sum())) + 65536
        for t in s["batch"].allocate(v, 6 * v, normals=case["iters"] > 0).values():
            if t is not None:
                t.zero_()
    else:
        s["density"], s["spheres"] = workloads.fit_batch(case["n"], dim=case["dim"], seed=seed % (1 << 31), device=ctx.device)
        s["plan"] = FitPlan(ctx, case["n"], case["dim"], iters=case["iters"])
        s["plan"].pos.zero_()
        s["plan"].idx.zero_()
        s["loss"] = torch.zeros(1, device=ctx.device)
        s["grad_pos"] = torch.zeros((s["plan"].vcap, 3), device=ctx.device)
        s["grad"] = torch.zeros_like(s["density"])
    return s


# --------------------------------------------------------------------------
# one pass
# --------------------------------------------------------------------------
def _stream():
    return ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)


def run(s):
    c, ctx = s["case"], s["ctx"]
    kind, lib, h = c["kind"], ctx.lib, ctx.h
    if kind == "chunk":
        m = s["mesh"]
        L.check(lib.bmf_extract_chunk(h, ctypes.byref(s["desc"]), ctypes.byref(s["field"]), ctypes.byref(s["opts"]),
                                      ctypes.byref(m), _stream()), h, lib)
        return dict(s["out"], n_verts=m.n_verts, n_idx=m.n_idx, contains_mesh=m.contains_mesh)
    if kind == "grid":
        m, d, w, st = s["mesh"], s["density"].data_ptr(), s["words"].data_ptr(), _stream()
        cm, cnt = ctypes.c_int32(0), ctypes.c_int64(0)
        L.check(lib.bmf_label_grid(h, c["dim"], d, w, ctypes.byref(cm), st), h, lib)
        L.check(lib.bmf_polygonize(h, c["dim"], d, w, MODE[c["mode"]], PLACE[c["place"]], ctypes.byref(m), st), h, lib)
        if c["iters"]:
            L.check(lib.bmf_process(h, ctypes.byref(m), c["iters"], 0, 1, st), h, lib)
        p, n, col = (t.data_ptr() for t in s["draw"])
        L.check(lib.bmf_format(h, ctypes.byref(m), int(c["mode"] == "Q"), int(c["iters"] > 0), p, n, col, s["cap"],
                               ctypes.byref(cnt), st), h, lib)
        return dict(s["out"], words=s["words"], draw_p=s["draw"][0], draw_n=s["draw"][1], draw_c=s["draw"][2],
                    n_verts=m.n_verts, n_idx=m.n_idx, contains_mesh=cm.value, drawn=cnt.value)
    if kind == "queue":
        nodes = s["gen"].process_queue(s["nodes"])
        for k, out in s["out"].items():
            if out is not None:
                parts = [n.vi[k] for n in nodes]
                torch.cat(parts, out=out[:sum(t.shape[0] for t in parts)])
        return dict(s["out"], meshes=sum(n.vi["contains_mesh"] for n in nodes))
    if kind == "update":
        b = s["batch"]
        b.set_descs(s["descs"])
        nv, ni = b.run(use_graph=True, sync=True)
        return dict(b.bufs, n_verts=nv, n_idx=ni)
    plan = s["plan"]
    plan.step_grad(s["density"], s["spheres"], s["loss"], s["grad_pos"], s["grad"])
    return dict(pos=plan.pos, idx=plan.idx, info=plan.info, loss=s["loss"], grad_pos=s["grad_pos"], grad=s["grad"])


# --------------------------------------------------------------------------
# what a pass cannot do without
# --------------------------------------------------------------------------
def work(case):
    """Bytes: inputs read once, outputs written once, with the measured surface
    density of these inputs (vertices per column).  Flops: one octave of
    noise (or one evaluation of the analytic field) per sample of a field;
    the sums and divisions of the smoothing sweeps; the QEF's products."""
    kind = case["kind"]
    q = case.get("mode") == "Q" or kind == "fit"
    iters = case["iters"]
    if kind in ("chunk", "grid"):
        cols, samples = case["dim"] ** 2, case["dim"] ** 3
    elif kind == "update":
        cols = samples = 0
        for d, f in ((33, 0.50), (65, 0.35), (129, 0.15)):
            cols += int(case["n"] * f * d * d)
            samples += int(case["n"] * f * d ** 3)
    else:
        cols, samples = case["n"] * case["dim"] ** 2, case["n"] * case["dim"] ** 3
    verts = (1.5 if not q else 0.9) * cols
    if kind in ("grid", "fit"):
        verts = 1.8 * cols
    idx = verts * (6 if not q else 4)
    out = verts * (12 + (12 if iters and kind != "fit" else 0) + 2) + 4 * idx
    flops = (verts + idx / 3) * iters * 20.0 + (verts * 300.0 if case.get("place") == "qef" or kind == "fit" else 0.0)
    if kind == "grid":
        out += 4 * samples + samples / 8 + 36 * verts * (4 if q else 1)  # the grid in, words and draw layout out
    elif kind == "fit":
        out += 8 * samples + 12 * verts  # the grids in, their gradient out
        flops = 3 * flops
    else:
        flops += 10.0 * samples
    return {"bytes": float(out), "flops": float(flops + samples)}


# --------------------------------------------------------------------------
# what a pass returns, in 64 bits
# --------------------------------------------------------------------------
def _crossing_positions(d):
    """Positions of the surface's edge crossings of grid d (dim^3, float64), in
    vertex order: samples in linear order, their x, y, z edges in turn."""
    n = d.shape[0]
    inside = d < 0
    mu = torch.zeros((n, n, n, 3), dtype=torch.float64, device=d.device)
    hit = torch.zeros((n, n, n, 3), dtype=torch.bool, device=d.device)
    for a in range(3):
        lo, hi = d.narrow(a, 0, n - 1), d.narrow(a, 1, n - 1)
        hit[..., a].narrow(a, 0, n - 1).copy_(inside.narrow(a, 0, n - 1) != inside.narrow(a, 1, n - 1))
        mu[..., a].narrow(a, 0, n - 1).copy_(-lo / (hi - lo))
    at = hit.nonzero()
    p = at[:, :3].to(torch.float64)
    return p + torch.nn.functional.one_hot(at[:, 3], 3) * mu[hit][:, None]


def exact(case, seed):
    """Only crossing positions of a caller's grid without smoothing have an
    independent 64-bit form: everywhere else topology, adjacency and the QEF's
    branches are the library's own discrete choices."""
    if case["kind"] != "grid" or case["mode"] != "R" or case["iters"]:
        return None
    d = _grid(case["dim"], seed, R.context().device).double().reshape((case["dim"],) * 3)
    p = torch.zeros((4 * case["dim"] ** 2 + 4096, 3), dtype=torch.float64, device=d.device)
    q = _crossing_positions(d)
    p[: q.shape[0]] = q
    return dict(pos=p, nrm=None, boundary=None, valence=None, idx=None, words=None, draw_p=p, draw_n=None, draw_c=None,
                n_verts=None, n_idx=None, contains_mesh=None, drawn=None)
