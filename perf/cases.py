"""Performance cases of the BVH build and ray-query engine.

Each case is one kind of work that a program using the engine has it do, at
one size, through the public entry points of `rq`:

  build_trace   build a BVH of a mesh (in place, as a program does that
                rebuilds what moves) and trace a ray buffer over it
  frame         deform, rebuild, primary rays to a G-buffer, shadow and AO rays
  visibility    deform, rebuild or refit, jittered primary rays
  batched       deform, build and trace many meshes at once
  serving       a burst of requests through the serving loop
  terrain       trace the reference's procedural rays over a kept BVH
  radv          build a RADV image of a vertex soup, and trace it
  effects       AO from a depth buffer, its blur, reflection rays
  instances     rebuild a top-level BVH over instances and trace it

`listed()` holds the benchmark's configurations and the ends of their ranges,
`draw()` other sizes of the same ranges.  All inputs come from the seed: the
meshes are height-field grids with vertex noise, the surface every
configuration of the benchmark uses.
"""
import math
import os
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, os.path.join(ROOT, "rdna2-accel-raster_b200"))

import rq  # noqa: E402
from rq import tune  # noqa: E402
from rq import workloads as W  # noqa: E402

DEV = "cuda"


# ------------------------------------------------------------------- the cases
def listed():
    return [
        # the plain method: a small dynamic mesh and a modest ray batch, bound by launches and latency
        dict(name="plain_4k", kind="build_trace", build="lbvh", qx=64, qy=32, rays=65536, any=False, mt=False),
        # the reference's own topology of a mid-size scene with occlusion queries over it
        dict(name="median_99k", kind="build_trace", build="median", qx=223, qy=223, rays=262144, any=True, mt=False),
        # the headline: the 1080p frame with a rebuild, 16 shadow rays and one AO ray per pixel
        dict(name="frame_1080p", kind="frame", qx=1118, qy=1118, width=1920, height=1080, lights=16, spp=1),
        # subpixel visibility of 8.3M triangles, rebuilt every frame, and refitted every frame
        dict(name="visibility_rebuild", kind="visibility", q=2040, width=1920, height=1080, refit=False),
        dict(name="visibility_refit", kind="visibility", q=2040, width=1920, height=1080, refit=True),
        # 512 deforming meshes of 64 to 65,536 triangles, 4,096 any-hit and 4,096 closest-hit rays each
        dict(name="batched_512", kind="batched", meshes=512, size_seed=2, rays_any=4096, rays_closest=4096),
        # a queue of requests over resident meshes of 64 to 1M triangles, 1k to 2M rays each
        dict(name="serving_64", kind="serving", meshes=24, requests=64, max_rays=2000000, size_seed=4),
        # the reference's micro-benchmark: incoherent rays, its triangle test
        dict(name="terrain_1m_incoherent", kind="terrain", q=707, rays=1 << 20, coherent=False, any=False, mt=True),
        # the fast builder on a small dynamic mesh that is then queried, and on the frame's mesh
        dict(name="radv_4k", kind="radv", qx=64, qy=32, rays=16384),
        dict(name="radv_2500k", kind="radv", qx=1118, qy=1118, rays=0),
        # screen-space AO replacement at 1080p, 2 samples, both blur passes, and reflections
        dict(name="effects_1080p", kind="effects", q=707, width=1920, height=1080, spp=2),
        # a scene of moving instances: the top level rebuilt, then one ray per pixel of a half-size view
        dict(name="instances_256", kind="instances", instances=256, meshes=8, max_tris=100000, size_seed=6,
             rays=518400, any=False),
    ]


def _log(rng, lo, hi):
    return int(math.exp(rng.uniform(math.log(lo), math.log(hi + 1))))


def _quads(rng, lo, hi):
    """A grid of about lo..hi triangles, of any aspect up to 3:1."""
    t = _log(rng, lo, hi)
    qx = max(1, int(math.sqrt(t / 2 * rng.uniform(0.6, 1.6))))
    return qx, max(1, t // (2 * qx))


def draw(rng):
    kind = rng.choice(["build_trace", "build_trace", "frame", "frame", "visibility", "visibility", "batched", "serving",
                       "terrain", "radv", "effects", "instances"])
    if kind == "build_trace":
        qx, qy = _quads(rng, 64, 1 << 20)
        return dict(kind=kind, build=rng.choice(["lbvh", "lbvh", "sah", "median"]), qx=qx, qy=qy,
                    rays=_log(rng, 1000, 2000000), any=rng.random() < 0.5, mt=rng.random() < 0.25)
    if kind == "frame":
        qx, qy = _quads(rng, 4096, 2499848)
        height = rng.randint(120, 1080)
        return dict(kind=kind, qx=qx, qy=qy, width=height * 16 // 9 - rng.randint(0, 7), height=height,
                    lights=rng.randint(1, 16), spp=rng.randint(0, 2))
    if kind == "visibility":
        height = rng.randint(360, 1080)
        return dict(kind=kind, q=_log(rng, 128, 2040), width=height * 16 // 9, height=height, refit=rng.random() < 0.5)
    if kind == "batched":
        return dict(kind=kind, meshes=_log(rng, 16, 512), size_seed=rng.randint(0, 999), rays_any=_log(rng, 100, 4096),
                    rays_closest=_log(rng, 100, 4096))
    if kind == "serving":
        return dict(kind=kind, meshes=rng.randint(4, 24), requests=_log(rng, 8, 64), max_rays=_log(rng, 20000, 2000000),
                    size_seed=rng.randint(0, 999))
    if kind == "terrain":
        return dict(kind=kind, q=_log(rng, 22, 707), rays=_log(rng, 1 << 15, 1 << 20), coherent=rng.random() < 0.5,
                    any=rng.random() < 0.5, mt=rng.random() < 0.5)
    if kind == "radv":
        qx, qy = _quads(rng, 64, 8323200)
        return dict(kind=kind, qx=qx, qy=qy, rays=_log(rng, 1000, 20000) if qx * qy <= 4096 else 0)
    if kind == "effects":
        height = rng.randint(240, 1080)
        return dict(kind=kind, q=_log(rng, 64, 1000), width=height * 16 // 9 - rng.randint(0, 7), height=height,
                    spp=rng.randint(1, 3))
    return dict(kind=kind, instances=_log(rng, 8, 512), meshes=rng.randint(1, 8), max_tris=100000,
                size_seed=rng.randint(0, 999), rays=_log(rng, 20000, 518400), any=rng.random() < 0.5)


# ---------------------------------------------------------------------- inputs
def _grid(qx, qy, gen):
    """The height field of rq.scene_grid with noise of this generator, made on the device."""
    x = torch.linspace(-1.0, 1.0, qx + 1, dtype=torch.float64, device=DEV)
    y = torch.linspace(-1.0, 1.0, qy + 1, dtype=torch.float64, device=DEV)
    z = W.AMP * torch.cos(W.FREQ * y)[:, None] * torch.sin(W.FREQ * x)[None, :]
    z = z + W.SIGMA * torch.randn(z.shape, generator=gen, dtype=torch.float32, device=DEV)
    pos = torch.stack([x[None, :].expand_as(z), y[:, None].expand_as(z), z], -1).reshape(-1, 3).float().contiguous()
    v = torch.arange((qx + 1) * (qy + 1), dtype=torch.int32, device=DEV).reshape(qy + 1, qx + 1)
    v00, v10, v01, v11 = v[:-1, :-1], v[:-1, 1:], v[1:, :-1], v[1:, 1:]
    idx = torch.stack([v00, v10, v01, v10, v11, v01], -1).reshape(-1, 3).contiguous()
    return pos, idx


def _rays_down(n, gen, tmax=1000.0):
    """The plain workload's rays: from z = 2 over the mesh, down within 0.3 of the vertical."""
    u = torch.rand((n, 4), generator=gen, dtype=torch.float32, device=DEV) * 2 - 1
    d = torch.cat([0.3 * u[:, 2:], torch.full((n, 1), -1.0, device=DEV)], 1)
    d = d / d.norm(dim=1, keepdim=True)
    o = torch.cat([u[:, :2], torch.full((n, 1), 2.0, device=DEV)], 1)
    return torch.cat([o, torch.full((n, 1), 0.01, device=DEV), d, torch.full((n, 1), tmax, device=DEV)], 1).contiguous()


def _hits(n):
    """A hit buffer and its distances as floats."""
    h = torch.empty((n, 4), dtype=torch.int32, device=DEV)
    return h, h.view(torch.float32)[:, 1]


def _lights(n, rng):
    xy = rng.uniform(-1.0, 1.0, (n, 2))
    return [(float(xy[k, 0]), float(xy[k, 1]), float(z), 100.0) for k, z in enumerate(rng.uniform(2.0, 2.5, n))]


def _flags(case):
    return (rq.RQ_TRACE_ANY if case.get("any") else 0) | (rq.RQ_TRI_MT if case.get("mt") else 0)


def _batch_meshes(case):
    sizes = W.batched_sizes(case["meshes"], seed=case["size_seed"])
    descs, v, t = [], 0, 0
    for s in sizes:
        qx, qy = W.grid_for_triangles(s)
        descs.append((v, (qx + 1) * (qy + 1), t, 2 * qx * qy, qx, qy))
        v, t = v + descs[-1][1], t + descs[-1][3]
    return descs


def _instance_sizes(case):
    rng = np.random.default_rng(case["size_seed"])
    return [W.grid_for_triangles(t) for t in W.log_uniform_int(rng, 500, case["max_tris"], case["meshes"])]


def _requests(case):
    """Mesh, kind and ray count of every request, and the meshes' sizes."""
    rng = np.random.default_rng(case["size_seed"])
    n = case["requests"]
    sizes = W.serving_catalogue(case["meshes"], seed=case["size_seed"])
    return sizes, rng.integers(0, len(sizes), n), rng.choice([1, 2, 3], size=n, p=list(W.SERVE_MIX)), \
        W.log_uniform_int(rng, 1000, case["max_rays"], n)


# --------------------------------------------------------------------- prepare
def prepare(case, seed):
    gen = torch.Generator(device=DEV).manual_seed(int(seed))
    rng = np.random.default_rng(int(seed))
    s = dict(case=case, ctx=rq.Context(torch.cuda.current_device()))
    globals()["_prepare_" + case["kind"]](s, case, gen, rng)
    return s


def _prepare_build_trace(s, case, gen, rng):
    s["pos"], s["idx"] = _grid(case["qx"], case["qy"], gen)
    s["mode"] = dict(median=case["build"] == "median", sah=case["build"] == "sah")
    s["bvh"] = rq.Bvh.build(s["ctx"], s["pos"], s["idx"], **s["mode"])
    s["rays"] = _rays_down(case["rays"], gen)
    s["hits"], s["t"] = _hits(case["rays"])


def _prepare_frame(s, case, gen, rng):
    s["base"], s["idx"] = _grid(case["qx"], case["qy"], gen)
    s["pos"] = s["base"].clone()
    s["time"] = float(rng.uniform(0.0, 6.0))
    s["bvh"] = rq.Bvh.build(s["ctx"], s["pos"], s["idx"], sah=True)
    s["cam"] = W.shadow_camera(case["width"], case["height"])
    s["params"] = rq.shade_params(case["width"], case["height"], _lights(case["lights"], rng), ao_spp=case["spp"],
                                  ao_tmax=0.5)
    shape = tune.lookup_shadow(tune.shadow_key(2 * case["qx"] * case["qy"], s["params"], True))
    if shape:
        s["ctx"].set_trace_tuning(**shape)
    n = case["width"] * case["height"]
    s["gbuf"] = torch.empty((n, 8), dtype=torch.int32, device=DEV)
    s["mask"] = torch.empty(n, dtype=torch.int32, device=DEV)
    s["ao"] = torch.empty(n, dtype=torch.float32, device=DEV)


def _prepare_visibility(s, case, gen, rng):
    s["base"], s["idx"] = _grid(case["q"], case["q"], gen)
    s["pos"] = s["base"].clone()
    s["time"] = float(rng.uniform(0.0, 6.0))
    s["bvh"] = rq.Bvh.build(s["ctx"], s["pos"], s["idx"])
    s["cam"] = W.visibility_camera(case["width"], case["height"], seed=int(rng.integers(1 << 31)))
    s["gbuf"] = torch.empty((case["width"] * case["height"], 8), dtype=torch.int32, device=DEV)


def _prepare_batched(s, case, gen, rng):
    descs = _batch_meshes(case)
    meshes = [_grid(d[4], d[5], gen) for d in descs]
    s["base"] = torch.cat([m[0] for m in meshes])
    s["idx"] = torch.cat([m[1] for m in meshes])
    s["pos"] = s["base"].clone()
    s["time"] = float(rng.uniform(0.0, 6.0))
    s["batch"] = rq.Batch(s["ctx"], [d[:4] for d in descs])
    a, c = case["rays_any"], case["rays_closest"]
    shape = tune.lookup(tune.workload_key([d[:4] for d in descs], a + c))
    if shape:
        s["batch"].set_tuning(shape)
    n = len(descs) * (a + c)
    s["rays"] = _rays_down(n, gen)
    s["mesh"] = torch.arange(len(descs), dtype=torch.int32, device=DEV).repeat_interleave(a + c)
    s["flags"] = (torch.arange(a + c, device=DEV) < a).int().repeat(len(descs))
    s["hits"], s["t"] = _hits(n)


def _prepare_serving(s, case, gen, rng):
    sizes, mesh, kind, rays = _requests(case)
    s["server"] = srv = rq.Server(device=torch.cuda.current_device())
    ids = []
    for t in sizes:
        pos, idx = _grid(*W.grid_for_triangles(t), gen)
        ids.append(srv.add_mesh(pos.cpu().numpy(), idx.cpu().numpy().view(np.uint32)))
    s["hits"], s["t"] = _hits(int(rays.sum()))
    first = np.concatenate([[0], np.cumsum(rays)])
    seeds = rng.integers(1 << 31, size=len(rays))
    s["requests"] = [srv.request(ids[mesh[k]], int(kind[k]), int(rays[k]), s["hits"][first[k]:first[k + 1]],
                                 seed=int(seeds[k]), user=k) for k in range(len(rays))]
    # the meshes become resident with their first request
    warm = torch.empty((32, 4), dtype=torch.int32, device=DEV)
    for m in ids:
        srv.submit(srv.request(m, rq.RQ_RAYS_CLOSEST, 32, warm))
    srv.completions()


def _prepare_terrain(s, case, gen, rng):
    pos, idx = _grid(case["q"], case["q"], gen)
    # the reference's terrain: 100 units wide, y up, heights a quarter of the grid's
    pos = torch.stack([50.0 * pos[:, 0], 12.5 * pos[:, 2], 50.0 * pos[:, 1]], 1).contiguous()
    s["pos"], s["idx"] = pos, idx
    s["bvh"] = rq.Bvh.build(s["ctx"], pos, idx)
    eye = [float(v) for v in rng.uniform([-3.0, 47.0, -48.0], [3.0, 53.0, -42.0])]
    s["rays"] = rq.gen_rays_procedural(s["ctx"], eye, [0, 0, 5], case["rays"], case["coherent"])
    s["hits"], s["t"] = _hits(case["rays"])


def _prepare_radv(s, case, gen, rng):
    pos, idx = _grid(case["qx"], case["qy"], gen)
    s["tri9"] = pos[idx.long()].reshape(-1).contiguous()
    s["image"] = torch.zeros(rq.radv_size(len(idx)), dtype=torch.uint8, device=DEV)
    s["rays"] = _rays_down(case["rays"], gen) if case["rays"] else None


def _prepare_effects(s, case, gen, rng):
    pos, idx = _grid(case["q"], case["q"], gen)
    ctx, w, h = s["ctx"], case["width"], case["height"]
    s["bvh"] = rq.Bvh.build(ctx, pos, idx, sah=True)
    cam = W.shadow_camera(w, h)
    s["gbuf"] = rq.render_gbuffer(ctx, s["bvh"], cam)
    s["view_proj"] = rq.view_proj_of(cam)
    s["ao_params"] = rq.ao_depth_params(cam, spp=case["spp"])
    s["reflect"] = rq.reflect_params(cam)
    s["depth"], s["ao"], s["half"], s["blurred"] = (torch.empty(w * h, dtype=torch.float32, device=DEV)
                                                    for _ in range(4))
    s["hits"], s["t"] = _hits(w * h)


def _prepare_instances(s, case, gen, rng):
    s["blas"] = []
    for qx, qy in _instance_sizes(case):
        pos, idx = _grid(qx, qy, gen)
        s["blas"].append(rq.Bvh.build(s["ctx"], pos, idx))
    s["instances"] = []
    for k in range(case["instances"]):
        q, _ = np.linalg.qr(rng.standard_normal((3, 3)))
        a = q @ np.diag(rng.uniform(0.5, 2.0, 3))
        t = rng.uniform(-8.0, 8.0, 3)
        s["instances"].append((np.hstack([a, t[:, None]]).astype(np.float32), 1000 + k, 0xFF,
                               s["blas"][int(rng.integers(len(s["blas"])))]))
    n = case["rays"]
    o = torch.rand((n, 3), generator=gen, device=DEV) * 24 - 12
    d = torch.randn((n, 3), generator=gen, device=DEV)
    d = d / d.norm(dim=1, keepdim=True)
    col = torch.ones((n, 1), device=DEV)
    s["rays"] = torch.cat([o, 0.01 * col, d, 1000.0 * col], 1).contiguous()
    s["hits"], s["t"] = _hits(n)


# ------------------------------------------------------------------------- run
def run(s):
    return globals()["_run_" + s["case"]["kind"]](s, s["ctx"])


def _run_build_trace(s, ctx):
    rq.Bvh.build(ctx, s["pos"], s["idx"], into=s["bvh"], **s["mode"])
    rq.trace(ctx, s["bvh"], s["rays"], flags=_flags(s["case"]), hits=s["hits"])
    return dict(hits=s["hits"], t=s["t"])


def _run_frame(s, ctx):
    rq.deform_wave(ctx, s["base"], s["pos"], s["time"], W.DEFORM_AMP, W.DEFORM_FREQ)
    rq.Bvh.build(ctx, s["pos"], s["idx"], into=s["bvh"], sah=True)
    rq.render_gbuffer(ctx, s["bvh"], s["cam"], s["gbuf"])
    rq.render_shadow_ao(ctx, s["bvh"], s["gbuf"], s["params"], s["mask"], s["ao"])
    return dict(gbuf=s["gbuf"], mask=s["mask"], ao=s["ao"])


def _run_visibility(s, ctx):
    rq.deform_wave(ctx, s["base"], s["pos"], s["time"], W.DEFORM_AMP, W.DEFORM_FREQ)
    if s["case"]["refit"]:
        s["bvh"].refit(s["pos"], s["idx"])
    else:
        rq.Bvh.build(ctx, s["pos"], s["idx"], into=s["bvh"])
    rq.render_gbuffer(ctx, s["bvh"], s["cam"], s["gbuf"])
    return dict(gbuf=s["gbuf"])


def _run_batched(s, ctx):
    rq.deform_wave(ctx, s["base"], s["pos"], s["time"], W.DEFORM_AMP, W.DEFORM_FREQ)
    s["batch"].build(s["pos"], s["idx"])
    s["batch"].trace(s["rays"], s["mesh"], s["flags"], hits=s["hits"])
    return dict(hits=s["hits"], t=s["t"])


def _run_serving(s, ctx):
    srv = s["server"]
    for r in s["requests"]:
        srv.submit(r)
    done = srv.completions()
    return dict(hits=s["hits"], t=s["t"], ok=sum(c["status"] == rq.RQ_OK for c in done.values()))


def _run_terrain(s, ctx):
    rq.trace(ctx, s["bvh"], s["rays"], flags=_flags(s["case"]), hits=s["hits"])
    return dict(hits=s["hits"], t=s["t"])


def _run_radv(s, ctx):
    rq.build_radv(ctx, s["tri9"], s["image"])
    if s["rays"] is None:
        return dict(image=s["image"])
    hits, _ = rq.trace_radv(ctx, s["image"], s["rays"])
    return dict(image=s["image"], hits=hits)


def _run_effects(s, ctx):
    w, h = s["case"]["width"], s["case"]["height"]
    rq.gbuffer_depth(ctx, s["gbuf"], s["view_proj"], s["depth"])
    rq.render_ao_depth(ctx, s["bvh"], s["depth"], s["ao_params"], s["ao"])
    rq.blur_ao(ctx, s["ao"], s["depth"], w, h, 1, 0, 0.01, s["half"])
    rq.blur_ao(ctx, s["half"], s["depth"], w, h, 0, 1, 0.01, s["blurred"])
    rq.render_reflect(ctx, s["bvh"], s["gbuf"], s["reflect"], s["hits"])
    return dict(depth=s["depth"], ao=s["ao"], blurred=s["blurred"], hits=s["hits"], t=s["t"])


def _run_instances(s, ctx):
    top = rq.Tlas(ctx, s["instances"])
    top.trace(s["rays"], flags=_flags(s["case"]), hits=s["hits"])
    top.destroy()
    return dict(hits=s["hits"], t=s["t"])


# ------------------------------------------------------------------------ work
RAY, HIT, PIXEL = 32, 16, 32
# a ray's least arithmetic: 4 boxes of 12 operations per level of a 4-wide tree, 4 triangle tests of 40
BOX4, TRIANGLES = 48, 160


def _ray_flops(n, tris):
    return n * (BOX4 * max(1.0, math.log(max(4, tris) / 4, 4)) + TRIANGLES)


def _mesh_bytes(tris, verts):
    return 12 * tris + 12 * verts


def work(case):
    k = case["kind"]
    if k == "batched":
        d = _batch_meshes(case)
        tris, verts = sum(x[3] for x in d), sum(x[1] for x in d)
        n = len(d) * (case["rays_any"] + case["rays_closest"])
        return dict(bytes=_mesh_bytes(tris, verts) + n * (RAY + 8 + HIT), flops=_ray_flops(n, tris / len(d)) + 60 * tris)
    if k == "serving":
        sizes, mesh, _, rays = _requests(case)
        return dict(bytes=float(rays.sum()) * HIT + 60.0 * sum(int(sizes[m]) for m in set(mesh.tolist())),
                    flops=sum(_ray_flops(int(r), int(sizes[m])) for r, m in zip(rays, mesh)))
    if k == "instances":
        tris = sum(2 * x * y for x, y in _instance_sizes(case))
        return dict(bytes=60 * tris + case["rays"] * (RAY + HIT), flops=_ray_flops(case["rays"], tris))
    qx, qy = case.get("qx", case.get("q")), case.get("qy", case.get("q"))
    tris, verts = 2 * qx * qy, (qx + 1) * (qy + 1)
    mesh = _mesh_bytes(tris, verts)
    if k == "radv":
        return dict(bytes=36 * tris + rq.radv_size(tris) + case["rays"] * (RAY + HIT),
                    flops=60 * tris + (_ray_flops(case["rays"], tris) if case["rays"] else 0))
    if k == "terrain":
        return dict(bytes=mesh + case["rays"] * (RAY + HIT), flops=_ray_flops(case["rays"], tris))
    if k == "build_trace":
        return dict(bytes=mesh + case["rays"] * (RAY + HIT), flops=_ray_flops(case["rays"], tris) + 60 * tris)
    n = case["width"] * case["height"]
    if k == "frame":
        return dict(bytes=mesh + 12 * verts + n * (PIXEL + 8),
                    flops=_ray_flops(n * (1 + case["lights"] + case["spp"]), tris) + 60 * tris)
    if k == "visibility":
        return dict(bytes=mesh + 12 * verts + n * PIXEL, flops=_ray_flops(n, tris) + 60 * tris)
    return dict(bytes=mesh + n * (PIXEL + 12 + HIT), flops=_ray_flops(n * (1 + case["spp"]), tris))


# ----------------------------------------------------------------------- exact
def _closest(tri, rays, mt):
    """Nearest crossing of each ray with the triangles (float64 [T,3,3]), -1 for a miss: every pair is solved."""
    v0, e1, e2 = tri[:, 0], tri[:, 1] - tri[:, 0], tri[:, 2] - tri[:, 0]
    n = torch.linalg.cross(e1, e2)
    out = torch.empty(len(rays), dtype=torch.float64, device=DEV)
    step = max(1, (1 << 25) // len(tri))
    for k in range(0, len(rays), step):
        r = rays[k:k + step]
        o, d = r[:, None, 0:3], r[:, None, 4:7]
        s = o - v0[None]
        det = -(d * n[None]).sum(-1)
        c = torch.linalg.cross(s, d.expand_as(s))
        u, v, t = (c * e2[None]).sum(-1) / det, -(c * e1[None]).sum(-1) / det, (s * n[None]).sum(-1) / det
        ok = (u >= 0) & (v >= 0) & (u + v <= 1) & (t >= r[:, None, 3]) & (t < r[:, None, 7])
        if mt:  # the reference's triangle test passes through triangles this close to parallel
            ok &= det.abs() >= 1e-7
        t = torch.where(ok, t, torch.inf).amin(1)
        out[k:k + step] = torch.where(t.isfinite(), t, -1.0)
    return out


def exact(case, seed):
    """Closest-hit distances of ray buffers over one mesh, where every pair of ray and triangle can be solved."""
    if case["kind"] != "build_trace" or case["any"] or 2.0 * case["qx"] * case["qy"] * case["rays"] > 6e9:
        return None
    gen = torch.Generator(device=DEV).manual_seed(int(seed))
    pos, idx = _grid(case["qx"], case["qy"], gen)
    rays = _rays_down(case["rays"], gen)
    return dict(hits=None, t=_closest(pos.double()[idx.long()], rays.double(), case["mt"]))
