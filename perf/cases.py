"""What a user of the renderer has it do, as cases that can be timed.

A case is a dict of plain values.  `listed()` gives the fixed ones, `draw(rng)`
one more of the same ranges, `prepare(case, seed)` what a program holds before
the call, `run(state)` one pass through the public entry points, `work(case)`
the bytes and operations a pass cannot do without and `exact(case, seed)` the
outputs in 64 bits where they are computed numbers with such a value.

Kinds:
  frame       Renderer.render / render_graph: the next frame of one view
  views       MultiViewRenderer.render: the next frame of several views
  edit        Renderer.erase and the frame after it
  build       Accel over a scene's tables, then pick rays through it
  visibility  ct_trace_visibility on a batch of shadow rays
  closest     ct_trace_closest on a batch of pick rays
  adjoint     AdjointRenderer.forward, with or without .backward
  nrc         NrcCache.infer / infer_encoded / encode_device
  nrc_frame   NrcRenderer.render: trace, online training, inference
"""
import ctypes
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "cube-tracing_b200"))

from cube_tracing import adjoint, native, nrc, scenes, views  # noqa: E402
from cube_tracing import layouts as L  # noqa: E402
from cube_tracing.frame import Accel, Renderer, SceneBuffers  # noqa: E402


# ---------------------------------------------------------------------------
# the cases

def listed():
    return [
        # an interactive preview of the small plain workload (64^3 grid,
        # 256x256, DI + PT to depth 4 + TAA), frames replayed from a graph:
        # launches and the latency of short queues count
        {"name": "frame_preview", "kind": "frame", "scene": "grid", "edge": 64, "width": 256, "height": 256,
         "depth": 4, "hybrid": False, "rounds": 1, "instances": 1, "graph": True},
        # the headline benchmark's frame: 256^3 terrain at 1920x1080, two DI
        # spatial rounds, ReSTIR PT with the hybrid shift to depth 8, TAA
        {"name": "frame_headline", "kind": "frame", "scene": "terrain", "edge": 256, "width": 1920, "height": 1080,
         "depth": 8, "hybrid": True, "rounds": 2, "instances": 1, "graph": False},
        # direct light only (the reference's shipped setting) at an odd size
        # over four instances with their own transforms
        {"name": "frame_direct_odd", "kind": "frame", "scene": "grid", "edge": 96, "width": 1277, "height": 719,
         "depth": 0, "hybrid": False, "rounds": 1, "instances": 4, "graph": False},
        # many small views per step, over shared scenes
        {"name": "views_batch", "kind": "views", "scenes": 3, "views": 8, "edge": 96, "width": 640, "height": 480,
         "depth": 6},
        # interactive editing: erase under the brush, rebuild, next frame
        {"name": "edit_frame", "kind": "edit", "scene": "terrain", "edge": 128, "width": 960, "height": 540,
         "depth": 4, "window": 50},
        # loading a scene: the acceleration structure of 4 M voxels, and the
        # first pick rays through it
        {"name": "build_terrain", "kind": "build", "scene": "terrain", "edge": 256, "rays": 16384},
        # a batch of shadow rays between surface points and lights
        {"name": "visibility_batch", "kind": "visibility", "scene": "terrain", "edge": 128, "rays": 1 << 20},
        # a pick under a brush: few rays, all latency
        {"name": "closest_pick", "kind": "closest", "scene": "grid", "edge": 64, "rays": 2001},
        # one gradient step's passes of the differentiable tracer
        {"name": "adjoint_step", "kind": "adjoint", "scene": "grid", "edge": 128, "width": 512, "height": 512,
         "spp": 8, "depth": 3, "backward": True},
        # the plain path tracer to depth 8, one sample per pixel
        {"name": "plain_trace", "kind": "adjoint", "scene": "terrain", "edge": 192, "width": 1277, "height": 719,
         "spp": 1, "depth": 8, "backward": False},
        # the radiance cache queried for every pixel of a 1080p frame
        {"name": "cache_query", "kind": "nrc", "op": "infer", "queries": 1920 * 1080},
        # a frame of the cache renderer with its online training
        {"name": "cache_frame", "kind": "nrc_frame", "scene": "terrain", "edge": 192, "width": 960, "height": 540,
         "paths": 1 << 14},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["frame", "frame", "views", "edit", "build", "visibility", "closest", "adjoint", "nrc",
                       "nrc_frame"])
    scene = rng.choice(["grid", "terrain"])
    c = {"kind": kind}
    if kind == "frame":
        depth = rng.choice([0, 2, 4, 6, 8])
        c.update(scene=scene, edge=_log(rng, 24, 160), width=_log(rng, 96, 1920), height=_log(rng, 80, 1080),
                 depth=depth, hybrid=bool(depth) and rng.random() < 0.5, rounds=rng.choice([1, 1, 2, 3]),
                 instances=rng.choice([1, 1, 2, 4]), graph=rng.random() < 0.5)
    elif kind == "views":
        c.update(scenes=rng.randint(1, 3), views=rng.randint(2, 8), edge=_log(rng, 48, 96),
                 width=_log(rng, 160, 640), height=_log(rng, 120, 480), depth=rng.choice([0, 4, 6]))
    elif kind == "edit":
        c.update(scene=scene, edge=_log(rng, 32, 128), width=_log(rng, 160, 960), height=_log(rng, 120, 540),
                 depth=rng.choice([0, 4]), window=rng.randint(5, 60))
    elif kind == "build":
        c.update(scene=scene, edge=_log(rng, 24, 200), rays=_log(rng, 1024, 16384))
    elif kind == "visibility":
        c.update(scene=scene, edge=_log(rng, 32, 160), rays=_log(rng, 1000, 1 << 20))
    elif kind == "closest":
        c.update(scene=scene, edge=_log(rng, 32, 160), rays=_log(rng, 1000, 1 << 20))
    elif kind == "adjoint":
        c.update(scene=scene, edge=_log(rng, 32, 160), width=_log(rng, 100, 512), height=_log(rng, 100, 512),
                 spp=rng.choice([1, 2, 4, 8]), depth=rng.randint(1, 6), backward=rng.random() < 0.6)
    elif kind == "nrc":
        c.update(op=rng.choice(["infer", "infer", "infer_encoded", "encode"]), queries=_log(rng, 500, 1 << 20))
    else:
        c.update(scene="terrain", edge=_log(rng, 64, 192), width=_log(rng, 200, 960), height=_log(rng, 160, 540),
                 paths=1 << rng.randint(10, 14))
    return c


# ---------------------------------------------------------------------------
# inputs

def _point_light(sc, edge, strength):
    pl = np.zeros(1, L.LIGHT)
    pl["position"] = (edge * 0.5, edge * 1.5, edge * 0.5)
    pl["emissive"] = (strength,) * 3
    pl["instance_id"] = L.MAX_INSTANCES
    pl["primitive_id"] = L.MAX_PRIMITIVES
    pl["type"] = L.LIGHT_POINT
    sc.point_lights = pl
    sc.light_config["point_light_count"] = 1


def _split(sc, parts, rng):
    """The scene's voxels over `parts` instances (slabs along z, which the
    voxels are ordered by), each turned a little about y and moved apart."""
    n = sc.aabbs.shape[0]
    z = sc.aabbs["minimum"][:, 2]
    cut = np.searchsorted(z, np.linspace(0, float(z.max()) + 1.0, parts + 1)[1:-1])
    first = np.concatenate([[0], cut, [n]]).astype(np.int64)
    inst = np.zeros(parts, L.INSTANCE)
    lights = sc.cube_lights.copy()
    prim = lights["primitive_id"].astype(np.int64)
    for i in range(parts):
        a = 0.0 if i == 0 else float(rng.uniform(-0.05, 0.05))
        m = np.eye(4)
        m[0, 0] = m[2, 2] = math.cos(a)
        m[0, 2], m[2, 0] = math.sin(a), -math.sin(a)
        m[:3, 3] = (0.0, 0.25 * i, 1.5 * i)
        inst["transform"][i] = m.astype(np.float32).reshape(-1, order="F")
        inst["first_primitive_index"][i] = first[i]
        inst["primitive_count"][i] = first[i + 1] - first[i]
        sel = (prim >= first[i]) & (prim < first[i + 1])
        p = np.concatenate([lights["position"][sel], np.ones((int(sel.sum()), 1), np.float32)], axis=1)
        lights["position"][sel] = (p @ m.T.astype(np.float32))[:, :3]
        lights["instance_id"][sel] = i
        lights["primitive_id"][sel] = (prim[sel] - first[i]).astype(np.uint32)
    sc.instances, sc.cube_lights = inst, lights


def _scene(c, seed):
    e = c["edge"]
    if c["kind"] in ("edit", "adjoint"):
        seed = 1  # their outputs have a row per voxel: the inputs vary in other ways
    if c["scene"] == "grid":
        sc = scenes.random_grid_scene(e, 0.3 if c["kind"] != "adjoint" else 0.25, emissive_fraction=0.02, seed=seed)
        _point_light(sc, e, 50.0)
    else:
        sc = scenes.heightfield_scene(e, base=e * 0.25, amplitude=e * 0.1875, emissive_fraction=0.005, seed=seed,
                                      radiance=(2.0, 20.0))
        _point_light(sc, e, 4.0)
    return sc


def _cameras(c, n, seed):
    """n frames of the kind's camera: a slow translation past the grid or an
    orbit over the terrain."""
    e, w, h = float(c["edge"]), c["width"], c["height"]
    if c["scene"] == "grid":
        return scenes.camera_path("translate", n, w, h, eye=(-e / 4 + seed % 7, e / 2, -e / 4), target=(e / 2,) * 3,
                                  step=(0.1, 0.0, 0.0))
    return scenes.camera_path("orbit", n, w, h, center=(e / 2, e * 0.234, e / 2), radius=e * 0.547,
                              elevation=e * 0.352, deg_per_frame=0.5, phi0=float(seed * 37 % 360))


def _view_sizes(c):
    """Resolutions of the case's views, log-uniform up to its largest."""
    rng = np.random.default_rng(c["views"] + c["width"])
    return [(int(math.exp(rng.uniform(math.log(128), math.log(c["width"])))),
             int(math.exp(rng.uniform(math.log(96), math.log(c["height"]))))) for _ in range(c["views"])]


def _pick_rays(c, seed):
    """Rays from a ring of eyes outside the grid to points inside it, as
    ct_ray_query records (10 words)."""
    n, e = c["rays"], float(c["edge"])
    g = torch.Generator("cuda").manual_seed(seed)
    u = torch.rand((n, 4), generator=g, device="cuda")
    az = u[:, 3] * (2 * math.pi)
    eye = torch.stack([e / 2 + 1.2 * e * torch.cos(az), 0.9 * e + 0.0 * az, e / 2 + 1.2 * e * torch.sin(az)], 1)
    target = u[:, :3] * torch.tensor([e, e * 0.3, e], device="cuda")
    d = target - eye
    q = torch.zeros((n, 10), device="cuda")
    q[:, 0:3] = eye
    q[:, 3] = 1e9
    q[:, 4:7] = d / d.norm(dim=1, keepdim=True)
    return q


def _shadow_rays(c, sc, seed):
    """Shadow rays from points just off the faces of emitters' neighbours to
    points on other emitters, which the query's target check lets through."""
    n = c["rays"]
    g = torch.Generator("cuda").manual_seed(seed)
    pos = torch.from_numpy(np.ascontiguousarray(sc.cube_lights["position"])).cuda()
    prim = torch.from_numpy(sc.cube_lights["primitive_id"].astype(np.int32)).cuda()
    a = torch.randint(0, pos.shape[0], (n,), generator=g, device="cuda")
    b = torch.randint(0, pos.shape[0], (n,), generator=g, device="cuda")
    j = torch.rand((n, 4), generator=g, device="cuda") - 0.5
    o = pos[a] + torch.stack([j[:, 0], torch.full_like(j[:, 0], 0.5005), j[:, 1]], 1)
    t = pos[b] + torch.stack([j[:, 2], torch.full_like(j[:, 2], 0.5), j[:, 3]], 1)
    d = t - o
    dist = d.norm(dim=1, keepdim=True).clamp(min=1e-6)
    q = torch.zeros((n, 10), device="cuda")
    q[:, 0:3], q[:, 3:4], q[:, 4:7] = o, dist, d / dist
    qi = q.view(torch.int32)
    qi[:, 7] = L.QUERY_CHECK_TARGET
    qi[:, 9] = prim[b]
    return q


def _renderer(c, seed):
    sc = _scene(c, seed)
    if c.get("instances", 1) > 1:
        _split(sc, c["instances"], np.random.default_rng(seed))
    params = {"spatial_passes": c.get("rounds", 1), "max_ris_cube_samples": 32}
    if c.get("hybrid"):
        params.update(taa_alpha=0.1, pt_shift_mapping=2, pt_near_field_distance=0.5)
    return Renderer(sc, c["width"], c["height"], params=params, indirect=c["depth"] > 0,
                    max_depth=c["depth"] or 3)


def _frame_outputs(r, image):
    """The image and the history the frame leaves for the next, the words of
    each record that are whole numbers apart from those that are floats."""
    def words(key, n, whole):
        w = r.buf[key].view(torch.int32).view(-1, n)
        real = [i for i in range(n) if i not in whole]
        return w[:, whole], w.view(torch.float32)[:, real]
    out = {"image": image}
    out["reservoir_ids"], out["reservoir"] = words("previous_reservoir", 9, [0, 1, 2])
    out["di_ids"], out["di"] = words("di", 15, [10, 11, 12, 13])
    if r.params.flags & native.CT_PARAM_INDIRECT:
        out["path_ids"], out["path"] = words("temporal_path_reservoir", 23, [2, 3, 11, 12, 13])
        out["indirect"] = r.buf["indirect_color"].view(torch.float32)
    return out


class _State:
    def __init__(self, **kw):
        self.__dict__.update(kw)


def _queries(case, seed):
    return nrc.random_queries(case["queries"], seed=seed)


def _cache(seed):
    return nrc.NrcCache((0.0, 0.0, 0.0), (256.0, 128.0, 256.0), seed=seed)


def prepare(case, seed):
    c, kind = case, case["kind"]
    if kind == "frame":
        # three frames in: a warm history, and the graph (if any) captured
        r, cams = _renderer(c, seed), _cameras(c, 64, seed)
        s = _State(kind=kind, r=r, cams=cams, draw=r.render_graph if c["graph"] else r.render)
        for k in range(3):
            s.draw(*cams[k])
        return s
    if kind == "views":
        scs, vs = views.views_workload(n_scenes=c["scenes"], n_views=c["views"], seed=seed,
                                       edge_range=(32, c["edge"]))
        for v, (w, h) in zip(vs, _view_sizes(c)):
            v["width"], v["height"] = w, h
        mv = views.MultiViewRenderer(scs, vs, indirect=c["depth"] > 0, max_depth=c["depth"] or 3)
        s = _State(kind=kind, mv=mv)
        for _ in range(3):
            mv.render(mv.cams(mv.frame))
        return s
    if kind == "edit":
        r, cams = _renderer(c, seed), _cameras(c, 64, seed)
        for k in range(2):
            r.render(*cams[k])
        sb = r.sb
        tables = [sb.instances, sb.primitives, sb.aabbs, sb.cube_lights, sb.light_config]
        return _State(kind=kind, r=r, cams=cams, tables=tables, saved=[t.clone() for t in tables],
                      pixel=(c["width"] // 2, c["height"] * 2 // 3), window=c["window"])
    if kind == "build":
        sc = _scene(c, seed)
        dev = [torch.from_numpy(np.ascontiguousarray(a).view(np.uint8).reshape(-1).copy()).cuda()
               for a in (sc.instances, sc.aabbs)]
        return _State(kind=kind, instances=dev[0], n_inst=sc.instances.shape[0], aabbs=dev[1],
                      n=sc.aabbs.shape[0], extent=sc.voxel_extent, q=_pick_rays(c, seed),
                      hits=torch.zeros((c["rays"], 4), dtype=torch.int32, device="cuda"))
    if kind in ("visibility", "closest"):
        sc = _scene(c, seed)
        sb = SceneBuffers(sc)
        if kind == "visibility":
            return _State(kind=kind, sb=sb, q=_shadow_rays(c, sc, seed),
                          out=torch.zeros(c["rays"], dtype=torch.uint8, device="cuda"))
        return _State(kind=kind, sb=sb, q=_pick_rays(c, seed),
                      hits=torch.zeros((c["rays"], 4), dtype=torch.int32, device="cuda"))
    if kind == "adjoint":
        sc = _scene(c, seed)
        iv, ip = _cameras(c, 1, seed)[0]
        a = adjoint.scene_tables(sc, iv, ip, c["width"], c["height"])
        r = adjoint.AdjointRenderer(a, spp=c["spp"], max_depth=c["depth"], seed=seed,
                                    miss_radiance=0.0 if c["backward"] else 0.5)
        g = torch.Generator("cuda").manual_seed(seed)
        return _State(kind=kind, r=r, backward=c["backward"],
                      albedo=torch.rand(a.albedo_target.shape, generator=g, device="cuda") * 0.8 + 0.1,
                      emission=torch.rand(a.emission_target.shape, generator=g, device="cuda") * 9.0 + 1.0,
                      target=torch.rand((c["height"], c["width"], 3), generator=g, device="cuda"))
    if kind == "nrc":
        cache, q = _cache(seed), _queries(c, seed)
        return _State(kind=kind, cache=cache, op=c["op"],
                      q=cache.encode_device(q) if c["op"] == "infer_encoded" else q)
    if kind == "nrc_frame":
        torch.manual_seed(seed)
        sc = _scene(c, seed)
        iv, ip = _cameras(c, 1, seed)[0]
        a = adjoint.scene_tables(sc, iv, ip, c["width"], c["height"])
        plain = adjoint.AdjointRenderer(a, spp=1, max_depth=8, seed=1, miss_radiance=0.5)
        cache = nrc.NrcCache((0.0, 0.0, 0.0), (float(c["edge"]),) * 3, seed=seed)
        # the cache serves from the second frame on; prepare renders that far
        r = nrc.NrcRenderer(plain, cache, train_paths=c["paths"], min_frames=1, diverge=1e9)
        s = _State(kind=kind, r=r, frame=0, seed=seed)
        for _ in range(2):
            run(s)
        return s
    raise ValueError(kind)


def _call(name, *args):
    native.check(name, getattr(native.lib(), name)(*args))


def _hits(h):
    return {"ids": h[:, :2], "t": h.view(torch.float32)[:, 2]}


def run(s):
    if s.kind == "frame":
        return _frame_outputs(s.r, s.draw(*s.cams[s.r.frame % 64]))
    if s.kind == "views":
        mv = s.mv
        mv.render(mv.cams(mv.frame))
        return [r.images[(r.frame - 1) % 2] for r in mv.r]
    if s.kind == "edit":
        for t, saved in zip(s.tables, s.saved):  # undo the last erase
            t.copy_(saved)
        s.r.erase(s.pixel, s.window)
        out = _frame_outputs(s.r, s.r.render(*s.cams[s.r.frame % 64]))
        out["tables"] = [s.r.sb.instances.view(torch.int32), s.r.sb.primitives.view(torch.int32),
                         s.r.sb.aabbs.view(torch.float32)]
        return out
    if s.kind == "build":
        acc = Accel(s.instances, s.n_inst, s.aabbs, s.n, s.extent)
        _call("ct_trace_closest", acc.handle, s.q.data_ptr(), s.q.shape[0], s.hits.data_ptr(),
              torch.cuda.current_stream().cuda_stream)
        i = acc.info()
        out = dict(_hits(s.hits), bricks=i.brick_count, voxels=i.voxel_count, exact=i.grid_exact,
                   grid=[int(v) for v in list(i.grid_min) + list(i.grid_dim)])
        acc.free()
        return out
    if s.kind == "visibility":
        _call("ct_trace_visibility", s.sb.accel.handle, s.q.data_ptr(), s.q.shape[0], s.out.data_ptr(),
              torch.cuda.current_stream().cuda_stream)
        return s.out
    if s.kind == "closest":
        _call("ct_trace_closest", s.sb.accel.handle, s.q.data_ptr(), s.q.shape[0], s.hits.data_ptr(),
              torch.cuda.current_stream().cuda_stream)
        return _hits(s.hits)
    if s.kind == "adjoint":
        img = s.r.forward(s.albedo, s.emission)
        if not s.backward:
            return img
        return [img, *s.r.backward(s.albedo, s.emission, 2.0 * (img - s.target))]
    if s.kind == "nrc":
        if s.op == "infer":
            return s.cache.infer(s.q)
        return s.cache.encode_device(s.q) if s.op == "encode" else s.cache.infer_encoded(s.q)
    s.frame += 1
    img, (loss, n) = s.r.render(1000 * s.seed + s.frame)
    return {"image": img, "loss": loss, "vertices": n, "query": s.r.query, "throughput": s.r.thp,
            "weights": [w.detach() for w in s.r.cache.mlp.weights], "packed": s.r.cache.weights}


# ---------------------------------------------------------------------------
# what a pass cannot do without, and its outputs in 64 bits

def _voxels(c):
    e = c["edge"]
    return (0.3 if c["scene"] == "grid" else 0.24) * e ** 3


def work(case):
    c, kind = case, case["kind"]
    if kind in ("frame", "edit"):
        px = c["width"] * c["height"]
        # records read and written once: DI 60 B (previous and new), reservoir
        # 36 B (two), velocity 8 B, images 16 B (three); with PT the path
        # reservoirs 92 B (two) and the indirect colour 12 B
        b = px * (2 * 60 + 2 * 36 + 8 + 3 * 16 + (2 * 92 + 12 if c["depth"] else 0))
        # 32 light candidates of ~60 operations, and per ray ~20 box steps of
        # ~30 operations for the camera, 2 + 8 per round shadow, depth bounces
        rays = 3 + 8 * c.get("rounds", 1) + c["depth"]
        f = px * (32 * 60 + rays * 600)
        if kind == "edit":
            b += 32 * _voxels(c) + 4 * c["edge"] ** 3
        return {"bytes": b, "flops": f}
    if kind == "views":
        px = sum(w * h for w, h in _view_sizes(c))
        return {"bytes": px * (444 if c["depth"] else 248), "flops": px * (32 * 60 + (11 + c["depth"]) * 600)}
    if kind == "build":
        # the AABBs read; the cell field (4 B a cell) and the voxel tables written
        return {"bytes": (24 + 4 + 4) * _voxels(c) + 4 * c["edge"] ** 3 + 56 * c["rays"], "flops": 0}
    if kind == "visibility":
        return {"bytes": 41 * c["rays"], "flops": 600 * c["rays"]}
    if kind == "closest":
        return {"bytes": 56 * c["rays"], "flops": 600 * c["rays"]}
    if kind == "adjoint":
        px = c["width"] * c["height"]
        b = px * 12 * (3 if c["backward"] else 1) + 12 * _voxels(c) * (2 if c["backward"] else 1)
        return {"bytes": b, "flops": px * c["spp"] * c["depth"] * 500 * (2 if c["backward"] else 1)}
    if kind == "nrc":
        n, mlp = c["queries"], 2 * (256 * 64 + 4 * 64 * 64 + 64 * 16)
        if c["op"] == "infer":
            return {"bytes": 60 * n, "flops": mlp * n}
        return {"bytes": 560 * n, "flops": 0} if c["op"] == "encode" else {"bytes": 524 * n, "flops": mlp * n}
    px = c["width"] * c["height"]
    mlp = 2 * (256 * 64 + 4 * 64 * 64 + 64 * 16)
    return {"bytes": px * (48 + 12 + 12 + 12) + c["paths"] * (5 * 48 + 4 * 24),
            "flops": mlp * (px + c["paths"] + 3 * 4 * 16384) + px * 2 * 500}


def _encode64(q, bmin, bext):
    """The cache's encoding of (n, 12) queries in 64 bits."""
    q = q.double()
    k = torch.arange(16, device=q.device, dtype=torch.float64)
    x = ((q[:, 0:3] - torch.tensor(bmin, device=q.device, dtype=torch.float64))
         / torch.tensor(bext, device=q.device, dtype=torch.float64)).clamp(0.0, 1.0)
    a = math.pi * torch.remainder(x[:, :, None] * 2.0 ** k, 2.0)
    parts = [torch.stack([torch.sin(a), torch.cos(a)], -1).reshape(q.shape[0], 96)]
    centres = (torch.arange(32, device=q.device, dtype=torch.float64) + 0.5) / 32.0
    for v in (q[:, 3:6], q[:, 6:9]):
        for u in (torch.atan2(v[:, 2], v[:, 0]) / (2.0 * math.pi) + 0.5, v[:, 1] / 2.0 + 0.5):
            parts.append(torch.exp(-0.5 * ((u[:, None] - centres) * 32.0) ** 2))
    parts += [q[:, 9:12], torch.zeros((q.shape[0], 29), device=q.device, dtype=torch.float64)]
    return torch.cat(parts, 1)


def _mlp64(x, weights):
    w = weights.double()
    at = 0
    for i, (o, n) in enumerate([(64, 256)] + [(64, 64)] * 4 + [(16, 64)]):
        x = x @ w[at:at + o * n].view(o, n).t()
        at += o * n
        if i < 5:
            x = torch.relu(x)
    return x[:, :3]


def _closest64(sc, q):
    """The nearest voxel box each ray enters: (ids, t), ties to the lowest id."""
    lo = torch.from_numpy(np.ascontiguousarray(sc.aabbs["minimum"])).cuda().double()
    hi = torch.from_numpy(np.ascontiguousarray(sc.aabbs["maximum"])).cuda().double()
    out = torch.empty(q.shape[0], dtype=torch.float64, device="cuda")
    for i in range(0, q.shape[0], 64):
        o, d = q[i:i + 64, None, 0:3].double(), q[i:i + 64, None, 4:7].double()
        a, b = (lo - o) / d, (hi - o) / d
        near, far = torch.minimum(a, b).amax(-1), torch.maximum(a, b).amin(-1)
        t = torch.where((near <= far) & (near > 0), near, math.inf).amin(1)
        out[i:i + 64] = torch.where(torch.isfinite(t), t, -1.0)
    return out


def exact(case, seed):
    """Rendered frames and gradients have none: which voxel a path meets
    turns on the last bits of its rays, and so does everything after it."""
    c, kind = case, case["kind"]
    if kind == "nrc":
        q, cache = _queries(c, seed), _cache(seed)
        if c["op"] == "infer_encoded":
            return _mlp64(cache.encode_device(q).double(), cache.weights)
        step = 1 << 17
        parts = [_encode64(q[i:i + step], cache.bbox_min, cache.bbox_extent) for i in range(0, q.shape[0], step)] \
            if c["op"] == "encode" else \
            [_mlp64(_encode64(q[i:i + step], cache.bbox_min, cache.bbox_extent), cache.weights)
             for i in range(0, q.shape[0], step)]
        return torch.cat(parts)
    if kind == "closest" and c["rays"] * _voxels(c) < 4e8:
        return {"ids": None, "t": _closest64(_scene(c, seed), _pick_rays(c, seed))}
    return None
