"""The measured cases: what a program that renders with this framework has it do.

A case names an entry point (``call``), a scene, and the sizes of one pass:

* ``query``       GpuScene.intersect: a batch of rays in host memory;
* ``rays``        gprt_intersect: a batch of rays in device memory;
* ``pass``        ProgressiveRaytracer.render_pass of a kept renderer: the RGBA image
                  of the next progressive pass;
* ``frame``       ProgressiveRaytracer.add_samples and the mean radiance image of a
                  kept renderer, path tracing or BDPT;
* ``progressive`` a whole progressive render, from the renderer's creation through
                  every pass with the adaptive stop, as the web front door runs it;
* ``serve``       a batch of requests through a RenderServer, each image read back.

``prepare`` builds the scene and the renderer or server that a program keeps between
passes; ``run`` is one pass.  The renderers draw new sample indices on each pass, so
no pass repeats another's work.
"""
import ctypes as C
import functools
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                                "go-progressive-raytracer_gb300"))
import gprt  # noqa: E402
from gprt import capi, scenes  # noqa: E402


def listed():
    return [
        # a picking or visibility query of a host program: a handful of rays in
        # host memory; the time is launches, copies and allocations
        {"name": "query_cornell_1000", "call": "query", "scene": "cornell_spheres", "rays": 1000, "any": False},
        # an occlusion batch on a medium mesh, a ragged number of rays
        {"name": "any_ico6_300007", "call": "rays", "scene": "ico", "level": 6, "rays": 300007, "any": True},
        # the benchmark's raw batch: 2^24 rays, half coherent, on 1.3 M triangles
        {"name": "closest_ico8_16m", "call": "rays", "scene": "ico", "level": 8, "rays": 1 << 24, "any": False},
        # the first thing that a viewer shows: 1 sample per pixel of a small image
        {"name": "preview_spheres_128", "call": "pass", "scene": "spheres", "width": 128, "height": 128, "spp": 1,
         "depth": 8},
        # a later progressive pass of the reference's built-in Cornell scene, as
        # configured there (depth 5, metal and glass)
        {"name": "pass_cornell_spheres_400", "call": "pass", "scene": "cornell_spheres", "width": 400, "spp": 8,
         "depth": 5},
        # the reference's default scene rendered as its front door does: adaptive
        # sampling, depth 50, thin lens, layered and glass spheres
        {"name": "progressive_default_400", "call": "progressive", "scene": "default", "width": 400, "spp": 16,
         "passes": 5},
        # the reference's textured test scene at an odd size: every shape kind
        {"name": "frame_textures_517", "call": "frame", "scene": "textures", "width": 517, "spp": 3, "depth": 10},
        # benchmark configuration: Cornell box, 64 samples per pixel
        {"name": "frame_cornell_400_64", "call": "frame", "scene": "cornell", "width": 400, "spp": 64, "depth": 8},
        # benchmark configuration: 1.3 M triangles, one material each, 16 samples per pixel
        {"name": "frame_ico8_1024_16", "call": "frame", "scene": "ico", "level": 8, "width": 1024, "spp": 16,
         "depth": 8},
        # a BDPT preview of the spot-light scene, odd size
        {"name": "bdpt_spot_131_2", "call": "frame", "scene": "spot", "width": 131, "spp": 2, "depth": 8,
         "bdpt": True},
        # benchmark configuration: Cornell boxes under BDPT, 64 samples per pixel
        {"name": "bdpt_boxes_512_64", "call": "frame", "scene": "boxes", "width": 512, "spp": 64, "depth": 8,
         "bdpt": True},
        # the headline's kind of load: requests of mixed sizes batched by the server
        {"name": "serve_32_jobs", "call": "serve", "scene": "spheres", "jobs": 32, "max_spp": 32, "depth": 8,
         "step_paths": 1 << 24},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    call = rng.choice(["query", "rays", "rays", "pass", "pass", "progressive", "frame", "frame", "bdpt", "serve"])
    if call == "query":
        return {"call": call, "scene": rng.choice(["cornell_spheres", "quadrics", "textures"]),
                "rays": _log_int(rng, 64, 20000), "any": rng.random() < 0.5}
    if call == "rays":
        c = {"call": call, "scene": rng.choice(["ico", "ico", "cornell", "quadrics"]),
             "rays": _log_int(rng, 3000, 6000000), "any": rng.random() < 0.5}
        if c["scene"] == "ico":
            c["level"] = rng.randint(3, 7)
        return c
    if call == "progressive":
        return {"call": call, "scene": rng.choice(["default", "grid"]), "width": rng.randint(160, 480),
                "spp": rng.randint(6, 20), "passes": rng.randint(2, 6)}
    if call == "serve":
        return {"call": call, "scene": "spheres", "jobs": rng.randint(3, 32), "max_spp": rng.randint(4, 32),
                "depth": rng.randint(5, 12), "step_paths": 1 << rng.randint(22, 24)}
    width = _log_int(rng, 48, 384 if call == "bdpt" else 640)
    c = {"call": "frame" if call == "bdpt" else call, "width": width,
         "spp": _log_int(rng, 1, max(1.0, min(64, 4e6 / width ** 2))), "depth": rng.randint(4, 12)}
    if call == "bdpt":
        c.update(scene=rng.choice(["boxes", "spot", "quadrics", "spheres"]), bdpt=True, depth=rng.randint(4, 9))
    else:
        c["scene"] = rng.choice(["cornell", "cornell_spheres", "spheres", "quadrics", "textures", "ico"])
    if c["scene"] == "ico":
        c["level"] = rng.randint(3, 7)
    if c["scene"] == "spheres":
        c["height"] = _log_int(rng, 48, 400)
    return c


# ---------------------------------------------------------------- scenes
@functools.lru_cache(maxsize=1)
def _context():
    return gprt.Context(0)  # a program has one


def _scene(case, seed):
    """The scene of a case; the seed varies what its family leaves open."""
    kind, width = case["scene"], case.get("width", 256)
    cam = gprt.CameraConfig(width=width)
    if kind == "cornell":
        s = scenes.cornell_baseline(width)
    elif kind == "cornell_spheres":
        s = scenes.cornell_scene(scenes.CORNELL_SPHERES, camera=cam)
    elif kind == "boxes":
        s = scenes.cornell_boxes_bdpt(width)
    elif kind == "spot":
        s = scenes.spot_scene(width)
    elif kind == "quadrics":
        s = scenes.quadric_scene(width)
    elif kind == "textures":
        s = scenes.texture_test_scene(cam)
    elif kind == "default":
        s = scenes.default_scene(cam)
    elif kind == "grid":
        s = scenes.sphere_grid_scene(10, camera=cam)
    elif kind == "ico":
        s = scenes.icosphere_scene(level=case["level"], width=width, noise_seed=7 + seed % 5, material_seed=seed)
    elif kind == "spheres":
        s = scenes.default_style_scene(seed, width, case.get("height", width))
    else:
        raise ValueError("unknown scene %r" % kind)
    if "depth" in case:  # fixed sampling; the others keep the scene's own adaptive settings
        s.sampling.max_depth = case["depth"]
        s.sampling.adaptive_min_samples, s.sampling.adaptive_threshold = 1.0, 0.0
    return s


def _bounds(scene):
    """A box around what the scene's rays start in: the mesh, or the space seen by its camera."""
    for sh in scene.shapes:
        if sh.mesh is not None:
            v = sh.mesh.placed_vertices()
            return v.min(0), v.max(0)
    c, a = np.array(scene.camera.center, dtype=np.float64), np.array(scene.camera.look_at, dtype=np.float64)
    r = 0.5 * np.linalg.norm(c - a)
    return a - r, a + r


def _rays(scene, n, seed):
    """n rays, (n, 8) float32 on the GPU: half coherent (jittered camera rays in
    scanline order), half incoherent (from points on the mesh, or within the
    scene, in uniform directions)."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    f = dict(device="cuda", generator=g, dtype=torch.float32)
    half = n // 2
    cam = scene.camera
    t = functools.partial(torch.tensor, device="cuda", dtype=torch.float32)
    o, at = t(cam.center), t(cam.look_at)
    w = (o - at) / torch.linalg.vector_norm(o - at)
    u = torch.linalg.cross(t(cam.up), w)
    u = u / torch.linalg.vector_norm(u)
    v = torch.linalg.cross(w, u)
    side = max(1, math.isqrt(max(1, half)))
    i = torch.arange(half, device="cuda")
    scale = 2.0 * math.tan(math.radians(cam.vfov) / 2)
    x = (((i % side) + torch.rand(half, **f)) / side - 0.5) * scale
    y = (0.5 - ((i // side) % side + torch.rand(half, **f)) / side) * scale
    d = x[:, None] * u + y[:, None] * v - w
    rays = torch.empty((n, 8), device="cuda")
    rays[:, 3], rays[:, 7] = 0.001, math.inf
    rays[:half, 0:3] = o
    rays[:half, 4:7] = d / torch.linalg.vector_norm(d, dim=1, keepdim=True)
    m = n - half
    mesh = next((sh.mesh for sh in scene.shapes if sh.mesh is not None), None)
    if mesh is not None:
        face = torch.from_numpy(mesh.faces.astype(np.int64)).cuda()[
            torch.randint(0, len(mesh.faces), (m,), device="cuda", generator=g)]
        vert = torch.from_numpy(mesh.placed_vertices()).cuda().float()
        r1, r2 = torch.rand(m, **f).sqrt()[:, None], torch.rand(m, **f)[:, None]
        rays[half:, 0:3] = vert[face[:, 0]] * (1 - r1) + vert[face[:, 1]] * (r1 * (1 - r2)) + vert[face[:, 2]] * (r1 * r2)
    else:
        lo, hi = (t(b) for b in _bounds(scene))
        rays[half:, 0:3] = lo + (hi - lo) * torch.rand((m, 3), **f)
    d = torch.randn((m, 3), **f)
    rays[half:, 4:7] = d / torch.linalg.vector_norm(d, dim=1, keepdim=True)
    return rays


def _request_sizes(case, seed):
    rng = np.random.default_rng(seed)
    sizes = [(128, 128), (256, 256), (512, 512), (1024, 768)]
    # the resolutions of the headline batch, each as often in every batch
    return [sizes[k % 4] + (int(rng.integers(1, case["max_spp"] + 1)), int(rng.integers(0, 2 ** 31 - 1)))
            for k in range(case["jobs"])]


# ---------------------------------------------------------------- one case
def prepare(case, seed):
    ctx = _context()
    call = case["call"]
    if call == "serve":
        req = [(gprt.GpuScene(ctx, scenes.default_style_scene(s, w, h, max_depth=case["depth"])),
                gprt.ProgressiveConfig(initial_samples=min(4, spp), max_samples_per_pixel=spp, max_passes=min(2, spp),
                                       seed=seed + k))
               for k, (w, h, spp, s) in enumerate(_request_sizes(case, seed))]
        return {"call": call, "server": gprt.RenderServer(ctx, step_paths=case["step_paths"]), "requests": req}
    scene = _scene(case, seed)
    g = gprt.GpuScene(ctx, scene)
    if call in ("query", "rays"):
        rays = _rays(scene, case["rays"], seed)
        if call == "query":
            return {"call": call, "scene": g, "any": case["any"], "rays": rays.cpu().numpy()}
        return {"call": call, "scene": g, "any": case["any"], "rays": rays, "ctx": ctx,
                "hits": torch.empty((case["rays"], 4), device="cuda"), "stream": torch.cuda.Stream()}
    if call == "progressive":
        return {"call": call, "scene": g,
                "config": gprt.ProgressiveConfig(max_samples_per_pixel=case["spp"], max_passes=case["passes"], seed=seed)}
    spp, many = case["spp"], 1 << 20  # a renderer that is asked for many passes of this size
    work = g.width * g.height * spp
    config = gprt.ProgressiveConfig(initial_samples=spp, max_samples_per_pixel=spp * many, max_passes=many, seed=seed,
                                    chunk_paths=min(work, 1 << 24))
    job = gprt.ProgressiveRaytracer(g, config, gprt.BDPTIntegrator() if case.get("bdpt") else None)
    return {"call": call, "job": job, "spp": spp, "pass": 0}


def run(state):
    call = state["call"]
    if call == "query":
        h = state["scene"].intersect(state["rays"], any_hit=state["any"])
        return {"t": h["t"], "uv": np.stack([h["u"], h["v"]], 1), "prim": h["prim"].astype(np.int64)}
    if call == "rays":
        lib, s = state["ctx"].lib, state["stream"]
        state["ctx"].check(lib.gprt_intersect(state["scene"].h, C.c_void_p(state["rays"].data_ptr()),
                                              len(state["rays"]), capi.ANY if state["any"] else capi.CLOSEST,
                                              C.c_void_p(state["hits"].data_ptr()), C.c_void_p(s.cuda_stream)))
        h = state["hits"]
        return {"t": h[:, 0], "uv": h[:, 2:4], "prim": h.view(torch.int32)[:, 1]}
    if call == "pass":
        state["pass"] += 1
        img, st = state["job"].render_pass(state["pass"])
        return {"rgba": img, "samples": st.total_samples}
    if call == "frame":
        state["job"].add_samples(state["spp"])
        return state["job"].image()
    if call == "progressive":
        r = gprt.ProgressiveRaytracer(state["scene"], state["config"])
        out = [{"rgba": p.image, "samples": p.stats.total_samples} for p in r.render_progressive()]
        r.close()
        return out
    server = state["server"]
    tickets = [server.submit(g, c) for g, c in state["requests"]]
    server.run_until_idle()
    out = [server.rgba8(t) for t in tickets]
    for t in tickets:
        server.release(t)
    return out


# ---------------------------------------------------------------- what a pass cannot do without
_PRIMS = {"cornell": 18, "cornell_spheres": 8, "boxes": 18, "spot": 5, "quadrics": 9, "textures": 14, "default": 9,
          "grid": 102, "spheres": 260}
_ASPECT = {"spot": 0.7, "textures": 16 / 9, "default": 16 / 9, "grid": 16 / 9}
# surfaces that a path meets, at most the depth: walls on every side, or a sky
_MEETS = {"cornell": 12.0, "cornell_spheres": 12.0, "boxes": 12.0}


def _prims(case):
    return 20 * 4 ** case["level"] + 1 if case["scene"] == "ico" else _PRIMS[case["scene"]]


def _ray_flops(prims):
    # a slab test (12 flops) of both children on each level of a binary tree, and two primitive tests
    return 24.0 * math.log2(prims + 1) + 2 * 50.0


def work(case):
    prims = _prims(case)
    scene = prims * (80.0 if case["scene"] != "ico" else 96.0)
    if case["call"] in ("query", "rays"):
        return {"bytes": 48.0 * case["rays"] + scene, "flops": case["rays"] * _ray_flops(prims)}
    if case["call"] == "serve":  # resolutions in equal parts, samples uniform up to max_spp
        pixels = case["jobs"] * (128 ** 2 + 256 ** 2 + 512 ** 2 + 1024 * 768) / 4.0
        samples = pixels * (case["max_spp"] + 1) / 2.0
        scene *= case["jobs"]
    else:
        w = case["width"]
        pixels = float(w * case.get("height", int(w / _ASPECT.get(case["scene"], 1.0))))
        samples = pixels * case["spp"]
    meets = min(float(case.get("depth", 50)), _MEETS.get(case["scene"], 2.5))
    flops = 2.0 * meets * _ray_flops(prims) + meets * 200.0  # to each surface and to a light; scatter and the light's sample
    if case.get("bdpt"):
        flops = 2 * flops + 0.5 * meets ** 2 * (_ray_flops(prims) + 150.0)  # two subpaths; a ray and a weight per connection
    # the film read and written once, the image out
    return {"bytes": scene + pixels * (2 * 24.0 + (12.0 if case["call"] == "frame" else 4.0)), "flops": samples * flops}


# ---------------------------------------------------------------- 64-bit answers
def exact(case, seed):
    """Closest hits of a ray batch by testing every primitive in 64 bits (triangles,
    quads and spheres).  Images have none: a path that a rounding sends past the edge
    of a shape goes elsewhere, so a 64-bit render is another draw of the same integral,
    and which hit an any-hit query reports is the traversal's choice."""
    if case["call"] not in ("query", "rays") or case["any"] or case["scene"] not in ("ico", "cornell", "cornell_spheres"):
        return None
    if case["rays"] * _prims(case) > 3e10:
        return None
    scene = _scene(case, seed)
    rays = _rays(scene, case["rays"], seed).double()
    tris, quads, spheres = _primitives(scene)
    t, uv = [], []
    step = max(1, int(4e7 // _prims(case)))
    for r in rays.split(step):
        a, b = _closest(r, tris, quads, spheres)
        t.append(a)
        uv.append(b)
    t, uv = torch.cat(t), torch.cat(uv)
    if case["call"] == "query":
        t, uv = t.cpu().numpy(), uv.cpu().numpy()
    return {"t": t, "uv": uv, "prim": None}


def _primitives(scene):
    """(triangles (a, ab, ac), quads (corner, u, v), spheres (centre, radius)) of a scene, 64 bits."""
    tris, quads, spheres = np.zeros((0, 9)), [], []
    for sh in scene.shapes + [lt.shape for lt in scene.lights if lt.shape is not None]:
        if sh.kind == capi.SHAPE_MESH:
            v, f = sh.mesh.placed_vertices(), sh.mesh.faces
            a = v[f[:, 0]]
            tris = np.concatenate([tris, np.concatenate([a, v[f[:, 1]] - a, v[f[:, 2]] - a], 1)])
        elif sh.kind == capi.SHAPE_QUAD and sh.p not in quads:
            quads.append(sh.p)
        elif sh.kind == capi.SHAPE_SPHERE and sh.p not in spheres:
            spheres.append(sh.p)
        elif sh.kind == capi.SHAPE_BOX:
            quads += _box_faces(sh.p)
    d = functools.partial(torch.tensor, device="cuda", dtype=torch.float64)
    return torch.from_numpy(tris).cuda(), d(quads).reshape(-1, 9), d(spheres).reshape(-1, 4)


def _box_faces(p):
    """The six faces of a box (centre, half extents, rotation about X, then Y, then Z); a face's
    u and v as the reference's NewBox has them (pkg/geometry/box.go:36-140)."""
    c, h, (rx, ry, rz) = np.array(p[0:3]), np.array(p[3:6]), p[6:9]

    def at(x, y, z):
        q = np.array([x, y, z]) * h
        q = np.array([q[0], q[1] * math.cos(rx) - q[2] * math.sin(rx), q[1] * math.sin(rx) + q[2] * math.cos(rx)])
        q = np.array([q[0] * math.cos(ry) + q[2] * math.sin(ry), q[1], -q[0] * math.sin(ry) + q[2] * math.cos(ry)])
        q = np.array([q[0] * math.cos(rz) - q[1] * math.sin(rz), q[0] * math.sin(rz) + q[1] * math.cos(rz), q[2]])
        return c + q

    corners = [((-1, -1, 1), (1, -1, 1), (-1, 1, 1)), ((1, -1, -1), (-1, -1, -1), (1, 1, -1)),
               ((1, -1, 1), (1, -1, -1), (1, 1, 1)), ((-1, -1, -1), (-1, -1, 1), (-1, 1, -1)),
               ((-1, 1, -1), (-1, 1, 1), (1, 1, -1)), ((-1, -1, 1), (-1, -1, -1), (1, -1, 1))]
    return [tuple(np.concatenate([at(*a), at(*b) - at(*a), at(*d) - at(*a)])) for a, b, d in corners]


def _closest(rays, tris, quads, spheres):
    """Nearest hit of each ray with t in [tmin, tmax]: t (-1 for none) and (u, v)."""
    n = len(rays)
    o, d, lo, hi = rays[:, None, 0:3], rays[:, None, 4:7], rays[:, None, 3], rays[:, None, 7]
    t = torch.full((n,), math.inf, device="cuda", dtype=torch.float64)
    uv = torch.zeros((n, 2), device="cuda", dtype=torch.float64)

    def offer(tt, u, v, ok):
        nonlocal t, uv
        if not tt.shape[1]:
            return
        tt = torch.where(ok & (tt >= lo) & (tt <= hi), tt, math.inf)
        best, k = tt.min(1)
        mine = torch.stack([x.gather(1, k[:, None])[:, 0] for x in (u, v)], 1)
        uv = torch.where((best < t)[:, None], mine, uv)
        t = torch.minimum(t, best)

    def dot(a, b):
        return (a * b).sum(-1)

    if len(tris):  # det = e1 . (d x e2), written with the triple products that need no (rays, triangles, 3) array of cross products
        a, e1, e2 = tris[:, 0:3], tris[:, 3:6], tris[:, 6:9]
        nrm = torch.linalg.cross(e1, e2)
        dd, oo = rays[:, 4:7], rays[:, 0:3]
        m = torch.linalg.cross(oo, dd)
        det = -(dd @ nrm.T)
        tt = (oo @ nrm.T - dot(a, nrm)[None]) / det
        # u = (s . (d x e2)) / det with s = o - a, and v = (d . (s x e1)) / det
        ae2, ae1 = torch.linalg.cross(a, e2), torch.linalg.cross(a, e1)
        u = (m @ e2.T + dd @ ae2.T) / det
        v = -(m @ e1.T + dd @ ae1.T) / det
        offer(tt, u, v, (det != 0) & (u >= 0) & (v >= 0) & (u + v <= 1))
    if len(quads):
        c, qu, qv = quads[None, :, 0:3], quads[None, :, 3:6], quads[None, :, 6:9]
        nn = torch.linalg.cross(qu, qv)
        tt = dot(c - o, nn) / dot(d, nn)
        h = o + tt[..., None] * d - c
        w = nn / dot(nn, nn)[..., None]
        u, v = dot(w, torch.linalg.cross(h, qv.expand_as(h))), dot(w, torch.linalg.cross(qu.expand_as(h), h))
        offer(tt, u, v, (u >= 0) & (u <= 1) & (v >= 0) & (v <= 1))
    if len(spheres):
        f = o - spheres[None, :, 0:3]
        a, hb = dot(d, d), dot(f, d)
        disc = hb * hb - a * (dot(f, f) - spheres[None, :, 3] ** 2)
        sq = disc.clamp(min=0).sqrt()
        near, far = (-hb - sq) / a, (-hb + sq) / a
        zero = torch.zeros_like(near)
        offer(torch.where(near >= lo, near, far), zero, zero, disc >= 0)
    return torch.where(torch.isinf(t), -1.0, t), uv
