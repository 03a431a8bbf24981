"""Timed cases of the render hot path, through the public Python entry points.

What a program does with this library falls into six kinds of call, each with
its own range of sizes:

  rays      batched ray queries against a built scene: picking and collision
            (few rays), occlusion tests with a bound per ray, baking and
            visibility (millions); rays resident on the device, or given and
            returned as host arrays
  frame     one image of one scene: reset, the frame's samples, the resolved image
  batch     many uneven render jobs in one device-driven run, every film read back
  inverse   one step of inverse rendering: loss and gradient
  rebuild   changed geometry: the acceleration structure rebuilt, then queried
  move      moved instances: the structure refitted, then queried

A scene, its accelerator, a ray buffer on the device and the arrays results are
read into are what such a program has in hand before the call (prepare); a pass
(run) is the call, up to the point where its results can be used.  Sizes are
those of the benchmark's workloads and of the tests, and sizes between them.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from vkpathtracer_b200 import scenes
from vkpathtracer_b200.tracer import BatchRenderer, CudaPathTracer, RenderTile, material_params


# ------------------------------------------------------------------- the cases
def _rays(n, mesh, size, mode="closest", test="mt", bvh="sah", host=False, **kw):
    """mesh "sphere": one displaced sphere of size x size vertices; "field":
    size x size displaced spheres on a ground plane; "box": the closed box."""
    return dict(kw, kind="rays", n=n, mesh=mesh, size=size, mode=mode, test=test, bvh=bvh, host=host)


def _frame(scene, size, width, height, spp, depth, bvh="sah", preview=False, **kw):
    """preview: one sample into a tone-mapped 8-bit image after a camera move
    (render_tile), else every sample of the frame into a linear float image."""
    return dict(kw, kind="frame", scene=scene, size=size, width=width, height=height, spp=spp, depth=depth, bvh=bvh,
                preview=preview)


def _batch(jobs, max_triangles, max_side, pool=0, block=0, stack=0, steps=0, occupancy=0, **kw):
    """The launch parameters are the ones a program keeps from the autotuner; 0: the defaults."""
    return dict(kw, kind="batch", jobs=jobs, max_triangles=max_triangles, max_side=max_side, pool=pool, block=block,
                stack=stack, steps=steps, occupancy=occupancy)


def listed():
    return [
        # a click or a handful of collision rays in an interactive scene: latency of one small call
        _rays(1000, "field", 16, name="pick_1k"),
        # ambient-occlusion style bounded visibility rays on a closed mesh, where the watertight test is wanted
        _rays(100_003, "sphere", 256, mode="any", test="watertight", bvh="reference", name="occlusion_100k"),
        # rays that a program computes on the host (IRayAccelerator::intersect in batches), results back on the host
        _rays(262_147, "field", 32, host=True, bvh="reference", name="host_rays_262k"),
        # the ray-query workload: 8,388,608 camera and random rays on the 1,046,904-triangle sphere
        _rays(8_388_608, "sphere", 724, name="closest_8m"),
        # the small closed-box image: 36 triangles, 16 samples, depth 8
        _frame("box", 1, 256, 256, 16, 8, bvh="reference", name="box_256"),
        # interactive preview: camera moved, one sample of a mid-sized scene, displayed
        _frame("field", 16, 1280, 720, 1, 6, bvh="reference", preview=True, name="preview_720p"),
        # a full-HD image of the 2,064,386-triangle sphere grid at depth 16, some of its 64 samples
        _frame("field", 64, 1920, 1080, 8, 16, name="full_hd_grid"),
        # sphere-traced SDF primitives next to triangles, an odd-sized window
        _frame("sdf", 1, 853, 479, 4, 8, bvh="reference", name="sdf_gallery"),
        # the 64-job batch of the benchmark, with the launch parameters of its autotuner, every film read back
        _batch(64, 500_000, 1024, pool=1 << 24, block=128, stack=8, steps=16, occupancy=4, name="batch_64_jobs"),
        # inverse rendering of the box room: 64 parameters, 128 x 128 pixels, 32 samples, forward and backward
        dict(kind="inverse", objects=16, side=128, spp=32, name="inverse_128"),
        # new geometry in a large scene: 2,064,386 triangles rebuilt with the SAH tree, one coarse view queried
        dict(kind="rebuild", size=64, bvh="sah", view=512, name="rebuild_2m"),
        # physics-driven objects: 1,024 instances moved (516,098 triangles refitted), one coarse view queried
        dict(kind="move", size=32, bvh="reference", view=256, name="move_1k_instances"),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["rays", "rays", "rays", "rays", "frame", "frame", "frame", "batch", "inverse", "rebuild",
                       "move"])
    bvh = rng.choice(["reference", "sah"])
    if kind == "rays":
        mesh = rng.choice(["sphere", "sphere", "field", "field", "box"])
        size = {"sphere": _log(rng, 24, 724), "field": _log(rng, 2, 64), "box": 1}[mesh]
        host = rng.random() < 0.2
        return _rays(_log(rng, 33, 600_000 if host else 8_000_000), mesh, size, rng.choice(["closest", "closest", "any"]),
                     rng.choice(["mt", "mt", "watertight"]), bvh, host)
    if kind == "frame":
        scene = rng.choice(["box", "field", "field", "sdf", "glass", "effects", "sky"])
        size = {"field": _log(rng, 3, 64), "sky": _log(rng, 2, 8)}.get(scene, 1)
        width, height = _log(rng, 61, 1921), _log(rng, 47, 1081)
        if rng.random() < 0.3:
            return _frame(scene, size, width, height, 1, rng.randint(2, 12), bvh, True)
        spp = max(1, min(64, int(rng.uniform(0.1, 1.0) * 1.6e7 / (width * height))))
        return _frame(scene, size, width, height, spp, rng.randint(2, 16), bvh)
    if kind == "batch":
        jobs, side = rng.randint(2, 24), _log(rng, 192, 640)
        if rng.random() < 0.5:
            return _batch(jobs, _log(rng, 4_000, 400_000), side)
        return _batch(jobs, _log(rng, 4_000, 400_000), side, 1 << rng.randint(20, 23), 128, 8, 16, 4)
    if kind == "inverse":
        return dict(kind="inverse", objects=rng.randint(4, 32), side=_log(rng, 33, 160), spp=rng.randint(2, 40))
    if kind == "rebuild":
        return dict(kind="rebuild", size=_log(rng, 2, 64), bvh=bvh, view=_log(rng, 33, 700))
    return dict(kind="move", size=_log(rng, 2, 48), bvh=bvh, view=_log(rng, 33, 500))


# ------------------------------------------------------------------- scenes
def _scene(kind, size, seed):
    if kind == "sphere":
        return scenes.displaced_sphere(size, seed=seed)
    if kind == "field":
        # the lights and their heights as the benchmark's jobs of this size have them; the full grid's are fixed
        if size >= 64:
            return scenes.sphere_grid(seed, size)
        return scenes.sphere_field(size, 15, 18, seed, n_lights=min(16, max(1, size)),
                                   light_size=max(1.0, 0.3 * size), light_height=max(4.0, 0.75 * size))
    if kind == "sdf" or kind == "glass":
        return scenes.sdf_gallery(seed, glass=kind == "glass")
    if kind == "effects":
        return scenes.effect_gallery(seed)
    if kind == "sky":
        return scenes.sky_scene(seed, size)
    return scenes.cornell_box(seed)


def _tracer(scene, settings, bvh, test="mt"):
    t = CudaPathTracer(bvh=bvh, triangle_test=test)
    for status in (t.configure(settings), t.load_scene_snapshot(scene), t.build_or_update_acceleration()):
        if not status.ok:
            raise RuntimeError(status.message)
    return t


def _unit(v):
    return v / v.norm(dim=1, keepdim=True)


def _camera_rays(camera, width, height):
    """Pinhole rays through the pixel centres, (width * height, 6) float32 on the device, row by row."""
    pos = torch.tensor(camera.position, dtype=torch.float64, device="cuda")
    fwd = _unit((torch.tensor(camera.target, dtype=torch.float64, device="cuda") - pos)[None])[0]
    right = _unit(torch.linalg.cross(fwd, torch.tensor(camera.up, dtype=torch.float64, device="cuda"))[None])[0]
    up = torch.linalg.cross(right, fwd)
    th = math.tan(0.5 * math.radians(camera.fov_deg))
    x = (2.0 * (torch.arange(width, device="cuda").double() + 0.5) / width - 1.0) * th * width / height
    y = (1.0 - 2.0 * (torch.arange(height, device="cuda").double() + 0.5) / height) * th
    d = _unit((fwd + x[None, :, None] * right + y[:, None, None] * up).reshape(-1, 3)).float()
    return torch.cat([pos.float().expand_as(d), d], dim=1).contiguous()


def _query_rays(scene, n, seed):
    """The first half camera rays (coherent), the rest random: origins in 1.5
    times the scene's bounding cube, directions uniform on the sphere."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    side = max(1, math.isqrt(n // 2))
    cam = _camera_rays(scene.camera, side, side)[: n // 2]
    m = n - cam.shape[0]
    v = np.asarray(scene.vertices, np.float64)
    lo, hi = v.min(axis=0), v.max(axis=0)
    mid = torch.tensor(0.5 * (lo + hi), device="cuda")
    half = 0.75 * float((hi - lo).max())
    o = mid + (2.0 * torch.rand(m, 3, generator=g, device="cuda", dtype=torch.float64) - 1.0) * half
    z = 1.0 - 2.0 * torch.rand(m, generator=g, device="cuda", dtype=torch.float64)
    ph = 2.0 * math.pi * torch.rand(m, generator=g, device="cuda", dtype=torch.float64)
    r = (1.0 - z * z).clamp(min=0.0).sqrt()
    d = _unit(torch.stack([r * ph.cos(), r * ph.sin(), z], dim=1)).float()
    rays = torch.cat([cam, torch.cat([o.float(), d], dim=1)]).contiguous()
    # bounds for occlusion queries: between a hundredth of the scene and all of it
    tmax = half * (0.02 + 2.0 * torch.rand(n, generator=g, device="cuda"))
    return rays, tmax


_ANY_SETTINGS = scenes.RenderSettings(width=8, height=8, spp=1)


class _Query:
    """Rays on the device and the buffers their hits go to, on a stream of the program's own."""

    def __init__(self, tracer, rays, tmax=None, mode=0):
        self.tracer, self.rays, self.tmax, self.mode = tracer, rays, tmax, mode
        self.n = rays.shape[0]
        self.prim = torch.empty(self.n, dtype=torch.int32, device="cuda")
        self.t = torch.empty(self.n, dtype=torch.float32, device="cuda")
        self.stream = torch.cuda.Stream()

    def __call__(self):
        self.tracer.trace_rays_device(self.rays.data_ptr(), 0 if self.tmax is None else self.tmax.data_ptr(), self.n,
                                      self.mode, self.prim.data_ptr(), self.t.data_ptr(), self.stream.cuda_stream)
        return {"prim": self.prim, "t": self.t}


# ------------------------------------------------------------------- prepare
def _batch_jobs(case, seed):
    """The benchmark's job set (its sizes belong to the case), each job with a
    moved camera and random numbers of its own."""
    jobs = scenes.batch_jobs(case["jobs"], max_triangles=case["max_triangles"], max_side=case["max_side"])
    for j, job in enumerate(jobs):
        job.settings.seed += seed + j
        job.scene.camera.position = tuple(p + 0.01 * (1 + (seed + j) % 7) for p in job.scene.camera.position)
    return jobs


def prepare(case, seed):
    k = case["kind"]
    if k == "rays":
        sc = _scene(case["mesh"], case["size"], seed % 1000)
        rays, tmax = _query_rays(sc, case["n"], seed)
        t = _tracer(sc, _ANY_SETTINGS, case["bvh"], case["test"])
        any_hit = case["mode"] == "any"
        if case["host"]:
            return {"case": case, "tracer": t, "rays": rays.cpu().numpy(), "tmax": tmax.cpu().numpy() if any_hit else None}
        return {"case": case, "query": _Query(t, rays, tmax if any_hit else None, int(any_hit))}
    if k == "frame":
        sc = _scene(case["scene"], case["size"], seed % 1000)
        st = scenes.RenderSettings(width=case["width"], height=case["height"], spp=case["spp"], max_depth=case["depth"],
                                   seed=seed + 1234, firefly_clamp=10.0 if case["size"] >= 64 else 0.0)
        cam = sc.camera
        step = 0.01 * (1 + seed % 7)
        moved = scenes.Camera(tuple(p + step for p in cam.position), cam.target, cam.up, cam.fov_deg)
        return {"case": case, "tracer": _tracer(sc, st, case["bvh"]), "camera": moved}
    if k == "batch":
        b = BatchRenderer(bvh="sah")
        jobs = _batch_jobs(case, seed)
        for j in jobs:
            b.add_job(j.scene, j.settings)
        px = [j.settings.width * j.settings.height for j in jobs]
        sums = torch.empty(3 * sum(px), dtype=torch.float32, pin_memory=True)
        counts = torch.empty(sum(px), dtype=torch.int32, pin_memory=True)
        off = np.concatenate([[0], np.cumsum(px)])
        s, c = sums.numpy(), counts.numpy()
        shapes = [(j.settings.height, j.settings.width) for j in jobs]
        return {"case": case, "batch": b, "sums": sums, "counts": counts,
                "sum_views": [s[3 * off[i]:3 * off[i + 1]].reshape(h, w, 3) for i, (h, w) in enumerate(shapes)],
                "count_views": [c[off[i]:off[i + 1]].reshape(h, w) for i, (h, w) in enumerate(shapes)],
                "tuning": dict(pool_paths=case["pool"], block_size=case["block"], stack_depth=case["stack"],
                               steps=case["steps"], occupancy=case["occupancy"])}
    if k == "inverse":
        sc = scenes.inverse_box_scene(seed=seed % 1000, n_objects=case["objects"])
        st = scenes.inverse_settings(case["side"], case["side"], case["spp"])
        t = _tracer(sc, st, "reference")
        target_params = material_params(sc.materials)
        t.adjoint_setup(case["spp"])
        _, target = t.forward(target_params, image=True)
        t.adjoint_setup(case["spp"], target)
        guess = target_params.copy()
        r = np.random.RandomState(seed % (1 << 31))
        own = slice(5, 5 + case["objects"])   # the objects' materials follow the room's five walls
        guess[own, :4] = r.uniform(0.1, 0.8, guess[own, :4].shape).astype(np.float32)
        return {"case": case, "tracer": t, "params": guess}
    if k == "rebuild":
        sc = _scene("field", case["size"], seed % 1000)
        t = _tracer(sc, _ANY_SETTINGS, case["bvh"])
        return {"case": case, "tracer": t, "query": _Query(t, _camera_rays(sc.camera, case["view"], case["view"]))}
    if k == "move":
        sc = scenes.dynamic_sphere_field(case["size"], seed=seed % 1000)
        t = _tracer(sc, _ANY_SETTINGS, case["bvh"])
        r = np.random.RandomState(seed % (1 << 31))
        tr = sc.instance_transforms.astype(np.float64)
        dynamic = [i for i in range(sc.instances.shape[0]) if sc.instance_local[i, 0] & 1]
        shift = r.uniform(-0.5, 0.5, (len(dynamic), 3))
        moves = [{"instance": i, "translation": tuple(float(x) for x in tr[i, 0:3] + shift[j]),
                  "rotation": tuple(float(x) for x in tr[i, 3:7]), "scale": tuple(float(x) for x in tr[i, 7:10])}
                 for j, i in enumerate(dynamic)]
        return {"case": case, "tracer": t, "moves": moves,
                "query": _Query(t, _camera_rays(sc.camera, case["view"], case["view"]))}
    raise ValueError(k)


# ------------------------------------------------------------------- run
def run(state):
    case = state["case"]
    k = case["kind"]
    if k == "rays":
        if not case["host"]:
            return state["query"]()
        prim, t = state["tracer"].trace_rays(state["rays"], int(case["mode"] == "any"), state["tmax"])
        return {"prim": prim.view(np.int32), "t": t}
    if k == "frame":
        t = state["tracer"]
        if case["preview"]:
            t.update_camera_state(state["camera"])
            t.reset_accumulation()
            if not t.render_tile(RenderTile(0, 0, case["width"], case["height"], 0)):
                raise RuntimeError(t.status().last_error)
            return {"image": t.resolve_ldr(tone_map="aces")}
        t.reset_accumulation()
        t.render_frame(0, case["spp"], sync=False)
        return {"image": t.resolve_hdr()}
    if k == "batch":
        state["batch"].run("loop", **state["tuning"])
        state["batch"].read_films(state["sum_views"], state["count_views"])
        return {"sums": state["sums"], "counts": state["counts"]}
    if k == "inverse":
        loss = state["tracer"].forward(state["params"])
        return {"loss": loss, "gradient": state["tracer"].backward()}
    if k == "rebuild":
        status = state["tracer"].build_or_update_acceleration()
        if not status.ok:
            raise RuntimeError(status.message)
        return state["query"]()
    state["tracer"].update_instance_transforms(state["moves"])
    return state["query"]()


# ------------------------------------------------------------------- work
def _triangles(case):
    kind = case.get("mesh") or case.get("scene") or "field"
    if kind == "sphere":
        return 2 * (case["size"] - 1) * case["size"]
    if kind in ("field", "sky"):
        return 504 * case["size"] ** 2
    return 36


def _query_work(rays, triangles):
    """Each ray read and its hit written once, each triangle's corners read
    once; per ray one box of every level of a four-wide tree and one triangle."""
    levels = max(1.0, math.log(max(2, triangles), 4))
    return 32.0 * rays + 36.0 * triangles, rays * (levels * 4 * 12 + 50.0)


def work(case):
    k = case["kind"]
    if k == "rays":
        b, f = _query_work(case["n"], _triangles(case))
        return {"bytes": b, "flops": f}
    if k == "frame":
        # a path has at least its camera ray, one light sample and the shading of one hit
        paths = case["width"] * case["height"] * case["spp"]
        b, f = _query_work(2 * paths, _triangles(case))
        return {"bytes": b - 64.0 * paths + 12.0 * case["width"] * case["height"], "flops": f + 200.0 * paths}
    if k == "batch":
        # the jobs' mean: side and triangles spread over their logarithms, 24.8 samples on average
        side2 = (case["max_side"] ** 2 - 128 ** 2) / (2 * math.log(case["max_side"] / 128))
        tris = (case["max_triangles"] - 1000) / math.log(case["max_triangles"] / 1000)
        b, f = _query_work(2 * 24.8 * side2, tris)
        return {"bytes": case["jobs"] * (b - 32.0 * 2 * 24.8 * side2 + 16.0 * side2),
                "flops": case["jobs"] * (f + 200.0 * 24.8 * side2)}
    if k == "inverse":
        # forward and backward, each with the camera ray and one light sample of every path
        paths = case["side"] ** 2 * case["spp"]
        b, f = _query_work(2 * paths, 12 * case["objects"] + 12)
        return {"bytes": b - 64.0 * paths + 24.0 * case["side"] ** 2, "flops": f + 600.0 * paths}
    triangles = 504 * case["size"] ** 2
    b, f = _query_work(case["view"] ** 2, triangles)
    # every triangle's box and normal, and the tree's nodes written once: 64 bytes a triangle
    return {"bytes": b + 64.0 * triangles, "flops": f + 60.0 * triangles}


# ------------------------------------------------------------------- exact
def _brute_force(scene, rays):
    """Distance of the closest hit in 64 bits over all triangles: Moller-Trumbore,
    |det| >= 1e-4, t > 1e-4; infinity for a miss."""
    v = torch.tensor(np.asarray(scene.vertices), device="cuda").double()
    tri = torch.tensor(np.asarray(scene.indices, np.int64).reshape(-1, 3), device="cuda")
    a, b, c = v[tri[:, 0]], v[tri[:, 1]], v[tri[:, 2]]
    e1, e2 = b - a, c - a
    nrm = torch.linalg.cross(e1, e2)
    out = []
    step = max(1, int(1.5e8 // max(1, tri.shape[0])))
    for k in range(0, rays.shape[0], step):
        o, d = rays[k:k + step, :3].double(), rays[k:k + step, 3:].double()
        det = -(d @ nrm.T)
        inv = 1.0 / det
        # e1 x e2 . (o - a); (o - a) x d . e2 and e1 as differences of per-ray and per-triangle products
        t = (o @ nrm.T - (a * nrm).sum(1)) * inv
        m = torch.linalg.cross(o, d)
        u = (m @ e2.T - d @ torch.linalg.cross(e2, a).T) * inv
        w = -(m @ e1.T - d @ torch.linalg.cross(e1, a).T) * inv
        ok = (det.abs() >= 1e-4) & (u >= 0) & (w >= 0) & (u + w <= 1) & (t > 1e-4)
        out.append(torch.where(ok, t, torch.inf).min(dim=1).values)
    return torch.cat(out)


def exact(case, seed):
    """Closest-hit distances by brute force where that is quick.  A path
    tracer's image is a sum over random decisions (no 64-bit value belongs to
    the 32-bit tracer's random paths), so images and gradients have none."""
    if case["kind"] != "rays" or case["mode"] != "closest" or case["test"] != "mt":
        return None
    if case["n"] * _triangles(case) > 3e10:
        return None
    sc = _scene(case["mesh"], case["size"], seed % 1000)
    rays, _ = _query_rays(sc, case["n"], seed)
    return {"prim": None, "t": _brute_force(sc, rays)}
