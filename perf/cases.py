"""The measured cases: what a program that uses this package has it do, each through the public entry points.

Ray queries against displaced-icosphere fields (one pick, host batches, device batches of camera and surface rays,
closest and any hit), rebuilding a scene whose geometry changed, and the three integrators from an interactive
preview to a still image, on plain, textured, environment-lit and instanced scenes.
"""
import functools
import math

import numpy as np
import torch

import selas_gb300 as sel
from selas_gb300 import scenes


def listed():
    return [
        # a click in a viewport: one ray from host memory, where the call's latency is all that counts
        dict(name="pick_one", kind="query", spheres=64, level=4, rays=1, set="primary", query="closest", where="host"),
        # a plugin's batch in ordinary host memory (rtcIntersect1M's usual caller), an odd count
        dict(name="host_batch", kind="query", spheres=64, level=5, rays=100_003, set="surface", query="closest",
             where="host"),
        # a frame's camera rays, resident in HBM, over 5.2 M triangles
        dict(name="camera_closest", kind="query", spheres=64, level=6, rays=2048 * 2048, set="primary",
             query="closest", where="device"),
        # secondary rays: bounces off random surface points, the incoherent half of any light transport
        dict(name="surface_closest", kind="query", spheres=64, level=6, rays=2048 * 2048, set="surface",
             query="closest", where="device"),
        # ambient occlusion / shadow batches: any hit of the same kind of rays, an odd count
        dict(name="surface_any", kind="query", spheres=64, level=6, rays=3_000_017, set="surface", query="any",
             where="device"),
        # animated geometry: every frame a scene of new vertices is attached, committed and traced
        dict(name="rebuild", kind="rebuild", spheres=32, level=5, rays=65_537),
        # the path tracer's interactive preview: one sample a pixel of a small window
        dict(name="pt_preview", kind="pt", scene="cornell", width=160, height=120, spp=1, bounces=8),
        # the path tracer's headline configuration: Cornell box, 512 x 512, 64 samples, depth 8
        dict(name="pt_still", kind="pt", scene="cornell", width=512, height=512, spp=64, bounces=8),
        # a textured production-like room (per-face Ptex, glass, Disney surfaces), progressive pass of 4 samples
        dict(name="pt_room", kind="pt", scene="room", width=1280, height=720, spp=4, bounces=8),
        # the deferred path tracer (4 x 4 correlated multi-jittered samples, its default bounce cap) under a sky
        # image, smooth normals and tangents, odd size
        dict(name="deferred_sky", kind="deferred", scene="sky", width=641, height=359, axis=4, bounces=64),
        # two passes of vertex connection and merging on the room
        dict(name="vcm_room", kind="vcm", scene="room", width=640, height=360, passes=2, length=10, merging=True),
        # a turntable of an instanced terrain: several cameras in one shared wavefront
        dict(name="terrain_views", kind="views", grid=1024, instances=2000, views=4, width=480, height=270, spp=4,
             bounces=8),
    ]


def _span(rng, lo, hi):
    """An integer spread over the logarithm of [lo, hi]."""
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["query", "query", "query", "query", "rebuild", "pt", "pt", "deferred", "vcm", "views"])
    if kind == "query":
        where = rng.choice(["device", "device", "host"])
        return dict(kind=kind, spheres=rng.randint(8, 64), level=rng.randint(3, 6),
                    rays=_span(rng, 1, 2048 * 2048 if where == "device" else 300_000),
                    set=rng.choice(["primary", "surface"]), query=rng.choice(["closest", "any"]), where=where)
    if kind == "rebuild":
        return dict(kind=kind, spheres=rng.randint(4, 32), level=rng.randint(3, 5), rays=_span(rng, 1, 262_144))
    if kind == "pt":
        return dict(kind=kind, scene=rng.choice(["cornell", "room", "sky"]), width=_span(rng, 33, 1280),
                    height=_span(rng, 33, 720), spp=_span(rng, 1, 8), bounces=rng.randint(2, 12))
    if kind == "deferred":
        return dict(kind=kind, scene=rng.choice(["cornell", "room", "sky"]), width=_span(rng, 33, 640),
                    height=_span(rng, 33, 360), axis=rng.randint(1, 4), bounces=rng.randint(4, 64))
    if kind == "vcm":
        return dict(kind=kind, scene=rng.choice(["cornell", "room", "sky"]), width=_span(rng, 33, 640),
                    height=_span(rng, 33, 360), passes=rng.randint(1, 2), length=rng.randint(3, 10),
                    merging=rng.random() < 0.75)
    return dict(kind=kind, grid=_span(rng, 64, 1024), instances=_span(rng, 10, 2000), views=rng.randint(2, 6),
                width=_span(rng, 33, 480), height=_span(rng, 33, 270), spp=rng.randint(1, 4), bounces=8)


# ---------------------------------------------------------------------------------------------------
# Inputs
# ---------------------------------------------------------------------------------------------------
@functools.lru_cache(maxsize=1)
def _device():
    return sel.Device(0)


@functools.lru_cache(maxsize=4)
def _render_scene(name):
    """The assets a program has loaded; cameras and seeds differ from state to state."""
    if name == "cornell":
        return scenes.cornell_box()
    if name == "room":
        return scenes.vcm_room(icospheres=8, level=5, log2=3)
    scene = scenes.smooth_spheres(count=6, level=4)
    scene.ibl = scenes.sky_ibl()
    return scene


@functools.lru_cache(maxsize=2)
def _terrain(grid, instances):
    return scenes.instanced_terrain(grid=grid, instances=instances)


class _State:
    """What the program keeps between calls; its scenes are released with it."""

    def __init__(self, case, **kept):
        self.case = case
        self.owned = []
        self.__dict__.update(kept)

    def __del__(self):
        torch.cuda.synchronize()
        for release in self.owned:
            release()


def _camera_rays(geometry, n, gen):
    """n pixels of a pinhole camera at a seeded place around the field, in pixel order; one ray alone is a pick, at
    a point of some sphere."""
    w = max(1, int(math.sqrt(n)))
    i = torch.arange(n, device="cuda")
    yaw = float(torch.rand((), generator=gen, device="cuda")) * 2.0 * math.pi
    cam = scenes.camera_basis([170.0 * math.sin(yaw), 70.0, -170.0 * math.cos(yaw)], [0.0, 40.0, 0.0],
                              [0.0, 1.0, 0.0], 60.0, w, max(1, -(-n // w)))
    x = ((i % w).double() + 0.5) / w
    y = ((i // w).double() + 0.5) / max(1, -(-n // w))
    ax = {k: torch.tensor(cam[k], device="cuda", dtype=torch.float64) for k in ("X", "Y", "Z", "position")}
    d = ax["Z"] - (2.0 * x - 1.0)[:, None] * ax["X"] + (1.0 - 2.0 * y)[:, None] * ax["Y"]
    if n == 1:
        _, v, f = geometry.meshes[int(torch.randint(len(geometry.meshes) - 1, (), generator=gen, device="cuda"))]
        face = f[int(torch.randint(f.shape[0], (), generator=gen, device="cuda"))]
        d = torch.from_numpy(v[face].mean(axis=0, dtype=np.float64)[None]).cuda() - ax["position"]
    d = d / d.norm(dim=1, keepdim=True)
    return ax["position"].expand(n, 3).float(), d.float()


def _surface_rays(geometry, n, gen):
    """Cosine-distributed directions from random points of random triangles, 1e-3 off the surface."""
    soup = np.concatenate([v[f].reshape(-1, 9) for _, v, f in geometry.meshes])
    soup = torch.from_numpy(soup).cuda()
    tri = torch.randint(soup.shape[0], (n,), generator=gen, device="cuda")
    v = soup[tri].view(n, 3, 3).double()
    u = torch.rand((n, 4), generator=gen, device="cuda", dtype=torch.float64)
    r1 = u[:, 0:1].sqrt()
    p = (1 - r1) * v[:, 0] + r1 * (1 - u[:, 1:2]) * v[:, 1] + r1 * u[:, 1:2] * v[:, 2]
    nrm = torch.linalg.cross(v[:, 1] - v[:, 0], v[:, 2] - v[:, 0])
    nrm = nrm / nrm.norm(dim=1, keepdim=True).clamp_min(1e-30)
    zero = torch.zeros_like(nrm[:, 0])
    t = torch.where((nrm[:, 0].abs() > nrm[:, 1].abs())[:, None], torch.stack([-nrm[:, 2], zero, nrm[:, 0]], 1),
                    torch.stack([zero, nrm[:, 2], -nrm[:, 1]], 1))
    t = t / t.norm(dim=1, keepdim=True).clamp_min(1e-30)
    b = torch.linalg.cross(nrm, t)
    rr, phi = u[:, 2:3].sqrt(), 2.0 * math.pi * u[:, 3:4]
    d = rr * phi.cos() * t + (1 - u[:, 2:3]).clamp_min(0).sqrt() * nrm + rr * phi.sin() * b
    d = d / d.norm(dim=1, keepdim=True).clamp_min(1e-30)
    return (p + 1e-3 * nrm).float(), d.float()


def _records(org, dirs, closest):
    """RTCRayHit (24 words) or RTCRay (12 words) records in HBM, as words."""
    n = org.shape[0]
    r = torch.zeros((n, 24 if closest else 12), device="cuda")
    r[:, 0:3], r[:, 4:7], r[:, 8] = org, dirs, math.inf
    ints = r.view(torch.int32)
    ints[:, 9] = -1  # mask
    if closest:
        ints[:, 17:21] = -1  # ids
    return r


def _field(case, seed):
    return scenes.displaced_icospheres(count=case["spheres"], level=case["level"], seed=seed)


def _query_inputs(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    geometry = _field(case, seed)
    n = case["rays"]
    org, dirs = _surface_rays(geometry, n, gen) if case.get("set", "surface") == "surface" else _camera_rays(geometry, n, gen)
    return geometry, org, dirs


def _view(camera, seed):
    """The scene's camera moved a little, as a viewer's hand moves it."""
    rng = np.random.default_rng(seed)
    c = dict(camera)
    reach = 0.05 * np.linalg.norm(np.asarray(c["position"], np.float64) - np.asarray(c["look_at"], np.float64))
    c["position"] = tuple(float(p) + reach * float(rng.uniform(-1, 1)) for p in c["position"])
    return c


def _camera(camera, case):
    return sel.camera(camera["position"], camera["look_at"], camera["up"], camera["fov_degrees"], case["width"],
                      case["height"])


def prepare(case, seed):
    dev, kind = _device(), case["kind"]
    if kind in ("query", "rebuild"):
        geometry, org, dirs = _query_inputs(case, seed)
        rays = _records(org, dirs, case.get("query", "closest") == "closest")
        if kind == "rebuild":
            return _State(case, meshes=[(g, np.ascontiguousarray(v, np.float32), np.ascontiguousarray(f, np.uint32))
                                        for g, v, f in geometry.meshes], rays=rays)
        scene = sel.Scene(dev)
        geometry.attach_to(scene)
        scene.commit()
        if case["where"] == "host":
            dtype = sel.RAYHIT_DTYPE if case["query"] == "closest" else sel.RAY_DTYPE
            rays = rays.cpu().numpy().view(dtype).reshape(-1)
        state = _State(case, scene=scene, rays=rays)
        state.owned.append(scene.release)
        return state
    if kind == "views":
        world = _terrain(case["grid"], case["instances"])
        built = world.build(sel, dev)
        cams = [_camera(_view(c, seed + k), case) for k, c in enumerate(scenes.terrain_views(world, case["views"]))]
        state = _State(case, scene=built[0], cameras=cams,
                       settings=sel.pt_settings(case["spp"], case["bounces"], seed=seed))
        state.owned.append(lambda: world.release(built))
        return state
    asset = _render_scene(case["scene"])
    scene = asset.build(sel, dev)
    if kind == "pt":
        settings = sel.pt_settings(case["spp"], case["bounces"], seed=seed)
    elif kind == "deferred":
        settings = sel.deferred_settings(case["axis"], case["bounces"], seed=seed)
    else:
        settings = sel.vcm_settings(case["passes"], case["length"], seed=seed, merging=case["merging"])
    state = _State(case, scene=scene, camera=_camera(_view(asset.camera, seed), case), settings=settings)
    state.owned.append(scene.release)
    return state


# ---------------------------------------------------------------------------------------------------
# One pass
# ---------------------------------------------------------------------------------------------------
def _hits(rays):
    if isinstance(rays, np.ndarray):
        words = rays.view(np.float32).reshape(rays.shape[0], -1)
        ints = words.view(np.int32)
    else:
        words, ints = rays, rays.view(torch.int32)
    if words.shape[1] == 12:
        return {"tfar": words[:, 8]}
    return {"tfar": words[:, 8], "ng": words[:, 12:15], "uv": words[:, 15:17], "ids": ints[:, 17:21]}


def run(state):
    case, kind = state.case, state.case["kind"]
    if kind == "query":
        rays, n = state.rays, case["rays"]
        if case["where"] == "host":
            rays["tfar"] = math.inf  # the records are traced again from the start
            if case["query"] == "closest":
                state.scene.intersect1M(rays)
            else:
                state.scene.occluded1M(rays)
            return _hits(rays)
        rays[:, 8] = math.inf
        stream = torch.cuda.current_stream().cuda_stream
        if case["query"] == "closest":
            state.scene.intersect_device(rays.data_ptr(), n, stream)
        else:
            state.scene.occluded_device(rays.data_ptr(), n, stream)
        return _hits(rays)
    if kind == "rebuild":
        scene = sel.Scene(_device())
        for geom, vertices, faces in state.meshes:
            scene.attach_triangle_mesh(geom, vertices, faces)
        scene.commit()
        state.rays[:, 8] = math.inf
        stream = torch.cuda.current_stream().cuda_stream
        scene.intersect_device(state.rays.data_ptr(), case["rays"], stream)
        scene.device.sync(stream)  # the frame's hits are wanted before its scene goes
        scene.release()
        return _hits(state.rays)
    if kind == "pt":
        return state.scene.pt_generate_image(state.camera, state.settings)
    if kind == "deferred":
        return state.scene.deferred_generate_image(state.camera, state.settings)
    if kind == "vcm":
        return state.scene.vcm_generate_image(state.camera, state.settings)
    return state.scene.render_views(state.cameras, state.settings)


# ---------------------------------------------------------------------------------------------------
# What a pass cannot do without
# ---------------------------------------------------------------------------------------------------
def _ray_flops(triangles):
    """A walk straight to the hit: one node of 8 boxes (6 multiply-adds each) a level, then one triangle."""
    return max(1, math.ceil(math.log(max(triangles, 8), 8))) * 8 * 12 + 60


def work(case):
    kind = case["kind"]
    if kind in ("query", "rebuild"):
        tris = case["spheres"] * 20 * 4 ** case["level"] + 2
        closest = case.get("query", "closest") == "closest"
        # per ray 32 bytes in; out the 24 (closest) or 4 (any) bytes of the hit; a rebuild also reads its triangles'
        # indices and vertices (12 bytes an index triple, 12 a vertex, half as many vertices)
        moved = case["rays"] * (56 if closest else 36) + (tris * 18 if kind == "rebuild" else 0)
        return {"bytes": moved, "flops": case["rays"] * _ray_flops(tris) + (tris * 60 if kind == "rebuild" else 0)}
    pixels = case["width"] * case["height"] * case.get("views", 1)
    if kind == "views":
        tris = 2 * case["grid"] ** 2 + case["instances"] * 20480
    else:
        tris = {"cornell": 34, "room": 215_000, "sky": 30_722}[case["scene"]]
    samples = {"pt": case.get("spp", 1), "views": case.get("spp", 1), "deferred": case.get("axis", 1) ** 2,
               "vcm": 2 * case.get("passes", 1)}[kind]
    bounces = min(case.get("bounces", case.get("length", 8)), 4)
    # per path about four segments, each with a shadow ray and a few hundred operations of surface and BSDF; the
    # image is written once
    per_path = bounces * (2 * _ray_flops(tris) + 400)
    return {"bytes": pixels * (24 if kind in ("pt", "views") else 12), "flops": pixels * samples * per_path}


def exact(case, seed):
    """Closest hits by brute force in 64 bits (t, u, v and the unnormalised normal), where that takes seconds; the
    integrators' random walks and any-hit bits have no 64-bit value."""
    if case["kind"] not in ("query", "rebuild") or case.get("query", "closest") != "closest":
        return None
    tris = case["spheres"] * 20 * 4 ** case["level"] + 2
    n = case["rays"]
    if n * tris > 4_000_000_000:
        return None
    geometry, org, dirs = _query_inputs(case, seed)
    soup = np.concatenate([v[f].reshape(-1, 9) for _, v, f in geometry.meshes])
    v = torch.from_numpy(soup).cuda().double().view(-1, 3, 3)
    e1, e2 = v[:, 1] - v[:, 0], v[:, 2] - v[:, 0]
    ng = torch.linalg.cross(e1, e2)
    t_all = torch.full((n,), math.inf, device="cuda", dtype=torch.float64)
    uv_all = torch.zeros((n, 2), device="cuda", dtype=torch.float64)
    ng_all = torch.zeros((n, 3), device="cuda", dtype=torch.float64)
    step = max(1, 40_000_000 // tris)
    for a in range(0, n, step):
        o, d = org[a:a + step].double()[:, None], dirs[a:a + step].double()[:, None]
        p = torch.linalg.cross(d.expand(-1, tris, 3), e2.expand(d.shape[0], -1, 3))
        det = (p * e1).sum(-1)
        s = o - v[:, 0]
        u = (s * p).sum(-1) / det
        q = torch.linalg.cross(s, e1.expand(d.shape[0], -1, 3))
        w = (q * d).sum(-1) / det
        t = (q * e2).sum(-1) / det
        t = torch.where((u >= 0) & (w >= 0) & (u + w <= 1) & (t >= 0), t, torch.full_like(t, math.inf))
        best, k = t.min(dim=1)
        hit = torch.isfinite(best)
        rows = torch.arange(best.shape[0], device="cuda")
        t_all[a:a + step] = best
        uv_all[a:a + step] = torch.where(hit[:, None], torch.stack([u[rows, k], w[rows, k]], 1), uv_all[a:a + step])
        ng_all[a:a + step] = torch.where(hit[:, None], ng[k], ng_all[a:a + step])
    return {"tfar": t_all, "ng": ng_all, "uv": uv_all, "ids": None}
