"""Workloads of the renderer, one pass each through its public entry points.

A case is a dict of plain values.  ``listed()`` gives the fixed ones,
``draw(rng)`` one more of the same ranges, ``prepare(case, seed)`` what a
user's program holds before the call (scene handles, rays on the device or in
host memory, output buffers), ``run(state)`` one pass and its outputs,
``work(case)`` the bytes and operations the pass cannot do without, and
``exact(case, seed)`` the outputs in 64 bits where that takes seconds.

Kinds of case:
  query   closest-hit or any-hit rays against one aggregate
  render  one frame of the direct-lighting renderer
  batch   renders and ray queries over many scenes in one launch
  served  a burst of requests against resident scenes
  rebuild an aggregate built on the device from new geometry, then queried
"""
from __future__ import annotations

import math
import random
from concurrent.futures import ThreadPoolExecutor

import numpy as np
import torch

from pbrt_rust_gb300 import generators as G
from pbrt_rust_gb300.batch import GpuBatch
from pbrt_rust_gb300.gpu import GpuBVHAccel, GpuSamplerRenderer, GpuScene
from pbrt_rust_gb300.scene import (Camera, DiffuseAreaLight, Film, Filter, MatteMaterial, PointLight, Primitive,
                                   Shape, StratifiedSampler)
from pbrt_rust_gb300.server import GpuServer
from pbrt_rust_gb300.transform import Transform


def listed() -> list[dict]:
    return [
        # a picking or collision probe: a handful of rays, all latency
        dict(name="query_few", kind="query", scene="soup", tris=4096, rays=257, any=False, buffers="device"),
        # the plain query workload: 4096 random triangles, 2^20 rays toward the centre
        dict(name="query_soup", kind="query", scene="soup", tris=4096, rays=1 << 20, any=False, buffers="device"),
        # incoherent rays against a terrain of a million triangles, rays and hits resident
        dict(name="query_mesh", kind="query", scene="mesh", tris=999698, rays=1 << 22, any=False, buffers="device"),
        # visibility over segments of such rays, a ragged count
        dict(name="query_mesh_any", kind="query", scene="mesh", tris=999698, rays=1500001, any=True,
             buffers="device"),
        # a host program that hands over pinned rays and reads pinned hits
        dict(name="query_mesh_host", kind="query", scene="mesh", tris=999698, rays=1 << 21, any=False,
             buffers="pinned"),
        # the smallest frame of the serving workload: a preview of a triangle soup
        dict(name="render_preview", kind="render", scene="soup", tris=20000, spheres=8, width=128, height=128,
             spp_side=1, lens=0.0, filter="box"),
        # the plain render: 64 matte spheres on a ground quad, point + area light, 512 squared, 4 spp
        dict(name="render_spheres", kind="render", scene="spheres", tris=0, spheres=64, width=512, height=512,
             spp_side=2, lens=0.0, filter="box"),
        # the large frame: terrain of a million triangles, 1024 squared, 16 spp
        dict(name="render_mesh", kind="render", scene="mesh", tris=999698, spheres=0, width=1024, height=1024,
             spp_side=4, lens=0.0, filter="box"),
        # instances, analytic shapes, depth of field and a wide filter at a ragged size
        dict(name="render_forest", kind="render", scene="forest", tris=2000, spheres=64, width=517, height=389,
             spp_side=2, lens=0.08, filter="gaussian"),
        # many scenes of uneven size, resolution and sample count in one launch
        dict(name="batch_scenes", kind="batch", scenes=24, mix=3, tri_lo=1000, tri_hi=256000, queries=4),
        # a burst of renders and ray batches against resident scenes
        dict(name="served_burst", kind="served", scenes=6, mix=9, tri_lo=10000, tri_hi=300000, requests=30, slots=2),
        # moving geometry: the tree is built anew on the device and queried
        dict(name="rebuild_mesh", kind="rebuild", scene="mesh", tris=180000, rays=100003),
    ]


def draw(rng: random.Random) -> dict:
    def log_int(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["query", "query", "query", "render", "render", "batch", "served", "rebuild"])
    if kind == "query":
        scene = rng.choice(["soup", "mesh", "forest"])
        tris = {"soup": log_int(1000, 300000), "mesh": log_int(5000, 1000000), "forest": log_int(200, 4000)}[scene]
        any_hit = rng.random() < 0.4
        rays = log_int(1000 if any_hit else 64, {"soup": 1 << 19, "mesh": 1 << 22, "forest": 1 << 20}[scene])
        return dict(kind=kind, scene=scene, tris=tris, rays=rays, any=any_hit,
                    buffers=rng.choice(["device", "device", "pinned", "pageable"]))
    if kind == "render":
        scene = rng.choice(["soup", "spheres", "mesh", "forest"])
        tris = {"soup": log_int(1000, 200000), "spheres": 0, "mesh": log_int(5000, 1000000),
                "forest": log_int(200, 4000)}[scene]
        spheres = {"soup": rng.randint(0, 32), "spheres": rng.randint(1, 64), "mesh": 0,
                   "forest": rng.randint(4, 128)}[scene]
        w = log_int(64, 700)
        h = max(64, min(700, int(w * rng.uniform(0.6, 1.4))))
        return dict(kind=kind, scene=scene, tris=tris, spheres=spheres, width=w, height=h,
                    spp_side=rng.choice([1, 2, 3, 4]), lens=rng.choice([0.0, 0.0, rng.uniform(0.02, 0.1)]),
                    filter=rng.choice(["box", "box", "gaussian", "mitchell"]))
    if kind == "batch":
        return dict(kind=kind, scenes=rng.randint(3, 24), mix=rng.randrange(1 << 20), tri_lo=1000,
                    tri_hi=log_int(4000, 200000), queries=rng.randint(0, 6))
    if kind == "served":
        return dict(kind=kind, scenes=rng.randint(2, 6), mix=rng.randrange(1 << 20), tri_lo=10000,
                    tri_hi=log_int(20000, 300000), requests=rng.randint(8, 30), slots=rng.randint(1, 3))
    return dict(kind=kind, scene="mesh", tris=log_int(2000, 180000), rays=log_int(1000, 100003))


# ---------------------------------------------------------------- scenes ---
def _mesh_side(tris: int) -> int:
    return max(3, int(round(math.sqrt(tris / 2.0))) + 1)


def _soup(rng: G.PCG32, tris: int, spheres: int, extent: float = 1.0):
    """A random-triangle soup and matte spheres, as in the multi-scene
    workload, with its two lights.  Returns (prims, lights)."""
    pts, idx = G.random_triangle_soup(rng, tris, extent=extent, offset=0.05 * extent)
    prims = [Primitive.geometric(Shape.triangle_mesh(Transform(), None, False, idx, pts),
                                 MatteMaterial(tuple(0.2 + 0.6 * rng.uniform(3))))]
    for u in rng.uniform(7 * spheres).reshape(spheres, 7):
        r = extent * (0.05 + 0.15 * u[0])
        o2w = Transform.translate(tuple(extent * (2.0 * u[1:4] - 1.0)))
        prims.append(Primitive.geometric(Shape.sphere(o2w, o2w.inverse(), False, r, -r, r, 360.0),
                                         MatteMaterial(tuple(0.2 + 0.6 * u[4:7]))))
    area = DiffuseAreaLight(Transform(), (10.0, 10.0, 10.0))
    lights = [PointLight(Transform.translate((0.0, 2.0 * extent, -extent)), (50.0 * extent * extent,) * 3), area]
    prims.append(Primitive.geometric_area_light(G.quad_light_mesh((0.0, 1.5 * extent, 0.0), extent),
                                                MatteMaterial((0, 0, 0)), area))
    return prims, lights


def _soup_eye(extent: float = 1.0) -> Transform:
    return Transform.look_at((0.0, 0.5 * extent, -3.5 * extent), (0.0, 0.0, 0.0), (0.0, 1.0, 0.0)).inverse()


def _geometry(case: dict, seed: int):
    """(prims, lights, camera-to-world, fov, eye-to-target distance)."""
    if case["scene"] == "soup":
        prims, lights = _soup(G.PCG32(seed), case["tris"], case.get("spheres", 0))
        return prims, lights, _soup_eye(), 60.0, 3.5
    if case["scene"] == "spheres":
        prims, lights, cam, _ = G.c1_scene(seed=seed, res=16, n_spheres=case["spheres"])
    elif case["scene"] == "mesh":
        prims, lights, cam, _, _ = G.heightfield(_mesh_side(case["tris"]), seed=seed, res=16, n_rays=0)
    else:
        prims, lights, cam, _, _ = G.instanced_forest(case.get("spheres", 64), case["tris"], seed=seed, res=16)
    return prims, lights, cam.camera_to_world, cam.fov, {"spheres": 6.2, "mesh": 15.6, "forest": 15.1}[case["scene"]]


_FILTERS = {"box": lambda: Filter.mean(0.5, 0.5), "gaussian": lambda: Filter.gaussian(2.0, 2.0, 2.0),
            "mitchell": lambda: Filter.mitchell(2.0, 2.0, 1.0 / 3.0, 1.0 / 3.0)}


def _renderer(c2w, fov: float, width: int, height: int, spp_side: int, lens: float = 0.0, focus: float = 1e30,
              filt: str = "box") -> GpuSamplerRenderer:
    film = Film.image(width, height, _FILTERS[filt]())
    cam = Camera.perspective(c2w, (-1.0, 1.0, -1.0, 1.0), 0.0, 1.0, lens, focus, fov, film)
    return GpuSamplerRenderer(StratifiedSampler.stratified(0, width, 0, height, spp_side, spp_side, True, 0.0, 1.0),
                              cam)


# ------------------------------------------------------------------ rays ---
def _unit(g: torch.Generator, n: int) -> torch.Tensor:
    v = torch.randn((n, 3), generator=g, device=g.device, dtype=torch.float32)
    return v / v.norm(dim=1, keepdim=True).clamp_min(1e-20)


def _rays(case: dict, seed: int, lo, hi) -> torch.Tensor:
    """(n, 8) float32 on the device: from a sphere around a soup toward its
    middle, or from anywhere in and about a scene's bounds in any direction;
    visibility rays end somewhere along the way, the others nowhere."""
    n = case["rays"]
    g = torch.Generator(device="cuda").manual_seed(seed)
    r = torch.empty((n, 8), device="cuda")
    r[:, 3] = 1e-4
    r[:, 7] = math.inf
    if case["scene"] == "soup":
        r[:, 0:3] = 3.0 * _unit(g, n)
        d = torch.rand((n, 3), generator=g, device="cuda") - 0.5 - r[:, 0:3]
        r[:, 4:7] = d / d.norm(dim=1, keepdim=True)
    else:
        lo = torch.tensor(np.asarray(lo) - 1.0, device="cuda", dtype=torch.float32)
        hi = torch.tensor(np.asarray(hi) + 1.0, device="cuda", dtype=torch.float32)
        r[:, 0:3] = lo + (hi - lo) * torch.rand((n, 3), generator=g, device="cuda")
        r[:, 4:7] = _unit(g, n)
    if case.get("any"):
        near, far = (1.0, 4.0) if case["scene"] == "soup" else (0.0, 16.0)
        r[:, 7] = near + (far - near) * torch.rand(n, generator=g, device="cuda")
    return r


# --------------------------------------------------------------- prepare ---
def prepare(case: dict, seed: int) -> dict:
    state = {"case": case, **globals()["_prepare_" + case["kind"]](case, seed)}
    torch.cuda.synchronize()
    return state


def _prepare_query(case, seed):
    bvh = GpuBVHAccel(_geometry(case, seed)[0], build_on_device=True)
    rays = _rays(case, seed, *bvh.world_bound())
    out = torch.empty(case["rays"] if case["any"] else (case["rays"], 4), device="cuda",
                      dtype=torch.uint8 if case["any"] else torch.float32)
    if case["buffers"] != "device":
        rays, out = rays.cpu(), out.cpu()
        if case["buffers"] == "pinned":
            rays, out = rays.pin_memory(), out.pin_memory()
    return dict(bvh=bvh, rays=rays, out=out)


def _prepare_render(case, seed):
    prims, lights, c2w, fov, dist = _geometry(case, seed)
    rend = _renderer(c2w, fov, case["width"], case["height"], case["spp_side"], case["lens"],
                     dist if case["lens"] else 1e30, case["filter"])
    return dict(scene=GpuScene(prims, lights, build_on_device=True), renderer=rend,
                out=torch.empty((case["height"], case["width"], 3), device="cuda"))


def _mix(case: dict) -> list[dict]:
    """The scenes of a batch or server: sizes from the case, not the seed."""
    rng = random.Random(case["mix"])
    lo, hi = math.log(case["tri_lo"]), math.log(case["tri_hi"])
    return [dict(tris=int(round(math.exp(rng.uniform(lo, hi)))), spheres=rng.randint(0, 32),
                 extent=rng.uniform(1.0, 4.0), res=rng.choice([128, 256, 512]), spp_side=rng.choice([1, 2, 4]))
            for _ in range(case["scenes"])]


def _requests(case: dict) -> list[dict]:
    """The request mix of the serving workload, as in the repository's
    generator, by the case's own mix number."""
    return G.serving_requests(case["requests"], case["scenes"], seed=case["mix"])


def _scenes(specs: list[dict], seed: int) -> list[GpuScene]:
    def one(k):
        prims, lights = _soup(G.PCG32(seed * 4096 + k), specs[k]["tris"], specs[k]["spheres"], specs[k]["extent"])
        return GpuScene(prims, lights, build_on_device=True)

    with ThreadPoolExecutor(8) as ex:  # the host side of a scene's creation releases the interpreter
        return list(ex.map(one, range(len(specs))))


_BATCH_RAYS = 60001


def _prepare_batch(case, seed):
    specs = _mix(case)
    scenes = _scenes(specs, seed)
    rend = [_renderer(_soup_eye(s["extent"]), 60.0, s["res"], s["res"], s["spp_side"]) for s in specs]
    px = sum(s["res"] ** 2 for s in specs)
    samples = sum(s["res"] ** 2 * s["spp_side"] ** 2 for s in specs)
    batch = GpuBatch(max_jobs=case["scenes"] + case["queries"], max_tasks=64 * case["scenes"], max_samples=samples,
                     max_light_samples=2 * samples, max_film_pixels=px)
    queries = []
    for q in range(case["queries"]):
        bvh = scenes[q % len(scenes)].aggregate()
        rays = _rays(dict(rays=_BATCH_RAYS, scene="any"), seed + 1 + q, *bvh.world_bound())
        out = (torch.empty(_BATCH_RAYS, device="cuda", dtype=torch.uint8) if q % 2
               else torch.empty((_BATCH_RAYS, 4), device="cuda"))
        queries.append((bvh, rays, bool(q % 2), out))
    return dict(batch=batch, scenes=scenes, renderers=rend, queries=queries,
                outs=[torch.empty((s["res"], s["res"], 3), device="cuda") for s in specs])


def _prepare_served(case, seed):
    specs = _mix(case)
    scenes = _scenes([dict(s, extent=1.0) for s in specs], seed)
    bvhs = [s.aggregate() for s in scenes]
    bounds = [b.world_bound() for b in bvhs]
    srv = GpuServer(slots=case["slots"], max_jobs=64, max_samples=1 << 22, max_film_pixels=1 << 20,
                    max_query_rays=1 << 18, max_tasks=1 << 12)
    cam = Camera.perspective(_soup_eye(), (-1.0, 1.0, -1.0, 1.0), 0.0, 1.0, 0.0, 1e30, 60.0,
                             Film.image(16, 16, Filter.mean(0.5, 0.5)))
    reqs = []
    for k, q in enumerate(_requests(case)):
        s = q["scene"]
        if q["kind"] == "render":
            c2w = G.orbit_camera(cam, q["radius"], q["azimuth"]).camera_to_world
            reqs.append((scenes[s], _renderer(c2w, 60.0, q["res"], q["res"], 1 if q["spp"] == 1 else 2),
                         torch.empty((q["res"], q["res"], 3), device="cuda")))
        else:
            rays = _rays(dict(rays=q["n"], scene="any"), seed + 1 + k, *bounds[s])
            reqs.append((bvhs[s], rays, torch.empty((q["n"], 4), device="cuda")))
    return dict(server=srv, scenes=scenes, requests=reqs)


def _prepare_rebuild(case, seed):
    pts, _, _ = G.heightfield_points(_mesh_side(case["tris"]), 8.0, seed)
    return dict(prims=_geometry(case, seed)[0], rays=_rays(case, seed, pts.min(axis=0), pts.max(axis=0)),
                out=torch.empty((case["rays"], 4), device="cuda"))


# ------------------------------------------------------------------- run ---
def _hits(h: torch.Tensor) -> dict:
    """A hit record by its parts: primitive (int32) and t, b1, b2."""
    return {"prim": h.view(torch.int32)[:, 0], "t_b1_b2": h[:, 1:]}


def run(state: dict):
    kind = state["case"]["kind"]
    if kind == "query":
        if state["case"]["any"]:
            return state["bvh"].intersect_p(state["rays"], out=state["out"])
        return _hits(state["bvh"].intersect(state["rays"], out=state["out"]))
    if kind == "render":
        return state["renderer"].render(state["scene"], out=state["out"])
    if kind == "batch":
        b = state["batch"]
        for scene, rend, out in zip(state["scenes"], state["renderers"], state["outs"]):
            b.add_render(scene, rend, out=out)
        for bvh, rays, any_hit, out in state["queries"]:
            b.add_query(bvh, rays, any_hit, out=out)
        outs = b.run()
        return outs[:len(state["scenes"])] + [o if q[2] else _hits(o)
                                              for q, o in zip(state["queries"], outs[len(state["scenes"]):])]
    if kind == "served":
        srv = state["server"]
        tickets = [(srv.submit_render if isinstance(a, GpuScene) else srv.submit_query)(a, b, out=out)
                   for a, b, out in state["requests"]]
        outs = [srv.wait(t) for t in tickets]
        return [o if isinstance(r[0], GpuScene) else _hits(o) for r, o in zip(state["requests"], outs)]
    bvh = GpuBVHAccel(state["prims"], build_on_device=True)
    return _hits(bvh.intersect(state["rays"], out=state["out"]))


# ------------------------------------------------------------------ work ---
# Nodes and primitives a ray has to test in the reference's tree, by scene
# (counted on the plain workloads: soup of 4096 triangles, terrain of a
# million; trees of other sizes grow with the logarithm of their size).
_TESTS = {"soup": (10.0, 3.0), "mesh": (1.7, 1.3), "forest": (4.0, 3.0), "spheres": (2.5, 1.5)}
_NODE_FLOPS, _PRIM_FLOPS, _SHADE_FLOPS = 25, 60, 400


def _tree_bytes(prims: int) -> int:
    return 32 * prims + 48 * prims  # a box per leaf and a record per primitive, each read once


def _ray_flops(scene: str, prims: int) -> float:
    nodes, tests = _TESTS[scene]
    return nodes * math.log2(max(prims, 2)) * _NODE_FLOPS + tests * _PRIM_FLOPS


def _query_work(scene: str, prims: int, rays: int, any_hit: bool) -> tuple[int, float]:
    # a call of few rays does not read the whole tree
    tree = min(_tree_bytes(prims), int(rays * 80 * _TESTS[scene][1] * math.log2(max(prims, 2))))
    return rays * (32 + (1 if any_hit else 16)) + tree, rays * _ray_flops(scene, prims)


def _render_work(scene: str, prims: int, pixels: int, spp: int, lights: int) -> tuple[int, float]:
    # camera rays, samples and radiances can stay on the chip: the image is
    # written once and the tree and the shading records are read once
    samples = pixels * spp
    tree = min(_tree_bytes(prims) + 48 * prims, int(samples * 128 * _TESTS[scene][1] * math.log2(max(prims, 2))))
    return 12 * pixels + tree, samples * ((1 + lights) * _ray_flops(scene, prims) + _SHADE_FLOPS)


def _prims(case: dict) -> int:
    return max(4, case["tris"] + case.get("spheres", 0)) if case["scene"] != "forest" else 2 * case["tris"] + 64


def work(case: dict) -> dict:
    kind = case["kind"]
    if kind == "query":
        b, f = _query_work(case["scene"], _prims(case), case["rays"], case["any"])
    elif kind == "render":
        b, f = _render_work(case["scene"], _prims(case), case["width"] * case["height"], case["spp_side"] ** 2,
                            1 if case["scene"] == "mesh" else 2)
    elif kind == "rebuild":
        n = 2 * (_mesh_side(case["tris"]) - 1) ** 2
        b, f = _query_work("mesh", n, case["rays"], False)
        b += 36 * n + 80 * n  # the vertices in, the tree out
        f += n * math.log2(max(n, 2)) * 12
    else:
        b, f = 0, 0.0
        specs = _mix(case)
        if kind == "batch":
            jobs = [(s["tris"], s["res"] ** 2, s["spp_side"] ** 2, 0, False) for s in specs]
            jobs += [(specs[q % len(specs)]["tris"], 0, 0, _BATCH_RAYS, bool(q % 2)) for q in range(case["queries"])]
        else:
            jobs = [(specs[q["scene"]]["tris"], q["res"] ** 2, q["spp"], 0, False) if q["kind"] == "render"
                    else (specs[q["scene"]]["tris"], 0, 0, q["n"], False) for q in _requests(case)]
        for tris, px, spp, rays, any_hit in jobs:
            jb, jf = _render_work("soup", tris, px, spp, 2) if px else _query_work("soup", tris, rays, any_hit)
            b += jb
            f += jf
    return {"bytes": int(b), "flops": float(f)}


# ----------------------------------------------------------------- exact ---
# The same results from plain torch and numpy in 64 bits: every primitive
# tested against every ray, no tree, no float32 and nothing of the package
# but the scene's own numbers.
_PAIRS = 5_000_000_000  # ray-primitive tests that take a few seconds


def exact(case: dict, seed: int):
    if case["kind"] == "query" and case["scene"] == "soup" and not case["any"]:
        if case["rays"] * case["tris"] > _PAIRS:
            return None
        geo = _Geometry64(_geometry(case, seed)[0])
        r = _rays(case, seed, None, None).double()
        h = geo.closest(r[:, 0:3], r[:, 4:7], r[:, 3], r[:, 7])
        out = torch.stack([h["t"], h["b1"], h["b2"]], dim=1)
        return {"prim": None, "t_b1_b2": out.cpu() if case["buffers"] != "device" else out}
    if case["kind"] == "render" and case["scene"] in ("soup", "spheres") and not case["lens"] and \
            case["filter"] == "box":
        samples = case["width"] * case["height"] * case["spp_side"] ** 2
        if 3 * samples * (case["tris"] + case["spheres"] + 4) > _PAIRS:
            return None
        return _render64(case, seed)
    return None


class _Geometry64:
    """Triangles and full spheres of a list of primitives, in the refined
    order (a mesh's triangles run over reversed index triples)."""

    def __init__(self, prims):
        tri, tid, sph, sid, kd, light = [], [], [], [], [], []
        n = 0
        for p in prims:
            s = p.shape
            if hasattr(s, "points") and s.points is not None and len(s.points):
                pts = np.asarray(s.points, np.float32).reshape(-1, 3).astype(np.float64)
                v = pts[np.asarray(s.indices).reshape(-1, 3)[:, ::-1].astype(np.int64)]
                tri.append(v)
                m = len(v)
                tid.append(np.arange(n, n + m))
            else:
                o = np.asarray(s.object_to_world.m, np.float32).reshape(4, 4).astype(np.float64)
                sph.append(np.concatenate([o[:3, 3], [float(np.float32(s.radius))]]))
                m = 1
                sid.append(n)
            c = p.material.kd if p.material is not None else (0.0, 0.0, 0.0)
            kd += [tuple(float(np.float32(x)) for x in c)] * m
            light += [p.area_light is not None] * m
            n += m
        dev = dict(device="cuda", dtype=torch.float64)
        self.tri = torch.tensor(np.concatenate(tri), **dev)
        self.tid = torch.tensor(np.concatenate(tid), device="cuda")
        self.sph = torch.tensor(np.array(sph).reshape(-1, 4), **dev)
        self.sid = torch.tensor(np.array(sid, np.int64), device="cuda")
        self.kd = torch.tensor(np.array(kd), **dev)
        self.light = torch.tensor(np.array(light), device="cuda")
        nt = torch.linalg.cross(self.tri[:, 1] - self.tri[:, 0], self.tri[:, 2] - self.tri[:, 0])
        self.tri_n = nt / nt.norm(dim=1, keepdim=True)

    def closest(self, o, d, tmin, tmax):
        n = o.shape[0]
        res = {"t": torch.zeros(n, device="cuda", dtype=torch.float64), "b1": torch.zeros_like(o[:, 0]),
               "b2": torch.zeros_like(o[:, 0]), "prim": torch.full((n,), -1, device="cuda", dtype=torch.int64),
               "tri": torch.full((n,), -1, device="cuda", dtype=torch.int64),
               "sph": torch.full((n,), -1, device="cuda", dtype=torch.int64)}
        step = max(1, (1 << 24) // (self.tri.shape[0] + self.sph.shape[0]))
        inf = math.inf
        a, e1, e2 = self.tri[:, 0], self.tri[:, 1] - self.tri[:, 0], self.tri[:, 2] - self.tri[:, 0]
        for lo in range(0, n, step):
            s = slice(lo, min(n, lo + step))
            oo, dd, t0, t1 = o[s], d[s], tmin[s, None], tmax[s, None]
            # Moeller-Trumbore by components: (rays, triangles) arrays
            dx, dy, dz = (dd[:, k:k + 1] for k in range(3))
            s1x, s1y, s1z = dy * e2[:, 2] - dz * e2[:, 1], dz * e2[:, 0] - dx * e2[:, 2], dx * e2[:, 1] - dy * e2[:, 0]
            inv = 1.0 / (s1x * e1[:, 0] + s1y * e1[:, 1] + s1z * e1[:, 2])
            sx, sy, sz = oo[:, 0:1] - a[:, 0], oo[:, 1:2] - a[:, 1], oo[:, 2:3] - a[:, 2]
            b1 = (s1x * sx + s1y * sy + s1z * sz) * inv
            s2x, s2y, s2z = sy * e1[:, 2] - sz * e1[:, 1], sz * e1[:, 0] - sx * e1[:, 2], sx * e1[:, 1] - sy * e1[:, 0]
            b2 = (dx * s2x + dy * s2y + dz * s2z) * inv
            t = (e2[:, 0] * s2x + e2[:, 1] * s2y + e2[:, 2] * s2z) * inv
            ok = (b1 >= 0) & (b2 >= 0) & (b1 + b2 <= 1) & (t >= t0) & (t <= t1)
            t, k = torch.where(ok, t, inf).min(dim=1)
            hit = t < inf
            row = torch.arange(len(k), device="cuda")
            res["t"][s] = torch.where(hit, t, 0.0)
            res["b1"][s] = torch.where(hit, b1[row, k], 0.0)
            res["b2"][s] = torch.where(hit, b2[row, k], 0.0)
            res["tri"][s] = torch.where(hit, k, -1)
            res["prim"][s] = torch.where(hit, self.tid[k], -1)
            if self.sph.shape[0]:
                oc = oo[:, None, :] - self.sph[None, :, :3]
                A = (dd * dd).sum(1, keepdim=True)
                B = 2.0 * (oc * dd[:, None, :]).sum(2)
                D = B * B - 4.0 * A * ((oc * oc).sum(2) - self.sph[:, 3] ** 2)
                q = torch.sqrt(D.clamp_min(0.0))
                u0, u1 = (-B - q) / (2.0 * A), (-B + q) / (2.0 * A)
                ts = torch.where(u0 >= t0, u0, u1)
                ts = torch.where((D >= 0) & (ts >= t0) & (ts <= t1), ts, inf)
                ts, k = ts.min(dim=1)
                near = ts < torch.where(hit, t, inf)
                res["t"][s] = torch.where(near, ts, res["t"][s])
                for key in ("b1", "b2"):
                    res[key][s] = torch.where(near, 0.0, res[key][s])
                res["tri"][s] = torch.where(near, -1, res["tri"][s])
                res["sph"][s] = torch.where(near, k, -1)
                res["prim"][s] = torch.where(near, self.sid[k], res["prim"][s])
        return res


def _keystream(task: int, words: int) -> np.ndarray:
    """The first `words` words of the ChaCha12 stream keyed by the task."""
    key, state, mask = [], task, (1 << 64) - 1
    for _ in range(8):  # the PCG32 seed expansion
        state = (state * 6364136223846793005 + 11634580027462260723) & mask
        x, rot = (((state >> 18) ^ state) >> 27) & 0xFFFFFFFF, state >> 59
        key.append(((x >> rot) | (x << ((32 - rot) & 31))) & 0xFFFFFFFF)
    blocks = (words + 15) // 16
    ctr = np.arange(blocks, dtype=np.uint64)
    init = [np.full(blocks, v, np.uint32) for v in (0x61707865, 0x3320646E, 0x79622D32, 0x6B206574, *key)]
    init += [ctr.astype(np.uint32), (ctr >> np.uint64(32)).astype(np.uint32), np.zeros(blocks, np.uint32),
             np.zeros(blocks, np.uint32)]
    x = [v.copy() for v in init]

    def quarter(a, b, c, d):
        for p, q, r, s in ((a, b, d, 16), (c, d, b, 12), (a, b, d, 8), (c, d, b, 7)):
            x[p] += x[q]
            x[r] ^= x[p]
            x[r] = (x[r] << np.uint32(s)) | (x[r] >> np.uint32(32 - s))

    for _ in range(6):
        for k in range(4):
            quarter(k, 4 + k, 8 + k, 12 + k)
        for k in range(4):
            quarter(k, 4 + (k + 1) % 4, 8 + (k + 2) % 4, 12 + (k + 3) % 4)
    return np.stack([v + i for v, i in zip(x, init)], axis=1).reshape(-1)[:words]


def _crop(num: int, count: int, aspect: float) -> list[float]:
    def split(asp):
        x, y = 1, count
        while y % 2 == 0 and 2 * asp * x < y:
            x, y = 2 * x, y // 2
        return x, y
    nx, ny = split(int(1.0 / aspect)) if aspect < 1.0 else split(int(aspect))[::-1]
    f = np.float32
    xo, yo = num % nx, num // nx
    return [f(xo) / f(nx), f(xo + 1) / f(nx), f(yo) / f(ny), f(yo + 1) / f(ny)]


def _render64(case: dict, seed: int) -> torch.Tensor:
    """The frame in 64 bits: the stratified samples of every task's stream,
    pinhole rays, every light sampled once, a box filter of radius 0.5."""
    prims, lights, c2w, fov, _ = _geometry(case, seed)
    geo = _Geometry64(prims)
    W, H, side, nl = case["width"], case["height"], case["spp_side"], len(lights)
    spp = side * side
    wpp = 9 * spp + 9 * nl * spp
    f = np.float32
    aspect = f(W) / f(H)
    num_tasks = (max(256, W * H // 256) - 1).bit_length()  # the renderer's task split for 8 cores
    cols = {"px": [], "u": [], "film": []}
    for task in range(num_tasks):
        c = _crop(task, num_tasks, float(aspect))
        win = [int(f(0) * (f(1) - c[k]) + f(n) * c[k]) for k, n in ((0, W), (1, W), (2, H), (3, H))]
        if win[0] == win[1] or win[2] == win[3]:
            continue
        film = [math.ceil(f(n) * c[k]) for k, n in ((0, W), (1, W), (2, H), (3, H))]
        film = [film[0], film[0] + max(film[1] - film[0], 1), film[2], film[2] + max(film[3] - film[2], 1)]
        w, h = win[1] - win[0], win[3] - win[2]
        u = (_keystream(task, w * h * wpp) >> np.uint32(8)).astype(np.float64).reshape(w * h, wpp) / 16777216.0
        y, x = np.divmod(np.arange(w * h), w)
        cols["px"].append(np.stack([x + win[0], y + win[2]], axis=1))
        cols["u"].append(u)
        cols["film"].append(np.broadcast_to(np.array(film), (w * h, 4)))
    dev = dict(device="cuda", dtype=torch.float64)
    px = torch.tensor(np.concatenate(cols["px"]), **dev)
    u = torch.tensor(np.concatenate(cols["u"]), **dev)
    film = torch.tensor(np.concatenate(cols["film"]), device="cuda")
    k = torch.arange(spp, device="cuda")
    strata = torch.stack([k % side, k // side], dim=1).double()
    im = ((strata + u[:, :2 * spp].reshape(-1, spp, 2)) / side + px[:, None, :]).reshape(-1, 2)
    ls = u[:, 9 * spp:].reshape(-1, spp, 9 * nl).reshape(-1, 9 * nl)
    film = film[:, None, :].expand(-1, spp, 4).reshape(-1, 4)
    m = torch.tensor(np.asarray(c2w.m, np.float32).reshape(4, 4).astype(np.float64), **dev)
    tan = math.tan(math.radians(fov) / 2.0)
    d = torch.stack([(2.0 * im[:, 0] / W - 1.0) * tan, (1.0 - 2.0 * im[:, 1] / H) * tan, torch.ones_like(im[:, 0])], 1)
    d = (d / d.norm(dim=1, keepdim=True)) @ m[:3, :3].T
    n = d.shape[0]
    o = m[:3, 3].expand(n, 3)
    zero, far = torch.zeros(n, **dev), torch.full((n,), 3.4028234663852886e38, **dev)
    h = geo.closest(o, d, zero, far)
    hit = h["prim"] >= 0
    p = o + d * h["t"][:, None]
    nn = geo.tri_n[h["tri"].clamp_min(0)]
    if geo.sph.shape[0]:
        ball = geo.sph[h["sph"].clamp_min(0)]
        nn = torch.where((h["sph"] >= 0)[:, None], (p - ball[:, :3]) / ball[:, 3:4], nn)
    kd = geo.kd[h["prim"].clamp_min(0)]
    cos_o = -(d * nn).sum(1)
    L = torch.zeros((n, 3), **dev)
    emit = [x for x in lights if isinstance(x, DiffuseAreaLight)]
    on_light = hit & geo.light[h["prim"].clamp_min(0)] & (cos_o > 0)
    if emit:
        L += torch.where(on_light[:, None], torch.tensor([float(v) for v in emit[0].radiance], **dev), 0.0)
    tri_of_light = geo.tri[geo.light[geo.tid]]
    for li, light in enumerate(lights):
        if isinstance(light, PointLight):
            lm = np.asarray(light.light_to_world.m, np.float32).reshape(4, 4).astype(np.float64)
            target = torch.tensor(lm[:3, 3], **dev).expand(n, 3)
            d2 = ((target - p) ** 2).sum(1)
            Li = torch.tensor([float(v) for v in light.intensity], **dev)[None] / d2[:, None]
            shrink = 1.0
        else:
            comp, s = ls[:, 3 * li], 3 * nl + 6 * li
            su = torch.sqrt(ls[:, s])
            b1, b2 = 1.0 - su, ls[:, s + 1] * su
            area = torch.linalg.cross(tri_of_light[:, 1] - tri_of_light[:, 0],
                                      tri_of_light[:, 2] - tri_of_light[:, 0]).norm(dim=1) / 2.0
            v = tri_of_light[(comp[:, None] >= torch.cumsum(area / area.sum(), 0)[None, :-1]).sum(1)]
            target = v[:, 0] * b1[:, None] + v[:, 1] * b2[:, None] + v[:, 2] * (1.0 - b1 - b2)[:, None]
            ns = torch.linalg.cross(v[:, 1] - v[:, 0], v[:, 2] - v[:, 0])
            ns = ns / ns.norm(dim=1, keepdim=True)
            w = target - p
            d2 = (w * w).sum(1)
            cs = -(ns * w).sum(1) / torch.sqrt(d2)
            Li = torch.where(cs > 0, cs * area.sum() / d2, 0.0)[:, None] * \
                torch.tensor([float(x) for x in light.radiance], **dev)[None]
            shrink = 1.0 - 1e-3
        w = target - p
        dist = torch.sqrt((w * w).sum(1))
        wi = w / dist[:, None]
        cos_i = (wi * nn).sum(1)
        want = hit & (cos_i * cos_o > 0) & (Li.sum(1) > 0) & (kd.sum(1) > 0)
        idx = want.nonzero()[:, 0]
        sh = geo.closest(p[idx], wi[idx], 5e-4 * h["t"][idx], shrink * dist[idx])
        free = idx[sh["prim"] < 0]
        L[free] += kd[free] / math.pi * Li[free] * cos_i[free].abs()[:, None]
    # the film: rgb -> xyz -> rgb by the renderer's two matrices (not quite inverses)
    to_xyz = torch.tensor([[0.412453, 0.357580, 0.180423], [0.212671, 0.715160, 0.072169],
                           [0.019334, 0.119193, 0.950227]], **dev)
    to_rgb = torch.tensor([[3.240479, -1.37150, -0.498535], [-0.969256, 1.875991, 0.041556],
                           [0.055648, -0.204043, 1.057311]], **dev)
    at = im.floor().long()
    inside = (at[:, 0] >= film[:, 0]) & (at[:, 0] < film[:, 1]) & (at[:, 1] >= film[:, 2]) & (at[:, 1] < film[:, 3])
    flat = (at[:, 1] * W + at[:, 0])[inside]
    acc = torch.zeros((H * W, 3), **dev).index_add_(0, flat, L[inside] @ to_xyz.T)
    cnt = torch.zeros(H * W, **dev).index_add_(0, flat, torch.ones_like(flat, dtype=torch.float64))
    return ((acc / cnt.clamp_min(1.0)[:, None]) @ to_rgb.T).clamp_min(0.0).reshape(H, W, 3)
