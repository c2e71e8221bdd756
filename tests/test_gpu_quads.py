"""The 4-wide walk over rounded boxes (trace4.cuh) where its argument is
tight: rays on box planes, axis-parallel rays with either zero, origins and
trees far from the origin, flat trees, leaves of several primitives, stacks
that overflow shared memory, rays that take the exact walk, trees past the
reach of the layout.  Hits, distances and barycentrics equal the oracle's bit
for bit, so no tolerance is involved."""
import ctypes as C

import numpy as np
import pytest

from pbrt_rust_gb300 import abi
from pbrt_rust_gb300.scene import InstanceDefinition, Primitive, Shape
from pbrt_rust_gb300.transform import Transform

pytestmark = pytest.mark.gpu


def mesh(pts):
    pts = np.asarray(pts, np.float32).reshape(-1, 3)
    return Shape.triangle_mesh(Transform(), None, False, np.arange(len(pts), dtype=np.uint32), pts)


def soup(rng, n, extent=1.0, size=0.1, center=(0, 0, 0)):
    c = rng.uniform(-extent, extent, (n, 1, 3)) + np.asarray(center)
    return c + rng.uniform(-size, size, (n, 3, 3))


def grid_floor(n=24):
    """Axis-aligned unit cells in the plane y = 0 and walls at integer x."""
    q = []
    for i in range(n):
        for j in range(n):
            a, b, c, d = (i, 0, j), (i + 1, 0, j), (i + 1, 0, j + 1), (i, 0, j + 1)
            q += [(a, b, c), (a, c, d)]
        q += [((i, 0, 0), (i, 2, 0), (i, 2, n)), ((i, 0, 0), (i, 2, n), (i, 0, n))]
    return np.array(q, np.float32)


def chain(n=220):
    """Triangles at geometrically growing distances: a tree that is one long
    chain, whose walk defers many children at once."""
    t = np.array([[0, 0, 0], [1, 0, 0], [0, 1, 0]], np.float64)
    return np.array([t * 1.09 ** k + np.array([0, 0, 1.09 ** k]) for k in range(n)], np.float32)


def scene(name):
    rng = np.random.default_rng(sum(map(ord, name)))
    if name == "floor":
        return [mesh(grid_floor())], (np.zeros(3), np.array([24.0, 2.0, 24.0]))
    if name == "chain":
        return [mesh(chain())], (np.array([-1.0, -1.0, 0.0]), np.array([8.0, 8.0, 60.0]))
    if name == "offset":  # small triangles a long way out
        c = np.array([2.0e5, -1.0e5, 3.0e5])
        return [mesh(soup(rng, 600, 4.0, 0.5, c))], (c - 5.0, c + 5.0)
    if name == "wide_range":  # tiny triangles inside a huge tree
        return [mesh(soup(rng, 300, 1.0, 0.1)), mesh(soup(rng, 40, 3.0e4, 4.0e3))], (np.full(3, -2.0), np.full(3, 2.0))
    if name == "past_reach":  # no 4-wide layout: the binary kernels take it
        return [mesh(soup(rng, 200, 1.0, 0.2)), mesh(soup(rng, 8, 4.0e12, 1.0e12))], (np.full(3, -2.0), np.full(3, 2.0))
    if name == "mixed":  # analytic leaves beside triangles
        prims = [mesh(soup(rng, 200, 1.0, 0.2))]
        for k in range(40):
            o = Transform.translate(tuple(rng.uniform(-1, 1, 3))) * Transform.rotate(float(rng.uniform(0, 360)),
                                                                                     (0.3, 1.0, 0.2))
            prims.append([Shape.sphere(o, None, False, 0.1, -0.1, 0.1, 360.0),
                          Shape.disk(o, None, False, 0.0, 0.2, 0.05, 300.0),
                          Shape.cylinder(o, None, False, 0.08, -0.1, 0.2, 360.0)][k % 3])
        return prims, (np.full(3, -1.2), np.full(3, 1.2))
    assert name == "instances"
    tree = InstanceDefinition([Primitive.simple(mesh(soup(rng, 60, 0.5, 0.2))),
                               Primitive.simple(Shape.sphere(Transform(), None, False, 0.3, -0.3, 0.3, 360.0))])
    flat = InstanceDefinition([Primitive.simple(mesh(grid_floor(4)))])
    prims = [Primitive.simple(mesh(soup(rng, 50, 2.0, 0.2)))]
    for k in range(12):
        place = Transform.translate(tuple(float(v) for v in rng.uniform(-2, 2, 3)))
        if k % 2:
            place = place * Transform.rotate(90.0 * k, (0.0, 1.0, 0.0))
        prims.append(Primitive.transformed(flat if k % 3 == 0 else tree, place.inverse()))
    return prims, (np.full(3, -2.5), np.full(3, 2.5))


def rays(box, n, seed, prims):
    """Random rays in and about the box; a quarter parallel to an axis or a
    plane with zeros of either sign, origins on the integer planes of the
    floor; some far away, with long or short directions, finite or negative
    segments, and some that the rounded walk must not take."""
    rng = np.random.default_rng(seed)
    lo, hi = box
    ext = hi - lo
    r = np.zeros(n, abi.RAY_DTYPE)
    o = lo - 0.25 * ext + 1.5 * ext * rng.random((n, 3))
    tgt = lo + ext * rng.random((n, 3))
    k = np.arange(n)
    far = k % 11 == 0
    o[far] += (rng.standard_normal((n, 3)) * 40.0 * ext)[far]
    d = tgt - o
    d[k % 3 == 0] *= 10.0 ** rng.uniform(-12, 9, (n, 1))[k % 3 == 0]
    snap = k % 4 == 1
    o[snap] = np.round(o[snap])
    zero = rng.random((n, 3)) < 0.5
    zero[np.arange(n), rng.integers(0, 3, n)] = False
    par = k % 4 == 1
    d[par] = np.where(zero[par], np.where(rng.random((par.sum(), 3)) < 0.5, 0.0, -0.0), d[par])
    r["o"], r["d"] = o, d
    r["tmin"] = np.where(k % 7 == 0, -5.0, 1e-4)
    r["tmax"] = np.where(k % 5 == 0, rng.uniform(0.1, 2.0, n), np.inf)
    odd = k % 97 == 0
    r["d"][odd & (k % 2 == 0), 1] = 1e-30
    r["d"][odd & (k % 2 == 1)] *= np.float32(1e22)
    r["o"][k % 193 == 5, 2] = np.nan
    r["d"][k % 389 == 7] = 0.0
    r["tmax"][k % 401 == 9] = np.nan
    return r


SCENES = ["floor", "chain", "offset", "wide_range", "past_reach", "mixed", "instances"]


def config(lib, kernel, reorder=0):
    """Sets the traversal; reorder = 1 keeps calls of few rays on the
    persistent kernel (and bins those of 32768 or more).  Returns the old
    configuration."""
    cfg = abi.PbrtTraceConfig()
    abi.check(lib.pbrtgpu_get_trace_config(C.byref(cfg)), lib)
    old = abi.PbrtTraceConfig.from_buffer_copy(cfg)
    cfg.kernel = abi.TRACE_KERNELS[kernel]
    cfg.reorder = reorder
    abi.check(lib.pbrtgpu_set_trace_config(C.byref(cfg)), lib)
    return old


@pytest.mark.parametrize("leaf", [(1, "sah"), (5, "middle")])
@pytest.mark.parametrize("name", SCENES)
def test_quad_walk_equals_oracle(lib, oracle, name, leaf):
    import torch
    from pbrt_rust_gb300.batch import GpuBatch
    from pbrt_rust_gb300.gpu import GpuBVHAccel
    prims, box = scene(name)
    bvh, ob = GpuBVHAccel(prims, *leaf), oracle.OracleBVH(prims, *leaf)
    r = rays(box, 6007, 5, prims)
    want, want_p = ob.intersect(r), ob.intersect_p(r)
    assert 300 < int((want["prim"] >= 0).sum()) < 5900
    dev = torch.from_numpy(r.view(np.float32).reshape(-1, 8).copy()).cuda()

    def check(hits, occ, what):
        got = hits.cpu().numpy().view(abi.HIT_DTYPE).reshape(-1)
        bad = np.nonzero((got["prim"] != want["prim"]))[0]
        assert len(bad) == 0, (what, bad[:5], r[bad[:3]], got[bad[:3]], want[bad[:3]])
        for f in ("t", "b1", "b2"):
            assert np.array_equal(got[f], want[f], equal_nan=True), (what, f)
        assert np.array_equal(occ.cpu().numpy(), want_p), what

    for kernel, reorder in (("w4pt", 1), ("w4pt", 0), ("w4", 0)):
        old = config(lib, kernel, reorder)
        try:
            check(bvh.intersect(dev), bvh.intersect_p(dev), (kernel, reorder))
        finally:
            abi.check(lib.pbrtgpu_set_trace_config(C.byref(old)), lib)
    for tuning in (dict(refill=32), dict(refill=8), dict(refill=8, stack=8, block=256)):
        b = GpuBatch(max_jobs=3, max_query_rays=0)
        b.set_tuning(extend_kernel="wide", **tuning)
        b.add_query(bvh, dev)
        b.add_query(bvh, dev, any_hit=True)
        hits, occ = b.run()
        check(hits, occ, tuning)


def test_shadow_rays_beside_axis_planes(oracle):
    """A render whose shadow rays run parallel to the floor's cells (a light
    straight above) equals the oracle's image bit for bit, alone and in a
    batch."""
    from pbrt_rust_gb300.batch import GpuBatch
    from pbrt_rust_gb300.gpu import GpuSamplerRenderer, GpuScene
    from pbrt_rust_gb300.scene import (Camera, Film, Filter, MatteMaterial, PointLight, SceneDescription,
                                       StratifiedSampler, default_num_tasks)
    prims = [Primitive.geometric(mesh(grid_floor(8)), MatteMaterial((0.5, 0.6, 0.7)))]
    lights = [PointLight(Transform.translate((4.0, 5.0, 4.0)), (60.0,) * 3)]
    cam = Camera.perspective(Transform.look_at((4.0, 6.0, -6.0), (4.0, 0.0, 4.0), (0.0, 1.0, 0.0)).inverse(),
                             (-1.0, 1.0, -1.0, 1.0), 0.0, 1.0, 0.0, 1e30, 60.0, Film.image(40, 40, Filter.mean(0.5, 0.5)))
    smp = StratifiedSampler.stratified(0, 40, 0, 40, 1, 1, False, 0.0, 1.0)
    nt = default_num_tasks(40, 40)
    want = oracle.render(SceneDescription(prims, lights), cam, smp, nt)
    sc, rn = GpuScene(prims, lights), GpuSamplerRenderer(smp, cam, num_tasks=nt)
    assert np.array_equal(rn.render(sc), want)
    for tuning in (dict(refill_shadow=8), dict(refill_shadow=32)):
        b = GpuBatch(max_jobs=2)
        b.set_tuning(shadow_kernel="wide", extend_kernel="wide", **tuning)
        b.add_render(sc, rn)
        assert np.array_equal(b.run()[0], want)


@pytest.mark.parametrize("n", [1, 33, 2128, 2129, 8513, 155648, 155649])
def test_calls_of_any_size(n, oracle):
    """Few rays are spread over more warps than they fill, in steps of the
    rays per warp, up to the count from which the persistent kernel takes over
    (the edges for 152 SMs): every ray gets its own hit, none past the end is
    written."""
    import torch
    from pbrt_rust_gb300.gpu import GpuBVHAccel
    prims, box = scene("mixed")
    bvh, ob = GpuBVHAccel(prims), oracle.OracleBVH(prims, 4, "sah")
    r = rays(box, n, 11, prims)
    want, want_p = ob.intersect(r), ob.intersect_p(r)
    dev = torch.from_numpy(r.view(np.float32).reshape(-1, 8).copy()).cuda()
    hits = torch.full((n + 64, 4), 7.0, device="cuda")
    occ = torch.full((n + 64,), 7, device="cuda", dtype=torch.uint8)
    bvh.intersect(dev, out=hits)
    bvh.intersect_p(dev, out=occ)
    got = hits[:n].cpu().numpy().view(abi.HIT_DTYPE).reshape(-1)
    for f in ("prim", "t", "b1", "b2"):
        assert np.array_equal(got[f], want[f], equal_nan=True), f
    assert np.array_equal(occ[:n].cpu().numpy(), want_p)
    assert bool((hits[n:] == 7.0).all()) and bool((occ[n:] == 7).all())
