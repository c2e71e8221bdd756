"""Rays and trees at the edges of what the 4-wide walk (trace4.cuh) takes: the
hits are the oracle's bit for bit whichever walk a ray ends up in, so no
tolerance is involved."""
import re

import numpy as np
import pytest

from pbrt_rust_gb300 import abi
from pbrt_rust_gb300.scene import InstanceDefinition, Primitive, Shape
from pbrt_rust_gb300.transform import Transform
from test_gpu_quads import mesh, soup

pytestmark = pytest.mark.gpu


def check(oracle, prims, r, max_prims=4, method="sah", on_device=False):
    """Every form of a query against the oracle: a call of few rays, the
    persistent kernel, and a batch of closest and any-hit jobs with and
    without refilling."""
    import torch

    from pbrt_rust_gb300.batch import GpuBatch
    from pbrt_rust_gb300.gpu import GpuBVHAccel
    bvh = GpuBVHAccel(prims, max_prims, method, build_on_device=on_device)
    ob = oracle.OracleBVH(prims, max_prims, method)
    want, want_p = ob.intersect(r), ob.intersect_p(r)
    dev = torch.from_numpy(r.view(np.float32).reshape(-1, 8).copy()).cuda()

    def same(hits, occ, what):
        got = hits.cpu().numpy().view(abi.HIT_DTYPE).reshape(-1)
        for f in ("prim", "t", "b1", "b2"):
            assert np.array_equal(got[f], want[f], equal_nan=True), (what, f, got[:3], want[:3])
        assert np.array_equal(occ.cpu().numpy(), want_p), what

    def called(what):
        hits, occ = bvh.intersect(dev), bvh.intersect_p(dev)
        torch.cuda.synchronize()
        same(hits, occ, what)

    called("few rays")
    before = abi.get_trace_config()
    abi.set_trace_config(reorder=True)  # keeps calls of few rays on the persistent kernel
    try:
        called("persistent")
    finally:
        abi.set_trace_config(**before)
    for tuning in (dict(refill=32), dict(refill=8)):
        b = GpuBatch(max_jobs=3, max_query_rays=0)
        b.set_tuning(extend_kernel="wide", **tuning)
        b.add_query(bvh, dev)
        b.add_query(bvh, dev, any_hit=True)
        same(*b.run(), tuning)
    return bvh, want


def flat_shape(kind):
    """A shape whose box has no thickness in y, at y = 1."""
    at = Transform.translate((0.0, 1.0, 0.0)) * Transform.scale(1.0, 1.0e-12, 1.0)
    if kind == "sphere":
        return Shape.sphere(at, None, False, 0.5, -0.5, 0.5, 360.0)
    if kind == "cylinder":
        return Shape.cylinder(at, None, False, 0.5, -0.5, 0.5, 360.0)
    lump = InstanceDefinition([Primitive.simple(mesh(soup(np.random.default_rng(3), 20, 0.4, 0.3)))])
    return Primitive.transformed(lump, at.inverse())


@pytest.mark.parametrize("max_prims", [1, 4])
@pytest.mark.parametrize("kind", ["sphere", "cylinder", "instance"])
@pytest.mark.parametrize("below", [False, True])
def test_rays_within_a_flat_box_on_the_boundary_of_the_boxes_around_it(oracle, kind, below, max_prims):
    """With a direction of -0 the reference rejects the boxes around, so that
    it never comes to the flat shape; with +0 it does."""
    s = -1.0 if below else 1.0
    rest = [mesh([[(3, 1 + s, 0), (4, 1 + s, 0), (3, 1 + 2 * s, 1)], [(3, 1, 4), (4, 1 + s / 2, 4), (3, 1 + 2 * s, 5)],
                  [(-3, 1 + s, 4), (-4, 1 + s / 2, 4), (-3, 1 + 2 * s, 5)]])]
    r = np.zeros(96, abi.RAY_DTYPE)
    r["o"] = (-2.0, 1.0, 0.0)
    r["o"][:, 2] = np.linspace(-0.45, 0.45, 96)
    r["d"] = (1.0, 0.0, 0.0)
    r["d"][::2, 1] = -0.0
    r["d"][::3, 2] = 0.05
    r["d"][1::3, 2] = -0.0
    r["tmax"] = np.inf
    _, want = check(oracle, [Primitive.simple(p) if not isinstance(p, Primitive) else p
                             for p in [flat_shape(kind)] + rest], r, max_prims)
    hit = want["prim"] >= 0
    assert hit[1::2].any() and not hit[::2].any()  # -0 finds nothing where +0 does


def funnel(n, ratio):
    """Triangles that shrink towards the origin, each `ratio` of the last: a
    tree that is one chain of nodes, the innermost far smaller than the walk's
    margins, where slots without a child pass too."""
    t = np.array([[0, 0, 0], [1, 0, 0], [0, 1, 0]], np.float64) + 1.0
    return np.array([t * float(ratio) ** -k for k in range(n)])


@pytest.mark.parametrize("where", ["alone", "instanced"])
@pytest.mark.parametrize("n,ratio", [(40, 3.0), (44, 3.0), (61, 3.0), (61, 2.0), (90, 2.0)])
def test_walks_whose_stack_runs_out(oracle, n, ratio, where):
    """Rays from the funnel's tip through every node of it, and from so far
    away that the margins exceed the whole tree."""
    rng = np.random.default_rng(n)
    r = np.zeros(300, abi.RAY_DTYPE)
    r["d"] = 1.0 + rng.uniform(-0.2, 0.2, (300, 3))
    far = np.arange(300) % 3 == 2
    r["o"][far] = -r["d"][far] * 10.0 ** rng.uniform(5, 7, (far.sum(), 1))
    r["tmax"] = np.inf
    prims = [Primitive.simple(mesh(funnel(n, ratio)))]
    if where == "instanced":
        lump = InstanceDefinition(prims)
        at = Transform.translate((0.0, 0.0, 2.0))
        prims = [Primitive.simple(mesh(funnel(n // 2, ratio))), Primitive.transformed(lump, Transform()),
                 Primitive.transformed(lump, at.inverse())]
    _, want = check(oracle, prims, r, 1, "middle")
    assert (want["prim"] >= 0).any()


@pytest.mark.parametrize("on_device", [False, True])
@pytest.mark.parametrize("kind", ["soup", "instanced"])
@pytest.mark.parametrize("offset", [0.0, 3.0e3, 2.0e5])
def test_rays_from_afar_and_trees_off_the_origin(oracle, offset, kind, on_device):
    """Margins from a small part of the boxes to many times the whole tree,
    beyond which rays take the exact walk, some of them axis-parallel."""
    rng = np.random.default_rng(8)
    at = np.array([offset, -0.5 * offset, 2.0 * offset])
    prims = [Primitive.simple(mesh(soup(rng, 400, 1.0, 0.15, at)))]
    if kind == "instanced":
        lump = InstanceDefinition([Primitive.simple(mesh(soup(rng, 200, 1.0, 0.15)))])
        for k in range(6):
            place = Transform.translate(tuple(float(v) for v in at + rng.uniform(-2, 2, 3))) * Transform.rotate(
                30.0 * k, (0.0, 1.0, 0.0))
            prims.append(Primitive.transformed(lump, place.inverse()))
    n = 3000
    u = rng.standard_normal((n, 3))
    u[::5] = np.eye(3)[rng.integers(0, 3, len(u[::5]))]
    u /= np.linalg.norm(u, axis=1, keepdims=True)
    far = 10.0 ** rng.uniform(0, 7, (n, 1))
    r = np.zeros(n, abi.RAY_DTYPE)
    r["o"] = at + rng.uniform(-1, 1, (n, 3)) + u * far
    r["d"] = -u * 10.0 ** rng.uniform(-3, 3, (n, 1))
    r["tmax"] = np.inf
    _, want = check(oracle, prims, r, on_device=on_device)
    hit = want["prim"] >= 0
    assert hit[far[:, 0] < 100].any() and hit[far[:, 0] > 1.0e5].any()


@pytest.mark.parametrize("method", ["sah", "middle"])
@pytest.mark.parametrize("n", [32, 33, 64, 2048, 2049, 5000])
def test_a_device_build_of_coincident_primitives_is_one_leaf(oracle, n, method):
    """Nothing to split at any size, so no small ranges either."""
    from pbrt_rust_gb300.gpu import GpuBVHAccel
    t = np.array([[-1, -1, 0], [1, -1, 0], [0, 1, 0]], np.float32)
    prims = [mesh(np.tile(t, (n, 1, 1)))]
    r = np.zeros(64, abi.RAY_DTYPE)
    r["o"] = np.random.default_rng(n).uniform(-0.7, 0.7, (64, 3)) + np.array([0, 0, 3])
    r["d"] = (0.0, 0.0, -1.0)
    r["tmax"] = np.inf
    dev, want = check(oracle, prims, r, 4, method, on_device=True)
    host = GpuBVHAccel(prims, 4, method)
    assert host.nodes().tobytes() == dev.nodes().tobytes() and len(host.nodes()) == 1
    assert np.array_equal(host.primitive_order(), dev.primitive_order())
    assert host.device_bytes() == dev.device_bytes()
    assert (want["prim"] >= 0).any()


@pytest.mark.parametrize("setting", [dict(kernel="w4spec"), dict(min_blocks=8)])
def test_settings_that_name_the_default_walk_take_its_kernels(setting):
    """The same kernels as by default, for calls of few rays and for pinned
    host buffers, and the same hits bit for bit."""
    import torch

    from pbrt_rust_gb300.gpu import GpuBVHAccel
    from test_gpu_render_choice import kernels_of
    bvh = GpuBVHAccel([mesh(soup(np.random.default_rng(5), 4000, 1.0, 0.1))])
    rng = np.random.default_rng(6)
    r = np.zeros(1 << 18, abi.RAY_DTYPE)
    r["o"], r["tmax"] = rng.uniform(-2, 2, (len(r), 3)), np.inf
    r["d"] = rng.uniform(-1, 1, (len(r), 3)) - r["o"]
    host = torch.from_numpy(r.view(np.float32).reshape(-1, 8)).pin_memory()
    few, out = host[:500].cuda(), torch.empty((len(r), 4)).pin_memory()

    def both():
        names = [set(re.findall(r"k_\w+(?:<[^>]*>)?", kernels_of(f)))
                 for f in (lambda: bvh.intersect(few), lambda: bvh.intersect(host, out=out))]
        return names, bvh.intersect(few).cpu().numpy().tobytes(), out.numpy().tobytes()
    want = both()
    before = abi.get_trace_config()
    abi.set_trace_config(**setting)
    try:
        got = both()
    finally:
        abi.set_trace_config(**before)
    assert got[1:] == want[1:]
    assert got[0] == want[0], (got[0], want[0])
