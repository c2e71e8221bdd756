"""Trees whose layout is made on the device (device_fill_layout), from single
leaves to sizes that leave the last of many blocks part full: the same hits
and sizes as the tree that the host lays out, so no tolerance is involved."""
import numpy as np
import pytest

from pbrt_rust_gb300.scene import InstanceDefinition, Primitive, Shape
from pbrt_rust_gb300.transform import Transform
from test_gpu_quads import mesh, rays, soup

pytestmark = pytest.mark.gpu


def sphere(rng, extent):
    o = Transform.translate(tuple(float(v) for v in rng.uniform(-extent, extent, 3)))
    return Shape.sphere(o, o.inverse(), False, 0.05, -0.05, 0.05, 360.0)


def scene(kind, n):
    rng = np.random.default_rng(n + len(kind))
    t = soup(rng, n, 2.0, 0.05)
    if kind == "triangles":
        return [mesh(t)]
    if kind == "clusters":  # leaves of several primitives
        t[:, :, :] = t[np.arange(n) % (n // 7)]
        return [mesh(t)]
    if kind == "coincident":  # half of them one leaf: laid out by the host
        t[: n // 2] = t[0]
        return [mesh(t)]
    if kind == "past_reach":  # no 4-wide layout
        t[n // 2] *= 1.0e13
        return [mesh(t)]
    if kind == "nan":
        t[n // 2, 1, 2] = np.nan
        return [mesh(t)]
    if kind == "mixed":
        return [mesh(t[: n // 2])] + [sphere(rng, 2.0) for _ in range(300)] + [mesh(t[n // 2:])]
    assert kind == "instances"
    big = InstanceDefinition([Primitive.simple(mesh(soup(rng, n, 0.5, 0.03))), Primitive.simple(sphere(rng, 0.3))])
    small = InstanceDefinition([Primitive.simple(mesh(soup(rng, 40, 0.5, 0.1)))])
    prims = [Primitive.simple(mesh(t))]
    for k in range(9):
        place = Transform.translate(tuple(float(v) for v in rng.uniform(-2, 2, 3)))
        prims.append(Primitive.transformed(small if k % 3 == 0 else big, place.inverse()))
    return prims


@pytest.mark.parametrize("kind,n,max_prims", [
    ("triangles", 1, 4), ("triangles", 2, 1), ("triangles", 3, 4), ("triangles", 5, 1), ("triangles", 129, 4),
    ("triangles", 130, 1), ("mixed", 40, 4), ("coincident", 200, 4), ("clusters", 257, 4),
    ("triangles", 16383, 4), ("triangles", 16384, 4), ("triangles", 16385, 1), ("triangles", 70001, 4),
    ("triangles", 300007, 2), ("clusters", 20011, 4), ("coincident", 16400, 4), ("past_reach", 16500, 4),
    ("nan", 16500, 4), ("mixed", 33333, 4), ("mixed", 16500, 1), ("instances", 16900, 4)])
def test_device_layout_equals_host_layout(kind, n, max_prims):
    import torch

    from pbrt_rust_gb300.abi import PbrtError
    from pbrt_rust_gb300.gpu import GpuBVHAccel

    def build(device):
        try:
            return GpuBVHAccel(scene(kind, n), max_prims, "sah", build_on_device=device)
        except PbrtError as e:  # refused by both
            return e.status
    host, dev = build(False), build(True)
    if isinstance(host, int) or isinstance(dev, int):
        assert host == dev
        return
    assert host.nodes().tobytes() == dev.nodes().tobytes()
    assert host.device_bytes() == dev.device_bytes()
    r = rays((np.full(3, -2.2), np.full(3, 2.2)), 20000, n, None)
    d = torch.from_numpy(r.view(np.uint8).reshape(-1, 32).copy()).cuda().view(torch.float32)
    for f in ("intersect", "intersect_p"):
        a, b = getattr(host, f)(d), getattr(dev, f)(d)
        torch.cuda.synchronize()
        assert torch.equal(a.view(torch.uint8), b.view(torch.uint8)), f
