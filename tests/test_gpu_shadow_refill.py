"""Frames whose shadow rays are walked by refilling warps (k_shadow4_refill):
the image of the binary kernels bit for bit, so no tolerance is involved.  The
instanced scene has a flat instance whose inverse scale takes rays beyond the
4-wide walk's reach, so that rays are marked and replayed."""
import numpy as np
import pytest

from pbrt_rust_gb300.scene import (Camera, DiffuseAreaLight, Film, Filter, InstanceDefinition, MatteMaterial, PointLight,
                                   Primitive, Shape, StratifiedSampler)
from pbrt_rust_gb300.transform import Transform
from test_gpu_quads import mesh, soup

pytestmark = pytest.mark.gpu


def scene(kind, n):
    from pbrt_rust_gb300 import generators as G
    rng = np.random.default_rng(n)
    matte = MatteMaterial((0.6, 0.5, 0.4))
    prims = [Primitive.geometric(mesh(soup(rng, n, 1.5, 0.06)), matte)]
    if kind == "instances":
        tree = InstanceDefinition([Primitive.geometric(mesh(soup(rng, 300, 0.4, 0.1)), matte)])
        slab = InstanceDefinition([Primitive.geometric(mesh(soup(rng, 60, 1.0, 0.3)), matte)])
        for k in range(20):
            place = Transform.translate(tuple(float(v) for v in rng.uniform(-1.5, 1.5, 3)))
            prims.append(Primitive.transformed(tree, place.inverse()))
        flat = Transform.translate((0.0, 0.3, 0.0)) * Transform.scale(1.0, 1.0e-19, 1.0)
        prims.append(Primitive.transformed(slab, flat.inverse()))
    area = DiffuseAreaLight(Transform(), (10.0, 10.0, 10.0))
    prims.append(Primitive.geometric_area_light(G.quad_light_mesh((0.0, 2.5, 0.0), 1.0), MatteMaterial((0, 0, 0)), area))
    return prims, [PointLight(Transform.translate((0.0, 3.0, -2.0)), (60.0, 60.0, 60.0)), area]


# samples x lights just above and at odd distances over the sizes where the
# refilling kernel begins
@pytest.mark.parametrize("kind,n,width,height,side", [
    ("soup", 16384, 513, 257, 4), ("soup", 40000, 517, 389, 4), ("instances", 500, 449, 439, 2),
    ("instances", 3000, 517, 389, 3)])
def test_refilled_shadow_rays_give_the_binary_kernels_image(kind, n, width, height, side):
    import torch

    from pbrt_rust_gb300 import abi
    from pbrt_rust_gb300.gpu import GpuSamplerRenderer, GpuScene
    prims, lights = scene(kind, n)
    cam2w = Transform.look_at((0.0, 0.8, -5.0), (0.0, 0.0, 0.0), (0.0, 1.0, 0.0)).inverse()
    a = width / height
    cam = Camera.perspective(cam2w, (-a, a, -1.0, 1.0), 0.0, 1.0, 0.0, 1.0e6, 50.0, Film.image(width, height, Filter()))
    smp = StratifiedSampler(0, width, 0, height, side, side, True)
    sc = GpuScene(prims, lights)
    old = abi.get_trace_config()["render_kernel"]
    images = {}
    try:
        for kernel in ("plain", "w4"):
            abi.set_trace_config(render_kernel=kernel)
            out = torch.full((height, width, 3), -1.0, device="cuda")
            GpuSamplerRenderer(smp, cam).render(sc, out=out)
            torch.cuda.synchronize()
            images[kernel] = out
    finally:
        abi.set_trace_config(render_kernel=old)
    assert float(images["w4"].max()) > 0.0
    assert torch.equal(images["plain"].view(torch.int32), images["w4"].view(torch.int32))
