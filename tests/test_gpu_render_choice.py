"""The choice of a render's traversal kernels: what a caller asks for is what
runs, on trees of any size, and gives the same image; the default goes by the
tree's size."""
import numpy as np
import pytest

from pbrt_rust_gb300 import abi, generators as G
from pbrt_rust_gb300.scene import MatteMaterial, Primitive
from test_gpu_quads import grid_floor, mesh, soup


def test_the_default_choice_is_one_that_can_be_set_again(lib):
    before = abi.get_trace_config()
    assert before["render_kernel"] == "auto"
    abi.set_trace_config(render_kernel="w4")
    assert abi.get_trace_config()["render_kernel"] == "w4"
    abi.set_trace_config(**before)
    assert abi.get_trace_config() == before
    with pytest.raises(abi.PbrtError):  # not a kernel of a query
        abi.set_trace_config(kernel="auto")


def kernels_of(fn):
    """Names of the kernels that fn launches (a process's first profile may
    come back empty)."""
    import torch
    names = ""
    for _ in range(2):
        with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CUDA]) as prof:
            fn()
            torch.cuda.synchronize()
        names = " ".join(e.key for e in prof.key_averages())
        if names:
            break
    return names


def scene(kind):
    """Geometry and a camera of the small test scene, with its two lights."""
    prims, lights, cam, smp = G.c1_scene(res=72, n_spheres=0)
    rng = np.random.default_rng(4)
    matte = MatteMaterial((0.6, 0.5, 0.4))
    if kind == "floor":
        shapes = [mesh(grid_floor(8) - np.array([4.0, 1.0, 4.0], np.float32))]
    else:
        shapes = [mesh(soup(rng, {"soup": 700, "large": 6000}[kind], 1.2, 0.12))]
    return prims + [Primitive.geometric(s, matte) for s in shapes], lights, cam, smp


@pytest.mark.gpu
@pytest.mark.parametrize("kind", ["floor", "soup", "large"])
def test_asked_for_kernels_run_and_give_the_oracles_image(oracle, kind):
    """Without analytic shapes every step is exact, so the images are equal:
    no tolerance is involved."""
    from pbrt_rust_gb300.gpu import GpuSamplerRenderer, GpuScene
    from pbrt_rust_gb300.scene import SceneDescription, default_num_tasks
    prims, lights, cam, smp = scene(kind)
    nt = default_num_tasks(72, 72)
    want = oracle.render(SceneDescription(prims, lights), cam, smp, nt)
    assert want.max() > 0.05
    sc, rn = GpuScene(prims, lights), GpuSamplerRenderer(smp, cam, num_tasks=nt)
    before = abi.get_trace_config()
    try:
        for choice, wide in (("w4", True), ("plain", False), ("auto", kind == "large")):
            abi.set_trace_config(render_kernel=choice)
            assert np.array_equal(rn.render(sc).view(np.uint32), want.view(np.uint32)), choice
            names = kernels_of(lambda: rn.render(sc))
            if "k_generate" not in names:
                pytest.skip("no kernel names to be had from the profiler")
            assert ("k_trace4" in names) == wide and ("k_shadow4" in names) == wide, (choice, names)
    finally:
        abi.set_trace_config(**before)
