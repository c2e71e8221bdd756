"""Instanced frames whose shadow rays are walked by refilling warps
(k_shadow4_refill and its replay) against walks that share none of their code:
the oracle's image, and the batch's, which takes instances over the binary
layout.  There are triangles only, so every step is exact and the images are
equal: no tolerance is involved.  One instance is flat with an inverse scale
that takes rays beyond the 4-wide walk's limits, so that rays are marked and
replayed."""
import numpy as np
import pytest

from pbrt_rust_gb300.scene import Camera, Film, Filter, SceneDescription, StratifiedSampler, default_num_tasks
from pbrt_rust_gb300.transform import Transform
from test_gpu_render_choice import kernels_of
from test_gpu_shadow_refill import scene

pytestmark = pytest.mark.gpu


# samples x lights just above and well above the size where refilling begins
@pytest.mark.parametrize("n,width,height,side", [(500, 449, 439, 2), (3000, 517, 389, 3)])
def test_refilled_shadow_rays_of_instanced_frames(oracle, n, width, height, side):
    import torch

    from pbrt_rust_gb300.batch import GpuBatch
    from pbrt_rust_gb300.gpu import GpuSamplerRenderer, GpuScene
    prims, lights = scene("instances", n)
    cam2w = Transform.look_at((0.0, 0.8, -5.0), (0.0, 0.0, 0.0), (0.0, 1.0, 0.0)).inverse()
    a = width / height
    cam = Camera.perspective(cam2w, (-a, a, -1.0, 1.0), 0.0, 1.0, 0.0, 1.0e6, 50.0, Film.image(width, height, Filter()))
    smp = StratifiedSampler(0, width, 0, height, side, side, True)
    nt = default_num_tasks(width, height)
    want = oracle.render(SceneDescription(prims, lights), cam, smp, nt)
    assert want.max() > 0.0
    sc, rn = GpuScene(prims, lights), GpuSamplerRenderer(smp, cam, num_tasks=nt)
    assert np.array_equal(rn.render(sc).view(np.uint32), want.view(np.uint32))
    samples = width * height * side * side
    batch = GpuBatch(max_jobs=1, max_tasks=nt, max_samples=samples, max_light_samples=2 * samples,
                     max_film_pixels=width * height)
    out = torch.empty((height, width, 3), device="cuda")

    def batched():
        batch.add_render(sc, rn, out=out)
        batch.run()
    batched()
    torch.cuda.synchronize()
    assert np.array_equal(out.cpu().numpy().view(np.uint32), want.view(np.uint32))
    alone, together = kernels_of(lambda: rn.render(sc)), kernels_of(batched)
    if "k_generate" not in alone or "kb_generate" not in together:
        pytest.skip("no kernel names to be had from the profiler")
    assert "k_shadow4_refill" in alone and "k_shadow_replay" in alone  # different walks indeed
    assert "4" not in "".join(w for w in together.split() if "kb_trace" in w).split("<")[0]
