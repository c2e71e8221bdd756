"""How large a frame pbrtgpu_render_noalloc takes: its scratch holds what the
kernels use and nothing else, so a frame of 313600 samples and two lights
(206 bytes per sample) fits its 64 MiB."""
import numpy as np
import pytest

from pbrt_rust_gb300 import abi, generators as G
from pbrt_rust_gb300.gpu import GpuSamplerRenderer, GpuScene
from test_zz_no_alloc import render_noalloc, same_bits

pytestmark = pytest.mark.gpu


def test_a_frame_that_just_fits_the_scratch(lib):
    prims, lights, cam, smp = G.c1_scene(res=280)
    scene, r = GpuScene(prims, lights), GpuSamplerRenderer(smp, cam)
    assert smp.x_samples * smp.y_samples == 4 and len(lights) == 2
    want = r.render(scene)
    got = np.full_like(want, -1.0)
    assert render_noalloc(lib, scene, r, got) == abi.PBRT_OK, lib.pbrtgpu_last_error()
    assert same_bits(got, want)
