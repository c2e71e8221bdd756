"""The device build's small ranges (one warp each, a lane per primitive) at
the sizes where they begin and end, with coincident, flat, gridded and NaN
primitives: the tree is the host build's node for node, so no tolerance is
involved."""
import numpy as np
import pytest

from pbrt_rust_gb300.scene import Shape
from pbrt_rust_gb300.transform import Transform

pytestmark = pytest.mark.gpu


def triangles(kind, n):
    rng = np.random.default_rng(100 * n + len(kind))
    c = rng.uniform(-1, 1, (n, 1, 3))
    if kind == "coincident":
        c[:] = c[0]
        c[n // 2:] += 1.0
    elif kind == "grid":  # many equal keys, zeros of both signs
        c = np.round(c * 2.0)
        c[::3] *= -1.0
    p = (c + rng.uniform(-0.1, 0.1, (n, 3, 3)) * (0.0 if kind == "grid" else 1.0)).astype(np.float32)
    if kind == "flat":
        p[:, :, 1] = 0.0
    if kind == "nan":
        p[::5, :, 0] = np.nan
        p[1::7, 1, 2] = np.inf
    return p


@pytest.mark.parametrize("method,max_prims", [("sah", 4), ("sah", 1), ("middle", 4)])
@pytest.mark.parametrize("kind", ["random", "coincident", "grid", "flat", "nan"])
def test_device_tree_equals_host_tree(kind, method, max_prims):
    from pbrt_rust_gb300.abi import PbrtError
    from pbrt_rust_gb300.gpu import GpuBVHAccel
    for n in (1, 2, 3, 4, 5, 8, 31, 32) + (() if kind == "nan" else (33, 64, 65, 97, 2049)):
        p = triangles(kind, n)
        mesh = Shape.triangle_mesh(Transform(), None, False, np.arange(3 * n, dtype=np.uint32), p)

        def build(device):
            try:
                return GpuBVHAccel([mesh], max_prims, method, build_on_device=device)
            except PbrtError as e:  # an empty partition is refused by both
                return e.status
        host, dev = build(False), build(True)
        if isinstance(host, int) or isinstance(dev, int):
            assert host == dev, (n, host, dev)
            continue
        assert np.array_equal(host.primitive_order(), dev.primitive_order()), n
        assert host.nodes().tobytes() == dev.nodes().tobytes(), n
