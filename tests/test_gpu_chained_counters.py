"""Counters of frames whose passes start early equal those of profiled frames,
whose launches are apart: 8, 4, 2 and 1 lanes per vertex, coloured and
uncoloured bends, contacts with a sphere."""
import numpy as np
import pytest

from xpbd_gb300 import scene
from xpbd_gb300.native import NativeXpbdSolver

pytestmark = pytest.mark.gpu


# 1,936 vertices (8 lanes), 4,489 (4), 4,624 and 130,321 (2), 131,769 (1)
@pytest.mark.parametrize("n", [44, 67, 68, 361, 363])
@pytest.mark.parametrize("uncoloured", [False, True])
def test_counters_equal_profiled_frames(n, uncoloured, gpu_lib):
    sc = scene.plain_grid_scene(n, 3)
    if uncoloured:
        sc.cloth.bend_color_offsets = np.asarray([0], np.int32)
    o = sc.options
    o.use_sphere, o.sphere_center, o.sphere_radius = True, (0.1, 0.0, -0.29), 0.3
    o.gravity = (0.0, 0.0, -60.0)
    a, b = (NativeXpbdSolver(sc.cloth, o, sc.static_triangles) for _ in range(2))
    a.set_launch_config({"fused_frame": 2 if n < 111 else 1})  # launched passes
    seen = np.zeros(38, np.uint64)
    for substeps, iterations in ((10, 2), (3, 1), (1, 3)):
        a.step(substeps, iterations, diagnostics=True)
        b.profile_frame(substeps, iterations)
        x, y = a.read_buffer(13, np.uint64, 38), b.read_buffer(13, np.uint64, 38)
        assert np.array_equal(x, y), (substeps, np.flatnonzero(x != y))
        seen += x
    assert np.count_nonzero(seen) >= 2  # clamped edges, bends or contacts among them
    a.close()
    b.close()
