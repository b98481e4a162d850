"""Vertex passes and bend colours may start while the launch before them
drains.  Positions, previous positions, velocities and all counters of frames
run that way equal those of profiled frames, whose launches are apart, bit for
bit: 8, 4, 2 and 1 lanes per vertex, coloured and uncoloured bends, normals
gathered (no prediction rides on a pass) and not, substep counts that end on
either position buffer."""
import numpy as np
import pytest

from xpbd_gb300 import scene
from xpbd_gb300.native import NativeXpbdSolver

pytestmark = pytest.mark.gpu


# 16,129 / 16,641 vertices (8 / 4 lanes), 32,761 / 33,124 (4 / 2), 131,044 / 131,769 (2 / 1)
@pytest.mark.parametrize("n", [112, 127, 129, 181, 182, 362, 363])
@pytest.mark.parametrize("kind", ["plain", "uncoloured", "pressure", "no graph"])
def test_frames_equal_profiled_frames(n, kind, gpu_lib):
    sc = scene.plain_grid_scene(n, 3)
    if kind == "uncoloured":
        sc.cloth.bend_color_offsets = np.asarray([0], np.int32)
    if kind == "pressure":
        sc.options.use_volume_pressure, sc.options.pressure_strength = True, 2.0
    sc.options.use_sphere, sc.options.sphere_center, sc.options.sphere_radius = True, (0.1, 0.0, -0.29), 0.3
    a, b = (NativeXpbdSolver(sc.cloth, sc.options, sc.static_triangles) for _ in range(2))
    if kind == "no graph":
        a.set_graph_capture(False)
    for substeps, iterations in ((10, 2), (3, 1), (1, 3)):
        a.step(substeps, iterations, diagnostics=True)
        b.profile_frame(substeps, iterations)
        for buf in (0, 1, 2):
            x, y = a.read_buffer(buf, np.float32, 4 * n * n), b.read_buffer(buf, np.float32, 4 * n * n)
            assert np.array_equal(x.reshape(-1, 4)[:, :3], y.reshape(-1, 4)[:, :3]), (substeps, buf)
    a.close()
    b.close()
