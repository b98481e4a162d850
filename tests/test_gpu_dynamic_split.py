"""The dynamic-collider pass gives a warp one vertex or several, by the number
of vertices: positions and the dynamic-collider counters must equal the
oracle's on both sides of the first change (152 x 64 = 9,728 vertices), for a
signed mesh with its inside passes, plain triangles and particles."""
import numpy as np
import pytest

import test_gpu_dynamic as base
from xpbd_gb300 import scene

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [5, 98, 99, 150])
@pytest.mark.parametrize("name", ["signed_with_particles", "unsigned_with_particles", "large_triangles"])
def test_vertices_per_warp(name, n, gpu_lib, oracle_lib):
    sc = scene.dynamic_scene(n, 2)
    gpu, ora = base._pair(sc, oracle_lib)
    p = sc.cloth.positions_world.copy()
    p[:, 2] -= np.float32(0.07)  # inside the colliders' reach from the first frame on
    gpu.update_positions(p)
    ora.update_positions(p)
    for f in range(2):
        kw = base.CASES[name](f)
        gpu.update_dynamic_colliders(**kw)
        ora.update_dynamic_colliders(**kw)
        gpu.step(sc.substeps, sc.iterations, diagnostics=True)
        ora.step(sc.substeps, sc.iterations)
        assert np.array_equal(gpu.download_positions(), ora.download_positions()), f
        cg, co = gpu.read_buffer(13, np.uint64, 38), ora.read_buffer(13, np.uint64, 38)
        assert np.array_equal(cg[base.DYN_SLOTS], co[base.DYN_SLOTS]), f
    if n > 5:
        assert cg[34] > 0 and cg[1] > 0
    gpu.close()
