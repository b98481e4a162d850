"""The self-collision queries give a warp 8, 16 or 32 items and a vertex of the
neighbour table 8, 4, 2 or 1 lanes, by the number of items.  On both sides of
each change positions and all counters must equal the oracle's, for a cloth
folded onto itself (every query finds contacts)."""
import numpy as np
import pytest

from xpbd_gb300 import scene
from xpbd_gb300.native import NativeXpbdSolver

pytestmark = pytest.mark.gpu


# vertices 6,084 / 6,241 (neighbour lanes 8 / 4), 20,449 / 20,736 (4 / 2),
# 48,841 / 49,284 (2 / 1); edges 64,237 / 65,121 (8 / 16 items per warp),
# 305,921 / 307,840 (16 / 32); 32,761 / 33,124 vertices (8 / 32)
@pytest.mark.parametrize("n", [63, 64, 78, 79, 143, 144, 147, 148, 156, 157, 181, 182, 221, 222, 253, 256, 320, 321])
@pytest.mark.parametrize("mode", [2, 1], ids=["strict", "fast"])
def test_folded(n, mode, gpu_lib, oracle_lib):
    sc = scene.drop_scene(12, 1, seed=1, self_mode=mode)
    sc.cloth = scene._unpinned_grid(n, 0.0, (n - 1) * 0.01)
    sc.options.self_collision_interval = 1
    gpu = NativeXpbdSolver(sc.cloth, sc.options, sc.static_triangles)
    ora = oracle_lib.OracleSolver.from_scene(sc.cloth, sc.options, sc.static_triangles)
    rng = np.random.default_rng(n)
    p = sc.cloth.positions_world.copy()
    right = p[:, 0] > 0.0
    p[right, 0] = -p[right, 0] + 0.001
    p[right, 2] += 0.0012
    p[:, :2] += rng.uniform(-2e-4, 2e-4, (len(p), 2)).astype(np.float32)
    p[:, 2] += np.float32(0.301)
    p = np.ascontiguousarray(p, np.float32)
    gpu.update_positions(p)
    ora.update_positions(p)
    steps = 2 if n < 100 else 1
    gpu.step(steps, 2, diagnostics=True)
    ora.step(steps, 2)
    assert np.array_equal(gpu.download_positions(), ora.download_positions())
    cg, co = gpu.read_buffer(13, np.uint64, 38), ora.read_buffer(13, np.uint64, 38)
    assert np.array_equal(cg, co), np.flatnonzero(cg != co)
    assert cg[2] > 0 and cg[0] + cg[1] > 0
    gpu.close()
