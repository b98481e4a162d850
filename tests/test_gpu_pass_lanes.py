"""The launched stretch pass gives a vertex 8, 4, 2 or 1 lanes by the number of
vertices, and the default schedule merges the next substep's prediction and
the last self-collision pass's pushes into a neighbouring pass.  On both sides
of each change the positions, previous positions, velocities and counters must
equal those of a launch per stage, and the positions the oracle's."""
import numpy as np
import pytest

from xpbd_gb300 import scene
from xpbd_gb300.native import NativeXpbdBatch, NativeXpbdSolver

pytestmark = pytest.mark.gpu


# vertices 16,384 / 16,641 (8 / 4 lanes), 32,761 / 33,124 (4 / 2), 130,321 /
# 131,769 (2 / 1); soft pins, wall and sphere contacts, capped corrections
@pytest.mark.parametrize("n", [128, 129, 181, 182, 361, 363])
def test_plain(n, gpu_lib, oracle_lib):
    sc = scene.plain_grid_scene(n, 2)
    w = np.zeros(n * n, np.float32)
    w[sc.cloth.pin_indices] = 1.0
    w[5 : n : 7] = 0.4
    sc.cloth = scene.build_cloth(sc.cloth.positions_world, sc.cloth.triangles, 0.2, w)
    o = sc.options
    o.use_sphere, o.sphere_center, o.sphere_radius = True, (0.1, 0.0, -0.295), 0.3
    o.use_wall, o.wall_origin, o.wall_normal = True, (-0.45, 0.0, 0.0), (1.0, 0.0, 0.2)
    o.gravity = (0.0, 0.0, -400.0)
    gpu, apart = (NativeXpbdSolver(sc.cloth, o, sc.static_triangles) for _ in range(2))
    apart.set_launch_config({"fused_frame": 2})
    ora = oracle_lib.OracleSolver.from_scene(sc.cloth, o, sc.static_triangles)
    for substeps, iterations in ((5, 2), (2, 1)):
        gpu.step(substeps, iterations, diagnostics=True)
        apart.step(substeps, iterations, diagnostics=True)
        ora.step(substeps, iterations)
        for buf in (0, 1, 2):
            a, b = (s.read_buffer(buf, np.float32, 4 * n * n).reshape(-1, 4)[:, :3] for s in (gpu, apart))
            assert np.array_equal(a, b), buf
        assert np.array_equal(gpu.download_positions(), ora.download_positions())
        cg = gpu.read_buffer(13, np.uint64, 38)
        assert np.array_equal(cg, apart.read_buffer(13, np.uint64, 38)) and np.array_equal(cg, ora.read_buffer(13, np.uint64, 38))
        assert gpu.last_step_launches() < apart.last_step_launches()
    gpu.close()
    apart.close()


@pytest.mark.parametrize("graphs", [True, False])
def test_mixed_batch(graphs, gpu_lib):
    """Fast and strict self collision at different intervals, a cloth without
    it, one inactive cloth, and dynamic colliders on one of them."""
    scs = [scene.drop_scene(20, 1, seed=1, self_mode=2), scene.drop_scene(26, 1, seed=2, self_mode=1), scene.plain_grid_scene(18, 1),
           scene.drop_scene(14, 1, seed=3, self_mode=2)]
    items = [(s.cloth, s.options, s.static_triangles) for s in scs]
    both = [NativeXpbdBatch(items) for _ in range(2)]
    both[1].set_launch_config({"fused_frame": 2})
    rng = np.random.default_rng(4)
    for k in (0, 1, 3):
        p = scs[k].cloth.positions_world.copy()
        right = p[:, 0] > 0.0
        p[right, 0] = -p[right, 0] + 0.001
        p[right, 2] += 0.0012
        p[:, :2] += rng.uniform(-2e-4, 2e-4, (len(p), 2)).astype(np.float32)
        for b in both:
            b.update_cloth_positions(k, np.ascontiguousarray(p, np.float32))
    for f in range(3):
        v, i = scene.icosphere((0.0, 0.0, 0.3 + 0.01 * f), 0.15, 2)
        for b in both:
            b.set_graph_capture(graphs)
            b.set_cloth_active(3, f != 1)
            if f == 2:
                b.update_cloth_dynamic_colliders(0, indexed=(v, i, False))
            b.step(4, 2, diagnostics=True)
        n = sum(len(s.cloth.positions_world) for s in scs)
        for buf in (0, 1, 2):
            x, y = (b.read_buffer(buf, np.float32, 4 * n).reshape(-1, 4)[:, :3] for b in both)
            assert np.array_equal(x, y), (f, buf)
        cg, ca = (b.read_buffer(13, np.uint64, 38) for b in both)
        assert np.array_equal(cg, ca), (f, np.flatnonzero(cg != ca))
        assert both[0].diagnostics()["abi41_max_smoothed_delta"] == both[1].diagnostics()["abi41_max_smoothed_delta"]
    for b in both:
        b.close()
