"""The fused frame runs as a thread-block cluster per cloth with an edge per
thread: 1 to 16 CTAs, up to 1,024 vertices in one CTA or 768 in each of
several, by the cloth's size and the number of cloths.  At the sizes where the
shape changes positions and all counters must equal the launched form's bit
for bit, and a cloth's positions the oracle's."""
import numpy as np
import pytest

from xpbd_gb300 import scene
from xpbd_gb300.native import NativeXpbdBatch, NativeXpbdSolver

pytestmark = pytest.mark.gpu


def _scene(n, extras, seed=0):
    """A hanging cloth; `extras` adds a sphere, an SDF box and a wall in its
    way, tethers, soft pins and bends without colours."""
    sc = scene.plain_grid_scene(n, 3)
    if not extras:
        return sc
    w = np.zeros(n * n, np.float32)
    w[sc.cloth.pin_indices] = 1.0
    w[1 :: max(n // 3, 2)] = np.maximum(w[1 :: max(n // 3, 2)], 0.4)
    sc.cloth = scene.build_cloth(sc.cloth.positions_world, sc.cloth.triangles, 0.2, w, tether_slack=1.01)
    if seed % 2:
        sc.cloth.bend_color_offsets = np.asarray([0], np.int32)
    o = sc.options
    o.lra_compliance = 1e-6
    o.use_sphere, o.sphere_center, o.sphere_radius = True, (0.1, 0.0, -0.29), 0.3
    o.use_wall, o.wall_origin, o.wall_normal = True, (-0.45, 0.0, 0.0), (1.0, 0.0, 0.2)
    o.gravity = (0.0, 0.0, -60.0)
    sc.static_triangles = scene.box_triangles((0.3, 0.0, -0.11), (0.1, 0.1, 0.1))
    o.static_sdf_max_resolution = 32
    return sc


def _item(sc):
    return (sc.cloth, sc.options, sc.static_triangles)


# vertices: 121 and 144 (one CTA, two), 1,024 and 1,089 (one launch, two),
# 2,025 and 2,116 (16 CTAs, the smallest share above 128), 8,100 and 8,281 (512
# vertices per CTA, more), 12,100 and 12,321 (cluster, launched)
@pytest.mark.parametrize("n", [2, 11, 12, 32, 33, 45, 46, 90, 91, 110, 111])
@pytest.mark.parametrize("extras", [False, True])
def test_single(n, extras, gpu_lib, oracle_lib):
    sc = _scene(n, extras, seed=n)
    gpu, launched = NativeXpbdSolver(*_item(sc)), NativeXpbdSolver(*_item(sc))
    launched.set_launch_config({"fused_frame": 2})
    ora = oracle_lib.OracleSolver.from_scene(*_item(sc)) if n < 50 else None
    for f in range(3):
        substeps, iterations = ((10, 2), (3, 1), (1, 3))[f]
        for s in (gpu, launched):
            s.step(substeps, iterations, diagnostics=True)
        assert np.array_equal(gpu.download_positions(), launched.download_positions()), f
        for buf in (1, 2):
            assert np.array_equal(gpu.read_buffer(buf, np.float32, 4 * n * n).reshape(-1, 4)[:, :3],
                                  launched.read_buffer(buf, np.float32, 4 * n * n).reshape(-1, 4)[:, :3]), (f, buf)
        cg, cl = gpu.read_buffer(13, np.uint64, 38), launched.read_buffer(13, np.uint64, 38)
        assert np.array_equal(cg, cl), (f, np.flatnonzero(cg != cl))
        if ora is not None:
            ora.step(substeps, iterations)
            assert np.array_equal(gpu.download_positions(), ora.download_positions()), f
    if n <= 110:
        assert launched.last_step_launches() > gpu.last_step_launches()
    gpu.close()
    launched.close()


@pytest.mark.parametrize("count,sizes", [(2, (70, 9)), (9, (33, 20, 46)), (19, (40, 12)), (20, (40, 12)), (76, (26, 32, 5)),
                                         (77, (26, 32, 5)), (160, (32, 8))])
def test_batch(count, sizes, gpu_lib):
    """Cloths of a batch share one shape; one of them is inactive for a frame."""
    scs = [_scene(sizes[k % len(sizes)], k % 3 == 1, seed=k) for k in range(count)]
    gpu, launched = (NativeXpbdBatch([_item(s) for s in scs]) for _ in range(2))
    launched.set_launch_config({"fused_frame": 2})
    for f in range(3):
        for s in (gpu, launched):
            s.set_cloth_active(count // 2, f != 1)
            s.step(4, 2, diagnostics=True)
        assert np.array_equal(gpu.download_positions(), launched.download_positions()), f
        assert np.array_equal(gpu.read_buffer(13, np.uint64, 38), launched.read_buffer(13, np.uint64, 38)), f
    gpu.close()
    launched.close()
