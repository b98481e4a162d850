"""Both sides of the lines where a launch changes its shape by size: threads of
the fused frame (128 and 288 vertices per CTA), vertices per warp of the flat
VT query (16,384 and 32,768), lanes per edge of the edge hash (307,200 edges).  Handles
stepped at once give what each gives alone."""
import numpy as np
import pytest

import test_gpu_frame_edges as frames
from xpbd_gb300 import scene
from xpbd_gb300.native import NativeXpbdSolver

pytestmark = pytest.mark.gpu


# 256 and 289 vertices: one CTA, four
@pytest.mark.parametrize("n", [16, 17, 44, 47, 67, 68])
@pytest.mark.parametrize("extras", [False, True])
def test_fused_frame_threads(n, extras, gpu_lib, oracle_lib):
    frames.test_single(n, extras, gpu_lib, oracle_lib)


def _folded(n, mode):
    sc = scene.drop_scene(n, 1, self_mode=mode)
    p = sc.cloth.positions_world.astype(np.float64).copy()
    right = p[:, 0] > 0.0
    p[right, 0] = -p[right, 0] + 0.001
    p[right, 2] += 0.0015
    p[:, 2] += 0.301
    p[:, :2] += np.random.default_rng(n).uniform(-2.0e-4, 2.0e-4, (len(p), 2))
    return sc, np.ascontiguousarray(p, np.float32)


@pytest.mark.parametrize("n", [128, 129, 181, 182])
def test_flat_vt_items(n, gpu_lib, oracle_lib):
    sc, p = _folded(n, 2)
    gpu = NativeXpbdSolver(sc.cloth, sc.options, sc.static_triangles)
    ora = oracle_lib.OracleSolver.from_scene(sc.cloth, sc.options, sc.static_triangles)
    for s in (gpu, ora):
        s.update_positions(p)
        s.step(2, 2)
    assert np.array_equal(gpu.download_positions(), ora.download_positions())
    assert np.array_equal(gpu.read_buffer(13, np.uint64, 38), ora.read_buffer(13, np.uint64, 38))
    gpu.close()


@pytest.mark.parametrize("n", [320, 321])
def test_edge_hash_lanes(n, gpu_lib):
    sc, p = _folded(n, 1)
    got = []
    for lanes in (0, 1, 16):
        s = NativeXpbdSolver(sc.cloth, sc.options, sc.static_triangles)
        if lanes:
            s.set_launch_config({"prim_lanes": lanes})
        else:
            assert s.launch_config()["prim_lanes"] == (4 if n == 320 else 8)
        s.update_positions(p)
        s.step(2, 2)
        got.append((s.download_positions().copy(), s.read_buffer(13, np.uint64, 38)))
        s.close()
    for x in got[1:]:
        assert np.array_equal(got[0][0], x[0]) and np.array_equal(got[0][1], x[1])


@pytest.mark.parametrize("kind", ["plain", "strict", "fast"])
def test_handles_stepped_at_once(kind, gpu_lib):
    mode = {"plain": 0, "strict": 2, "fast": 1}[kind]
    items = []
    for n in (12, 46, 64, 70, 100, 112) if mode == 0 else (12, 37, 64, 70):
        sc, p = _folded(n, mode) if mode else (scene.plain_grid_scene(n, 3), None)
        items.append(((sc.cloth, sc.options, sc.static_triangles), sc.cloth.positions_world if p is None else p))
    alone, handles = [], []
    for item, p in items:
        s = NativeXpbdSolver(*item)
        s.update_positions(p)
        for _ in range(3):
            s.step(10, 2)
        alone.append(s.download_positions().copy())
        s.close()
    for item, p in items * 3:
        handles.append(NativeXpbdSolver(*item))
        handles[-1].update_positions(p)
    for _ in range(3):
        for s in handles:
            s.step(10, 2, diagnostics=False, synchronize=False)
    for k, s in enumerate(handles):
        assert np.array_equal(s.download_positions(), alone[k % len(items)]), k
        s.close()
