"""Bucket scans by one block up to 4,096 counts, by two launches beyond: the
start tables equal the oracle's on both sides (a vertex table of 4,096 buckets
for 1,024 vertices, of 8,192 for 1,025), and so do the edge buckets of cells
so crowded that they overflow their slots."""
import numpy as np
import pytest

from xpbd_gb300 import scene
from xpbd_gb300.native import NativeXpbdSolver

pytestmark = pytest.mark.gpu


def _strip(v):
    i = np.arange(v - 2, dtype=np.int32)
    k = np.arange(v)
    pos = np.stack([0.01 * (k // 2), 0.01 * (k % 2), np.zeros(v)], 1).astype(np.float32)
    return scene.build_cloth(pos, np.stack([i, i + 1, i + 2], 1), 0.2, np.zeros(v, np.float32))


@pytest.mark.parametrize("v", [200, 256, 257, 1023, 1024, 1025, 2049])
@pytest.mark.parametrize("crowded", [False, True])
def test_tables(v, crowded, gpu_lib, oracle_lib):
    sc = scene.drop_scene(12, 1, seed=1, self_mode=2)
    cloth = _strip(v)
    gpu = NativeXpbdSolver(cloth, sc.options, sc.static_triangles)
    ora = oracle_lib.OracleSolver.from_scene(cloth, sc.options, sc.static_triangles)
    p = cloth.positions_world + np.float32([0.0, 0.0, 0.5])
    if crowded:
        p = np.random.default_rng(v).uniform(0.4, 0.41, (v, 3)).astype(np.float32)
    for s in (gpu, ora):
        s.update_positions(p)
        s.build_self_structures()
    vb, tb, eb = (int(x) for x in gpu.hash_info()[:3])
    for start, ent, nb in ((4, 5, vb), (6, 7, tb), (8, 9, eb)):
        a, b = gpu.read_buffer(start, np.int32, nb + 1), ora.read_buffer(start, np.int32, nb + 1)
        assert np.array_equal(a, b), start
        n = int(a[-1])
        ga, gb = gpu.read_buffer(ent, np.int32, n), ora.read_buffer(ent, np.int32, n)
        for k in np.flatnonzero(np.diff(a)):
            assert np.array_equal(np.sort(ga[a[k]:a[k + 1]]), np.sort(gb[a[k]:a[k + 1]])), (ent, k)
    for s in (gpu, ora):
        s.update_positions(p)
        s.step(1, 1)
    assert np.array_equal(gpu.download_positions(), ora.download_positions())
    assert np.array_equal(gpu.read_buffer(13, np.uint64, 38), ora.read_buffer(13, np.uint64, 38))
