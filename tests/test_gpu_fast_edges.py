"""Fast edge-edge query in rounds of 32 pairs: an item's budget and its up to
16 cluster keys carry over from round to round.  Crowded cloths (buckets of
more than 32 edges, items that span rounds), budgets from 1 to 32 and 8, 16 or
32 items per warp: positions and all counters equal the oracle's."""
import numpy as np
import pytest

from xpbd_gb300 import scene
from xpbd_gb300.native import NativeXpbdBatch, NativeXpbdSolver

pytestmark = pytest.mark.gpu


def _item(n, budget, margin=1.0):
    sc = scene.drop_scene(12, 1, seed=1, self_mode=1)
    sc.cloth = scene._unpinned_grid(n, 0.0, (n - 1) * 0.05)  # at rest only edges that share a vertex are near
    sc.options.self_collision_interval = 1
    sc.options.use_sphere = False
    sc.options.max_self_collision_neighbors = budget
    sc.options.cloth_thickness *= margin
    return sc.cloth, sc.options, sc.static_triangles


def _crowd(n, side, seed):
    rng = np.random.default_rng(seed)
    p = rng.uniform(0.0, side, (n * n, 3))
    p[:, 2] += 0.4
    return np.ascontiguousarray(p, np.float32)


@pytest.mark.parametrize("budget", [1, 2, 5, 16, 31, 32])
@pytest.mark.parametrize("n,side", [(9, 0.004), (14, 0.01), (23, 0.004), (23, 0.03)])
def test_crowds(n, side, budget, gpu_lib, oracle_lib):
    item = _item(n, budget)
    gpu, ora = NativeXpbdSolver(*item), oracle_lib.OracleSolver.from_scene(*item)
    p = _crowd(n, side, n + budget)
    for s in (gpu, ora):
        s.update_positions(p)
        s.step(2, 1)
    assert np.array_equal(gpu.download_positions(), ora.download_positions())
    cg, co = gpu.read_buffer(13, np.uint64, 38), ora.read_buffer(13, np.uint64, 38)
    assert np.array_equal(cg, co), np.flatnonzero(cg != co)


@pytest.mark.parametrize("count", [1, 60, 300])  # 8, 16 and 32 items per warp
def test_batches(count, gpu_lib, oracle_lib):
    items = [_item(23 if k % 3 else 19, 1 + (5 * k) % 32, 1.0 + 0.1 * (k % 4)) for k in range(count)]
    batch = NativeXpbdBatch(items)
    crowds = [_crowd(23 if k % 3 else 19, 0.02, k % 7) for k in range(count)]
    batch.update_positions(np.concatenate(crowds))
    batch.step(1, 1, diagnostics=True)
    for k in range(0, count, max(count // 12, 1)):
        ora = oracle_lib.OracleSolver.from_scene(*items[k])
        ora.update_positions(crowds[k])
        ora.step(1, 1)
        assert np.array_equal(batch.download_cloth_positions(k), ora.download_positions()), k
