"""Neighbour table and strict VV with 1 to 32 lanes per vertex (32 vertices to
one per warp): the table, all counters and the positions equal the oracle's,
for loose vertices, for vertices of a warp with very uneven numbers of members
around them, and for cells so crowded that buckets hold more than 32 members
and the table overflows.  Cloth sizes that are no multiple of a warp's
vertices, and a batch whose cloths meet within a warp."""
import numpy as np
import pytest

from xpbd_gb300 import scene
from xpbd_gb300.native import NativeXpbdBatch, NativeXpbdSolver

pytestmark = pytest.mark.gpu

LANES = [1, 2, 4, 8, 16, 32]


def _scene(n, mode):
    sc = scene.drop_scene(12, 1, seed=1, self_mode=mode)
    sc.cloth = scene._unpinned_grid(n, 0.0, (n - 1) * 0.05)  # at rest no two vertices are neighbours
    sc.options.self_collision_interval = 1
    sc.options.use_sphere = False
    return sc


def _positions(n, pose, seed):
    """`even`: about one vertex per cell; `uneven`: a ninth of them packed
    into one corner; `crowded`: tens of vertices per cell."""
    rng = np.random.default_rng(seed)
    cell = 1.8 * 0.002
    side = {"even": (n * n) ** (1 / 3), "uneven": (n * n) ** (1 / 3), "crowded": 3.0}[pose] * cell
    p = rng.uniform(0.0, side, (n * n, 3))
    if pose == "uneven":
        p[::9] = rng.uniform(0.0, 2.0 * cell, (len(p[::9]), 3))
    p[:, 2] += 0.4
    return np.ascontiguousarray(p, np.float32)


def _table(s, v):
    s.build_self_structures()
    count = s.read_buffer(10, np.int32, v)
    idx = s.read_buffer(11, np.int32, 32 * v).reshape(v, 32)
    return count, np.where(np.arange(32)[None, :] < count[:, None], idx, -1)


@pytest.mark.parametrize("pose", ["even", "uneven", "crowded"])
@pytest.mark.parametrize("n", [12, 23])
@pytest.mark.parametrize("mode", [2, 1], ids=["strict", "fast"])
def test_lanes(n, pose, mode, gpu_lib, oracle_lib):
    sc = _scene(n, mode)
    p = _positions(n, pose, n)
    ora = oracle_lib.OracleSolver.from_scene(sc.cloth, sc.options, sc.static_triangles)
    ora.update_positions(p)
    count, idx = _table(ora, n * n)
    assert count.max() == 32 if (n == 23 and pose != "even") else count.max() >= 8  # the scene is what it says
    ora.update_positions(p)
    ora.step(1, 1)
    want, counters = ora.download_positions(), ora.read_buffer(13, np.uint64, 38)
    for lanes in LANES:
        gpu = NativeXpbdSolver(sc.cloth, sc.options, sc.static_triangles)
        gpu.set_launch_config({"neighbor_lanes": lanes})
        gpu.update_positions(p)
        c, i = _table(gpu, n * n)
        assert np.array_equal(c, count) and np.array_equal(i, idx), lanes
        gpu.update_positions(p)
        gpu.step(1, 1, diagnostics=True)
        assert np.array_equal(gpu.download_positions(), want), lanes
        got = gpu.read_buffer(13, np.uint64, 38)
        assert np.array_equal(got, counters), (lanes, np.flatnonzero(got != counters))
        gpu.close()


@pytest.mark.parametrize("lanes", LANES)
def test_cloths_that_share_a_warp(lanes, gpu_lib, oracle_lib):
    sizes, modes = (12, 13, 12, 17), (2, 1, 2, 2)
    scs = [_scene(n, m) for n, m in zip(sizes, modes)]
    for k, sc in enumerate(scs):
        sc.options.cloth_thickness *= 1.0 + 0.25 * k  # their own cell sizes
    batch = NativeXpbdBatch([(s.cloth, s.options, s.static_triangles) for s in scs])
    batch.set_launch_config({"neighbor_lanes": lanes})
    oras = [oracle_lib.OracleSolver.from_scene(s.cloth, s.options, s.static_triangles) for s in scs]
    for k, n in enumerate(sizes):
        p = _positions(n, "uneven", 50 + k)
        batch.update_cloth_positions(k, p)
        oras[k].update_positions(p)
    batch.step(2, 1, diagnostics=True)
    for k, o in enumerate(oras):
        o.step(2, 1)
        assert np.array_equal(batch.download_cloth_positions(k), o.download_positions()), k
    counters = sum(o.read_buffer(13, np.uint64, 38) for o in oras)
    assert np.array_equal(batch.read_buffer(13, np.uint64, 38), counters)
