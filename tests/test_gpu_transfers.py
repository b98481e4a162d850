"""Positions and pins in and out, where the way they travel changes: up to
64 KB (5,461 vertices) through page-locked memory that a kernel reads or
writes, beyond by a copy; up to 128 pin changes as kernel arguments, beyond by
a staging copy; whole batches in the caller's order of the cloths in either."""
import numpy as np
import pytest

from xpbd_gb300 import scene
from xpbd_gb300.native import NativeXpbdBatch, NativeXpbdSolver

pytestmark = pytest.mark.gpu


def _strip(v, mode=0):
    i = np.arange(v - 2, dtype=np.int32)
    k = np.arange(v)
    pos = np.stack([0.01 * (k // 2), 0.01 * (k % 2), np.zeros(v)], 1).astype(np.float32)
    w = np.zeros(v, np.float32)
    w[0] = 1.0
    cloth = scene.build_cloth(pos, np.stack([i, i + 1, i + 2], 1), 0.2, w)
    opt = scene.SolverOptions(dt=1.0 / 60.0, use_ground=False)
    if mode:
        opt.self_collision, opt.self_collision_mode, opt.cloth_thickness = True, mode, 0.002
    return cloth, opt, np.empty((0, 3, 3), np.float32)


def _rows(s, buf, n):
    return s.read_buffer(buf, np.float32, 4 * n).reshape(-1, 4)


@pytest.mark.parametrize("v", [3, 256, 257, 5461, 5462, 9000])
def test_positions_round_trip(v, gpu_lib):
    item = _strip(v)
    s = NativeXpbdSolver(*item)
    rest = _rows(s, 0, v)
    rng = np.random.default_rng(v)
    for _ in range(2):
        p = rng.normal(0.0, 1.0, (v, 3)).astype(np.float32)
        s.update_positions(p)
        assert np.array_equal(s.download_positions(), p)
        for buf in (0, 1):
            got = _rows(s, buf, v)
            assert np.array_equal(got[:, :3], p) and np.array_equal(got[:, 3], rest[:, 3])
    s.step(2, 1, diagnostics=True)
    assert np.abs(_rows(s, 2, v)[:, :3]).max() > 0.0
    s.reset()
    assert np.array_equal(s.download_positions(), rest[:, :3])
    assert np.array_equal(_rows(s, 0, v), rest) and np.array_equal(_rows(s, 1, v), rest)
    assert not _rows(s, 2, v).any() and not s.read_buffer(13, np.uint64, 38).any()


@pytest.mark.parametrize("sizes", [(40, 300, 17), (3000, 2461, 1), (4000, 900, 2000)])
def test_batch_in_the_callers_order(sizes, gpu_lib):
    sizes = [max(v, 3) for v in sizes]
    batch = NativeXpbdBatch([_strip(v, mode) for v, mode in zip(sizes, (2, 0, 1))])  # stored as 0, 1, 2
    rng = np.random.default_rng(sum(sizes))
    p = rng.normal(0.0, 1.0, (sum(sizes), 3)).astype(np.float32)
    at = np.concatenate([[0], np.cumsum(sizes)])
    batch.update_positions(p)
    assert np.array_equal(batch.download_positions(), p)
    p = p[::-1].copy()
    for k in range(3):
        batch.update_cloth_positions(k, p[at[k]:at[k + 1]])
        assert np.array_equal(batch.download_cloth_positions(k), p[at[k]:at[k + 1]])
    assert np.array_equal(batch.download_positions(), p)


@pytest.mark.parametrize("pins", [1, 2, 127, 128, 129, 131, 400])
def test_pin_updates(pins, gpu_lib, oracle_lib):
    item = _strip(600)
    gpu, ora = NativeXpbdSolver(*item), oracle_lib.OracleSolver.from_scene(*item)
    rng = np.random.default_rng(pins)
    for f in range(3):
        # the changes are the pins cleared and the pins set: `pins` of them in all
        new = rng.permutation(np.arange(1, 600))[: pins if f == 0 else pins // 2].astype(np.int32)
        if len(new):
            new[-1] = new[0]  # a vertex listed twice keeps its last entry
        to = (item[0].positions_world[new] + rng.uniform(-0.01, 0.01, (len(new), 3))).astype(np.float32)
        w = rng.choice(np.float32([0.3, 0.7, 1.0]), len(new)).astype(np.float32)
        for s in (gpu, ora):
            s.update_pin_targets(new, to, w)
            s.step(4, 2)
        assert np.array_equal(gpu.download_positions(), ora.download_positions()), f


@pytest.mark.parametrize("sizes", [[1365] * 9, [5461, 40, 5461], [300] * 40])
def test_uploads_one_after_another(sizes, gpu_lib):
    """More small uploads than the page-locked memory holds at once, each from
    a buffer that is overwritten as soon as the call returns."""
    batch = NativeXpbdBatch([_strip(v) for v in sizes])
    rng = np.random.default_rng(len(sizes))
    at = np.concatenate([[0], np.cumsum(sizes)])
    for _ in range(3):
        want = rng.normal(0.0, 1.0, (at[-1], 3)).astype(np.float32)
        for k in range(len(sizes)):
            p = want[at[k]:at[k + 1]].copy()
            batch.update_cloth_positions(k, p)
            p[:] = np.nan
        assert np.array_equal(batch.download_positions(), want)
        assert np.array_equal(_rows(batch, 1, at[-1])[:, :3], want)
