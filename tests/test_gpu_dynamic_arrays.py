"""A dynamic collider upload has read the caller's arrays when it returns, also
where frames are still queued before it: the arrays are overwritten at once,
and the frames after it equal those of a solver whose arrays were left alone.
Page-locked arrays too, which an asynchronous copy reads late.  Sizes on both
sides of the hashes (64) and of what the solver copies at once (1 MB)."""
import numpy as np
import pytest
import torch

from xpbd_gb300 import scene
from xpbd_gb300.native import NativeXpbdSolver

pytestmark = pytest.mark.gpu


def _array(a, locked):
    if not locked:
        return a.copy()
    t = torch.empty(a.shape, dtype=torch.from_numpy(a).dtype, pin_memory=True)
    t.numpy()[:] = a
    return t.numpy()


def _inputs(kind, count, f):
    rng = np.random.default_rng(count + f)
    if kind == "particles":
        pos = rng.uniform((-0.5, -0.5, -0.06), (0.5, 0.5, -0.01), (count, 3)).astype(np.float32)
        return {"particles": [pos, rng.uniform(0.01, 0.02, count).astype(np.float32)]}
    if kind == "indexed":
        v, t = scene.icosphere((0.0, 0.0, -0.16 + 0.01 * f), 0.15, {20: 0, 1280: 3, 5120: 4}[count])
        return {"indexed": [np.asarray(v, np.float32), np.asarray(t, np.int32), f == 0]}
    at = rng.uniform((-0.5, -0.5, -0.03), (0.5, 0.5, -0.01), (count, 1, 3))
    return {"triangles": [(at + rng.uniform(-0.02, 0.02, (count, 3, 3))).astype(np.float32)]}


@pytest.mark.parametrize("locked", [False, True])
@pytest.mark.parametrize("kind,count", [("particles", 40), ("particles", 500), ("particles", 9000), ("indexed", 20),
                                        ("indexed", 1280), ("indexed", 5120), ("triangles", 40), ("triangles", 700),
                                        ("triangles", 24000)])
def test_arrays_may_change_after_the_call(kind, count, locked, gpu_lib):
    pos, tris = scene.grid_mesh(48, 1.0, 0.0)
    cloth = scene.build_cloth(pos, tris, 0.2, np.zeros(48 * 48, np.float32))
    opt = scene.SolverOptions(dt=1.0 / 60.0, cloth_thickness=0.002, collision_margin=0.005, contact_friction=0.2)
    a, b = (NativeXpbdSolver(cloth, opt, np.empty((0, 3, 3), np.float32)) for _ in range(2))
    moved = False
    for f in range(3):
        given = _inputs(kind, count, f)
        (key, arrays), = given.items()
        mine = [_array(x, locked) if isinstance(x, np.ndarray) else x for x in arrays]
        call = lambda s, x: s.update_dynamic_colliders(**{key: x[0] if key == "triangles" else tuple(x)})
        for s in (a, b):  # frames queued before the upload
            for _ in range(4):
                s.step(10, 2, diagnostics=False, synchronize=False)
        call(a, mine)
        for x in mine:  # valid, but other, colliders
            if isinstance(x, np.ndarray):
                x[:] = x[::-1].copy() if x.dtype == np.int32 else x * np.float32(0.5)
        call(b, arrays)
        b.synchronize()
        for s in (a, b):
            s.step(10, 2, diagnostics=True)
        assert np.array_equal(a.download_positions(), b.download_positions()), f
        moved |= a.diagnostics()["candidate_count"] > 0
    assert moved
    a.close()
    b.close()
