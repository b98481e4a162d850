"""A frame whose cluster barrier gave up is an error of the calls that wait for
it, hand its state out or go on from it, until the whole solver is reset.  The
kernels report through a word of host memory; here the host sets it."""
import numpy as np
import pytest

from xpbd_gb300 import scene
from xpbd_gb300.native import NativeSolverError, NativeXpbdBatch, NativeXpbdSolver

pytestmark = pytest.mark.gpu


def _scene(kind):
    if kind == "plain":
        return scene.plain_grid_scene(32, 2)
    return scene.hardness_grid_scene(20, 1.0 if kind == "caps" else 0.4, 2)


def _calls(s):
    yield lambda: s.step(2, 1, diagnostics=False, synchronize=False)
    yield lambda: s.step(2, 1, diagnostics=True)
    yield s.synchronize
    yield s.download_positions
    yield lambda: s.read_buffer(0, np.float32, 4096)


@pytest.mark.parametrize("kind", ["plain", "caps", "solve", "batch"])
def test_reported_until_reset(kind, gpu_lib):
    if kind == "batch":
        scs = [scene.plain_grid_scene(n, 2) for n in (8, 20)]
        s = NativeXpbdBatch([(x.cloth, x.options, x.static_triangles) for x in scs])
    else:
        sc = _scene(kind)
        s = NativeXpbdSolver(sc.cloth, sc.options, sc.static_triangles)
    word = s._lib.xpbd_gb300_barrier_word(s._handle)
    assert word
    s.step(10, 2)
    want = s.download_positions().copy()
    assert word[0] == 0
    for call in _calls(s):
        word[0] = 1
        with pytest.raises(NativeSolverError, match="timed out"):
            call()
        assert word[0] == 1
    if kind == "batch":  # the other cloths' state is as undefined as before
        s.reset_cloth(0)
        assert word[0] == 1
    s.reset()
    assert word[0] == 0
    s.step(10, 2)
    assert np.array_equal(s.download_positions(), want)
    s.close()


def test_no_cluster_form_no_word(gpu_lib):
    sc = scene.drop_scene(24, 2)
    s = NativeXpbdSolver(sc.cloth, sc.options, sc.static_triangles)
    assert not s._lib.xpbd_gb300_barrier_word(s._handle)
    s.close()
