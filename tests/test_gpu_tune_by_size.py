"""Lanes of the neighbour table are chosen by size, for the fast cloths and for
the strict ones: the launch configuration reports what an untuned frame uses,
and setting another slot, or tuning, starts from there."""
import pytest

from xpbd_gb300 import scene
from xpbd_gb300.native import NativeXpbdBatch

pytestmark = pytest.mark.gpu


def _batch(*cloths):
    scs = [scene.drop_scene(n, 1, self_mode=mode) for n, mode in cloths]
    return NativeXpbdBatch([(s.cloth, s.options, s.static_triangles) for s in scs])


def _lanes(b):
    return b.launch_config()["neighbor_lanes"]


@pytest.mark.parametrize("n", [24, 100, 160, 240])
def test_fast_cloths_report_their_own_size(n, gpu_lib):
    fast, strict = _batch((n, 1)), _batch((n, 2))
    assert _lanes(fast) == _lanes(strict) > 0
    for b in (fast, strict):
        b.close()


def test_mixed_batch_stays_by_size(gpu_lib):
    b = _batch((24, 1), (240, 2))
    assert _lanes(b) == 0
    b.set_launch_config({"vertex_block": 64})
    assert _lanes(b) == 0 and b.launch_config()["vertex_block"] == 64
    b.set_launch_config({"neighbor_lanes": 2})
    assert _lanes(b) == 2
    b.close()


def test_a_set_value_is_reported(gpu_lib):
    sc = scene.plain_grid_scene(8, 1)
    b = NativeXpbdBatch([(sc.cloth, sc.options, sc.static_triangles)])
    b.set_launch_config({"neighbor_lanes": 4})
    assert _lanes(b) == 4
    b.close()
