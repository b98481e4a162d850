"""Frames with self collision ask for one share of L1 as shared memory, launch
by launch where other frames use the same kernels: making such a solver leaves
the launched passes' own preference as it was, and a plain solver's frames as
they were."""
import ctypes

import numpy as np
import pytest

from xpbd_gb300 import scene
from xpbd_gb300.native import NativeXpbdSolver

pytestmark = pytest.mark.gpu


def test_other_solvers_kernels_keep_their_preference(gpu_lib):
    sc = scene.plain_grid_scene(120, 1)
    plain = NativeXpbdSolver(sc.cloth, sc.options, sc.static_triangles)
    plain.step(10, 2)
    want = plain.download_positions().copy()
    share = plain._lib.xpbd_gb300_pass_carveout
    share.restype = ctypes.c_int
    assert share() == -1
    drop = scene.drop_scene(24, 1)
    strict = NativeXpbdSolver(drop.cloth, drop.options, drop.static_triangles)
    strict.step(10, 2)
    assert share() == -1
    plain.reset()
    plain.step(10, 2)
    assert np.array_equal(plain.download_positions(), want)
    strict.close()
    plain.close()
