"""Device preprocessing where its joint lists change hands: both halves of a
list scanned in one go at the edges of a scan tile (2 V at and around 4,096
and 8,192), a single triangle, unused vertices, no bend output asked for, and
the first of several bad indices reported."""
import ctypes

import numpy as np
import pytest

from xpbd_gb300 import scene

pytestmark = pytest.mark.gpu


def _strip(v, unused):
    """A triangle strip over v vertices, `unused` more after it; every fifth
    triangle listed twice with the other winding."""
    rng = np.random.default_rng(v)
    pos = rng.normal(0.0, 0.3, (v + unused, 3)).astype(np.float32)
    i = np.arange(v - 2, dtype=np.int32)
    tris = np.stack([i, i + 1, i + 2], 1)
    tris = np.concatenate([tris, tris[::5, ::-1]])
    return pos, np.ascontiguousarray(tris[rng.permutation(len(tris))])


def _bits(a):
    return np.ascontiguousarray(a).view(np.uint8).tobytes()


@pytest.mark.parametrize("v,unused", [(3, 0), (4, 1), (2047, 0), (2048, 0), (2049, 0), (2040, 8), (4096, 0), (4099, 1000)])
def test_joint_lists_at_scan_tile_edges(v, unused, gpu_lib):
    pos, tris = _strip(v, unused)
    hard = np.zeros(len(pos), bool)
    hard[::7] = True
    e_ref, r_ref = scene.edge_constraints(tris, pos)
    inv_ref = scene.vertex_inverse_mass(pos, tris, 0.2, hard).astype(np.float32)
    b_ref, br_ref = scene.bend_constraints(tris, pos)
    e, r, inv, b, br = scene.cloth_inputs_device(pos, tris, 0.2, hard)
    assert e.shape == (len(e_ref), 2) and b.shape == (len(b_ref), 2)
    assert _bits(e) == _bits(e_ref.astype(np.int32)) and _bits(r) == _bits(r_ref.astype(np.float32))
    assert _bits(inv) == _bits(inv_ref)
    assert _bits(b) == _bits(b_ref.astype(np.int32)) and _bits(br) == _bits(br_ref.astype(np.float32))


def test_without_bends_and_without_triangles(gpu_lib):
    pos, tris = _strip(100, 3)
    e_ref, r_ref = scene.edge_constraints(tris, pos)
    lib = scene._native_prep()
    pf, pi = ctypes.POINTER(ctypes.c_float), ctypes.POINTER(ctypes.c_int)
    edges, rest = np.empty((3 * len(tris), 2), np.int32), np.empty(3 * len(tris), np.float32)
    inv = np.empty(len(pos), np.float32)
    args = (0.2, 1.0e-7, None, edges.ctypes.data_as(pi), rest.ctypes.data_as(pf), inv.ctypes.data_as(pf), None, None, None)
    n = lib.xpbd_gb300_prepare_cloth_device(pos.ctypes.data_as(pf), len(pos), tris.ctypes.data_as(pi), len(tris), *args)
    assert n == len(e_ref)
    assert _bits(edges[:n]) == _bits(e_ref.astype(np.int32)) and _bits(rest[:n]) == _bits(r_ref.astype(np.float32))
    n = lib.xpbd_gb300_prepare_cloth_device(pos.ctypes.data_as(pf), len(pos), tris.ctypes.data_as(pi), 0, *args)
    assert n == 0 and (inv == 1.0).all()
    e, r, inv, b, br = scene.cloth_inputs_device(pos, np.empty((0, 3), np.int32), 0.2, np.zeros(len(pos), bool))
    assert e.shape == (0, 2) and b.shape == (0, 2) and len(r) == len(br) == 0 and (inv == 1.0).all()


@pytest.mark.parametrize("first", [0, 1, 2, 298, 401])
def test_first_bad_index_is_reported(first, gpu_lib):
    pos, tris = _strip(200, 0)
    tris = tris.copy()
    flat = tris.reshape(-1)
    flat[first:][::11] = -5
    flat[first] = 777
    with pytest.raises(RuntimeError, match="triangle index 777 outside the 200 vertices"):
        scene.cloth_inputs_device(pos, tris, 0.2, np.zeros(len(pos), bool))
    with pytest.raises(RuntimeError, match="triangle index 777 outside the 0 vertices"):
        flat[0] = 777
        scene.cloth_inputs_device(np.empty((0, 3), np.float32), tris, 0.2, np.zeros(0, bool))
