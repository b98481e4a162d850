"""Bucket scans of more than 33,554,432 counts scan their blocks' sums in a
launch of their own.  Device preprocessing scans two counts per vertex: a mesh
whose few triangles lie scattered over 16,777,216 vertices (the largest of two
launches) and over one more."""
import numpy as np
import pytest

from xpbd_gb300 import scene

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("v", [1 << 24, (1 << 24) + 1])
def test_scattered_triangles(v, gpu_lib):
    rng = np.random.default_rng(v)
    used = np.unique(np.concatenate([[0, 1, v - 2, v - 1], rng.integers(0, v, 4000)]))
    corner = rng.integers(0, len(used), (6000, 3))
    corner = corner[(corner[:, 0] != corner[:, 1]) & (corner[:, 1] != corner[:, 2]) & (corner[:, 2] != corner[:, 0])]
    corner[0] = (0, 1, len(used) - 1)
    small = rng.normal(0.0, 0.3, (len(used), 3)).astype(np.float32)
    pos = np.zeros((v, 3), np.float32)
    pos[used] = small
    hard = np.zeros(v, bool)
    hard[used[::9]] = True
    # the same mesh without its unused vertices, by the host's builders
    e_ref, r_ref = scene.edge_constraints(corner.astype(np.int32), small)
    b_ref, br_ref = scene.bend_constraints(corner.astype(np.int32), small)
    inv_ref = scene.vertex_inverse_mass(small, corner.astype(np.int32), 0.2, hard[used]).astype(np.float32)
    e, r, inv, b, br = scene.cloth_inputs_device(pos, used[corner].astype(np.int32), 0.2, hard)
    assert np.array_equal(e, used[e_ref]) and np.array_equal(r, r_ref.astype(np.float32))
    assert np.array_equal(b, used[b_ref]) and np.array_equal(br, br_ref.astype(np.float32))
    assert np.array_equal(inv[used], inv_ref)
    rest = np.ones(v, bool)
    rest[used] = False
    assert (inv[rest] == 1.0).all()
