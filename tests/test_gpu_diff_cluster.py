"""The rollout and its adjoint run as one thread-block cluster for cloths of up
to 12,288 vertices (1 to 16 CTAs, up to 384 or 768 vertices each) and as
launched kernels for larger ones.  At the sizes where the shape changes the
forward must equal the solver bit for bit, and the gradients the launched
form's."""
import numpy as np
import pytest
import torch

from xpbd_gb300 import scene
from xpbd_gb300.diff import DiffCloth
from xpbd_gb300.native import NativeXpbdSolver

pytestmark = pytest.mark.gpu


# vertices: 4; 121 and 144 (one CTA, two); 2,025 and 2,116 (16 CTAs, the
# smallest share above 128); 6,084 and 6,241 (384 vertices per CTA, more);
# 12,100 and 12,321 (cluster, launched)
@pytest.mark.parametrize("n", [2, 11, 12, 45, 46, 78, 79, 110, 111])
def test_forward_equals_solver(n, gpu_lib):
    sc = scene.diff_scene(n, 2)
    dc = DiffCloth(sc.cloth, sc.options)
    ks = torch.full((len(sc.cloth.edges),), sc.options.stretch_compliance, dtype=torch.float32, device="cuda")
    kb = torch.full((len(sc.cloth.bends),), sc.options.bend_compliance, dtype=torch.float32, device="cuda")
    solver = NativeXpbdSolver(sc.cloth, sc.options, sc.static_triangles)
    for _ in range(2):
        solver.step(10, 2, diagnostics=False, synchronize=True)
    x = dc.rollout(ks, kb, 2, 10, 2)
    assert np.array_equal(x.cpu().numpy(), solver.download_positions())
    # the checkpoints are the states the launched form keeps
    first, last = dc.checkpoint(0).cpu().numpy(), dc.checkpoint(2).cpu().numpy()
    assert np.array_equal(first[0, :, :3], sc.cloth.positions_world) and np.array_equal(first[0], first[1])
    assert np.array_equal(last[0, :, :3], x.cpu().numpy())
    assert np.array_equal(last[0], solver.read_buffer(0, np.float32, 4 * n * n).reshape(-1, 4))
    assert np.array_equal(last[2], solver.read_buffer(2, np.float32, 4 * n * n).reshape(-1, 4))


def _with_padding(n):
    """The n x n cloth alone, and as the first part of a mesh with a separate
    112 x 112 cloth, which is too large for the cluster form: the same
    vertices, constraints and constraint order for the first part."""
    pos, tris = scene.grid_mesh(n, 1.0, 0.0)
    w = np.zeros(len(pos), np.float32)
    w[(n - 1) * n] = w[n * n - 1] = 1.0
    pad, pad_tris = scene.grid_mesh(112, 1.0, 5.0)
    alone = scene.build_cloth(pos, tris, 0.2, w)
    both = scene.build_cloth(np.concatenate([pos, pad]), np.concatenate([tris, pad_tris + len(pos)]), 0.2,
                             np.concatenate([w, np.zeros(len(pad), np.float32)]))
    return alone, both


@pytest.mark.parametrize("n,substeps,iterations", [(2, 10, 2), (11, 1, 1), (12, 3, 1), (12, 2, 3), (45, 4, 2), (46, 4, 2), (78, 3, 2),
                                                   (79, 3, 2), (110, 2, 2)])
def test_gradients_equal_launched_form(n, substeps, iterations, gpu_lib):
    """Same arithmetic in the same order: the cluster form's positions and
    gradients are the launched form's bit for bit."""
    options = scene.diff_scene(4, 1).options
    alone, both = _with_padding(n)
    rng = np.random.default_rng(n)
    g = rng.normal(size=alone.positions_world.shape).astype(np.float32)
    got = []
    for cloth in (alone, both):
        V = n * n
        res = []
        fields = []
        for pairs, seed in ((cloth.edges, 5), (cloth.bends, 6)):
            # a value per vertex pair, the same in both meshes; every seventh is rigid
            mine = (pairs < V).all(axis=1)
            key = np.where(mine, pairs[:, 0].astype(np.int64) * V + pairs[:, 1], 0)
            unit = ((key * 2654435761 + seed) % 1000003) / 1000003.0
            k = (3e-3 * 10.0 ** (2.0 * unit - 1.0)).astype(np.float32)
            k[key % 7 == 3] = 0.0
            fields.append((torch.tensor(k, device="cuda"), mine, key))
        grad = np.zeros((len(cloth.positions_world), 3), np.float32)
        grad[:V] = g
        dc = DiffCloth(cloth, options)
        x = dc.rollout(fields[0][0], fields[1][0], 3, substeps, iterations)
        gs, gb = dc.backward(torch.tensor(grad, device="cuda"))
        res.append(x.cpu().numpy()[:V])
        for values, (_, mine, key) in zip((gs, gb), fields):
            order = np.argsort(key[mine], kind="stable")
            res.append(values.cpu().numpy()[mine][order])
        got.append(res)
    for a, b in zip(*got):
        assert a.shape == b.shape and np.array_equal(a, b)
    assert np.abs(got[0][1]).max() > 0.0
