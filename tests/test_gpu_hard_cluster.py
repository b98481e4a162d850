"""The hard-stretch solve has a cluster form (one thread-block cluster of 1 to
16 CTAs per cloth, one, two or four vertices per thread) for solvers whose
solving cloths have at most 32,768 vertices each (20,480 without caps), and a
launched form for the others.  Positions and all counters must equal the
oracle's at the sizes where the form or its shape changes, with a caller's
edge colouring and without one, and with edges short enough for the tiny caps."""
import numpy as np
import pytest

from xpbd_gb300 import scene
from xpbd_gb300.native import NativeXpbdBatch, NativeXpbdSolver

pytestmark = pytest.mark.gpu


def _check(sc, frames, oracle_lib):
    gpu = NativeXpbdSolver(sc.cloth, sc.options, sc.static_triangles)
    ora = oracle_lib.OracleSolver.from_scene(sc.cloth, sc.options, sc.static_triangles)
    for f in range(frames):
        gpu.step(sc.substeps, sc.iterations, diagnostics=True)
        ora.step(sc.substeps, sc.iterations)
        assert np.array_equal(gpu.download_positions(), ora.download_positions()), f
        assert np.array_equal(gpu.read_buffer(13, np.uint64, 38), ora.read_buffer(13, np.uint64, 38)), f
    gpu.close()


# 625 and 676 vertices: one vertex per thread of one CTA, two; 1,024 and 1,089:
# one CTA, 16; 10,201 and 10,404: one vertex per thread, two; 16,384 and 16,641:
# two, four; 20,449 and 20,736: cluster, launched (no caps); 32,761 and 33,124:
# cluster, launched (caps)
@pytest.mark.parametrize("n", [2, 25, 26, 32, 33, 101, 102, 128, 129, 143, 144, 181, 182])
@pytest.mark.parametrize("hardness", [0.4, 1.0])
def test_sizes(n, hardness, gpu_lib, oracle_lib):
    _check(scene.hardness_grid_scene(n, hardness, 1), 2 if n < 100 else 1, oracle_lib)


@pytest.mark.parametrize("n,side,colours", [(33, 0.02, True), (33, 0.02, False), (40, 1.0, False), (40, 0.03, True)])
def test_caps(n, side, colours, gpu_lib, oracle_lib):
    """0.02 m over 33 vertices: sides of 0.625 mm (tiny caps) and diagonals of
    0.88 mm (normal caps) in one cloth."""
    sc = scene.hardness_grid_scene(n, 1.0, 3)
    pos, tris = scene.grid_mesh(n, side, 0.0)
    w = np.zeros(n * n, np.float32)
    w[sc.cloth.pin_indices] = 1.0
    sc.cloth = scene.build_cloth(pos, tris, 0.2, w, tether_slack=1.0)
    if not colours:
        sc.cloth.edge_color_offsets = np.asarray([0], np.int32)
    sc.options.gravity = (0.0, 0.0, -60.0)
    _check(sc, 3, oracle_lib)


def test_batch_of_sizes(gpu_lib):
    """Cloths of a batch share the largest one's cluster size; each equals its
    own solver."""
    scs = [scene.hardness_grid_scene(n, h, 2) for n, h in ((8, 1.0), (40, 0.4), (70, 1.0), (33, 1.0))]
    scs.append(scene.plain_grid_scene(20, 2))
    batch = NativeXpbdBatch([(s.cloth, s.options, s.static_triangles) for s in scs])
    for _ in range(2):
        batch.step(10, 2)
    for k, s in enumerate(scs):
        solo = NativeXpbdSolver(s.cloth, s.options, s.static_triangles)
        for _ in range(2):
            solo.step(10, 2)
        assert np.array_equal(batch.download_cloth_positions(k), solo.download_positions()), k
        solo.close()
    batch.close()
