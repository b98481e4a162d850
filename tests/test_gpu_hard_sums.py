"""Sums of the hard-stretch solve's cluster form where some of its warps hold
no vertex: solves without caps always take 16 CTAs, so small cloths leave
whole CTAs without one, and in a batch the largest cloth decides how many
warps a CTA has.  Positions and counters equal the oracle's, and a
batch's cloths their own solvers'."""
import numpy as np
import pytest

from xpbd_gb300 import scene
from xpbd_gb300.native import NativeXpbdBatch, NativeXpbdSolver

pytestmark = pytest.mark.gpu


# 25 vertices in one of 16 CTAs; 144 and 256 in 5 and 8; 289 in 10; 529 in 9 of
# two warps each; 1,089 in 12 of three
@pytest.mark.parametrize("n", [5, 12, 16, 17, 23, 33])
@pytest.mark.parametrize("hardness", [0.4, 0.7])
def test_ctas_without_vertices(n, hardness, gpu_lib, oracle_lib):
    sc = scene.hardness_grid_scene(n, hardness, 3)
    gpu = NativeXpbdSolver(sc.cloth, sc.options, sc.static_triangles)
    ora = oracle_lib.OracleSolver.from_scene(sc.cloth, sc.options, sc.static_triangles)
    for f in range(3):
        gpu.step(sc.substeps, sc.iterations, diagnostics=True)
        ora.step(sc.substeps, sc.iterations)
        assert np.array_equal(gpu.download_positions(), ora.download_positions()), f
        assert np.array_equal(gpu.read_buffer(13, np.uint64, 38), ora.read_buffer(13, np.uint64, 38)), f
    gpu.close()


@pytest.mark.parametrize("sizes", [(2, 12, 101, 5), (140, 2, 33, 17), (24,) * 9 + (3, 60)])
def test_uneven_batches(sizes, gpu_lib):
    scs = [scene.hardness_grid_scene(n, 0.4, 2) for n in sizes]
    batch = NativeXpbdBatch([(s.cloth, s.options, s.static_triangles) for s in scs])
    for _ in range(3):
        batch.step(10, 2)
    for k, s in enumerate(scs):
        solo = NativeXpbdSolver(s.cloth, s.options, s.static_triangles)
        for _ in range(3):
            solo.step(10, 2)
        assert np.array_equal(batch.download_cloth_positions(k), solo.download_positions()), k
        solo.close()
    batch.close()
