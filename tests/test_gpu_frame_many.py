"""The fused frame of more cloths than the GPU has SMs: blocks of as few
threads as let all cloths run at once, down to a thread per vertex.  Positions
and counters equal the launched form's bit for bit."""
import numpy as np
import pytest

from xpbd_gb300 import scene
from xpbd_gb300.native import NativeXpbdBatch

pytestmark = pytest.mark.gpu


# 155 of 8 x 8: an edge per thread; 1,000: fewer; 400 of 16 x 16: a thread per
# vertex, in waves; 160 of 24 x 24 and 30 x 30: the larger block
@pytest.mark.parametrize("sizes", [(8,) * 155, (2, 5, 8) * 333 + (8,), (16, 9) * 200, (24,) * 160, (30, 4) * 80])
def test_equal_launched_form(sizes, gpu_lib):
    made = {n: scene.plain_grid_scene(n, 2) for n in set(sizes)}
    items = [(made[n].cloth, made[n].options, made[n].static_triangles) for n in sizes]
    fused, launched = NativeXpbdBatch(items), NativeXpbdBatch(items)
    launched.set_launch_config({"fused_frame": 2})
    rng = np.random.default_rng(len(sizes))
    p = fused.download_positions().copy()
    p[:, 2] += rng.uniform(-1.0e-3, 1.0e-3, len(p)).astype(np.float32)
    for b in (fused, launched):
        b.update_positions(p)
    for substeps, iterations in ((10, 2), (3, 1)):
        for b in (fused, launched):
            b.step(substeps, iterations, diagnostics=True)
        assert np.array_equal(fused.download_positions(), launched.download_positions()), substeps
        assert np.array_equal(fused.read_buffer(13, np.uint64, 38), launched.read_buffer(13, np.uint64, 38)), substeps
    fused.close()
    launched.close()
