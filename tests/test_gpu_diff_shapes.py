"""The rollout's cluster form runs in blocks of 512 threads up to 512 vertices
per CTA (8,100 vertices on 16 CTAs) and of 768 beyond (8,281): forward and
gradients on both sides."""
import pytest

import test_gpu_diff_cluster as shapes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [90, 91])
def test_forward_equals_solver(n, gpu_lib):
    shapes.test_forward_equals_solver(n, gpu_lib)


@pytest.mark.parametrize("n,substeps,iterations", [(90, 3, 2), (91, 3, 2)])
def test_gradients_equal_launched_form(n, substeps, iterations, gpu_lib):
    shapes.test_gradients_equal_launched_form(n, substeps, iterations, gpu_lib)
