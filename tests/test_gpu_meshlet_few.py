"""The meshlet split's steps of ten triangles (limits of few triangles or few
vertices a meshlet) on the index lists of test_gpu_meshlet_steps: limits at the
step's size, one past it, and few vertices with many triangles, which only
triangles that repeat a vertex reach over several steps."""
import pytest

import test_gpu_meshlet_steps as steps

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("limits", [(64, 1), (4, 2), (30, 9), (64, 10), (29, 10), (8, 11), (3, 126), (8, 1024), (7, 20)])
@pytest.mark.parametrize("kind", ["strip", "repeats", "spread", "stride", "one"])
def test_few_triangles_match_oracle(ctx, oracle, kind, limits):
    steps.test_meshlet_steps_match_oracle(ctx, oracle, kind, limits)
