"""The projector's wide float32 volumes at the borders of their own rules: scans of far apart views
that go by samples where a cell holds few, in tiles of 4 views x 4 rows (remainders of both, and
fewer rows than a tile has), the same tiles without copies at every step; against the float64
oracle, within the bounds of the walk by cells."""
import pytest

from test_gpu_cell_walk import test_projection_by_cells_matches_the_sum_over_samples as project

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nv", [1, 2, 5])
@pytest.mark.parametrize("n,views,step", [(255, 9, 1.09), (256, 9, 1.08), (256, 9, 1.09), (257, 7, 2.1), (257, 258, 1.09),
                                          (257, 6, 0.36), (257, 6, 0.37), (257, 4, 0.1)])
def test_wide_walks(n, views, step, nv, cuda):
    project(n, 6, 17, nv, views, step, "f32", True, cuda)
