"""The projector's ray tiles and walks at the borders of the rules that choose them: scans that
leave much of a tile of 16 views x 1 row (16-bit cells: 4 x 4) outside, walks by samples in
tiles of 8 views (fan beam and without copies too), and wide volumes whose long scans go by
samples and short ones in windows; against the float64 oracle, within the bounds of the walk
by cells."""
import pytest

from test_gpu_cell_walk import test_projection_by_cells_matches_the_sum_over_samples as project

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,nz,nu,nv,views,step,storage,cone", [
    # views and rows outside the tile: 8 x 2 and 4 x 4 instead of 16 x 1, 16 x 1 instead of 4 x 4
    (34, 8, 37, 16, 23, 0.2, "f32", True), (34, 8, 37, 16, 9, 0.2, "f32", True), (34, 8, 37, 15, 5, 0.2, "f32", True),
    (34, 6, 37, 2, 33, 0.2, "bf16", True), (34, 6, 37, 1, 32, 0.2, "f16", True), (34, 6, 37, 5, 33, 0.2, "bf16", True),
    (34, 17, 37, 17, 23, 0.3, "f32", False), (34, 16, 37, 16, 4, 0.3, "f32", False),
    # by samples: both sides of the sample count, views around the tile's 8
    (40, 8, 35, 9, 7, 0.5, "f32", True), (40, 8, 35, 9, 41, 0.8, "f32", True), (33, 5, 40, 7, 24, 0.36, "f32", True),
    (40, 8, 17, 9, 17, 0.28, "f16", True), (255, 6, 17, 3, 5, 0.3, "f16", True), (256, 6, 17, 3, 5, 0.3, "f16", True),
    (40, 8, 17, 9, 17, 0.29, "bf16", True), (40, 8, 17, 2, 9, 0.8, "bf16", True),
    (34, 3, 37, 3, 30, 0.44, "f32", False), (34, 3, 37, 3, 30, 0.45, "f32", False), (260, 2, 41, 2, 9, 0.5, "f32", False),
    (34, 9, 17, 9, 9, 1.7, "f32", False),
    # wide volumes: long scans between 0.6 and 1.2 samples a cell by samples
    (256, 6, 17, 3, 255, 0.5, "f32", True), (256, 6, 17, 3, 256, 0.5, "f32", True), (257, 6, 9, 2, 257, 0.36, "f32", True),
    (257, 6, 9, 2, 257, 0.37, "f32", True), (257, 6, 9, 2, 257, 0.72, "f32", True), (257, 6, 9, 2, 257, 0.73, "f32", True)])
def test_ray_tiles(n, nz, nu, nv, views, step, storage, cone, cuda):
    project(n, nz, nu, nv, views, step, storage, cone, cuda)
