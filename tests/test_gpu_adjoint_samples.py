"""The adjoint on both sides of the rules that choose its walk, by cells or by samples: the sample
count per cell, small grids, the image's width and the detector's, against the float64 oracle
within the bounds of the walk by cells."""
import pytest

from test_gpu_adjoint_walk import test_adjoint_by_cells_matches_the_sum_over_samples as adjoint

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,nz,nu,nv,views,step,cone", [
    # grids of fewer than 4000 and 60000 rays, and more
    (33, 7, 40, 7, 12, 0.27, True), (33, 7, 40, 7, 15, 0.27, True), (33, 7, 40, 7, 15, 0.37, True),
    (33, 7, 60, 33, 30, 0.37, True), (33, 7, 64, 33, 30, 0.37, True),
    # wide grids by image width and step
    (31, 9, 64, 33, 30, 0.3, True), (63, 9, 64, 33, 30, 0.37, True), (64, 9, 64, 33, 30, 0.72, True),
    (64, 9, 64, 33, 30, 0.73, True), (111, 5, 64, 33, 30, 0.8, True), (112, 5, 140, 33, 13, 1.2, True),
    (112, 5, 141, 33, 13, 1.2, True), (64, 9, 64, 33, 30, 0.96, True), (64, 9, 64, 33, 30, 0.97, True),
    (34, 9, 128, 9, 36, 0.45, False), (34, 9, 128, 9, 60, 1.5, False), (34, 3, 37, 3, 30, 0.6, False)])
def test_adjoint_walks(n, nz, nu, nv, views, step, cone, cuda):
    adjoint(n, nz, nu, nv, views, step, cone, cuda)
