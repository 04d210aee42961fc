"""The adjoint's workspace as one place per cell (by samples) and as faces (by cells), on both sides
of the rule between them, where a voxel's sum could miss one of its 8 cells: volumes of few planes
and of few columns, and odd sizes; against the float64 oracle within the bounds of the walk by cells."""
import pytest

from test_gpu_adjoint_walk import test_adjoint_by_cells_matches_the_sum_over_samples as adjoint

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,nz,nu,nv,views,step", [
    (63, 9, 64, 33, 30, 0.72), (63, 9, 64, 33, 30, 0.73), (64, 9, 64, 33, 30, 0.73), (64, 9, 64, 33, 30, 1.08),
    (64, 9, 64, 33, 30, 1.09), (65, 3, 64, 33, 30, 1.3), (3, 40, 33, 37, 60, 1.9), (130, 6, 97, 7, 9, 0.5)])
def test_sums_by_cell(n, nz, nu, nv, views, step, cuda):
    adjoint(n, nz, nu, nv, views, step, True, cuda)
