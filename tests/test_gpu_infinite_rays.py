"""The adjoint of a sinogram that holds infinite values (a detector element that saw nothing): a
voxel that such a ray gives a weight is infinite, the others are as without the ray."""
import numpy as np
import pytest

from test_gpu_nonfinite_geometry import _scan

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("workspace", [True, None])
@pytest.mark.parametrize("cone,step", [(True, 0.2), (True, 0.9), (False, 0.2), (False, 0.9)])
def test_an_infinite_ray_gives_infinite_voxels(cone, step, workspace, cuda):
    import torch
    from reconstruction_program_taichi_gb300 import ops
    dg = _scan(cone, step)
    y = torch.zeros(dg.sgm_shape, device="cuda")
    for row, view, col in ((2, 3, 17), (1, 9, 11), (0, 14, 25)):
        y[row, view, col] = 1.0
    one = ops.fp_adjoint(dg, y, workspace=workspace)
    got = ops.fp_adjoint(dg, torch.where(y > 0, float("inf"), 0.0), workspace=workspace)
    # weights far above rounding, and voxels without a neighbour that has one (a sample within
    # rounding of a face may be taken from the cell on its other side)
    hit = one > 1e-3
    away = torch.nn.functional.max_pool3d(one.abs()[None], 3, 1, 1)[0] == 0
    assert hit.sum() > 50 and away.any()
    assert (got[hit] == np.inf).all()
    assert (got[away] == 0).all()
