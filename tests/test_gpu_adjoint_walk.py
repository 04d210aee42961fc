"""The adjoint's walk by cells against the float64 oracle's transpose of its sum over samples,
where the two could part: steps that leave many samples or none in a cell (and so cross faces
one at a time or several at once), volumes of few cells along an axis, rays of all octants,
rows and columns that do not fill the blocks of rays, fan beam, and both places the corner
sums go to (face buffers, or straight into the volume)."""
import numpy as np
import pytest

from conftest import rel_l2
from oracle import fpj_ops as P
from test_gpu_parity import _cone_obj

pytestmark = pytest.mark.gpu

# float32 sample positions are within 3 * 2^-24 * n (2.3e-5 voxel at n = 130) of the float64
# ones and enter a weight of 0.35 on average: 7e-5.  Compared off the faces, where a sample
# whose inside test flips has no weight.
TOL = 1e-4


@pytest.mark.parametrize("n,nz,nu,nv,views,step,cone", [
    (32, 9, 40, 11, 24, 0.05, True), (32, 9, 40, 11, 24, 0.9, True), (33, 5, 40, 7, 24, 2.5, True),
    (17, 40, 33, 37, 24, 0.2, True), (64, 3, 65, 3, 40, 0.2, True), (3, 3, 31, 5, 24, 0.1, True),
    (4, 17, 9, 4, 24, 0.7, True), (130, 6, 97, 1, 9, 0.2, True),
    (34, 3, 37, 3, 30, 0.2, False), (33, 1, 65, 1, 30, 1.7, False), (3, 2, 33, 2, 30, 0.05, False)])
def test_adjoint_by_cells_matches_the_sum_over_samples(n, nz, nu, nv, views, step, cone, cuda):
    import torch
    from reconstruction_program_taichi_gb300 import geometry, ops
    kw = {} if cone else {"ConeBeam": False}
    o = _cone_obj(n=n, nz=nz, nu=nu, nv=nv, views=views, ForwardProjectionStepSize=step,
                  DetectorElementWidth=1.3 * n * 0.5 * 550 / 300 / nu, DetectorElementHeight=0.9 * nz * 0.5 * 550 / 300 / nv, **kw)
    dg = geometry.fpj_geometry(o)
    rng = np.random.default_rng(n + views)
    y = (rng.uniform(-1, 1, dg.sgm_shape) + 0.5).astype(np.float32)
    mask = (rng.uniform(0, 1, dg.sgm_shape) > 0.1).astype(np.float32)
    ref = np.zeros(dg.vol_shape)
    for j in range(views):
        P.march(None, j, dg.host["angles"], dg.host["u"], dg.host["v"], nx=n, nz=nz, px=o.img_pix_size,
                pz=o.img_voxel_height, cx=o.img_center_x, cy=o.img_center_y, cz_view=o.array_img_center_z[j],
                sid=o.source_isocenter_dis, sdd=o.source_det_dis, step=step, cone_beam=cone, rows=dg.geom.nv,
                K=dg.geom.fp_steps, mask=mask[:, j, :], mode="adjoint", ray_values=y[:, j, :], out=ref)
    yt, m = torch.from_numpy(y).cuda(), torch.from_numpy(mask).cuda()
    inner = (slice(1, -1) if cone else slice(None), slice(1, -1), slice(1, -1))
    assert np.abs(ref[inner]).max() > 0
    for ws in (True, None):
        got = ops.fp_adjoint(dg, yt, mask=m, workspace=ws).cpu().numpy()
        assert rel_l2(got[inner], ref[inner]) < TOL


@pytest.mark.parametrize("step", [0.36, 0.37, 0.44, 0.45])
def test_fan_beam_adjoint_on_both_sides_of_the_walk_by_samples(step, cuda):
    test_adjoint_by_cells_matches_the_sum_over_samples(34, 3, 37, 3, 30, step, False, cuda)
