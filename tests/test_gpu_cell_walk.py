"""The forward projector's walk by cells against the float64 oracle's sum over samples, where
the two could part: steps that leave many samples or none in a cell, volumes on both sides of
the widths where the copies' rows are padded (128) and the rays are walked in windows (256),
scans on both sides of the ray tiles' rule (256 views), one-cell-thick volumes, fan beam, and
each storage type."""
import numpy as np
import pytest

from conftest import rel_l2
from oracle import fpj_ops as P
from test_gpu_parity import _cone_obj

pytestmark = pytest.mark.gpu

# float32 sample positions are within 3 * 2^-24 * n (5e-5 voxel at n = 256) of the float64
# ones; on a noise volume (values and differences of the same size) that bounds the relative
# error of a ray by about as much.  The outer two voxel layers are 0, so that a sample whose
# inside test flips carries nothing.  Storage rounds each value by 2^-11 / 2^-8 at most.
TOL = {"f32": 5e-5, "f16": 2.0 ** -11, "bf16": 2.0 ** -8}


@pytest.mark.parametrize("n,nz,nu,nv,views,step,storage,cone", [
    (32, 9, 40, 11, 24, 0.05, "f32", True), (32, 9, 40, 11, 24, 0.9, "f32", True), (33, 5, 40, 7, 24, 2.5, "f32", True),
    (127, 6, 17, 5, 9, 0.2, "f32", True), (128, 6, 17, 5, 9, 0.2, "f32", True), (130, 6, 17, 5, 9, 0.2, "bf16", True),
    (255, 6, 17, 3, 5, 0.2, "f32", True), (256, 6, 17, 3, 5, 0.2, "f32", True), (257, 6, 33, 3, 5, 0.2, "f32", True),
    (40, 8, 35, 9, 255, 0.2, "f32", True), (40, 8, 35, 9, 257, 0.2, "f32", True), (40, 8, 35, 9, 257, 0.2, "bf16", True),
    (40, 8, 35, 9, 30, 0.2, "f16", True),
    (40, 8, 35, 9, 30, 0.3, "bf16", True), (131, 6, 17, 5, 9, 0.5, "bf16", True), (40, 8, 35, 9, 30, 0.5, "f16", True), (40, 6, 35, 9, 30, 0.1, "f32", True),
    (34, 3, 37, 3, 30, 0.2, "f32", False), (130, 1, 41, 1, 9, 0.1, "f32", False), (260, 2, 41, 2, 5, 0.3, "f32", False)])
def test_projection_by_cells_matches_the_sum_over_samples(n, nz, nu, nv, views, step, storage, cone, cuda):
    import torch
    from reconstruction_program_taichi_gb300 import geometry, ops
    kw = {} if cone else {"ConeBeam": False}
    o = _cone_obj(n=n, nz=nz, nu=nu, nv=nv, views=views, ForwardProjectionStepSize=step,
                  DetectorElementWidth=1.3 * n * 0.5 * 550 / 300 / nu, DetectorElementHeight=0.9 * nz * 0.5 * 550 / 300 / nv, **kw)
    dg = geometry.fpj_geometry(o)
    rng = np.random.default_rng(n + views)
    vol = np.zeros(dg.vol_shape, np.float32)
    zs = slice(2, -2) if cone else slice(None)
    vol[zs, 2:-2, 2:-2] = rng.uniform(-1, 1, vol[zs, 2:-2, 2:-2].shape) + 0.5
    mask = (rng.uniform(0, 1, dg.sgm_shape) > 0.1).astype(np.float32)
    dtype = {"f32": ops.MCT_F32, "f16": ops.MCT_F16, "bf16": ops.MCT_BF16}[storage]
    x, m = torch.from_numpy(vol).cuda(), torch.from_numpy(mask).cuda()
    got = [ops.fp(dg, x, mask=m, dtype=dtype)]
    if storage == "f32":
        got.append(ops.fp(dg, x, mask=m, workspace=None))
    some = sorted({0, 1, views // 3, views // 2, views - 1})
    ref = np.stack([P.march(vol, j, dg.host["angles"], dg.host["u"], dg.host["v"], nx=n, nz=nz, px=o.img_pix_size,
                            pz=o.img_voxel_height, cx=o.img_center_x, cy=o.img_center_y,
                            cz_view=o.array_img_center_z[j], sid=o.source_isocenter_dis, sdd=o.source_det_dis,
                            step=step, cone_beam=cone, rows=dg.geom.nv, K=dg.geom.fp_steps, mask=mask[:, j, :])
                    for j in some], axis=1)
    for g in got:
        assert rel_l2(g.cpu().numpy()[:, some], ref) < TOL[storage]


@pytest.mark.parametrize("n,nz,nu,nv,views,step", [
    (40, 8, 35, 9, 39, 0.36), (40, 8, 35, 9, 39, 0.37), (40, 8, 35, 9, 40, 0.5), (128, 6, 17, 5, 9, 0.5),
    (255, 6, 17, 3, 5, 0.5), (256, 6, 17, 3, 5, 0.5), (9, 5, 33, 3, 20, 1.7)])
def test_float32_projection_by_samples_matches_the_sum_over_samples(n, nz, nu, nv, views, step, cuda):
    """Both sides of the step, width and view count that decide how float32 quads are walked."""
    test_projection_by_cells_matches_the_sum_over_samples(n, nz, nu, nv, views, step, "f32", True, cuda)
