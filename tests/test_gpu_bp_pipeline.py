"""The cone-beam backprojector's software-pipelined view loop where it could go wrong: scans of
fewer views than a run of views, of one more and one less, columns that leave the detector in
the first, a middle or the last view of a run, curved detectors, 16-bit operands, and
detectors too tall for row indices from the float32 rounding constant."""
import numpy as np
import pytest

from conftest import rel_l2
from oracle import fbp_ops as F
from oracle import ir_ops as I
from test_gpu_parity import _cone_obj

pytestmark = pytest.mark.gpu

# float32 sums against float64: 1e-4 as for the other operators; 16-bit operands round the base
# value of each cell by 2^-9 (bf16) or 2^-12 (float16) of its size, on noise with zero mean by
# up to twice that relative to the sum.
TOL = {"f32": 1e-4, "bf16": 2.0 ** -8, "f16": 2.0 ** -11}


@pytest.mark.parametrize("views,storage,kw", [
    (2, "f32", {}), (31, "f32", {}), (32, "f32", {}), (33, "f32", {"CurvedDetector": True}), (65, "f32", {}),
    (65, "bf16", {}), (33, "bf16", {"CurvedDetector": True}), (33, "f16", {"ReconViewMode": "coronal"}),
    (40, "f32", {"TotalScanAngle": 220, "ReconViewMode": "sagittal"})])
def test_backprojection_matches_the_oracle_with_truncated_columns(views, storage, kw, cuda):
    import torch
    from reconstruction_program_taichi_gb300 import geometry, ops
    # the detector is narrower than the image: its corners and edges leave it in some view
    o = _cone_obj(n=37, nz=18, nu=34, nv=30, views=views, **kw)
    dg = geometry.fbp_geometry(o)
    g = dg.geom
    rng = np.random.default_rng(views)
    f = rng.normal(0, 1, (views, g.nv, g.nu)).astype(np.float32)
    dtype = {"f32": ops.MCT_F32, "bf16": ops.MCT_BF16, "f16": ops.MCT_F16}[storage]
    x = torch.from_numpy(f).cuda()
    got = ops.fdk_bp(dg, ops.pack(dg, x, dtype), dtype).cpu().numpy()
    u, v, ang = geometry.fbp_arrays(o)
    ref = F.fdk_bp(f.transpose(1, 0, 2), ang, u, v, nx=o.img_dim, nz=o.img_dim_z, px=o.img_pix_size,
                   pz=o.img_voxel_height, cx=o.img_center_x, cy=o.img_center_y, cz=o.img_center_z,
                   sid=o.source_isocenter_dis, sdd=o.source_det_dis, dv=o.det_elem_height, img_rot=o.img_rot,
                   total_scan_angle=o.total_scan_angle, short_scan=o.short_scan, cone_beam=True,
                   curved=o.curved_dect, view_mode=o.recon_view_mode)
    assert 0.05 < np.mean(ref == 0) < 0.95
    # voxels within float32 rounding of the detector's edge may fall on either side
    assert np.mean((got == 0) != (ref == 0)) < 1e-3
    both = (got != 0) & (ref != 0)
    assert rel_l2(got[both], ref[both]) < TOL[storage]


def test_detector_of_more_than_2_22_rows_gives_the_same_volume(cuda):
    """A detector whose first rows are the small one's and hold everything the volume reads:
    the same row indices through the tall detectors' floor, so the same bits."""
    import torch
    from reconstruction_program_taichi_gb300 import geometry, ops
    o = _cone_obj(n=8, nz=4, nu=8, nv=24, views=2, DetectorElementWidth=2.0)
    dg = geometry.fbp_geometry(o)
    rng = np.random.default_rng(3)
    f = torch.from_numpy(rng.normal(0, 1, (2, 24, 8)).astype(np.float32)).cuda()
    small = ops.fdk_bp(dg, ops.pack(dg, f))
    dg.geom = dg.geom.copy(nv=(1 << 22) + 3)
    tall = torch.zeros((2, dg.geom.nv, 8), device="cuda")
    tall[:, :24] = f
    got = ops.fdk_bp(dg, ops.pack(dg, tall))
    assert float((small != 0).float().mean()) > 0.5
    assert torch.equal(got, small)


@pytest.mark.parametrize("views,storage", [(2, "f32"), (31, "f32"), (32, "f32"), (33, "f32"), (65, "f32"), (33, "bf16"),
                                           (33, "f16")])
def test_solver_backprojection_matches_the_oracle_off_the_detector(views, storage, cuda):
    """The solver's backprojector in the same loop: columns that leave the detector are zero,
    rows that leave it are skipped."""
    import torch
    from reconstruction_program_taichi_gb300 import geometry, ops
    o = _cone_obj(n=37, nz=18, nu=34, nv=12, views=views)
    dg = geometry.ir_geometry(o)
    rng = np.random.default_rng(views)
    sgm = rng.normal(0, 1, dg.sgm_shape).astype(np.float32)
    dtype = {"f32": ops.MCT_F32, "bf16": ops.MCT_BF16, "f16": ops.MCT_F16}[storage]
    got = ops.bp_unmatched_packed(dg, ops.pack_sinogram(dg, torch.from_numpy(sgm).cuda(), dtype), dtype).cpu().numpy()
    ref = I.bp_unmatched(sgm, dg.host["angles"], dg.host["u"], dg.host["v"], o.array_img_center_z, nx=o.img_dim,
                         nz=o.img_dim_z, px=o.img_pix_size, pz=o.img_voxel_height, cx=o.img_center_x, cy=o.img_center_y,
                         sid=o.source_isocenter_dis, sdd=o.source_det_dis, dv=o.det_elem_height, img_rot=o.img_rot,
                         cone_beam=True)
    assert 0.05 < np.mean(ref == 0) < 0.95
    # voxels within float32 rounding of the detector's edge may fall on either side
    assert np.mean((got == 0) != (ref == 0)) < 1e-3
    both = (got != 0) & (ref != 0)
    assert rel_l2(got[both], ref[both]) < 5 * TOL[storage]  # a row at the edge in or out: one view of `views`


@pytest.mark.parametrize("n,nz,views,kw", [
    (7, 5, 255, {}), (8, 16, 256, {}), (9, 17, 257, {"CurvedDetector": True}), (17, 3, 513, {"ReconViewMode": "coronal"})])
def test_backprojection_at_the_edges_of_blocks_and_view_tables(n, nz, views, kw, cuda):
    """Volumes of one column less and more than a block, scans of one view less and more than
    the block's table of views."""
    import torch
    from reconstruction_program_taichi_gb300 import geometry, ops
    o = _cone_obj(n=n, nz=nz, nu=3 * n, nv=2 * nz, views=views, **kw)
    dg = geometry.fbp_geometry(o)
    g = dg.geom
    f = np.random.default_rng(views).normal(0, 1, (views, g.nv, g.nu)).astype(np.float32)
    got = ops.fdk_bp(dg, ops.pack(dg, torch.from_numpy(f).cuda())).cpu().numpy()
    u, v, ang = geometry.fbp_arrays(o)
    ref = F.fdk_bp(f.transpose(1, 0, 2), ang, u, v, nx=o.img_dim, nz=o.img_dim_z, px=o.img_pix_size,
                   pz=o.img_voxel_height, cx=o.img_center_x, cy=o.img_center_y, cz=o.img_center_z,
                   sid=o.source_isocenter_dis, sdd=o.source_det_dis, dv=o.det_elem_height, img_rot=o.img_rot,
                   total_scan_angle=o.total_scan_angle, short_scan=o.short_scan, cone_beam=True,
                   curved=o.curved_dect, view_mode=o.recon_view_mode)
    assert np.mean((got == 0) != (ref == 0)) < 1e-3
    both = (got != 0) & (ref != 0)
    assert both.sum() > 0.2 * both.size
    assert rel_l2(got[both], ref[both]) < TOL["f32"]


@pytest.mark.parametrize("n,nz,storage,kw", [
    (16, 8, "f32", {}), (20, 16, "f32", {}), (20, 17, "bf16", {}), (20, 25, "f32", {"CurvedDetector": True}),
    (33, 9, "f16", {"ReconViewMode": "sagittal"}), (200, 16, "f32", {}), (200, 24, "f32", {}), (200, 17, "f32", {"CurvedDetector": True})])
def test_columns_of_8_and_of_16_slices_match_the_oracle(n, nz, storage, kw, cuda):
    """Both sides of the rule that picks the slices of a column: few and many blocks, last
    slices that fill 16 or half of them."""
    import torch
    from reconstruction_program_taichi_gb300 import geometry, ops
    o = _cone_obj(n=n, nz=nz, nu=40, nv=2 * nz, views=5, PixelSize=24.0 / n, DetectorElementWidth=1.6, **kw)
    dg = geometry.fbp_geometry(o)
    g = dg.geom
    f = np.random.default_rng(n + nz).normal(0, 1, (5, g.nv, g.nu)).astype(np.float32)
    dtype = {"f32": ops.MCT_F32, "bf16": ops.MCT_BF16, "f16": ops.MCT_F16}[storage]
    got = ops.fdk_bp(dg, ops.pack(dg, torch.from_numpy(f).cuda(), dtype), dtype).cpu().numpy()
    u, v, ang = geometry.fbp_arrays(o)
    ref = F.fdk_bp(f.transpose(1, 0, 2), ang, u, v, nx=o.img_dim, nz=o.img_dim_z, px=o.img_pix_size,
                   pz=o.img_voxel_height, cx=o.img_center_x, cy=o.img_center_y, cz=o.img_center_z,
                   sid=o.source_isocenter_dis, sdd=o.source_det_dis, dv=o.det_elem_height, img_rot=o.img_rot,
                   total_scan_angle=o.total_scan_angle, short_scan=o.short_scan, cone_beam=True,
                   curved=o.curved_dect, view_mode=o.recon_view_mode)
    assert np.mean((got == 0) != (ref == 0)) < 1e-3
    both = (got != 0) & (ref != 0)
    assert both.sum() > 0.2 * both.size
    assert rel_l2(got[both], ref[both]) < TOL[storage]


@pytest.mark.parametrize("n,nz,views,storage", [
    (7, 8, 255, "f32"), (9, 16, 257, "f32"), (20, 17, 40, "bf16"), (200, 16, 5, "f32"), (201, 17, 5, "f32"), (200, 30, 5, "f16")])
def test_solver_backprojection_at_the_edges_of_its_blocks(n, nz, views, storage, cuda):
    """Blocks of 8 x 8 columns, view tables of 256 entries, columns of 8 and of 16 slices."""
    import torch
    from reconstruction_program_taichi_gb300 import geometry, ops
    o = _cone_obj(n=n, nz=nz, nu=60, nv=2 * nz, views=views, PixelSize=12.0 / n, DetectorElementWidth=1.0)
    dg = geometry.ir_geometry(o)
    sgm = np.random.default_rng(n + views).normal(0, 1, dg.sgm_shape).astype(np.float32)
    dtype = {"f32": ops.MCT_F32, "bf16": ops.MCT_BF16, "f16": ops.MCT_F16}[storage]
    got = ops.bp_unmatched_packed(dg, ops.pack_sinogram(dg, torch.from_numpy(sgm).cuda(), dtype), dtype).cpu().numpy()
    ref = I.bp_unmatched(sgm, dg.host["angles"], dg.host["u"], dg.host["v"], o.array_img_center_z, nx=o.img_dim,
                         nz=o.img_dim_z, px=o.img_pix_size, pz=o.img_voxel_height, cx=o.img_center_x, cy=o.img_center_y,
                         sid=o.source_isocenter_dis, sdd=o.source_det_dis, dv=o.det_elem_height, img_rot=o.img_rot,
                         cone_beam=True)
    assert np.mean((got == 0) != (ref == 0)) < 1e-3
    both = (got != 0) & (ref != 0)
    assert both.sum() > 0.2 * both.size
    assert rel_l2(got[both], ref[both]) < 5 * TOL[storage]  # a row at the edge in or out, as above
