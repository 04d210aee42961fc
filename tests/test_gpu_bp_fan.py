"""The fan-beam backprojector's pairs of rows, view groups and inside shortcut at their edges:
images of an odd number of rows and of a warp's width and one more, fewer views than groups,
more views than a table holds, one to nine slices, detectors that hold every pixel, lose the
image's edge, or are shifted so that only some warps are inside, curved detectors and 16-bit
operands."""
import numpy as np
import pytest

from conftest import rel_l2
from oracle import fbp_ops as F
from test_gpu_parity import _cone_obj

pytestmark = pytest.mark.gpu

# float32 sums against float64: 1e-4 as for the other operators; 16-bit operands round the base
# value of each pair by 2^-9 (bf16) or 2^-12 (float16), on zero-mean noise up to twice that.
TOL = {"f32": 1e-4, "bf16": 2.0 ** -8, "f16": 2.0 ** -11}


@pytest.mark.parametrize("n,nz,views,wide,storage,kw", [
    (32, 1, 2, 2.0, "f32", {}), (33, 1, 7, 2.0, "f32", {}), (35, 1, 8, 1.0, "f32", {}), (64, 1, 513, 2.0, "f32", {}),
    (37, 1, 40, 1.1, "f32", {}), (70, 1, 40, 1.3, "f32", {"DetectorOffsetHorizontal": 9.0}),
    (37, 1, 40, 1.1, "f32", {"CurvedDetector": True}), (37, 1, 40, 2.0, "f32", {"CurvedDetector": True}),
    (33, 3, 17, 2.0, "f32", {}), (34, 8, 17, 1.1, "f32", {}), (35, 9, 24, 1.1, "f32", {"CurvedDetector": True}),
    (33, 1, 30, 1.1, "bf16", {}), (33, 9, 30, 2.0, "bf16", {}), (33, 1, 30, 2.0, "f16", {}),
    (33, 2, 30, 1.1, "f32", {"TotalScanAngle": 220})])
def test_fan_backprojection_matches_the_oracle(n, nz, views, wide, storage, kw, cuda):
    import torch
    from reconstruction_program_taichi_gb300 import geometry, ops
    nu = 90
    o = _cone_obj(n=n, nz=nz, nu=nu, nv=nz, views=views, ConeBeam=False,
                  DetectorElementWidth=wide * n * 0.5 * 550 / 300 / nu, **kw)
    dg = geometry.fbp_geometry(o)
    rng = np.random.default_rng(n + views)
    f = rng.normal(0, 1, (views, nz, nu)).astype(np.float32)
    dtype = {"f32": ops.MCT_F32, "bf16": ops.MCT_BF16, "f16": ops.MCT_F16}[storage]
    x = torch.from_numpy(f).cuda()
    got = ops.fdk_bp(dg, ops.pack(dg, x, dtype), dtype).cpu().numpy()
    u, v, ang = geometry.fbp_arrays(o)
    ref = F.fdk_bp(f.transpose(1, 0, 2), ang, u, v, nx=n, nz=nz, px=o.img_pix_size, pz=0.0, cx=o.img_center_x,
                   cy=o.img_center_y, cz=0.0, sid=o.source_isocenter_dis, sdd=o.source_det_dis, dv=1.0,
                   img_rot=o.img_rot, total_scan_angle=o.total_scan_angle, short_scan=o.short_scan, cone_beam=False,
                   curved=o.curved_dect)
    assert np.mean(ref != 0) > 0.2
    # pixels within float32 rounding of the detector's edge may fall on either side
    assert np.sum((got == 0) != (ref == 0)) <= 2 * nz
    both = (got != 0) & (ref != 0)
    assert rel_l2(got[both], ref[both]) < TOL[storage]
