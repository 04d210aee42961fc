"""The tensor-core filter's column tiles and epilogue, and the weighting fused into its operand
split, at their edges: rows of one to several tiles, few enough for the 64-column tiles and
enough for the 256-column ones, columns below, at and past a chunk and a tile, 16-byte aligned
rows and others, blocks of operand rows within one, two and many detector rows."""
import numpy as np
import pytest

from conftest import rel_l2
from oracle import fbp_ops as F
from test_gpu_parity import _cone_obj

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nv,views,nu,kw", [
    (2, 3, 31, {}), (2, 64, 33, {}), (3, 43, 64, {}), (3, 100, 65, {}), (2, 129, 127, {"CurvedDetector": True}),
    (50, 5, 130, {}), (3, 200, 257, {"TotalScanAngle": 220}), (41, 320, 66, {}), (41, 320, 97, {"CurvedDetector": True}),
    (7, 90, 701, {"CurvedDetector": True, "TotalScanAngle": 220}),
    (4, 70, 99, {"BeamHardeningCorrectionCoefficients": [0.0, 1.0, 0.05]})])
@pytest.mark.parametrize("parts", ["tc3", "tc"])
def test_weighted_and_filtered_rows_match_the_oracle(nv, views, nu, kw, parts, cuda):
    import torch
    from reconstruction_program_taichi_gb300 import fbp, geometry
    o = _cone_obj(n=16, nz=4, nu=nu, nv=nv, views=views, **kw)
    rng = np.random.default_rng(nu)
    sgm = rng.uniform(0, 1, (nv, views, nu)).astype(np.float32)
    got = fbp.FdkPipeline(o, filter_impl=parts).filter(torch.from_numpy(sgm).cuda()).cpu().numpy()
    u, v, ang = geometry.fbp_arrays(o)
    x = sgm.astype(np.float64)
    if o.bool_bh_correction:
        x = sum(float(c) * x ** (k + 1) for k, c in enumerate(o.array_bh_coefficients))
    w = F.weight_sgm(x, u, v, ang, o.source_det_dis, o.curved_dect, o.short_scan, o.total_scan_angle)
    ref = F.filter_rows(w, geometry.recon_taps(o), o.det_elem_width).transpose(1, 0, 2)
    # float32 accumulation of nu products of which the ramp cancels most: a few 2^-24 times the
    # sum of their sizes over the result (about 30 on noise of mean 1/2); two parts drop 2^-16
    assert rel_l2(got, ref) < {"tc3": 1e-5, "tc": 5e-4}[parts]
