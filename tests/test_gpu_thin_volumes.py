"""Cone-beam volumes of the fewest slices in the projector and its adjoint: one slice holds no
cell, so nothing is summed and nothing is written; two slices hold one layer of cells, compared
in both of them.  The adjoint's volume is the front of a larger buffer whose rest stays 0."""
import numpy as np
import pytest

from conftest import rel_l2
from oracle import fpj_ops as P
from test_gpu_parity import _cone_obj

pytestmark = pytest.mark.gpu


def _scan(n, nz, nu, nv, views, step, high, **kw):
    from reconstruction_program_taichi_gb300 import geometry
    o = _cone_obj(n=n, nz=nz, nu=nu, nv=nv, views=views, ForwardProjectionStepSize=step,
                  DetectorElementWidth=1.3 * n * 0.5 * 550 / 300 / nu, DetectorElementHeight=high * nz * 0.5 * 550 / 300 / nv, **kw)
    return o, geometry.fpj_geometry(o)


def _adjoint(dg, y, mask, workspace):
    """P^T y, written to the front of a buffer with four planes behind it."""
    import torch
    from reconstruction_program_taichi_gb300 import ops
    nz, n, _ = dg.vol_shape
    whole = torch.zeros((nz + 4, n, n), device="cuda")
    ops.fp_adjoint(dg, y, mask=mask, out=whole[:nz], accumulate=True, workspace=workspace)
    assert not whole[nz:].any()
    return whole[:nz].cpu().numpy()


@pytest.mark.parametrize("n,nu,nv,views,cz", [(32, 40, 33, 12, 0.11), (64, 48, 32, 4, 0.22), (2, 9, 9, 13, 0.1)])
def test_one_slice_projects_nothing(n, nu, nv, views, cz, cuda):
    import torch
    from reconstruction_program_taichi_gb300 import ops
    _, dg = _scan(n, 1, nu, nv, views, 0.2, 4.0, ImageCenterZ=cz)
    y = torch.ones(dg.sgm_shape, device="cuda")
    x = torch.ones(dg.vol_shape, device="cuda")
    for ws in (True, None):
        assert not _adjoint(dg, y, None, ws).any()
        assert not ops.fp(dg, x, workspace=ws).any()
    assert ops.fp_count_samples(dg) == 0


def _clear_rays(o, dg, step):
    """1 for the rays all of whose samples keep 1e-3 voxel from the volume's faces: there an
    inside test flips with the rounding of the position."""
    g = dg.geom
    h = dg.host
    n, nz, px, pz = g.nx, g.nz, o.img_pix_size, o.img_voxel_height
    lmin = g.sid - np.sqrt(2 * (n * px) ** 2 + (nz * pz) ** 2) / 2
    l = np.arange(g.fp_steps) * step * np.sqrt(2 * px * px + pz * pz) + lmin
    out = np.ones(dg.sgm_shape, np.float32)
    for j in range(g.views):
        sz, ux, uy, uz, _ = P._ray_dirs(h["u"], h["v"], g.nv, g.sid, g.sdd, False, 0.0, j)
        c, s = np.cos(h["angles"][j]), np.sin(h["angles"][j])
        x, y, z = g.sid + ux[..., None] * l, uy[..., None] * l, sz + uz[..., None] * l
        fx = (x * c - y * s + (n - 1) / 2 * px - g.cx) / px
        fy = (y * c + x * s - (n - 1) / 2 * px - g.cy) / -px
        fz = (z + (nz - 1) / 2 * pz - o.array_img_center_z[j]) / pz
        near = np.zeros(fx.shape, bool)
        for f, m in ((fx, n), (fy, n), (fz, nz)):
            near |= (np.abs(f) < 1e-3) | (np.abs(f - (m - 1)) < 1e-3)
        # only where the other axes do not already put the sample outside
        reach = np.ones(fx.shape, bool)
        for f, m in ((fx, n), (fy, n), (fz, nz)):
            reach &= (f > -1e-3) & (f < m - 1 + 1e-3)
        out[:, j] = 1.0 - (near & reach).any(-1)
    return out


# float32 sample positions are within 3 * 2^-24 * n of the float64 ones (1.2e-5 voxel at n = 64);
# with values and differences of the same size that bounds a ray's relative error by about as
# much, a voxel's by 3 times that (weights of 0.35).  Storage rounds by 2^-11 / 2^-8 at most.
TOL = {"f32": 5e-5, "f16": 2.0 ** -11, "bf16": 2.0 ** -8}


@pytest.mark.parametrize("nz,nv", [(2, 7), (3, 8)])
@pytest.mark.parametrize("step", [0.05, 0.2, 0.5, 1.3])
def test_one_and_two_layers_of_cells(nz, nv, step, cuda):
    import torch
    from reconstruction_program_taichi_gb300 import ops
    n, nu, views = 40, 35, 24
    o, dg = _scan(n, nz, nu, nv, views, step, 1.1, ImageCenterZ=0.13)
    mask = _clear_rays(o, dg, step)
    assert mask.mean() > 0.5
    rng = np.random.default_rng(nz)
    vol = (rng.uniform(-1, 1, dg.vol_shape) + 0.5).astype(np.float32)
    y = (rng.uniform(-1, 1, dg.sgm_shape) + 0.5).astype(np.float32)

    def march(j, **kw):
        return P.march(vol if "out" not in kw else None, j, dg.host["angles"], dg.host["u"], dg.host["v"], nx=n, nz=nz,
                       px=o.img_pix_size, pz=o.img_voxel_height, cx=o.img_center_x, cy=o.img_center_y,
                       cz_view=o.array_img_center_z[j], sid=o.source_isocenter_dis, sdd=o.source_det_dis, step=step,
                       cone_beam=True, rows=nv, K=dg.geom.fp_steps, mask=mask[:, j], **kw)

    ref = np.stack([march(j) for j in range(views)], axis=1)
    back = np.zeros(dg.vol_shape)
    for j in range(views):
        march(j, mode="adjoint", ray_values=y[:, j], out=back)
    x, m, yt = torch.from_numpy(vol).cuda(), torch.from_numpy(mask).cuda(), torch.from_numpy(y).cuda()
    for storage, kw in (("f32", {}), ("f32", dict(workspace=None)), ("bf16", dict(dtype=ops.MCT_BF16)),
                        ("f16", dict(dtype=ops.MCT_F16))):
        assert rel_l2(ops.fp(dg, x, mask=m, **kw).cpu().numpy(), ref) < TOL[storage]
    for ws in (True, None):
        assert rel_l2(_adjoint(dg, yt, m, ws), back) < 3 * TOL["f32"]


@pytest.mark.parametrize("n,nz,nu,nv,step", [(41, 3, 41, 3, 0.2), (41, 9, 41, 7, 0.1), (9, 41, 41, 41, 0.3), (40, 5, 41, 1, 0.9)])
def test_rays_along_planes(n, nz, nu, nv, step, cuda):
    """A centred scan of an odd number of planes, rows and columns: the middle row's rays stay
    on a plane, some views' middle column's on a column of voxels, with fractions that round to
    0 or to 1 - 2^-24."""
    import torch
    from reconstruction_program_taichi_gb300 import ops
    views = 8
    o, dg = _scan(n, nz, nu, nv, views, step, 0.8, ImageCenterZ=0.0, DetectorOffsetVertical=0.0, ImageCenter=[0.0, 0.0],
                  DetectorOffsetHorizontal=0.0, ImageRotation=0)
    mask = _clear_rays(o, dg, step)
    assert mask[nv // 2].mean() > 0.5
    rng = np.random.default_rng(n)
    vol = (rng.uniform(-1, 1, dg.vol_shape) + 0.5).astype(np.float32)
    y = (rng.uniform(-1, 1, dg.sgm_shape) + 0.5).astype(np.float32)
    kw = dict(nx=n, nz=nz, px=o.img_pix_size, pz=o.img_voxel_height, cx=0.0, cy=0.0, sid=o.source_isocenter_dis,
              sdd=o.source_det_dis, step=step, cone_beam=True, rows=nv, K=dg.geom.fp_steps)
    tables = dg.host["angles"], dg.host["u"], dg.host["v"]
    ref = np.stack([P.march(vol, j, *tables, cz_view=o.array_img_center_z[j], mask=mask[:, j], **kw) for j in range(views)], 1)
    back = np.zeros(dg.vol_shape)
    for j in range(views):
        P.march(None, j, *tables, cz_view=o.array_img_center_z[j], mask=mask[:, j], mode="adjoint", ray_values=y[:, j],
                out=back, **kw)
    x, m, yt = torch.from_numpy(vol).cuda(), torch.from_numpy(mask).cuda(), torch.from_numpy(y).cuda()
    for storage, a in (("f32", {}), ("f32", dict(workspace=None)), ("bf16", dict(dtype=ops.MCT_BF16)),
                       ("f16", dict(dtype=ops.MCT_F16))):
        assert rel_l2(ops.fp(dg, x, mask=m, **a).cpu().numpy(), ref) < TOL[storage]
    for ws in (True, None):
        assert rel_l2(_adjoint(dg, yt, m, ws), back) < 3 * TOL["f32"]


def test_volume_of_more_planes_than_the_float_floor_holds(cuda):
    """2^22 + 4096 planes without a workspace: the samples near the top, where adding 1.5 x 2^23 is
    no floor, are taken from their own planes.  A ramp that is 0 at plane 2^22 gives each ray its
    plane times its length; float32 places a plane there to within one, of about 1000."""
    import torch
    from reconstruction_program_taichi_gb300 import _lib, ops
    nz, px, pz, plane, views, nu = (1 << 22) + 4096, 10.0, 0.01, (1 << 22) + 1000, 4, 5
    steps = int(np.sqrt(2 * (2 * px) ** 2 + (nz * pz) ** 2) / (0.2 * np.sqrt(2 * px * px + pz * pz)))
    g = _lib.Geom(nu=nu, nv=1, views=views, nv_total=1, nx=2, nz=nz, flags=_lib.MCT_CONE, view_mode=1, fp_steps=steps, du=1.0,
                  dv=1.0, px=px, pz=pz, cz=(nz - 1) / 2 * pz - plane * pz, sid=300.0, sdd=550.0, total_scan_angle=2 * np.pi,
                  fp_step=0.2)
    dg = ops.DeviceGeometry(g, angles=0.3 + np.arange(views) * np.pi / 2, u=np.arange(nu) - 2.0, v=[0.0])
    z = torch.arange(nz, device="cuda", dtype=torch.float32) - float(1 << 22)
    ramp = z.clamp(min=0)[:, None, None].expand(nz, 2, 2).contiguous()
    one = torch.ones_like(ramp)
    length = ops.fp(dg, one, workspace=None)
    assert (length > 5.0).all()
    assert ((ops.fp(dg, ramp, workspace=None) / length - 1000).abs() < 2).all()
    back = ops.fp_adjoint(dg, torch.ones(dg.sgm_shape, device="cuda"), workspace=None)
    hit = back.sum((1, 2)).nonzero().flatten()
    assert ((hit - plane).abs() <= 2).all()
    assert abs(float(back.sum()) / float(length.sum()) - 1) < 1e-4
