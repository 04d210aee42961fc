"""Scans whose tables hold an entry that is no finite number: the views (columns, rows) it
belongs to have no positions.  The adjoint adds nothing for them, the projector gives NaN for
their rays that meet the volume, and everything else is what it is without them.  Buffers are the
front of larger ones whose rest stays as it was."""
import numpy as np
import pytest

from conftest import rel_l2
from test_gpu_parity import _cone_obj

pytestmark = pytest.mark.gpu

BAD_VIEW = 5


def _scan(cone, step=0.2, **kw):
    from reconstruction_program_taichi_gb300 import geometry
    n, nz = 32, 9 if cone else 3
    o = _cone_obj(n=n, nz=nz, nu=40, nv=11 if cone else 3, views=24, ForwardProjectionStepSize=step,
                  DetectorElementWidth=1.3 * n * 0.5 * 550 / 300 / 40, DetectorElementHeight=0.9 * nz * 0.5 * 550 / 300 / 11,
                  **({} if cone else {"ConeBeam": False}), **kw)
    return geometry.fpj_geometry(o)


def _front(shape, value=0.0):
    """A tensor of this shape at the front of a buffer of `value`, and the rest of the buffer."""
    import torch
    whole = torch.full((2 * int(np.prod(shape)) + 4096,), value, device="cuda")
    n = int(np.prod(shape))
    return whole[:n].view(shape), whole[n:]


@pytest.mark.parametrize("bad", [float("nan"), float("inf")])
@pytest.mark.parametrize("table,cone,step", [("angles", True, 0.2), ("angles", True, 0.9), ("angles", False, 0.2),
                                             ("angles", False, 0.9), ("cz", True, 0.2), ("u", True, 0.2), ("v", True, 0.2)])
def test_rays_without_a_position(table, cone, step, bad, cuda):
    import torch
    from reconstruction_program_taichi_gb300 import ops
    good, dg = _scan(cone, step), _scan(cone, step)
    gen = torch.Generator("cuda").manual_seed(3)
    x = torch.rand(dg.vol_shape, device="cuda", generator=gen) + 0.5
    y = torch.rand(dg.sgm_shape, device="cuda", generator=gen) + 0.5
    i = BAD_VIEW if table in ("angles", "cz") else 2
    dg._keep[table][i] = bad
    hit = {"u": np.s_[:, :, i], "v": np.s_[i]}.get(table, np.s_[:, i])
    keep = torch.ones(dg.sgm_shape, device="cuda")
    keep[hit] = 0.0

    variants = [dict(workspace=None), {}]
    if cone:
        variants += [dict(dtype=ops.MCT_BF16), dict(dtype=ops.MCT_F16)]
    for kw in variants:
        out, rest = _front(dg.sgm_shape, 3.0)
        ops.fp(dg, x, out=out, **kw)
        want = ops.fp(good, x, **kw)
        assert (rest == 3.0).all()
        assert torch.equal(out[keep > 0], want[keep > 0])
        broken, lines = out[keep == 0], want[keep == 0]
        assert (torch.isnan(broken) | (broken == 0)).all()
        # an infinite centre or row puts the volume out of the rays' reach
        assert torch.isnan(broken[lines > 0.5]).any() != (table in ("cz", "v") and bad == float("inf"))

    for ws in (True, None):
        out, rest = _front(dg.vol_shape)
        ops.fp_adjoint(dg, y, out=out, accumulate=True, workspace=ws)
        want = ops.fp_adjoint(good, y, mask=keep, workspace=ws)
        assert not rest.any()
        # the same additions in another order: 24 views of at most about 10 per voxel
        assert rel_l2(out.cpu().numpy(), want.cpu().numpy()) < 1e-6
    assert ops.fp_count_samples(dg) == ops.fp_count_samples(good, mask=keep)


def _fan(n, nz, views, curved=False, wide=2.0, **kw):
    from reconstruction_program_taichi_gb300 import geometry
    o = _cone_obj(n=n, nz=nz, nu=90, nv=nz, views=views, ConeBeam=False, CurvedDetector=curved,
                  DetectorElementWidth=wide * n * 0.5 * 550 / 300 / 90, **kw)
    return geometry.fbp_geometry(o)


@pytest.mark.parametrize("bad", [float("nan"), float("inf")])
@pytest.mark.parametrize("n,nz,views,curved,view", [(33, 1, 40, False, 7), (33, 1, 40, True, 39), (64, 1, 600, False, 0),
                                                    (34, 9, 40, False, 7), (34, 3, 40, True, 20)])
def test_a_fan_beam_view_without_an_angle_leaves_no_pixel(n, nz, views, curved, view, bad, cuda):
    """It sees every pixel off the detector, so all are written as 0; in chunks too, where the
    other chunks' pixels are inside the detector in each of their views."""
    import torch
    from reconstruction_program_taichi_gb300 import ops
    dg = _fan(n, nz, views, curved)
    f = torch.rand((views, nz, 90), device="cuda", generator=torch.Generator("cuda").manual_seed(1)) + 0.5
    for dtype in (ops.MCT_F32, ops.MCT_BF16):
        good = ops.fdk_bp(dg, ops.pack(dg, f, dtype), dtype)
        assert (good != 0).float().mean() > 0.9
    dg._keep["angles"][view] = bad
    for dtype in (ops.MCT_F32, ops.MCT_BF16, ops.MCT_F16):
        out, rest = _front(dg.vol_shape, 3.0)
        ops.fdk_bp(dg, ops.pack(dg, f, dtype), dtype, out=out)
        assert not out.any() and (rest == 3.0).all()
    vol = torch.zeros(dg.vol_shape, device="cuda")
    for b in range(0, views, 30):
        c = ops.ViewChunk(dg, b, min(30, views - b), accumulate=True)
        ops.fdk_bp(c, ops.pack(c, f[b:b + 30].contiguous()), out=vol)
    assert not ops.fdk_bp_finish(dg, vol).any()


@pytest.mark.parametrize("curved", [False, True])
def test_fan_beam_of_a_far_source_drops_the_pixels_off_the_detector(curved, cuda):
    """sid^2 is beyond float32; the rays are parallel, the magnification 2."""
    import torch
    from reconstruction_program_taichi_gb300 import ops
    dg = _fan(64, 1, 40, curved, wide=0.5)
    dg.geom.sid, dg.geom.sdd = 2e19, 4e19
    g = dg.geom
    f = torch.ones((40, 1, 90), device="cuda")
    got = ops.fdk_bp(dg, ops.pack(dg, f)).cpu().numpy()[0]
    i = np.arange(64)
    x = (i[None, :] - 31.5) * g.px + g.cx
    y = -(i[:, None] - 31.5) * g.px + g.cy
    a = dg.host["angles"][:, None, None]
    index = (2 * (y * np.cos(a) - x * np.sin(a)) - g.u0) / g.u_step
    edge = np.minimum(np.abs(index), np.abs(index - 88)).min(0) < 1e-3
    seen = ((index >= 0) & (index + 1 <= 89)).all(0)
    assert 0.1 < seen.mean() < 0.9
    assert not got[~seen & ~edge].any()
