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
