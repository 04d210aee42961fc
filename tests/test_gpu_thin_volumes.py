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
