"""The passes around the filter, which take several elements per thread, at the edges of their
tiles: the packed copies (64 columns x 16 rows of a view, lines of 128 threads), the helical
rebinning (1024 columns), the weighting (aligned rows 16 bytes at a time).  Each is a few
float32 operations per element, so results are compared bit for bit."""
import ctypes

import numpy as np
import pytest

from test_gpu_parity import _cone_obj

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nu,nv,views", [(2, 2, 1), (65, 15, 3), (66, 16, 2), (64, 17, 3), (130, 33, 2), (1026, 5, 2)])
@pytest.mark.parametrize("storage", ["f32", "bf16"])
def test_packed_cells_at_tile_edges(nu, nv, views, storage, cuda):
    import torch
    from reconstruction_program_taichi_gb300 import geometry, ops
    dtype, td = {"f32": (ops.MCT_F32, torch.float32), "bf16": (ops.MCT_BF16, torch.bfloat16)}[storage]
    for cone in (True, False):
        o = _cone_obj(n=8, nz=2, nu=nu, nv=nv, views=views, ConeBeam=cone, **({} if cone else {"ImageDimensionZ": nv}))
        dg = geometry.fbp_geometry(o)
        nv_ = dg.geom.nv
        f = torch.randn((views, nv_, nu), device="cuda", generator=torch.Generator("cuda").manual_seed(nu))
        a = f[..., :-1].to(td).float()
        b = f[..., 1:]
        if cone:
            c, d = f[:, 1:, :-1], f[:, 1:, 1:]
            a, b = a[:, :-1], b[:, :-1]
            want = torch.stack([a, c - a, b - a, (d - c) - (b - a)], -1).to(td)
            got = ops.pack(dg, f, dtype)[:ops.packed_bytes(dg, dtype)].view(td).reshape(views, nv_, nu - 1, 4)
            strided = ops.pack_sinogram(dg, f.transpose(0, 1).contiguous(), dtype)[:ops.packed_bytes(dg, dtype)]
            assert torch.isnan(got[:, -1].float()).all()
            assert torch.equal(strided.view(torch.uint8), got.contiguous().view(torch.uint8).flatten())
            got = got[:, :-1]
        else:
            want = torch.stack([a, b - a], -1).to(td)
            got = ops.pack(dg, f, dtype)[:ops.packed_bytes(dg, dtype)].view(td).reshape(views, nv_, nu - 1, 2)
        # the order of the four coefficients in memory is the kernels' own
        assert torch.equal(torch.sort(got.float(), -1)[0], torch.sort(want.float(), -1)[0])


@pytest.mark.parametrize("nu", [1, 127, 1023, 1024, 1025, 2100])
def test_helical_rebinning_treats_columns_alike(nu, cuda):
    """A detector's columns rebinned one block of 50 at a time give the same bits."""
    import torch
    from reconstruction_program_taichi_gb300 import _lib, ops

    def rebin(x, z):
        h = _lib.Helical(nu=x.shape[2], nv=x.shape[0], views=x.shape[1], view_count=7, n_slices=z.numel(), dv=1.0, sdd=500.0,
                         mag=1.5, det_offset_vertical=0.3, dis_per_view=0.4)
        out = torch.full((z.numel(), 7, x.shape[2]), 7.0, device="cuda")
        _lib.call("mct_helical_rebin", ctypes.byref(h), ops._ptr(x), ops._ptr(z), ops._ptr(out),
                  torch.cuda.current_stream().cuda_stream)
        return out

    x = torch.randn((4, 20, nu), device="cuda", generator=torch.Generator("cuda").manual_seed(nu))
    z = torch.tensor([-3.0, 0.5, 3.1, 8.0], device="cuda")
    got = rebin(x, z)
    want = torch.cat([rebin(x[..., c:c + 50].contiguous(), z) for c in range(0, nu, 50)], -1)
    assert torch.equal(got, want)
    assert float((got == 0).float().mean()) < 0.9 and not (got == 7.0).any()


@pytest.mark.parametrize("nu,kw", [(64, {}), (60, {}), (68, {"TotalScanAngle": 220}), (52, {"CurvedDetector": True})])
def test_weighting_of_aligned_and_unaligned_rows_agrees(nu, kw, cuda):
    import torch
    from reconstruction_program_taichi_gb300 import geometry, ops
    o = _cone_obj(n=16, nz=4, nu=nu, nv=6, views=20, **kw)
    dg = geometry.fbp_geometry(o)
    x = torch.rand((6, 20, nu), device="cuda", generator=torch.Generator("cuda").manual_seed(nu))
    shifted = torch.empty(x.numel() + 1, device="cuda")[1:].reshape(x.shape)
    shifted.copy_(x)
    assert x.data_ptr() % 16 == 0 and shifted.data_ptr() % 16 == 4
    taps = torch.from_numpy(np.asarray(geometry.recon_taps(o), np.float32)).cuda()
    fil = ops.TcFilter(dg, taps, ops.MCT_F32)
    want = fil(ops.weight(dg, x, 20 * nu, nu))
    for src in (x, shifted):
        assert torch.equal(fil.weight_filter(src, 20 * nu, nu), want)
