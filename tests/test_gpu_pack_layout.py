"""The packed operands element by element, in their documented order and bit for bit: cone beam
{A, C-A, B-A, (D-C)-(B-A)}, fan beam {A, B-A} with A as stored, each type, the float16 operand
with its power-of-two scale; at the edges of the lines and tiles that a block takes."""
import numpy as np
import pytest

from test_gpu_parity import _cone_obj

pytestmark = pytest.mark.gpu


def _packed(dg, f, storage):
    """The operand and its elements as float32: what is stored, times the scale."""
    import torch
    from reconstruction_program_taichi_gb300 import ops
    dtype, td = {"f32": (ops.MCT_F32, torch.float32), "bf16": (ops.MCT_BF16, torch.bfloat16),
                 "f16": (ops.MCT_F16, torch.float16)}[storage]
    g = dg.geom
    k = 4 if g.flags & 1 else 2
    n = g.views * g.nv * (g.nu - 1) * k
    a, b = ops.pack(dg, f, dtype), ops.pack_sinogram(dg, f.transpose(0, 1).contiguous(), dtype)
    m = float(f.abs().max())
    scale = 2.0 ** (12 - int(np.floor(np.log2(m)))) if storage == "f16" else 1.0
    ops_ = [t.view(torch.uint8)[:n * td.itemsize].clone().view(td).reshape(g.views, g.nv, g.nu - 1, k) for t in (a, b)]
    assert torch.equal(ops_[0].view(torch.uint8), ops_[1].view(torch.uint8))
    return ops_[0], td, scale


CASES = [(2, 2, 1), (5, 3, 7), (9, 1, 130), (17, 4, 33), (33, 5, 70), (34, 13, 3), (65, 2, 19), (66, 12, 5), (70, 9, 31),
         (97, 3, 11), (98, 6, 9), (129, 7, 10), (130, 4, 9), (131, 17, 3), (520, 2, 5)]


@pytest.mark.parametrize("nu,nv,views", CASES)
@pytest.mark.parametrize("storage", ["f32", "bf16", "f16"])
@pytest.mark.parametrize("cone", [True, False])
def test_packed_operand_in_its_documented_order(nu, nv, views, storage, cone, cuda):
    import torch
    from reconstruction_program_taichi_gb300 import _lib, geometry
    if cone and nv < 2:
        pytest.skip("cone beam has at least 2 rows")
    assert _lib.MCT_CONE == 1
    o = _cone_obj(n=8, nz=2, nu=nu, nv=nv, views=views, ConeBeam=cone, **({} if cone else {"ImageDimensionZ": nv}))
    dg = geometry.fbp_geometry(o)
    f = torch.randn((views, dg.geom.nv, nu), device="cuda", generator=torch.Generator("cuda").manual_seed(nu + nv))
    got, td, scale = _packed(dg, f, storage)
    f = f * scale  # a power of two
    a, b = f[..., :-1].to(td).float(), f[..., 1:]
    if cone:
        assert torch.isnan(got[:, -1].float()).all()
        got, a, b, c, d = got[:, :-1], a[:, :-1], b[:, :-1], f[:, 1:, :-1], f[:, 1:, 1:]
        want = torch.stack([a, c - a, b - a, (d - c) - (b - a)], -1).to(td)
    else:
        want = torch.stack([a, b - a], -1).to(td)
    assert torch.equal(got, want)
