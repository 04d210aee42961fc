"""Performance cases of the reconstruction framework: what a scan's user has it do, each
through the public entry points, from one small 2D slice to the full benchmark volume.

Five kinds of work:
  fbp      filtered backprojection of a device-resident sinogram (FdkPipeline.run): 2D fan
           beam and cone beam (FDK), flat and curved detectors, full and short scans, the
           three view modes, float32 and 16-bit operands
  fp       forward projection of a volume (ops.fp), cone and fan beam, float32 and 16-bit
  grad     the differentiable projector, forward and backward (autograd.Projector)
  ir       an IRN-CGLS-TV solve (Mgfbp_ir.solve_tv)
  helical  helical FBP by rebinning (Mgfbp_helical.reconstruct)

All scans share the benchmark's gantry (source to isocentre 600 mm, to detector 1100 mm),
its fields of view (cone beam 204.8 mm, fan beam 128 mm) and its phantom: 20 seeded
ellipsoids with 1e5-photon noise.  A case chooses the grid and the options.
"""
import math

import numpy as np
import torch

from reconstruction_program_taichi_gb300 import autograd, config, fbp, geometry, ops
from reconstruction_program_taichi_gb300.helical import Mgfbp_helical
from reconstruction_program_taichi_gb300.ir import Mgfbp_ir

PI = 3.1415926536  # the framework's constant: angles, scan ranges and taps are built from it
SID, SDD = 600.0, 1100.0
HELICAL_SID = 600.5  # so that no slice lies exactly half way between two views
PHOTONS = 1e5
DEV = "cuda"

CASE = dict(kind="fbp", cone=True, nx=0, nz=1, nu=0, nv=1, views=0, scan=360.0, curved=False, mode="axial", offset=0.0,
            hamming=1.0, storage="float32", step=0.2, pitch=1.0, irn=1, cg=3)


def _case(name=None, **kw):
    c = dict(CASE, **kw)
    return dict(c, name=name) if name else c


def listed():
    return [
        # the smallest reconstruction: one 2D slice, as an interactive user or a request to a
        # server asks for; launches and latency count
        _case("fan_256", cone=False, nx=256, nu=512, views=720),
        # a large 2D slice in mixed precision, the biggest 2D request of a server
        _case("fan_1024_mixed", cone=False, nx=1024, nu=2048, views=1440, storage="bfloat16"),
        # a small cone-beam volume: previews, parameter searches
        _case("fdk_128", nx=128, nz=64, nu=256, nv=64, views=270),
        # an ordinary scan with none of the sizes round: curved detector, short scan with
        # Parker weights, a shifted detector, a soft kernel
        _case("fdk_333_short_curved", nx=333, nz=101, nu=701, nv=157, views=500, scan=220.0, curved=True, offset=3.1,
              hamming=0.54),
        # a cubic volume in coronal view mode with 16-bit operands
        _case("fdk_256_coronal_mixed", nx=256, nz=256, nu=512, nv=256, views=360, mode="coronal", storage="bfloat16"),
        # the benchmark reconstruction: a full scan of 1080 views
        _case("fdk_512", nx=512, nz=256, nu=1024, nv=256, views=1080),
        # forward projection of a preview volume
        _case("fp_128", kind="fp", nx=128, nz=64, nu=256, nv=64, views=270),
        # a sparse-view projection in 16-bit storage, as the few-view solvers apply it
        _case("fp_512_sparse_mixed", kind="fp", nx=512, nz=128, nu=1024, nv=128, views=90, storage="bfloat16"),
        # the benchmark projection: a full scan simulated from a reconstructed volume
        _case("fp_512", kind="fp", nx=512, nz=256, nu=1024, nv=256, views=1080),
        # one training step's projector: forward, and the exact adjoint backward, odd sizes
        _case("grad_250", kind="grad", nx=250, nz=45, nu=501, nv=47, views=181),
        # an iterative reconstruction: the plain CGLS solve and one TV reweighting
        _case("ir_256", kind="ir", nx=256, nz=64, nu=512, nv=64, views=180),
        # a helical scan of three rounds
        _case("helical_512", kind="helical", nx=512, nz=1, nu=1024, nv=64, views=2160, scan=1080.0),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    while True:
        kind = rng.choice(["fan", "fbp", "fbp", "fp", "fp", "fp_fan", "grad", "ir", "helical"])
        nx = _log(rng, 96, 512)
        nz = max(8, int(nx * rng.uniform(0.1, 0.6)))
        nu = int(nx * rng.uniform(1.6, 2.2))
        nv = max(8, int(nz * rng.uniform(0.7, 1.3)))
        c = dict(nx=nx, nz=nz, nu=nu, nv=nv, views=_log(rng, 60, 1080), curved=rng.random() < 0.25,
                 offset=rng.choice([0.0, 0.0, 1.3, -2.6]))
        if kind == "fan":
            nx, nz = _log(rng, 128, 1024), rng.choice([1, 1, 1, 3, 8, 20])
            c.update(kind="fbp", cone=False, nx=nx, nz=nz, nv=nz, nu=int(nx * rng.uniform(1.6, 2.2)),
                     views=_log(rng, 180, 1440), hamming=rng.choice([1.0, 0.54]), scan=rng.choice([360.0, 360.0, 220.0]),
                     storage=rng.choice(["float32", "float32", "bfloat16", "float16"]))
        elif kind == "fbp":
            c.update(kind="fbp", hamming=rng.choice([1.0, 0.54]), scan=rng.choice([360.0, 360.0, 220.0]),
                     mode=rng.choice(["axial", "axial", "axial", "coronal", "sagittal"]),
                     storage=rng.choice(["float32", "float32", "float32", "bfloat16", "float16"]))
            if c["mode"] != "axial":
                c["nv"] = int(nx * rng.uniform(0.7, 1.3))
        elif kind == "fp":
            c.update(kind="fp", step=rng.choice([0.1, 0.2, 0.2, 0.2, 0.3, 0.5]),
                     storage=rng.choice(["float32", "float32", "float32", "bfloat16", "float16"]))
        elif kind == "fp_fan":
            nz = rng.choice([1, 1, 4, 16])
            c.update(kind="fp", cone=False, nz=nz, nv=nz, step=rng.choice([0.1, 0.2, 0.2, 0.3]))
        elif kind == "grad":
            c.update(kind="grad", step=rng.choice([0.2, 0.2, 0.3]), views=_log(rng, 60, 360))
        elif kind == "ir":
            c.update(kind="ir", views=_log(rng, 60, 360), curved=False, cg=rng.choice([2, 3]),
                     storage=rng.choice(["float32", "float32", "bfloat16"]))
        else:
            rounds = rng.choice([2, 3, 4])
            c.update(kind="helical", nz=1, nv=rng.choice([16, 33, 64]), views=rounds * rng.choice([180, 360, 501, 720]),
                     scan=360.0 * rounds, curved=False, offset=0.0, pitch=rng.choice([1.0, 1.0, 0.75]))
        c = _case(**c)
        # no more than the largest listed case takes; at most a few GB of inputs
        if _seconds(c) <= 0.15 and _sgm_elems(c) <= 3e8:
            return c


# ---------------------------------------------------------------- geometry

def _geo(c):
    """Sizes and spacings of a case."""
    fov, width = (204.8, 819.2) if c["cone"] else (128.0, 409.6)
    g = dict(c, px=fov / c["nx"], du=width / c["nu"], sid=SID)
    g["pz"] = g["px"] if c["cone"] else 0.0
    # the detector is twice as high as the volume (the benchmark's proportion), whose height is
    # the image's row axis in the coronal and sagittal view modes
    high = c["nz"] if c["mode"] == "axial" else c["nx"]
    g["dv"] = 2.0 * high * g["px"] / c["nv"] if c["cone"] else 0.0
    if c["kind"] == "helical":
        g.update(sid=HELICAL_SID, dv=51.2 / c["nv"], pz=0.4)
    return g


def _sgm_elems(c):
    return c["nv"] * c["views"] * c["nu"]


def _config(c):
    g = _geo(c)
    cfg = {"InputDir": "/tmp", "OutputDir": "/tmp/mandoct_perf", "InputFiles": "none", "OutputFilePrefix": "",
           "OutputFileReplace": ["sgm", "rec"], "DetectorElementCountHorizontal": c["nu"], "DetectorElementWidth": g["du"],
           "DetectorOffsetHorizontal": c["offset"], "DetectorElementCountVertical": c["nv"], "Views": c["views"],
           "TotalScanAngle": c["scan"], "SourceIsocenterDistance": g["sid"], "SourceDetectorDistance": SDD,
           "ImageDimension": c["nx"], "PixelSize": g["px"], "CurvedDetector": c["curved"], "HammingFilter": c["hamming"],
           "ConeBeam": c["cone"], "ReconViewMode": c["mode"], "ForwardProjectionStepSize": c["step"]}
    if c["cone"]:
        cfg.update(DetectorElementHeight=g["dv"], DetectorOffsetVertical=0.0, ImageDimensionZ=c["nz"],
                   VoxelHeight=g["pz"])
    if c["kind"] == "ir":
        cfg.update(Lambda=1e-3, BetaTV=1e-6, NumberOfIRNIterations=c["irn"], NumberOfIterations=c["cg"],
                   StoragePrecision=c["storage"])
    if c["kind"] == "helical":
        cfg.update(HelicalPitch=c["pitch"])
    return cfg


class _Obj:
    verbose = False


def _parsed(c):
    o, cfg = _Obj(), _config(c)
    config.parse_fbp(o, cfg)
    config.parse_fpj(o, cfg)
    config.parse_fpj_v3(o, cfg)
    return o


def _arrays(g, dtype=torch.float64):
    """Detector columns, rows and view angles as the framework orders them."""
    s = dict(device=DEV, dtype=dtype)
    u = -(torch.arange(g["nu"], **s) - (g["nu"] - 1) / 2) * g["du"] - g["offset"]
    v = (torch.arange(g["nv"], **s) - (g["nv"] - 1) / 2) * g["dv"]
    if g["kind"] == "ir":
        v = -v
    ang = torch.arange(g["views"], **s) * (g["scan"] / 180.0 * PI / g["views"])
    return u, v, ang


# ---------------------------------------------------------------- inputs

def _ellipsoids(g, seed):
    rng = np.random.default_rng(seed)
    fov, zext = g["nx"] * g["px"] / 2, max(g["nz"] * g["pz"] / 2, 1.0)
    if g["kind"] == "helical":
        zext = 60.0
    out = []
    for _ in range(20):
        r, a = 0.6 * fov * math.sqrt(rng.uniform()), rng.uniform(0, 2 * math.pi)
        ax, ay = rng.uniform(0.05, 0.4, 2) * fov
        az, cz = (rng.uniform(0.05, 0.4) * zext, rng.uniform(-0.4, 0.4) * zext) if g["cone"] else (1e7, 0.0)
        out.append((r * math.cos(a), r * math.sin(a), cz, ax, ay, az, rng.uniform(0, math.pi), rng.uniform(0.01, 0.05)))
    return out


def _sinogram(g, seed):
    """Noisy line integrals [rows, views, columns] of the seeded phantom."""
    u, v, ang = _arrays(g, torch.float32)
    gen = torch.Generator(device=DEV).manual_seed(int(seed))
    cb, sb = torch.cos(ang)[:, None], torch.sin(ang)[:, None]
    if g["curved"]:
        du, dp = SDD * torch.sin(u / SDD), SDD * torch.cos(u / SDD)
    else:
        du, dp = u, torch.full_like(u, SDD)
    dx, dy = -dp * cb - du * sb, -dp * sb + du * cb  # source to detector element, [views, columns]
    ox, oy = g["sid"] * cb, g["sid"] * sb
    oz = torch.zeros(g["views"], device=DEV)
    if g["kind"] == "helical":
        oz = torch.arange(g["views"], device=DEV) * _helical(g)["dpv"]
        oz = oz - oz.mean()
    v3, oz3 = v[:, None, None], oz[None, :, None]
    sgm = torch.zeros(g["nv"], g["views"], g["nu"], device=DEV)
    for x, y, z, a, b, h, phi, mu in _ellipsoids(g, seed):
        c, s = math.cos(phi), math.sin(phi)
        px, py = ((ox - x) * c + (oy - y) * s) / a, (-(ox - x) * s + (oy - y) * c) / b
        qx, qy = (dx * c + dy * s) / a, (-dx * s + dy * c) / b
        A = (qx * qx + qy * qy)[None] + (v3 / h) ** 2
        B = (px * qx + py * qy)[None] + (oz3 - z) * v3 / (h * h)
        disc = B * B - A * ((px * px + py * py - 1.0)[None] + ((oz3 - z) / h) ** 2)
        del B
        sgm += disc.clamp_(min=0.0).sqrt_().mul_(2.0 * mu).div_(A)
        del A, disc
    sgm *= torch.sqrt((du * du + dp * dp)[None, None] + v3 * v3)
    sgm += torch.sqrt(torch.exp(sgm) / PHOTONS) * torch.randn(sgm.shape, device=DEV, generator=gen)
    return sgm


def _volume(g, seed):
    """The seeded phantom at the voxel centres, with the noise of a reconstruction."""
    gen = torch.Generator(device=DEV).manual_seed(int(seed) + 1)
    nx, nz = g["nx"], g["nz"]
    s = dict(device=DEV, dtype=torch.float32)
    x = ((torch.arange(nx, **s) - (nx - 1) / 2) * g["px"])[None, None, :]
    y = (((nx - 1) / 2 - torch.arange(nx, **s)) * g["px"])[None, :, None]
    z = ((torch.arange(nz, **s) - (nz - 1) / 2) * g["pz"])[:, None, None]
    vol = torch.randn(nz, nx, nx, generator=gen, **s) * 5e-4
    for ex, ey, ez, a, b, h, phi, mu in _ellipsoids(g, seed):
        c, sn = math.cos(phi), math.sin(phi)
        px, py = ((x - ex) * c + (y - ey) * sn) / a, (-(x - ex) * sn + (y - ey) * c) / b
        vol += ((px * px + py * py) + ((z - ez) / h) ** 2 <= 1.0).float() * mu
    return vol


def _inputs(c, seed):
    g = _geo(c)
    if c["kind"] in ("fbp", "helical"):
        return dict(sgm=_sinogram(g, seed))
    if c["kind"] == "fp":
        return dict(vol=_volume(g, seed))
    if c["kind"] == "grad":
        gen = torch.Generator(device=DEV).manual_seed(int(seed) + 2)
        # the upstream gradient of a data-fidelity loss: a residual of measurement size
        return dict(vol=_volume(g, seed), up=torch.randn(c["nv"], c["views"], c["nu"], device=DEV, generator=gen) * 0.05)
    x0 = _volume(g, seed)
    return dict(sgm=_sinogram(g, seed), x0=torch.nn.functional.avg_pool3d(x0[None, None], 3, 1, 1)[0, 0].contiguous())


def prepare(case, seed):
    c = dict(CASE, **case)
    st = dict(kind=c["kind"], **_inputs(c, seed))
    dtype = {"float32": ops.MCT_F32, "bfloat16": ops.MCT_BF16, "float16": ops.MCT_F16}[c["storage"]]
    if c["kind"] == "fbp":
        filt = "tc3" if c["storage"] == "float32" else "tc"
        st["pipe"] = fbp.FdkPipeline(_parsed(c), storage=c["storage"], filter_impl=filt).allocate()
    elif c["kind"] == "fp":
        st["dg"], st["dtype"] = geometry.fpj_geometry(_parsed(c)), dtype
        st["out"] = torch.empty(st["dg"].sgm_shape, device=DEV)
        ops.fp_workspace(st["dg"], dtype)
    elif c["kind"] == "grad":
        st["projector"] = autograd.Projector(geometry.fpj_geometry(_parsed(c)))
        st["vol"].requires_grad_(True)
    elif c["kind"] == "ir":
        st["ir"] = Mgfbp_ir(_config(c), verbose=False)
        st["ir"].system
    else:
        st["helical"] = Mgfbp_helical(_config(c), verbose=False)
    return st


def run(st):
    kind = st["kind"]
    if kind == "fbp":
        return st["pipe"].run(st["sgm"])
    if kind == "fp":
        return ops.fp(st["dg"], st["vol"], out=st["out"], dtype=st["dtype"])
    if kind == "grad":
        y = st["projector"](st["vol"])
        (g,) = torch.autograd.grad(y, st["vol"], st["up"])
        return y.detach(), g
    if kind == "ir":
        return st["ir"].solve_tv(st["sgm"], st["x0"])
    return st["helical"].reconstruct(st["sgm"], save_rebinned=False)


# ---------------------------------------------------------------- work

def _samples(c):
    """In-volume samples of one projection: the volume's extent times the density of the
    samples (rays per area at the isocentre, steps per length)."""
    g, mag = _geo(c), SDD / SID
    step = c["step"] * math.sqrt(2 * g["px"] ** 2 + g["pz"] ** 2)
    area = (c["nx"] * g["px"]) ** 2
    if c["cone"]:
        return c["views"] * area * c["nz"] * g["pz"] * mag * mag / (g["du"] * g["dv"]) / step
    return c["views"] * area * c["nz"] * mag / g["du"] / step


def _helical(g):
    """Slices and per-slice views of a helical scan, as run_mgfbp_helical.py:61-95 derives them."""
    mag = SDD / g["sid"]
    cover = g["nv"] * g["dv"] / mag
    scan = g["scan"] / 180.0 * PI
    per_view, rounds = scan / g["views"], scan / (2 * PI)
    dpv = g["pitch"] * cover / (g["views"] / rounds)
    gamma = 2 * np.arctan(0.5 * g["nu"] * g["du"] / SDD) / PI
    short = max(2 * PI / g["pitch"], PI + gamma)
    z = np.arange(cover / 2.0, dpv * g["views"] - cover / 2.0, g["pz"], dtype=np.float32)
    vc = int(np.ceil(short / per_view))
    return dict(mag=mag, dpv=dpv, z=z, vc=vc, per_view=per_view, scan=vc * per_view)


def _updates(c):
    """Voxel x view updates of one backprojection."""
    if c["kind"] == "helical":
        h = _helical(_geo(c))
        return len(h["z"]) * c["nx"] ** 2 * h["vc"]
    return c["nx"] ** 2 * c["nz"] * c["views"]


def work(case):
    c = dict(CASE, **case)
    vol, sgm = c["nx"] ** 2 * c["nz"], _sgm_elems(c)
    if c["kind"] in ("fbp", "helical"):
        rows = sgm / c["nu"]
        if c["kind"] == "helical":
            h = _helical(_geo(c))
            vol, rows = c["nx"] ** 2 * len(h["z"]), len(h["z"]) * h["vc"]
        # bilinear interpolation and the weight per update; the row filter as two FFTs
        return {"bytes": 4.0 * (vol + sgm), "flops": 8.0 * _updates(c) + rows * 20.0 * c["nu"] * math.log2(2 * c["nu"])}
    per = 15.0 if c["cone"] else 7.0  # trilinear (bilinear) interpolation and the sum
    if c["kind"] == "fp":
        return {"bytes": 4.0 * (vol + sgm), "flops": per * _samples(c)}
    if c["kind"] == "grad":
        return {"bytes": 8.0 * (vol + sgm), "flops": 2 * per * _samples(c)}
    n = (c["irn"] + 1) * (c["cg"] + 1)
    return {"bytes": 4.0 * (2 * vol + sgm), "flops": n * (per * _samples(c) + 12.0 * _updates(c))}


def _seconds(c):
    """Rough cost of a pass, for draw()."""
    if c["kind"] in ("fbp", "helical"):
        return _updates(c) / (1e12 if c["cone"] and c["kind"] == "fbp" else 4e11)
    if c["kind"] == "fp":
        return _samples(c) / 7e11
    if c["kind"] == "grad":
        return _samples(c) / 2e11
    return (c["irn"] + 1) * (c["cg"] + 1) * (_samples(c) / 7e11 + _updates(c) / 1e12)


# ---------------------------------------------------------------- the same in 64 bits

F64 = dict(device=DEV, dtype=torch.float64)


def _taps(g):
    """Apodised ramp of run_mgfbp.py:877-914, taps -(nu-1) .. nu-1."""
    nu, du, t = g["nu"], g["du"], g["hamming"]
    n = np.arange(2 * nu - 1, dtype=np.int64) - (nu - 1)
    h = np.zeros(n.shape)
    h[n == 0] = t / (4.0 * du * du)
    m = n[n % 2 != 0].astype(np.float64)
    a = m * du / SDD
    h[n % 2 != 0] = -t / (PI * SDD * (a - a ** 3 / 6.0 + a ** 5 / 120.0)) ** 2 if g["curved"] else -t / (PI * m * du) ** 2
    p, q = 1.0 / (1.0 + 2.0 * n), 1.0 / (1.0 - 2.0 * n)
    sgn = np.where(n % 2 == 0, 1.0, -1.0)
    return h + (1.0 - t) * (sgn / (2 * PI * du * du) * (p + q) - (p * p + q * q) / (PI * PI * du * du))


def _parker(g, beta, u, scan):
    """Weights of an over- or short scan, run_mgfbp.py:971-1011; [views, columns]."""
    gamma = -u / SDD if g["curved"] else torch.atan2(-u, torch.full_like(u, SDD))
    beta, gamma = beta[:, None], gamma[None]
    nr = math.floor(scan / (2 * PI))
    ra = scan - nr * 2 * PI
    one = torch.ones_like(beta + gamma)
    if ra <= PI:
        if nr == 0:
            return one
        end = 2 * PI * nr + ra
        w = torch.where(beta < ra, beta / ra * one, one)
        return torch.where(beta < 2 * PI * nr, w, (end - beta) / ra * one)
    gm = ra - PI
    a, b = gm - 2 * gamma, PI * (2 * nr + 1) - 2 * gamma
    up = torch.sin(PI / 2 * beta / a) ** 2
    down = torch.sin(PI / 2 * (PI + gm - (beta - 2 * PI * nr)) / (gm + 2 * gamma)) ** 2
    return torch.where(beta < a, up, torch.where(beta < b, one, down))


def _filtered(g, sgm, scan, beta, full):
    """Weighted and filtered view-major sinogram [views, rows, columns] in 64 bits."""
    u, v, _ = _arrays(g)
    u3, v3 = u[None, None, :], v[:, None, None]
    if g["curved"]:
        wt = SDD * SDD * torch.cos(u3 / SDD) / torch.sqrt(SDD * SDD + v3 * v3)
    else:
        wt = SDD * SDD / torch.sqrt(SDD * SDD + u3 * u3 + v3 * v3)
    if not full:
        wt = wt * _parker(g, beta, u, scan)[None]
    nu, taps = g["nu"], torch.from_numpy(_taps(g)).to(DEV)
    n = 1 << (3 * nu).bit_length()
    H = torch.fft.rfft(taps, n)
    out = torch.empty(sgm.shape[1], sgm.shape[0], nu, **F64)
    step = max(1, int(2e7 // (sgm.shape[0] * n)))
    for j in range(0, sgm.shape[1], step):
        x = sgm[:, j:j + step].double() * (wt[:, j:j + step] if wt.shape[1] > 1 else wt)
        y = torch.fft.irfft(torch.fft.rfft(x, n) * H, n)[..., nu - 1:2 * nu - 1]
        out[j:j + step] = y.permute(1, 0, 2) * g["du"]
    return out


def _columns(g):
    """x and y of the voxel columns ([cb, nx]) and z of the slices, for the view mode."""
    nx, nz = g["nx"], g["nz"]
    i, k = torch.arange(nx, **F64) - (nx - 1) / 2, torch.arange(nz, **F64) - (nz - 1) / 2
    if g["mode"] == "axial":
        return (i * g["px"])[None, :].expand(nx, nx), (-i * g["px"])[:, None].expand(nx, nx), k * g["pz"]
    if g["mode"] == "coronal":
        return (i * g["px"])[None, :].expand(nz, nx), (-k * g["pz"])[:, None].expand(nz, nx), -i * g["px"]
    return (k * g["pz"])[:, None].expand(nz, nx), (-i * g["px"])[None, :].expand(nz, nx), -i * g["px"]


def _detector(g, x, y, b):
    L = g["sid"] - x * math.cos(b) - y * math.sin(b)
    t = -x * math.sin(b) + y * math.cos(b)
    u = SDD * torch.atan2(t, L) if g["curved"] else SDD * t / L
    ui = (u + g["offset"]) / -g["du"] + (g["nu"] - 1) / 2
    return L, t, ui


def _gather(F, ui, vi):
    """Bilinear samples F(vi, ui) of one view: F [rows, columns], ui [n], vi [slices, n]."""
    grid = torch.empty(1, *vi.shape, 2, **F64)
    grid[0, ..., 0] = ui * (2.0 / (F.shape[1] - 1)) - 1.0
    torch.mul(vi, 2.0 / (F.shape[0] - 1), out=grid[0, ..., 1])
    grid[0, ..., 1] -= 1.0
    return torch.nn.functional.grid_sample(F[None, None], grid, align_corners=True)[0, 0]


def _backproject(g, F, angles, dbeta, div, rot=0.0):
    """Pixel-driven backprojection of F [views, rows, columns]; zero where any view misses."""
    x, y, z = _columns(g)
    if rot:
        x, y = x * math.cos(rot) + y * math.sin(rot), -x * math.sin(rot) + y * math.cos(rot)
    shape, x, y = x.shape, x.reshape(-1), y.reshape(-1)
    acc = torch.zeros(len(z) if g["cone"] else F.shape[1], x.numel(), **F64)
    dead = torch.zeros(x.numel(), dtype=torch.bool, device=DEV)
    lo, hi = torch.full_like(x, 1e30), torch.full_like(x, -1e30)
    for j, b in enumerate(angles):
        L, t, ui = _detector(g, x, y, b)
        dead |= (ui < 0) | (ui + 1 > g["nu"] - 1)
        w = g["sid"] / (L * L + t * t if g["curved"] else L * L) * (dbeta[j] * div)
        if g["cone"]:
            mag = SDD / L
            lo, hi = torch.minimum(lo, mag), torch.maximum(hi, mag)
            vi = z[:, None] * (mag / g["dv"])[None]
            vi += (g["nv"] - 1) / 2
            acc.addcmul_(_gather(F[j], ui, vi), w[None])
            del vi
        else:
            i0 = ui.floor().clamp(0, g["nu"] - 2).long()
            r = ui - i0
            acc.addcmul_(F[j][:, i0] * (1 - r) + F[j][:, i0 + 1] * r, w[None])
    acc[:, dead] = 0.0
    if g["cone"]:
        for m in (lo, hi):
            vi = z[:, None] * (m / g["dv"])[None] + (g["nv"] - 1) / 2
            acc[(vi < 0) | (vi >= g["nv"] - 1)] = 0.0
    acc = acc.reshape(-1, *shape)
    return acc if g["mode"] == "axial" else acc.permute(1, 0, 2).contiguous()


def _redundancy(scan, full):
    rounds = math.floor(scan / (2 * PI) + 1e-12)
    if full:
        return 1.0 / (2.0 * rounds)
    if scan < 2 * PI:
        return 1.0
    return 1.0 / (2.0 * rounds) if scan - rounds * 2 * PI < PI else 1.0 / (2.0 * rounds + 1.0)


def _fbp64(g, sgm):
    _, _, ang = _arrays(g)
    scan = g["scan"] / 180.0 * PI
    full = abs(scan % (2 * PI)) < 0.01 / 180 * PI
    F = _filtered(g, sgm, scan, ang - ang[0], full)
    db = [scan / g["views"]] * g["views"]
    return _backproject(g, F, ang.tolist(), db, _redundancy(scan, full))


def _helical64(g, sgm):
    h = _helical(g)
    vc, nz = h["vc"], len(h["z"])
    z = torch.from_numpy(h["z"]).to(DEV).double()
    v0 = z / h["dpv"]
    idx = torch.floor(v0 - 0.5 * vc + 0.5)[:, None] + torch.arange(vc, **F64)[None]
    ok = (idx >= 0) & (idx <= g["views"] - 2)
    v_pos = (z[:, None] - idx * h["dpv"]) * h["mag"]
    vi = (-v_pos / g["dv"] + (g["nv"] - 1.0) / 2.0).clamp(0, g["nv"] - 1)
    i0 = vi.floor().clamp(max=g["nv"] - 2).long()
    r = (vi - i0)[..., None]
    j = idx.clamp(0, g["views"] - 1).long()
    scale = (ok * SDD / torch.sqrt(SDD * SDD + v_pos * v_pos))[..., None]
    stack = torch.empty(nz, vc, g["nu"], **F64)
    for s in range(nz):  # [views, columns] of one slice
        stack[s] = (sgm[i0[s], j[s]].double() * (1 - r[s]) + sgm[i0[s] + 1, j[s]].double() * r[s]) * scale[s]
    full = abs(h["scan"] % (2 * PI)) < 0.01 / 180 * PI
    base = (torch.arange(vc, **F64) * (h["scan"] / vc)).tolist()
    fan = dict(g, cone=False, nv=1, views=vc, scan=h["scan"] / PI * 180.0)
    F = _filtered(dict(fan, dv=0.0), stack, h["scan"], torch.tensor(base, **F64), full)
    rots = np.floor(h["z"].astype(np.float64) / h["dpv"] - 0.5 * (vc - 1.0)) * h["per_view"]
    one = dict(fan, nz=1)
    return torch.stack([_backproject(one, F[:, s:s + 1], base, [h["scan"] / vc] * vc, _redundancy(h["scan"], full),
                                     float(rots[s]))[0] for s in range(nz)])


def _steps(g):
    size = math.sqrt(2 * (g["nx"] * g["px"]) ** 2 + (g["nz"] * g["pz"]) ** 2)
    vd = math.sqrt(2 * g["px"] ** 2 + g["pz"] ** 2)
    return size, g["step"] * vd, int(math.floor(size / (g["step"] * vd)))


def _ray(g, u, v, b):
    """Voxel index at step 0 and its increment per step, for the rays of one view: [.., 3]."""
    size, step, _ = _steps(g)
    if g["curved"]:
        ex, ey = -SDD * torch.cos(u / SDD), SDD * torch.sin(u / SDD)
    else:
        ex, ey = torch.full_like(u, -SDD), u
    norm = torch.sqrt(ex * ex + ey * ey + v[:, None] ** 2)
    c, s, l0 = math.cos(b), math.sin(b), g["sid"] - size / 2
    dx, dy, dz = (ex * c - ey * s) / norm, (ey * c + ex * s) / norm, v[:, None] / norm
    n, px = g["nx"], g["px"]
    f0 = [(g["sid"] * c + l0 * dx) / px + (n - 1) / 2, -(g["sid"] * s + l0 * dy) / px + (n - 1) / 2]
    df = [dx * step / px, -dy * step / px]
    if g["cone"]:
        f0.append(l0 * dz / g["pz"] + (g["nz"] - 1) / 2)
        df.append(dz * step / g["pz"])
    return torch.stack(f0, -1), torch.stack(df, -1)


def _points(g, u, v, b):
    """Sample positions [rows, columns, steps, axes] of one view, and which lie inside."""
    f0, df = _ray(g, u, v, b)
    k = torch.arange(_steps(g)[2], **F64)
    f = f0[..., None, :] + df[..., None, :] * k[:, None]
    inside = torch.ones(f.shape[:-1], dtype=torch.bool, device=DEV)
    for a in range(f.shape[-1]):
        i = torch.floor(f[..., a])
        inside &= (i >= 0) & (i + 1 < (g["nx"], g["nx"], g["nz"])[a])
    return f, inside


def _project_view(g, vol, u, v, b):
    f, inside = _points(g, u, v, b)
    size = torch.tensor([g["nx"], g["nx"], g["nz"]][:f.shape[-1]], **F64)
    f.mul_(2.0 / (size - 1)).sub_(1.0)
    if g["cone"]:
        s = torch.nn.functional.grid_sample(vol[None, None], f[None], align_corners=True)[0, 0]
    else:
        s = torch.nn.functional.grid_sample(vol[:, None], f, align_corners=True)[:, 0]
    return (s * inside).sum(-1) * _steps(g)[1]


def _project64(g, vol):
    u, v, ang = _arrays(g)
    return torch.stack([_project_view(g, vol, u, v, b) for b in ang.tolist()], 1)


def _adjoint64(g, up):
    u, v, ang = _arrays(g)
    total = torch.zeros(g["nz"], g["nx"], g["nx"], **F64)
    x = torch.zeros_like(total, requires_grad=True)
    for j, b in enumerate(ang.tolist()):
        total += torch.autograd.grad(_project_view(g, x, u, v, b), x, up[:, j].double())[0]
    return total


def _ray_map(g):
    """1 for the rays that do not leave the reconstructed cylinder through its ends."""
    u, v, ang = _arrays(g)
    keep = torch.empty(g["nv"], g["views"], g["nu"], **F64)
    n, h = g["nx"], g["nx"] / 2.0
    for j, b in enumerate(ang.tolist()):
        f = torch.floor(_points(g, u, v, b)[0])
        x, y, z = f.unbind(-1)
        inside = (x >= 0) & (x + 1 < n) & (y >= 0) & (y + 1 < n) & ((x - h) ** 2 + (y - h) ** 2 < h * h)
        keep[:, j] = (~(inside & ((z < 0) | (z + 1 >= g["nz"]))).any(-1)).double()
    return keep


def _unmatched64(g, sgm):
    """The solver's backprojector: distance-weighted bilinear gathers, zero where u misses."""
    _, _, ang = _arrays(g)
    x, y, z = (a.reshape(-1) for a in _columns(g))
    acc, dead = torch.zeros(len(z), x.numel(), **F64), torch.zeros(x.numel(), dtype=torch.bool, device=DEV)
    for j, b in enumerate(ang.tolist()):
        L, _, ui = _detector(g, x, y, b)
        dead |= (ui < 0) | (ui + 1 > g["nu"] - 1)
        qx, qy = x - g["sid"] * math.cos(b), y - g["sid"] * math.sin(b)
        w = torch.sqrt(qx * qx + qy * qy + z[:, None] ** 2) / torch.maximum(qx.abs(), qy.abs()) * g["px"]
        vi = -z[:, None] * (SDD / L / g["dv"])[None] + (g["nv"] - 1) / 2
        w *= (vi >= 0) & (vi < g["nv"] - 1)
        acc.addcmul_(_gather(sgm[:, j], ui, vi), w)
    acc[:, dead] = 0.0
    return acc.reshape(-1, g["nx"], g["nx"])


def _diffs(x):
    d = [torch.zeros_like(x) for _ in range(3)]
    d[0][:, :-1], d[1][:, :, :-1] = x[:, 1:] - x[:, :-1], x[:, :, 1:] - x[:, :, :-1]
    if x.shape[0] > 2:
        d[2][:-1] = x[1:] - x[:-1]
    return d


def _dtwd(x, w):
    a, b, c = (w * d for d in _diffs(x))
    r = torch.zeros_like(x)
    r[:, 1:-1] -= a[:, 1:-1] - a[:, :-2]
    r[:, :, 1:-1] -= b[:, :, 1:-1] - b[:, :, :-2]
    if x.shape[0] > 2:
        r[1:-1] -= c[1:-1] - c[:-2]
    return r


def _solve64(g, sgm, x):
    keep = _ray_map(g)
    lam = 1e-3 * _sgm_elems(g) / (g["nz"] * g["nx"] ** 2)
    rhs, w = _unmatched64(g, sgm.double() * keep), torch.ones_like(x)

    def apply(d):
        return _unmatched64(g, _project64(g, d) * keep) + lam * _dtwd(d, w)

    for k in range(g["irn"] + 1):
        if k:
            w = 1.0 / torch.sqrt(sum(d * d for d in _diffs(x)) + 1e-6)
        d = rhs - apply(x)
        r = d.clone()
        for _ in range(g["cg"]):
            q, rr = apply(d), (r * r).sum()
            a = rr / (d * q).sum()
            x, r = x + a * d, r - a * q
            d = r + (r * r).sum() / rr * d
    return x


def exact(case, seed):
    c = dict(CASE, **case)
    g = _geo(c)
    points = c["nv"] * c["views"] * c["nu"] * _steps(g)[2]
    if c["kind"] == "fbp":
        return _fbp64(g, _sinogram(g, seed)) if _updates(c) <= 8e10 else None
    if c["kind"] == "helical":
        return _helical64(g, _sinogram(g, seed)) if _updates(c) <= 3e10 else None
    if c["kind"] == "fp":
        return _project64(g, _volume(g, seed).double()) if points <= 4e10 else None
    inp = _inputs(c, seed)
    if c["kind"] == "grad":
        return (_project64(g, inp["vol"].double()), _adjoint64(g, inp["up"])) if points <= 1e10 else None
    return _solve64(g, inp["sgm"], inp["x0"].double()) if points * (c["irn"] + 1) * (c["cg"] + 1) <= 6e10 else None
