"""The rule by which the fan-beam backprojector leaves out the detector test (csrc/fan.cuh,
compiled here for the host): a pixel that it calls inside has an index in [0, nu - 2] in every
view, computed in float32 as the kernel computes it, whatever the geometry holds."""
import ctypes
import subprocess

import numpy as np
import pytest

from reconstruction_program_taichi_gb300 import _build

SOURCE = r"""
#include "fan.cuh"

extern "C" void fan_inside(int n, const float* x, const float* y, float sid, float sdd, float u0, float inv_ustep, int nu,
                           int curved, unsigned char* out) {
    for (int i = 0; i < n; ++i)
        out[i] = curved ? mct::fan_pair_inside<true>(x[i], y[i], x[i], y[i], sid, sdd, u0, inv_ustep, nu)
                        : mct::fan_pair_inside<false>(x[i], y[i], x[i], y[i], sid, sdd, u0, inv_ustep, nu);
}
"""


@pytest.fixture(scope="module")
def host_lib(tmp_path_factory):
    d = tmp_path_factory.mktemp("fan")
    (d / "fan.cu").write_text(SOURCE)
    out = str(d / "libfan.so")
    subprocess.run([_build.nvcc_path(), "-std=c++17", "-O1", "-shared", "-Xcompiler", "-fPIC", "-I", _build.CSRC,
                    str(d / "fan.cu"), "-o", out], check=True)
    return ctypes.CDLL(out)


def inside(lib, x, y, sid, sdd, u0, inv, nu, curved):
    x, y = np.ascontiguousarray(x, np.float32), np.ascontiguousarray(y, np.float32)
    out = np.zeros(x.size, np.uint8)
    f = [ctypes.c_float(float(a)) for a in (sid, sdd, u0, inv)]
    lib.fan_inside(x.size, x.ctypes.data_as(ctypes.c_void_p), y.ctypes.data_as(ctypes.c_void_p), *f, nu, int(curved),
                   out.ctypes.data_as(ctypes.c_void_p))
    return out.astype(bool)


def indices(x, y, sid, sdd, u0, inv, curved, angles):
    """Detector indices [pixel][view] in float32."""
    f = np.float32
    cb, sb = np.cos(angles).astype(f)[None], np.sin(angles).astype(f)[None]
    x, y = x.astype(f)[:, None], y.astype(f)[:, None]
    with np.errstate(all="ignore"):
        L = (f(sid) - x * cb) - y * sb
        t = y * cb - x * sb
        u = f(sdd) * np.arctan2(t, L) if curved else (f(sdd) * (f(1) / L)) * t
        return (u - f(u0)) * f(inv)


SCANS = [  # sid, sdd, nu, u_step, image radius over the radius that fills the detector
    (600.0, 1100.0, 512, -0.8, 1.1), (300.0, 550.0, 90, 0.5, 1.3), (300.0, 550.0, 65536, 1e-3, 1.01),
    (600.0, 1100.0, 40000, 0.1, 1.05), (1.0, 1e6, 2048, 900.0, 1.1), (-300.0, 550.0, 1024, 1.0, 0.9),
    (300.0, -550.0, 512, 1.0, 1.1), (1e25, 2e25, 512, 1.0, 1e30), (2e19, 4e19, 512, 1e16, 1.5), (float("inf"), 550.0, 512, 1.0, 1.0),
    (float("nan"), 550.0, 512, 1.0, 1.0), (300.0, float("nan"), 512, 1.0, 1.0), (300.0, 550.0, 1 << 22, 1e-3, 1.01),
    (1e-30, 2e-30, 512, 1e-32, 1.1), (1e-3, 1e38, 512, 1.0, 1.0)]


@pytest.mark.parametrize("sid,sdd,nu,u_step,wide", SCANS)
@pytest.mark.parametrize("curved", [False, True])
def test_inside_pixels_have_a_column_in_every_view(sid, sdd, nu, u_step, wide, curved, host_lib):
    rng = np.random.default_rng(7)
    with np.errstate(all="ignore"):
        half = abs(u_step) * (nu - 1) / 2
        angle = min(half / abs(sdd), 1.4) if curved else np.arctan(half / abs(sdd))
        full = wide * abs(sid) * np.sin(angle) if np.isfinite(sid) and np.isfinite(sdd) else 100.0
    full = float(min(max(full, 1e-37), 1e37)) if np.isfinite(full) else 100.0
    # pixels over the disc, near its rim (the detector's edge among them), and the axis
    rho = np.concatenate([full * np.sqrt(rng.uniform(0, 1, 300)), full / wide * (1 + rng.normal(0, 2.0 / nu, 300)), [0.0]])
    phi = rng.uniform(0, 2 * np.pi, rho.size)
    x, y = (rho * np.cos(phi)).astype(np.float32), (rho * np.sin(phi)).astype(np.float32)
    u0, inv = np.float32(-u_step * (nu - 1) / 2), np.float32(1.0 / u_step)
    got = inside(host_lib, x, y, sid, sdd, u0, inv, nu, curved)
    angles = np.concatenate([np.arange(720) * 2 * np.pi / 720, rng.uniform(0, 2 * np.pi, 300)])
    i = np.floor(indices(x[got], y[got], sid, sdd, u0, inv, curved, angles))
    assert ((i >= 0) & (i <= nu - 2)).all()
    if 1 <= sid < 1e4 and 0 < sdd < 1e7 and nu <= 65536:
        assert 0.2 < got.mean() < 1.0  # the rule is of use for the scans it is meant for
