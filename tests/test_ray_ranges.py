"""The step range that the projector and its adjoint walk without testing each sample
(csrc/ray.cuh, compiled here for the host): every sample of it lies in a cell of the volume."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

from conftest import ROOT
from reconstruction_program_taichi_gb300 import _build, _lib

SOURCE = r"""
#include "ray.cuh"

extern "C" void ray_ranges(const mct_geom* g, const float* angles, const float* u, const float* v, const float* czv,
                           const float* pa, const float* pxs, int32_t* steps, float* terms) {
    const mct::FpParams p = mct::ray_params(g);
    for (int j = 0; j < p.views; ++j)
        for (int iv = 0; iv < p.nv; ++iv)
            for (int iu = 0; iu < p.nu; ++iu, steps += 4, terms += 6) {
                mct::Ray r{};
                int kis = 1, kie = 0;
                const bool any = mct::setup_ray(p, iu, iv, j, angles, u, v, czv, pa, pxs, true, r);
                if (any) mct::interior_range(p, r, p.cone, kis, kie);
                const int32_t s[4] = {any ? r.ks : 0, any ? r.ke : -1, kis, kie};
                const float t[6] = {r.fx0, r.dfx, r.fy0, r.dfy, r.fz0, r.dfz};
                for (int i = 0; i < 4; ++i) steps[i] = s[i];
                for (int i = 0; i < 6; ++i) terms[i] = t[i];
            }
}
"""


@pytest.fixture(scope="module")
def host_lib(tmp_path_factory):
    d = tmp_path_factory.mktemp("rays")
    (d / "rays.cu").write_text(SOURCE)
    out = str(d / "librays.so")
    subprocess.run([_build.nvcc_path(), "-std=c++17", "-O1", "-shared", "-Xcompiler", "-fPIC", "-I", _build.CSRC, "-I",
                    os.path.join(ROOT, "include"), str(d / "rays.cu"), "-o", out], check=True)
    return ctypes.CDLL(out)


def geom(nx, nz, nu, nv, views, step=0.2, cone=True, px=0.5, pz=0.5, wide=1.3, high=0.9, cz=0.0, sid=300.0, sdd=550.0):
    """A scan of `views` views whose detector spans wide x high times the image, and its tables."""
    du, dv = wide * nx * px * sdd / sid / nu, high * nz * pz * sdd / sid / nv
    vd = np.sqrt(2 * px * px + pz * pz)
    steps = int(np.sqrt(2 * (nx * px) ** 2 + (nz * pz) ** 2) / (step * vd))
    g = _lib.Geom(nu=nu, nv=nv, views=views, nv_total=nv, nx=nx, nz=nz, flags=_lib.MCT_CONE if cone else 0, view_mode=1,
                  fp_steps=steps, du=du, dv=dv, px=px, pz=pz, cz=cz, sid=sid, sdd=sdd, total_scan_angle=2 * np.pi,
                  fp_step=step)
    u = ((np.arange(nu) - (nu - 1) / 2) * du).astype(np.float32)
    v = ((np.arange(nv) - (nv - 1) / 2) * dv if cone else np.zeros(nv)).astype(np.float32)
    return g, dict(angles=(2 * np.pi * np.arange(views) / views).astype(np.float32), u=u, v=v, cz=None, pa=None, pxs=None)


def ranges(lib, g, t):
    n = g.views * g.nv * g.nu
    steps, terms = np.zeros((n, 4), np.int32), np.zeros((n, 6), np.float32)
    ptr = [None if a is None else np.ascontiguousarray(a, np.float32) for a in
           (t["angles"], t["u"], t["v"], t["cz"], t["pa"], t["pxs"])]
    lib.ray_ranges(ctypes.byref(g), *[None if a is None else a.ctypes.data_as(ctypes.c_void_p) for a in ptr],
                   steps.ctypes.data_as(ctypes.c_void_p), terms.ctypes.data_as(ctypes.c_void_p))
    return steps, terms


def check_inside(g, steps, terms):
    """Positions as the kernels compute them (one rounding) at both ends of each range: linear in
    the step, so the samples between lie between them.  Returns the rays that have a range."""
    rays = steps[:, 2] <= steps[:, 3]
    s, t = steps[rays].astype(np.float64), terms[rays].astype(np.float64)
    assert np.isfinite(t).all()
    for axis, n in enumerate((g.nx, g.nx, g.nz)[:3 if g.flags & _lib.MCT_CONE else 2]):
        for k in (s[:, 2], s[:, 3]):
            f = (t[:, 2 * axis] + k * t[:, 2 * axis + 1]).astype(np.float32)
            assert (np.floor(f) >= 0).all() and (np.floor(f) <= n - 2).all()
    return rays


@pytest.mark.parametrize("nx,nz,nu,nv,views,step,cone", [
    (32, 9, 40, 11, 24, 0.2, True), (2, 2, 9, 7, 13, 0.1, True), (9, 40, 9, 33, 13, 1.1, True),
    (129, 2, 40, 16, 9, 0.2, True), (33, 4, 40, 4, 24, 0.2, False), (2, 1, 9, 1, 13, 0.05, False),
    (8192, 1, 64, 1, 8, 0.2, False)])
def test_every_sample_of_the_range_lies_in_a_cell(nx, nz, nu, nv, views, step, cone, host_lib):
    g, t = geom(nx, nz, nu, nv, views, step, cone)
    assert check_inside(g, *ranges(host_lib, g, t)).sum() > 0


@pytest.mark.parametrize("nx,nu,nv,views,high,cz", [(256, 48, 32, 4, 8.0, 0.22), (32, 40, 33, 12, 4.0, 0.1), (3, 9, 9, 13, 6.0, 0.267)])
def test_a_cone_beam_volume_of_one_slice_has_no_cells(nx, nu, nv, views, high, cz, host_lib):
    """Its only plane lies on both z faces at once: no sample passes the inside test."""
    g, t = geom(nx, 1, nu, nv, views, px=0.8, pz=0.4, high=high, cz=cz)
    steps, terms = ranges(host_lib, g, t)
    assert (steps[:, 0] <= steps[:, 1]).any()  # rays reach the plane
    assert not (steps[:, 2] <= steps[:, 3]).any()


@pytest.mark.parametrize("bad", [np.nan, np.inf, -np.inf])
@pytest.mark.parametrize("table", ["angles", "cz", "u", "v", "pa", "pxs"])
def test_a_ray_without_a_position_has_no_range(table, bad, host_lib):
    """A table entry that is no finite number takes the ranges of its rays, and of no others."""
    g, t = geom(32, 9, 16, 7, 8)
    t["cz"] = np.linspace(-0.1, 0.1, 8)
    if table in ("pa", "pxs"):  # matrices that put the rays where the circular scan has them
        g.flags |= _lib.MCT_PMATRIX
        m = np.zeros((8, 9))
        for j, a in enumerate(t["angles"].astype(np.float64)):
            for i, (w, eu, ev) in enumerate(((-550.0, 0.0, 0.0), (t["u"][0], g.du, 0.0), (t["v"][0], 0.0, g.dv))):
                m[j, 3 * i:3 * i + 3] = eu, ev, w
            c, s = np.cos(a), np.sin(a)
            x, y = m[j, 0:3].copy(), m[j, 3:6].copy()
            m[j, 0:3], m[j, 3:6] = c * x - s * y, s * x + c * y
        t["pa"] = m
        t["pxs"] = np.stack([300 * np.cos(t["angles"]), 300 * np.sin(t["angles"]), 0 * t["angles"]], 1)
    good, terms = ranges(host_lib, g, t)
    assert check_inside(g, good, terms).mean() > 0.3
    a = t[table]
    a[3 if a.ndim == 1 else (3, 0)] = bad
    steps, _ = ranges(host_lib, g, t)
    has = (steps[:, 2] <= steps[:, 3]).reshape(8, 7, 16)
    hit = {"u": np.s_[:, :, 3], "v": np.s_[:, 3]}.get(table, np.s_[3])
    rest = np.ones_like(has)
    rest[hit] = False
    assert not has[hit].any()
    assert (steps.reshape(8, 7, 16, 4)[rest] == good.reshape(8, 7, 16, 4)[rest]).all()


@pytest.mark.parametrize("nx", [8191, 20001, 40001, 46339])
def test_the_last_row_of_a_wide_image_is_no_cell(nx, host_lib):
    """A ray along the last row of voxels: above 2^15 columns 1e-3 is less than half a float there."""
    g, t = geom(nx, 1, 9, 1, 4, cone=False, wide=1e-4)
    for axis, name in ((0, "cx"), (1, "cy")):
        for sign in (-1, 1):
            g.cx = g.cy = 0.0
            setattr(g, name, sign * (nx - 1) / 2 * g.px)
            steps, terms = ranges(host_lib, g, t)
            middle = terms.reshape(4, 9, 6)[:, 4]
            assert (np.abs(middle[:, [0, 2]] - (nx - 1)) < 0.01).any() or (np.abs(middle[:, [0, 2]]) < 0.01).any()
            check_inside(g, steps, terms)


@pytest.mark.parametrize("nz,walked", [((1 << 22) - 1, True), (1 << 22, True), ((1 << 22) + 1, False), ((1 << 22) + 4096, False)])
def test_planes_that_the_float_floor_does_not_hold_are_not_walked(nz, walked, host_lib):
    """Adding 1.5 x 2^23 is exactly the floor below 2^22; in taller volumes each sample is tested
    and takes its index from a conversion."""
    g, t = geom(2, nz, 5, 3, 4, px=10.0, pz=0.01, high=1e-6, cz=(nz - 1) / 2 * 0.01 - (nz - 100) * 0.01)
    steps, terms = ranges(host_lib, g, t)
    middle = (terms[:, 4] + steps[:, :2].mean(1) * terms[:, 5])[steps[:, 0] <= steps[:, 1]]
    assert middle.size and (np.abs(middle - (nz - 100)) < 10).all()  # the rays lie just below the top
    assert (steps[:, 2] <= steps[:, 3]).any() == walked


def test_long_marches_are_not_walked(host_lib):
    """Step indices are exact in float32 up to 2^23."""
    for steps_, walked in (((1 << 23) - 1, True), (1 << 23, False)):
        g, t = geom(32, 9, 9, 3, 4)
        g.fp_steps = steps_
        steps, _ = ranges(host_lib, g, t)
        assert (steps[:, 2] <= steps[:, 3]).any() == walked
