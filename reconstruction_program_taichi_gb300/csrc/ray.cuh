// The forward projector's rays: parameters, set-up and step ranges, also compiled for the host
// (the tests check the ranges there).
#pragma once
#include <cmath>

#include "mandoct_gb300.h"

#define MCT_HD __host__ __device__ __forceinline__

namespace mct {
namespace {

struct FpParams {
    float sid, sdd, cx, cy, cz;
    float stepvd, l_min, inv_px, inv_pz;
    float x0, y0, zoff;  // voxel (0,0) centre x, y; z0 = zoff + cz_view
    float zpv;
    int nx, nz, nu, nv, views, K, cone, curved, pmat;
    // fp_kernel's ray tiles: a block of 2^ls rays is 16 detector columns x 2^vshift views x
    // 2^(ls - 4 - vshift) detector rows, a warp 2^wcs columns x 2^(5 - wcs) of the block's
    // (view, row) slots; blockIdx.y runs over 2^rs row tiles within each view group (the
    // block order is column tile, row tile, view group, row group)
    int ls, vshift, wcs, rs;
    int pitch;  // elements per row of the volume or its copies (a plane is nx rows)
};

struct Ray {
    float fx0, dfx, fy0, dfy, fz0, dfz;  // fractional voxel index = f0 + k*df
    int ks, ke;                          // clipped step range [ks, ke]
};

// Ray set-up shared by all ray kernels, following run_mgfpj_v3.py:221-324.
MCT_HD bool setup_ray(const FpParams& p, int iu, int iv, int j, const float* __restrict__ angles,
                      const float* __restrict__ u_arr, const float* __restrict__ v_arr, const float* __restrict__ czv,
                      const float* __restrict__ pa, const float* __restrict__ pxs, bool clip_z, Ray& r) {
    float sb, cb;
    sincosf(angles[j], &sb, &cb);
    const float zj = p.zpv * (float)j;
    const float uval = u_arr[iu];
    float dx, dy;
    if (p.curved) {
        const float g = (-uval) / p.sdd;
        float sg, cg;
        sincosf(g, &sg, &cg);
        dx = -p.sdd * cg + p.sid;
        dy = -p.sdd * sg;
    } else {
        dx = -(p.sdd - p.sid);
        dy = uval;
    }
    const float dz = v_arr[iv] + zj;
    const float ex = dx - p.sid, ey = dy, ez = dz - zj;
    const float dist = sqrtf(ex * ex + ey * ey + ez * ez);
    float Ox, Oy, Oz, Dx, Dy, Dz;
    if (p.pmat) {
        float s0, c0;
        sincosf(angles[0], &s0, &c0);
        const float* A = pa + 9 * j;
        const float* xs = pxs + 3 * j;
        const float fu = (float)iu, fv = (float)iv;
        const float ax = A[0] * fu + A[1] * fv + A[2];
        const float ay = A[3] * fu + A[4] * fv + A[5];
        const float az = A[6] * fu + A[7] * fv + A[8];
        Ox = xs[0] * c0 - xs[1] * s0;
        Oy = xs[1] * c0 + xs[0] * s0;
        Oz = xs[2] + zj;
        Dx = (ax * c0 - ay * s0) / dist;
        Dy = (ay * c0 + ax * s0) / dist;
        Dz = az / dist;
    } else {
        const float ux = ex / dist, uy = ey / dist, uz = ez / dist;
        Ox = p.sid * cb;
        Oy = p.sid * sb;
        Oz = zj;
        Dx = ux * cb - uy * sb;
        Dy = uy * cb + ux * sb;
        Dz = uz;
    }
    const float z0 = p.zoff + (czv ? czv[j] : p.cz);
    r.fx0 = (Ox + p.l_min * Dx - p.x0) * p.inv_px;
    r.dfx = p.stepvd * Dx * p.inv_px;
    r.fy0 = (Oy + p.l_min * Dy - p.y0) * (-p.inv_px);
    r.dfy = p.stepvd * Dy * (-p.inv_px);
    r.fz0 = (Oz + p.l_min * Dz - z0) * p.inv_pz;
    r.dfz = p.stepvd * Dz * p.inv_pz;
    // clip k so that f in [0, n-1) on each axis (conservative by one step)
    float klo = -1.0f, khi = (float)p.K;
    auto clip = [&](float f0, float df, float n) -> bool {
        if (fabsf(df) < 1e-20f) return f0 >= 0.0f && f0 < n - 1.0f;
        float t1 = (0.0f - f0) / df, t2 = (n - 1.0f - f0) / df;
        klo = fmaxf(klo, fminf(t1, t2));
        khi = fminf(khi, fmaxf(t1, t2));
        return true;
    };
    bool any = clip(r.fx0, r.dfx, (float)p.nx) && clip(r.fy0, r.dfy, (float)p.nx);
    if (clip_z && p.cone) any = any && clip(r.fz0, r.dfz, (float)p.nz);
    if (!any || !(klo <= khi)) {
        r.ks = 0;
        r.ke = -1;
        return false;
    }
    r.ks = max(0, (int)floorf(klo) - 1);
    r.ke = min(p.K - 1, (int)ceilf(khi) + 1);
    return r.ks <= r.ke;
}

// Above this many steps a ray's indices are no longer exact in float32 (and would not advance one
// by one), above this many planes its positions' floors: such rays are sampled one sample at a
// time, each tested.
constexpr int kMaxWalkSteps = 1 << 23, kMaxWalkPlanes = 1 << 22;

// Steps [kis, kie] whose sample lies at least 1e-3 voxel (a float, if that is more) inside the
// box on every tested axis (and one more step in from both ends): for them the reference's inside
// test certainly passes, far beyond float rounding, so it can be skipped.  A ray with a term
// that is no finite number (from an angle, a centre, a matrix) has no such steps, so no index
// is taken from it; false is returned if the terms that are finite would leave it some.
MCT_HD bool interior_range(const FpParams& p, const Ray& r, bool test_z, int& kis, int& kie) {
    float lo = -3.0e38f, hi = 3.0e38f;
    bool empty = false, finite = true;
    auto axis = [&](float f0, float df, float n) {
        finite = finite && fabsf(f0) <= 3.4e38f && fabsf(df) <= 3.4e38f;
        const float eps = fmaxf(1e-3f, n * 0x1p-23f);  // at least a float below n - 1
        const float a = eps, b = n - 1.0f - eps;
        if (!(a <= b)) empty = true;  // one plane: no cell (t1, t2 would span the plane's two sides)
        if (fabsf(df) < 1e-20f) {
            if (!(f0 >= a && f0 <= b)) empty = true;
            return;
        }
        const float t1 = (a - f0) / df, t2 = (b - f0) / df;
        lo = fmaxf(lo, fminf(t1, t2));
        hi = fminf(hi, fmaxf(t1, t2));
    };
    axis(r.fx0, r.dfx, (float)p.nx);
    axis(r.fy0, r.dfy, (float)p.nx);
    if (test_z) axis(r.fz0, r.dfz, (float)p.nz);
    lo = fmaxf(lo, (float)r.ks - 2.0f);
    hi = fminf(hi, (float)r.ke + 2.0f);
    kis = 1;
    kie = 0;
    if (!empty && lo <= hi) {
        kis = max(r.ks, (int)ceilf(lo) + 1);
        kie = min(r.ke, (int)floorf(hi) - 1);
    }
    const bool lost = !finite && kis <= kie;
    if (lost || kis > kie || p.K >= kMaxWalkSteps || (test_z && p.nz > kMaxWalkPlanes)) {
        kis = r.ke + 1;
        kie = r.ke;
    }
    return !lost;
}

// The launch parameters of a geometry, without a ray tile.
inline FpParams ray_params(const mct_geom* g) {
    FpParams p{};
    p.nx = g->nx; p.nz = g->nz; p.nu = g->nu; p.nv = g->nv; p.views = g->views; p.K = g->fp_steps;
    p.cone = (g->flags & MCT_CONE) != 0;
    p.curved = (g->flags & MCT_CURVED) != 0;
    p.pmat = (g->flags & MCT_PMATRIX) != 0;
    p.sid = g->sid; p.sdd = g->sdd; p.cx = g->cx; p.cy = g->cy; p.cz = g->cz;
    // run_mgfpj_v3.py:210-239 in double, then rounded
    const double px = g->px, pz = p.cone ? g->pz : 0.0;
    const double img_dimension = g->nx * px, image_dimension_z = g->nz * (double)g->pz;
    const double vd = std::sqrt(2 * px * px + (double)g->pz * g->pz);
    p.stepvd = (float)(g->fp_step * vd);
    p.l_min = (float)(g->sid - std::sqrt(2 * img_dimension * img_dimension + image_dimension_z * image_dimension_z) / 2.0);
    p.inv_px = (float)(1.0 / px);
    p.inv_pz = p.cone ? (float)(1.0 / pz) : 0.0f;
    p.x0 = (float)(-(g->nx - 1.0) / 2.0 * px + g->cx);
    p.y0 = (float)(-(g->nx - 1.0) / 2.0 * (-px) + g->cy);
    p.zoff = (float)(-(g->nz - 1.0) / 2.0 * (double)g->pz);
    p.zpv = g->fp_z_per_view;
    p.pitch = g->nx;
    return p;
}

}  // namespace
}  // namespace mct
