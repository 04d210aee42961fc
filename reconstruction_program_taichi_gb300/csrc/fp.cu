// Ray-driven trilinear forward projector, its exact adjoint, the effective ray map,
// binning/noise, and analytic ellipsoid projections.
//
// Reference kernels replaced: Mgfpj_v3.ForwardProjectionBilinear
// (run_mgfpj_v3.py:184-366), its masked copy in Mgfbp_ir
// (run_mgfbp_iterative_recon_IRN_CGLS.py:494-676), the effective-map agent (:679-833),
// BinSinogram / AddPossionNoise (run_mgfpj_v3.py:368-391).
//
// All views are projected in ONE launch (the reference launches once per view).
// A ray's sample positions are affine in the step index k, so each ray first clips
// its step range to the volume's bounding box (with a one-step margin) and then
// applies the reference's per-sample inside test exactly; samples outside the box
// contribute 0 in the reference too.
#include <cmath>
#include <type_traits>

#include "common.cuh"
#include "ray.cuh"

namespace mct {
namespace {

// Direction (in object x, y) along which neighbouring detector columns spread.
__device__ __forceinline__ bool spread_along_y(const FpParams& p, int j, const float* __restrict__ angles,
                                               const float* __restrict__ pa) {
    if (p.pmat) {
        float s0, c0;
        sincosf(angles[0], &s0, &c0);
        const float* A = pa + 9 * j;
        const float ex = A[0] * c0 - A[3] * s0, ey = A[3] * c0 + A[0] * s0;
        return fabsf(ey) > fabsf(ex);
    }
    float sb, cb;
    sincosf(angles[j], &sb, &cb);
    return fabsf(cb) > fabsf(sb);  // d(x, y)/du is (-sin b, cos b)
}

// Grid of the other ray kernels: x = 32-column detector tiles, y = views, z = 8-row
// detector tiles.  Blocks are scheduled x, then y, then z, so the blocks resident at
// one time cover many views of the same detector rows; those rays cross only a thin
// z-slab of the volume, which then stays in L2 across views.  fp_kernel takes tiles of
// 16 columns, several consecutive views and rows (x = column tiles, y = view groups, z =
// row tiles).
//
// One thread per ray (u, v) of view j.  vol is [z][y][x]; vol_t, when
// given, is the same volume as [z][x][y]: views whose detector columns spread along
// y read vol_t so that neighbouring rays touch consecutive addresses.  With ZP
// (cone beam, workspace given) the volume is read from copies zp_x ([z][y][x]) and
// zp_y ([z][x][y]): float32 quads (two adjacent 16-byte elements per cell) or
// 16-bit cells (the whole 2x2x2 trilinear cell in one 16-byte element), below.

// float32 quad copy, indexed in a (slow s, fast f) frame: (s, f) = (y, x) for views whose
// detector columns spread along x (copy cx, [z][y][x]) and (x, y) for the others (copy
// cy, [z][x][y]), so that neighbouring rays read neighbouring elements.  Element
// (z, s, f) holds the voxel and its forward differences along z, s and both,
//   {V, Dz V, Ds V, Dz Ds V}(z, s, f)    (16 bytes),
// and the neighbour along f is the next element: a cell is two adjacent 16-byte loads,
// and its f-differences are taken in registers.  Whole 32-byte cells would double the
// copies, and half as many cells fit L1 and L2.  Differences instead of the four values
// themselves: the interpolation then needs no z-subtractions (five of about 50
// instructions per cell; 171.9 -> 158.9 ms at 512x512x256 / 1080 views).
struct __align__(16) Quad16 {
    float v[4];
};

// bf16 cell copy: element (z, y, x) of either orientation holds the whole 2x2x2 cell
// whose lowest corner is voxel (z, y, x), as four bf16 pairs {lower, upper z-plane}:
//   .x = e00 = {V[z][y][x], V[z+1][y][x]}      .y = g00 = e01 - e00' (x+1 corner)
//   .z = e10 = {V[z][y+1][x], V[z+1][y+1][x]}  .w = g10 = e11 - e10' (x+1, y+1)
// (x, y as in the volume; e' is e rounded to bf16, so the x+1 corners are restored to
// the bf16 precision of the differences).  A reload is one 16-byte gather.
__device__ __forceinline__ uint32_t pack_bf16x2(float lo, float hi) {
    __nv_bfloat162 b = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<uint32_t*>(&b);
}

// How a ray's interior samples are summed: by cells, by cells in windows, or one by one.
enum Walk { kCells, kWindows, kSamples };

// Resident blocks per SM that the register allocation of fp_kernel targets: 5 (48
// registers) with copies.  512x512x256 / 1080 views, float32: 4 blocks 160.6 ms, 5
// 158.9, 6 164.7; 512x512x64 / 360 views, bf16: 4 blocks 13.55 ms, 5 13.41, 6 14.27.
// The fan-beam path needs 40 registers (6 blocks), the walk of 16-bit cells by samples 62
// (4; 5 blocks cost it 10 %); that of float32 quads is 3 to 4 % faster with 5 than with 4.
template <bool CONE, typename ZT, int WALK>
constexpr int fp_min_blocks() {
    return WALK == kSamples && sizeof(ZT) == 16 && !std::is_same<ZT, Quad16>::value ? 4 : CONE ? 5 : 6;
}

// Planes along the rays' main axis per window (WIN, below).
constexpr int kWinPlanes = 64;

// A ray's sum over its samples, cell by cell.  The samples are equally spaced (step df)
// and the interpolant of one 2x2x2 cell is trilinear, so the n samples that fall into a
// cell need not be taken one by one: with m their midpoint and s^2 = (n^2 - 1) / 12 the
// variance of n consecutive integers,
//     sum = n [ V(m) + s^2 (dx dy Vxy(m) + dx dz Vxz(m) + dy dz Vyz(m)) ]
// exactly (the odd central moments vanish, the second differences along one axis too).
// n is the number of steps to the nearest face the ray leaves the cell through.  At the
// default step of 0.2 voxel diagonals a cell holds 2.2 samples on average (0.1: 4.4,
// 0.5: 0.9), and every lane of a warp loads a cell in every iteration, where a walk by
// samples has some lane entering a cell at almost every sample, with the others idle.
// A sample within rounding of a face may be taken from the cell before it: the
// interpolant is continuous there.
//
// What bounds it: L1 data-pipe wavefronts (84 % for float32 at 128^3, 93 % at 256x256x64
// / 180 views), then issue (62 %, 49 %).  A warp's loads take a tag lookup per 4 lines
// and a wavefront per conflicting 16-byte bank, so the copies' rows are padded to an odd
// number of elements (copy_pitch), a warp's rays are neighbours (ray tiles, below), and
// with WIN the lanes are kept together: they cross the volume in windows of kWinPlanes
// planes along their main axis and wait for each other at the end of each, which keeps
// rays whose cells are counted differently in the same rows of the copy.  The wait costs
// what the rays' entry points differ by, so it pays for wide volumes.
//   ms, by samples / by cells / with windows:
//     512x512x256, 1080 views, float32     237.6 / 159.0 / 153.0
//     128x128x64, 270 views, float32       1.036 / 0.699 / 0.738
//     512x512x64, 360 views, bf16          18.32 / 13.41 / 14.9 (windows: 16-bit cells lose)
//     512^2 fan beam, 720 views            1.34 / 0.80 / 0.66
//     256x256x128, 360 views, step 0.1     18.83 / 7.19;  step 0.5: 6.20 / 5.95
// Where a step leaves about one sample per cell or fewer, the sum over cells saves nothing
// and costs its second-order terms: from the step on where it is the faster
// (walk_by_samples below), a ray is walked by samples and keeps its cell in registers until
// it enters another.
template <bool CONE, bool ZP, typename ZT, int WALK>
__global__ void __launch_bounds__(256, fp_min_blocks<CONE, ZT, WALK>())
fp_kernel(FpParams p, const float* __restrict__ angles, const float* __restrict__ u_arr,
          const float* __restrict__ v_arr, const float* __restrict__ czv, const float* __restrict__ pa,
          const float* __restrict__ pxs, const float* __restrict__ vol, const float* __restrict__ vol_t,
          const ZT* __restrict__ zp_x, const ZT* __restrict__ zp_y, const float* __restrict__ mask,
          float* __restrict__ sgm, const uint32_t* __restrict__ f16_max) {
    // ray of this thread: column tx and (view, row) slot ty of the block's tile, warps
    // of 2^wcs columns x 2^(5 - wcs) slots
    const int tid = threadIdx.y * 32 + threadIdx.x;
    const int warp = tid >> 5, lane = tid & 31;
    const int gpr = 4 - p.wcs;  // log2 of the warps across the tile's columns
    const int tx = ((warp & ((1 << gpr) - 1)) << p.wcs) + (lane & ((1 << p.wcs) - 1));
    const int ty = ((warp >> gpr) << (5 - p.wcs)) + (lane >> p.wcs);
    const int iu = (blockIdx.x << 4) + tx;
    const int vs = p.vshift;
    const int vg = blockIdx.y >> p.rs, rsub = blockIdx.y & ((1 << p.rs) - 1);  // view group, row tile in it
    const int iv = ((((int)blockIdx.z << p.rs) + rsub) << (p.ls - 4 - vs)) + (ty >> vs);
    const int j = (vg << vs) + (ty & ((1 << vs) - 1));
    if (iu >= p.nu || iv >= p.nv || j >= p.views) return;
    const int64_t oidx = ((int64_t)iv * p.views + j) * p.nu + iu;
    if (mask && mask[oidx] != 1.0f) {
        sgm[oidx] = 0.0f;
        return;
    }
    const int nx = p.nx;
    const bool tr = (ZP || vol_t != nullptr) && spread_along_y(p, j, angles, pa);
    // quad copies are addressed in their (slow, fast) frame: the ray's x and y swap for
    // the transposed copy, so the fast axis is always "x" below (both axes span
    // [0, nx - 1), so the clipping and inside tests are unchanged)
    constexpr bool kQuad = ZP && std::is_same<ZT, Quad16>::value;
    const float* __restrict__ V = tr ? vol_t : vol;
    const ZT* __restrict__ V2 = tr ? zp_y : zp_x;
    const int sx = (tr && !kQuad) ? p.pitch : 1, sy = (tr && !kQuad) ? 1 : p.pitch;
    const int plane = p.pitch * nx;  // volumes and copies below 2^31 elements (checked on the host)
    Ray r;
    float acc = 0.0f;
    if (setup_ray(p, iu, iv, j, angles, u_arr, v_arr, czv, pa, pxs, true, r)) {
        if (kQuad && tr) {
            float t = r.fx0;
            r.fx0 = r.fy0;
            r.fy0 = t;
            t = r.dfx;
            r.dfx = r.dfy;
            r.dfy = t;
        }
        const float xmax = (float)(nx - 1), zmax = (float)(p.nz - 1);
        struct Cell {
            // float32 quads: corner, x, y and xy difference, each {value, z-difference}; the
            // others: corner and x-difference of row y (e, ex) and of row y + 1 (ey, exy), each
            // {lower plane, upper plane}
            float2 e, ex, ey, exy;
        };
        auto load_cell = [&](int off, Cell& c) {
            if constexpr (kQuad) {
                const float4 q0 = __ldg(reinterpret_cast<const float4*>(V2 + off));
                const float4 q1 = __ldg(reinterpret_cast<const float4*>(V2 + off + 1));
                c.e = make_float2(q0.x, q0.y);
                c.ey = make_float2(q0.z, q0.w);
                c.ex = __fadd2_rn(make_float2(q1.x, q1.y), make_float2(-q0.x, -q0.y));
                c.exy = __fadd2_rn(make_float2(q1.z, q1.w), make_float2(-q0.z, -q0.w));
            } else if constexpr (ZP && std::is_same<ZT, uint4>::value) {
                const uint4 q = __ldg(V2 + off);
                c.e = bf16x2_to_float2(q.x);
                c.ex = bf16x2_to_float2(q.y);
                c.ey = bf16x2_to_float2(q.z);
                c.exy = bf16x2_to_float2(q.w);
            } else if constexpr (ZP && std::is_same<ZT, h16x8>::value) {
                const uint4 q = __ldg(reinterpret_cast<const uint4*>(V2 + off));
                c.e = h16x2_to_float2(q.x);
                c.ex = h16x2_to_float2(q.y);
                c.ey = h16x2_to_float2(q.z);
                c.exy = h16x2_to_float2(q.w);
            } else {
                const float* b = V + off;
                const float a00 = __ldg(b), a01 = __ldg(b + sx), a10 = __ldg(b + sy), a11 = __ldg(b + sx + sy);
                float c00 = 0.f, c01 = 0.f, c10 = 0.f, c11 = 0.f;
                if (CONE) {
                    const float* u = b + plane;
                    c00 = __ldg(u); c01 = __ldg(u + sx); c10 = __ldg(u + sy); c11 = __ldg(u + sx + sy);
                }
                c.e = make_float2(a00, c00);
                c.ey = make_float2(a10, c10);
                c.ex = __fadd2_rn(make_float2(a01, c01), make_float2(-a00, -c00));
                c.exy = __fadd2_rn(make_float2(a11, c11), make_float2(-a10, -c10));
            }
        };
        auto sub2 = [](float2 a, float2 b) { return __fadd2_rn(a, make_float2(-b.x, -b.y)); };
        // the cell's value at fractions (xw, yw, zw)
        auto interp = [&](const Cell& c, float xw, float yw, float zw) -> float {
            const float2 x2 = make_float2(xw, xw), y2 = make_float2(yw, yw);
            const float2 l = __ffma2_rn(x2, c.ex, c.e);
            const float2 l1 = __ffma2_rn(x2, c.exy, c.ey);
            if constexpr (kQuad) {
                const float2 pl = __ffma2_rn(y2, l1, l);
                return fmaf(zw, pl.y, pl.x);
            }
            const float2 pl = __ffma2_rn(y2, sub2(l1, l), l);
            return CONE ? fmaf(zw, pl.y - pl.x, pl.x) : pl.x;
        };
        Cell cur;       // the last sample's cell: kSamples reloads it only when a ray enters another
        int cell = -1;
        cur.e = cur.ex = cur.ey = cur.exy = make_float2(0.0f, 0.0f);
        // Checked samples at the ends of the range, where the inside test decides; the range
        // between them (at least 1e-3 voxel inside on every axis) is walked cell by cell.
        auto sample = [&](int k) {
            const float fk = (float)k;
            const float fx = fmaf(fk, r.dfx, r.fx0);
            const float fy = fmaf(fk, r.dfy, r.fy0);
            const float xf = floorf(fx), yf = floorf(fy);
            bool ok = xf >= 0.0f && xf < xmax && yf >= 0.0f && yf < xmax;
            const int xi = min(max((int)xf, 0), nx - 2), yi = min(max((int)yf, 0), nx - 2);
            int zi = iv;
            float zw = 0.0f;
            if (CONE) {
                const float fz = fmaf(fk, r.dfz, r.fz0);
                const float zf = floorf(fz);
                ok = ok && zf >= 0.0f && zf < zmax;
                zi = min(max((int)zf, 0), p.nz - 2);
                zw = fz - zf;
            }
            const int off = zi * plane + yi * sy + xi * sx;
            if (WALK != kSamples || off != cell) load_cell(off, cur);
            cell = off;
            const float v = interp(cur, fx - xf, fy - yf, zw);
            acc += ok ? v : 0.0f;
        };
        int kis, kie;
        if (!interior_range(p, r, CONE, kis, kie)) acc = __int_as_float(0x7fffffff);  // its values have no weights
        for (int k = r.ks; k < kis; ++k) sample(k);
        if (kis <= kie) {
            // Positions come from f = fma(k, df, f0) and floors from adding M = 1.5 * 2^23
            // rounded toward minus infinity (exactly M + floor(f) for |f| < 2^22), on the FMA
            // pipe; x and y travel as one f32x2 pair.  The element offset is summed in
            // unsigned arithmetic (the bias terms wrap, the total is the offset, below 2^31).
            const float M = 12582912.0f;
            const unsigned MB = 0x4B400000u;  // bit pattern of M
            const unsigned obias =
                CONE ? MB * (unsigned)(plane + sy + sx) : MB * (unsigned)(sy + sx) - (unsigned)(iv * plane);
            const float2 M2 = make_float2(M, M), nM2 = make_float2(-M, -M);
            const float2 dxy = make_float2(r.dfx, r.dfy), fxy0 = make_float2(r.fx0, r.fy0);
            // steps from fraction w to the face that the ray leaves the cell through: A + w * B.
            // The bound keeps an axis without motion finite and is far enough that it never ends
            // a run (at 1e6 a ray along a plane, whose fraction rounds to 1 - 2^-24, took its
            // samples one by one: bf16 141x141x3, 129 views of 3 rows 115 us, now 66; float32 132, 73).
            const float ix = fminf(1.0f / fabsf(r.dfx), 1e30f), iy = fminf(1.0f / fabsf(r.dfy), 1e30f);
            const float iz = fminf(1.0f / fabsf(r.dfz), 1e30f);
            const float2 B2 = make_float2(r.dfx < 0.0f ? ix : -ix, r.dfy < 0.0f ? iy : -iy);
            const float2 A2 = make_float2(r.dfx < 0.0f ? 0.0f : ix, r.dfy < 0.0f ? 0.0f : iy);
            const float Bz = r.dfz < 0.0f ? iz : -iz, Az = r.dfz < 0.0f ? 0.0f : iz;
            const float cxy = r.dfx * r.dfy * (1.0f / 12.0f);
            const float cxz = r.dfx * r.dfz * (1.0f / 12.0f), cyz = r.dfy * r.dfz * (1.0f / 12.0f);
            const float kend = (float)kie;
            // midpoint: n1 / 2 steps; the 16-bit kernels scale n1 instead of the step (two
            // registers fewer: 48, without spills)
            constexpr float kN = ZP && !kQuad ? 0.5f : 1.0f, kD = ZP && !kQuad ? 1.0f : 0.5f;
            const float2 hd = make_float2(kD * r.dfx, kD * r.dfy);
            const float hdz = kD * r.dfz;
            struct Run {
                Cell c;
                float2 m;      // fractions of the run's midpoint
                float mz, n;   // and its number of samples
            };
            // element of sample fk's cell and the sample's fractions in it
            auto locate = [&](float fk, float2& w, float& zw) -> int {
                const float2 f = __ffma2_rn(make_float2(fk, fk), dxy, fxy0);
                const float2 m = __fadd2_rd(f, M2);
                const float2 fl = __fadd2_rn(m, nM2);
                w = __fadd2_rn(f, make_float2(-fl.x, -fl.y));
                unsigned off = (unsigned)__float_as_int(m.x) * (unsigned)sx + (unsigned)__float_as_int(m.y) * (unsigned)sy - obias;
                zw = 0.0f;
                if (CONE) {
                    const float fz = fmaf(fk, r.dfz, r.fz0);
                    const float mz = __fadd_rd(fz, M);
                    zw = fz - (mz - M);
                    off += (unsigned)__float_as_int(mz) * (unsigned)plane;
                }
                return (int)off;
            };
            // the run of samples from fk on that lie in one cell; fk moves past it
            auto next_run = [&](float& fk, Run& q) {
                float2 w;
                float zw;
                load_cell(locate(fk, w, zw), q.c);
                const float2 t2 = __ffma2_rn(w, B2, A2);
                float t = fminf(fminf(t2.x, t2.y), kend - fk);
                if (CONE) t = fminf(t, fmaf(zw, Bz, Az));
                const float n1 = __fadd_rd(t, M) - M;  // steps to the run's last sample
                q.n = n1 + 1.0f;
                const float h = kN * n1;
                q.m = __ffma2_rn(make_float2(h, h), hd, w);
                if (CONE) q.mz = fmaf(h, hdz, zw);
                fk += q.n;
            };
            auto add_run = [&](const Run& q) {
                const float2 x2 = make_float2(q.m.x, q.m.x), y2 = make_float2(q.m.y, q.m.y);
                const float2 l = __ffma2_rn(x2, q.c.ex, q.c.e);
                float v, corr;
                if constexpr (kQuad) {
                    const float2 gy = __ffma2_rn(x2, q.c.exy, q.c.ey);
                    const float2 pl = __ffma2_rn(y2, gy, l);
                    v = fmaf(q.mz, pl.y, pl.x);
                    corr = fmaf(cxy, fmaf(q.mz, q.c.exy.y, q.c.exy.x),
                                fmaf(cxz, fmaf(q.m.y, q.c.exy.y, q.c.ex.y), cyz * gy.y));
                } else {
                    const float2 gxy = sub2(q.c.exy, q.c.ex);
                    const float2 gy = __ffma2_rn(x2, gxy, sub2(q.c.ey, q.c.e));
                    const float2 pl = __ffma2_rn(y2, gy, l);
                    v = pl.x;
                    corr = cxy * gxy.x;
                    if (CONE) {
                        const float2 gx = __ffma2_rn(y2, gxy, q.c.ex);
                        v = fmaf(q.mz, pl.y - pl.x, pl.x);
                        corr = fmaf(cxy, fmaf(q.mz, gxy.y - gxy.x, gxy.x), fmaf(cxz, gx.y - gx.x, cyz * (gy.y - gy.x)));
                    }
                }
                acc = fmaf(q.n, fmaf(fmaf(q.n, q.n, -1.0f), corr, v), acc);
            };
            float fk = (float)kis;
            if constexpr (WALK == kSamples) {
// 256x256x64 / 360 views, bf16, step 0.3: 3.28 / 3.22 / 3.29 ms unrolled 2 / 3 / 4
#pragma unroll 3
                for (int k = kis; k <= kie; ++k, fk += 1.0f) {
                    float2 w;
                    float zw;
                    const int off = locate(fk, w, zw);
                    if (off != cell) load_cell(off, cur);
                    cell = off;
                    acc += interp(cur, w.x, w.y, zw);
                }
            }
            if constexpr (WALK == kWindows) {
                // window i ends at plane i * kWinPlanes along the rays' main axis, counted
                // from the side that they enter through: step w0 + i * wi
                const float ds = tr && !kQuad ? r.dfx : r.dfy, s0 = tr && !kQuad ? r.fx0 : r.fy0;
                const float is = tr && !kQuad ? ix : iy;
                const float wi = (float)kWinPlanes * is, w0 = -(ds < 0.0f ? xmax - s0 : s0) * is;
                for (int i = 1; i * kWinPlanes < nx; ++i) {
                    const float wend = fminf(fmaf((float)i, wi, w0), kend + 0.5f);
                    while (fk < wend) {
                        Run q;
                        next_run(fk, q);
                        add_run(q);
                    }
                }
            }
            while (WALK != kSamples && fk <= kend) {
                Run q;
                next_run(fk, q);
                add_run(q);
            }
        }
        for (int k = max(kie + 1, kis); k <= r.ke; ++k) sample(k);
    }
    if constexpr (IsF16<ZT>::value) acc *= ldexpf(1.0f, -f16_scale_exp(*f16_max));  // float16 cells hold v * 2^e
    sgm[oidx] = acc * p.stepvd;
}

// Largest |v| of the volume as float bits into *maxbits (zeroed by the caller).
template <typename TIN>
__global__ void vol_absmax_kernel(int64_t n, const TIN* __restrict__ v, uint32_t* __restrict__ maxbits) {
    uint32_t m = 0;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        m = max(m, __float_as_uint(ldv(v, i)) & 0x7fffffffu);
    m = __reduce_max_sync(0xffffffffu, m);
    if ((threadIdx.x & 31) == 0) atomicMax(maxbits, m);
}

// 16-bit cell copies (layout above; float16 cells hold v * 2^e, see f16_scale_exp): cx[z][y][x] and cy[z][x][y] both hold the cell at
// voxel (z, y, x); corners outside the volume are 0 (no in-volume sample uses them).
// 32x32 tiles, the transposed copy through shared memory.
template <bool F16, typename TIN = float>
__global__ void cell16_kernel(int nx, int nz, int pitch, const TIN* __restrict__ v, uint4* __restrict__ cx,
                              uint4* __restrict__ cy, const uint32_t* __restrict__ f16_max) {
    __shared__ uint4 tile[32][33];
    const int64_t plane = (int64_t)nx * nx;
    const int z = blockIdx.z;
    const int x0 = blockIdx.x * 32, y0 = blockIdx.y * 32;
    const float sc = F16 ? ldexpf(1.0f, f16_scale_exp(*f16_max)) : 1.0f;
    auto at = [&](int zz, int yy, int xx) -> float {
        return (zz < nz && yy < nx && xx < nx) ? ldv(v, zz * plane + (int64_t)yy * nx + xx) * sc : 0.0f;
    };
    auto rb = [](float a) {
        return F16 ? __half2float(__float2half_rn(a)) : __bfloat162float(__float2bfloat16_rn(a));
    };
    auto pk = [](float lo, float hi) { return F16 ? pack_h16x2(lo, hi) : pack_bf16x2(lo, hi); };
    for (int i = threadIdx.y; i < 32; i += blockDim.y) {
        const int y = y0 + i, x = x0 + threadIdx.x;
        if (y < nx && x < nx) {
            const float a0 = rb(at(z, y, x)), a1 = rb(at(z + 1, y, x));
            const float c0 = rb(at(z, y + 1, x)), c1 = rb(at(z + 1, y + 1, x));
            uint4 q;
            q.x = pk(a0, a1);
            q.y = pk(at(z, y, x + 1) - a0, at(z + 1, y, x + 1) - a1);
            q.z = pk(c0, c1);
            q.w = pk(at(z, y + 1, x + 1) - c0, at(z + 1, y + 1, x + 1) - c1);
            cx[((int64_t)z * nx + y) * pitch + x] = q;
            tile[i][threadIdx.x] = q;
        }
    }
    __syncthreads();
    for (int i = threadIdx.y; i < 32; i += blockDim.y) {
        const int x = x0 + i, y = y0 + threadIdx.x;
        if (y < nx && x < nx) cy[((int64_t)z * nx + x) * pitch + y] = tile[threadIdx.x][i];
    }
}

// float32 quad copies (layout at Quad16): cx[z][y][x] with fast axis x and s = y, cy[z][x][y]
// with fast axis y and s = x; corners outside the volume count as 0 (no in-volume sample
// uses them).  32x32 tiles, the transposed copy through shared memory.
template <typename TIN = float>
__global__ void quad32_kernel(int nx, int nz, int pitch, const TIN* __restrict__ v, float4* __restrict__ cx,
                              float4* __restrict__ cy) {
    __shared__ float4 tile[32][33];
    const int64_t plane = (int64_t)nx * nx;
    const int z = blockIdx.z;
    const int x0 = blockIdx.x * 32, y0 = blockIdx.y * 32;
    auto at = [&](int zz, int yy, int xx) -> float {
        return (zz < nz && yy < nx && xx < nx) ? ldv(v, zz * plane + (int64_t)yy * nx + xx) : 0.0f;
    };
    for (int i = threadIdx.y; i < 32; i += blockDim.y) {
        const int y = y0 + i, x = x0 + threadIdx.x;
        if (y < nx && x < nx) {
            const float a0 = at(z, y, x), az = at(z + 1, y, x) - a0;
            auto quad = [&](float b0, float b1) {
                const float d = b0 - a0;
                return make_float4(a0, az, d, (b1 - b0) - az);
            };
            cx[((int64_t)z * nx + y) * pitch + x] = quad(at(z, y + 1, x), at(z + 1, y + 1, x));
            tile[i][threadIdx.x] = quad(at(z, y, x + 1), at(z + 1, y, x + 1));
        }
    }
    __syncthreads();
    for (int i = threadIdx.y; i < 32; i += blockDim.y) {
        const int x = x0 + i, y = y0 + threadIdx.x;
        if (y < nx && x < nx) cy[((int64_t)z * nx + x) * pitch + y] = tile[threadIdx.x][i];
    }
}

// vt[z][x][y] = v[z][y][x], 32x32 tiles through shared memory.
__global__ void transpose_xy_kernel(int nx, int nz, const float* __restrict__ v, float* __restrict__ vt) {
    __shared__ float tile[32][33];
    const int64_t plane = (int64_t)nx * nx;
    const int z = blockIdx.z;
    const int x0 = blockIdx.x * 32, y0 = blockIdx.y * 32;
    for (int i = threadIdx.y; i < 32; i += blockDim.y) {
        const int y = y0 + i, x = x0 + threadIdx.x;
        if (y < nx && x < nx) tile[i][threadIdx.x] = v[z * plane + (int64_t)y * nx + x];
    }
    __syncthreads();
    for (int i = threadIdx.y; i < 32; i += blockDim.y) {
        const int x = x0 + i, y = y0 + threadIdx.x;
        if (y < nx && x < nx) vt[z * plane + (int64_t)x * nx + y] = tile[threadIdx.x][i];
    }
}

// 16-byte vector reduction (sm_90 and later): four float adds at one aligned address,
// one L2 atomic request instead of four.
__device__ __forceinline__ void red_add_v4(float* q, float a, float b, float c, float d) {
    asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(q), "f"(a), "f"(b), "f"(c), "f"(d)
                 : "memory");
}

__device__ __forceinline__ void red_add_v2(float* q, float a, float b) {
    asm volatile("red.global.add.v2.f32 [%0], {%1, %2};" ::"l"(q), "f"(a), "f"(b) : "memory");
}

// One ray of the adjoint.  Corners are kept by its direction, 0 behind and 1 ahead on each
// axis; fx, fy, fz tell where behind is the higher index.  They are template arguments: as
// run-time values they cost 16 selects per cell.
template <bool CONE, bool CELLS, bool fx, bool fy, bool fz>
__device__ __forceinline__ void adjoint_ray(const FpParams& p, const Ray& r, int iv, float yv, float* __restrict__ out) {
    const int nx = p.nx;
    const int plane = nx * nx;
    const int stepx = fx ? -1 : 1, stepy = fy ? -nx : nx, stepz = fz ? -plane : plane;
    const int first = (fx ? 1 : 0) + (fy ? nx : 0) + (CONE && fz ? plane : 0);  // from the cell to its corner behind on all axes
    const unsigned xf = fx ? 1u : 0u;                                            // XF of the face behind
    const unsigned yf = (unsigned)p.nz * (unsigned)plane + (fy ? (unsigned)nx : 0u);  // YF of the face behind
    int cell = -1;
    float2 s00 = make_float2(0.f, 0.f), s01 = s00, s10 = s00, s11 = s00;  // s<x><z> = {y behind, y ahead}
    auto order = [](bool flip, float a, float b) { return flip ? make_float2(b, a) : make_float2(a, b); };
    auto face = [&](unsigned element, float2 behind, float2 ahead) {  // pairs at z behind and ahead
        float* q = out + (size_t)element * 4;
        const float2 lo = fz ? ahead : behind, hi = fz ? behind : ahead;
        red_add_v4(q, lo.x, lo.y, hi.x, hi.y);
    };
    auto flush = [&]() {  // all corners
        if (cell < 0) return;
        if constexpr (CONE && CELLS) {
            face((unsigned)cell + xf, order(fy, s00.x, s00.y), order(fy, s01.x, s01.y));
            face((unsigned)cell + 1u - xf, order(fy, s10.x, s10.y), order(fy, s11.x, s11.y));
        } else if constexpr (CELLS) {
            const float2 lo = order(fx, s00.x, s10.x), hi = order(fx, s00.y, s10.y);  // y behind, ahead
            red_add_v4(out + (size_t)cell * 4, fy ? hi.x : lo.x, fy ? hi.y : lo.y, fy ? lo.x : hi.x, fy ? lo.y : hi.y);
        } else {
            float* q = out + (cell + first);
            atomicAdd(q, s00.x);
            atomicAdd(q + stepx, s10.x);
            atomicAdd(q + stepy, s00.y);
            atomicAdd(q + stepx + stepy, s10.y);
            if (CONE) {
                q += stepz;
                atomicAdd(q, s01.x);
                atomicAdd(q + stepx, s11.x);
                atomicAdd(q + stepy, s01.y);
                atomicAdd(q + stepx + stepy, s11.y);
            }
        }
        s00 = s01 = s10 = s11 = make_float2(0.f, 0.f);
    };
    auto enter = [&](int off) {
        if (off == cell) return;
        const int d = off - cell;
        if ((CONE || !CELLS) && cell >= 0 && (d == stepx || d == stepy)) {
            const bool x = d == stepx;
            const float b0 = x ? s00.y : s10.x, b1 = x ? s01.y : s11.x;  // the face's other corner, z behind and ahead
            if constexpr (CELLS) {
                const bool f = x ? fy : fx;
                face((unsigned)cell + (x ? xf : yf), order(f, s00.x, b0), order(f, s01.x, b1));
            } else {
                float* q = out + (cell + first);
                const int t = x ? stepy : stepx;
                atomicAdd(q, s00.x);
                atomicAdd(q + t, b0);
                if (CONE) {
                    atomicAdd(q + stepz, s01.x);
                    atomicAdd(q + stepz + t, b1);
                }
            }
            s00 = make_float2(x ? s10.x : s00.y, x ? s10.y : 0.0f);
            s10 = make_float2(x ? 0.0f : s10.y, 0.0f);
            s01 = make_float2(x ? s11.x : s01.y, x ? s11.y : 0.0f);
            s11 = make_float2(x ? 0.0f : s11.y, 0.0f);
        } else if (CONE && cell >= 0 && d == stepz) {
            if constexpr (CELLS) {
                float* q = out + ((size_t)((unsigned)cell + xf) * 4 + (fz ? 2 : 0));
                const float2 a = order(fy, s00.x, s00.y), b = order(fy, s10.x, s10.y);
                red_add_v2(q, a.x, a.y);
                red_add_v2(out + ((size_t)((unsigned)cell + 1u - xf) * 4 + (fz ? 2 : 0)), b.x, b.y);
            } else {
                float* q = out + (cell + first);
                atomicAdd(q, s00.x);
                atomicAdd(q + stepy, s00.y);
                atomicAdd(q + stepx, s10.x);
                atomicAdd(q + stepx + stepy, s10.y);
            }
            s00 = s01;
            s10 = s11;
            s01 = s11 = make_float2(0.f, 0.f);
        } else {
            flush();
        }
        cell = off;
    };
    const float dx = fabsf(r.dfx), dy = fabsf(r.dfy), dzz = fabsf(r.dfz);
    const float kxy = dx * dy * (1.0f / 12.0f), kxz = dx * dzz * (1.0f / 12.0f), kyz = dy * dzz * (1.0f / 12.0f);
    // n samples with midpoint fractions (x, y, z) towards the corners ahead
    auto add = [&](float n, float x, float y, float z) {
        const float g = n * yv, h = fmaf(n, n, -1.0f), c = h * g;
        const float a = c * kxy, gy = g * y;
        const float2 v = make_float2(g - gy, gy);
        const float2 p1 = __ffma2_rn(make_float2(x, x), v, make_float2(-a, a));  // x ahead, both z
        const float2 p0 = __fadd2_rn(v, make_float2(-p1.x, -p1.y));
        if (CONE) {
            const float b = h * kxz, e = c * kyz, ex = e * x;  // v holds g already
            const float2 z2 = make_float2(z, z);
            const float2 t = __ffma2_rn(z2, v, make_float2(-e, e));  // z ahead, both x
            const float2 q1 = __ffma2_rn(z2, p1, __ffma2_rn(make_float2(b, b), v, make_float2(-ex, ex)));
            const float2 q0 = __fadd2_rn(t, make_float2(-q1.x, -q1.y));
            s11 = __fadd2_rn(s11, q1);
            s01 = __fadd2_rn(s01, q0);
            s10 = __fadd2_rn(s10, __fadd2_rn(p1, make_float2(-q1.x, -q1.y)));
            s00 = __fadd2_rn(s00, __fadd2_rn(p0, make_float2(-q0.x, -q0.y)));
        } else {
            s10 = __fadd2_rn(s10, p1);
            s00 = __fadd2_rn(s00, p0);
        }
    };
    // samples at the ends of the range, where the inside test decides
    auto sample = [&](int k) {
        const float fk = (float)k;
        const float px = fmaf(fk, r.dfx, r.fx0), py = fmaf(fk, r.dfy, r.fy0);
        const float xf_ = floorf(px), yf_ = floorf(py);
        if (!(xf_ >= 0.0f && xf_ + 1.0f < (float)nx && yf_ >= 0.0f && yf_ + 1.0f < (float)nx)) return;
        int zi = iv;
        float zw = 0.0f;
        if (CONE) {
            const float pz = fmaf(fk, r.dfz, r.fz0);
            const float zf_ = floorf(pz);
            if (!(zf_ >= 0.0f && zf_ + 1.0f < (float)p.nz)) return;
            zi = (int)zf_;
            zw = pz - zf_;
        }
        enter(zi * plane + (int)yf_ * nx + (int)xf_);
        const float xw = px - xf_, yw = py - yf_;
        add(1.0f, fx ? 1.0f - xw : xw, fy ? 1.0f - yw : yw, fz ? 1.0f - zw : zw);
    };
    int kis, kie;
    interior_range(p, r, CONE, kis, kie);
    for (int k = r.ks; k < kis; ++k) sample(k);
    if (kis <= kie) {
        const float M = 12582912.0f;
        const unsigned MB = 0x4B400000u;  // bit pattern of M
        const unsigned obias = CONE ? MB * (unsigned)(plane + nx + 1) : MB * (unsigned)(nx + 1) - (unsigned)(iv * plane);
        const float2 dxy = make_float2(r.dfx, r.dfy), fxy0 = make_float2(r.fx0, r.fy0);
        const float2 flip = make_float2(fx ? -1.0f : 1.0f, fy ? -1.0f : 1.0f), base = make_float2(fx ? 1.0f : 0.0f, fy ? 1.0f : 0.0f);
        const float2 hd = make_float2(0.5f * dx, 0.5f * dy);
        const float hdz = 0.5f * dzz;
        const float ix = fminf(1.0f / dx, 1e30f), iy = fminf(1.0f / dy, 1e30f), iz = fminf(1.0f / dzz, 1e30f);  // as in fp_kernel
        const float kend = (float)kie;
        float fk = (float)kis;
        while (fk <= kend) {
            const float2 f = __ffma2_rn(make_float2(fk, fk), dxy, fxy0);
            const float2 m = __fadd2_rd(f, make_float2(M, M));
            const float2 fl = __fadd2_rn(m, make_float2(-M, -M));
            const float2 w = __ffma2_rn(__fadd2_rn(f, make_float2(-fl.x, -fl.y)), flip, base);
            unsigned off = __float_as_uint(m.x) + __float_as_uint(m.y) * (unsigned)nx - obias;
            float zw = 0.0f;
            if (CONE) {
                const float pz = fmaf(fk, r.dfz, r.fz0);
                const float mz = __fadd_rd(pz, M);
                zw = pz - (mz - M);
                if (fz) zw = 1.0f - zw;
                off += __float_as_uint(mz) * (unsigned)plane;
            }
            // steps to the face ahead
            float t = fminf(fminf(fmaf(w.x, -ix, ix), fmaf(w.y, -iy, iy)), kend - fk);
            if (CONE) t = fminf(t, fmaf(zw, -iz, iz));
            const float n1 = fmaxf(__fadd_rd(t, M) - M, 0.0f);
            const float2 mid = __ffma2_rn(make_float2(n1, n1), hd, w);
            enter((int)off);
            add(n1 + 1.0f, mid.x, mid.y, fmaf(n1, hdz, zw));
            fk += n1 + 1.0f;
        }
    }
    for (int k = max(kie + 1, kis); k <= r.ke; ++k) sample(k);
    flush();
}

template <bool CONE, bool CELLS, bool fx, bool fy>
__device__ __forceinline__ void adjoint_ray_z(const FpParams& p, const Ray& r, int iv, float yv, float* __restrict__ out) {
    if (CONE && r.dfz < 0.0f)
        adjoint_ray<CONE, CELLS, fx, fy, CONE>(p, r, iv, yv, out);
    else
        adjoint_ray<CONE, CELLS, fx, fy, false>(p, r, iv, yv, out);
}

// One ray of the adjoint sample by sample: a cell's corner sums are kept in registers and all
// added when the ray enters another, to the volume or to the workspace: with FACES to XF of
// fp_adjoint_kernel (the faces behind and ahead along x), else to the cell's own 8 (fan beam: 4)
// sums, x first.
template <bool CONE, bool CELLS, bool FACES>
__device__ __forceinline__ void adjoint_ray_samples(const FpParams& p, const Ray& r, int iv, float yv,
                                                    float* __restrict__ out) {
    const int nx = p.nx;
    const int plane = nx * nx;
    int cell = -1;
    float s00 = 0.f, s01 = 0.f, s10 = 0.f, s11 = 0.f, t00 = 0.f, t01 = 0.f, t10 = 0.f, t11 = 0.f;  // <y><x>; t: z ahead
    auto flush = [&]() {
        if (cell < 0) return;
        if constexpr (CELLS) {
            float* c = out + (int64_t)cell * (CONE && !FACES ? 8 : 4);
            if (CONE && FACES) {
                red_add_v4(c, s00, s10, t00, t10);
                red_add_v4(c + 4, s01, s11, t01, t11);
            } else {
                red_add_v4(c, s00, s01, s10, s11);
                if (CONE) red_add_v4(c + 4, t00, t01, t10, t11);
            }
        } else {
            float* b = out + cell;
            atomicAdd(b, s00);
            atomicAdd(b + 1, s01);
            atomicAdd(b + nx, s10);
            atomicAdd(b + nx + 1, s11);
            if (CONE) {
                float* c = b + plane;
                atomicAdd(c, t00);
                atomicAdd(c + 1, t01);
                atomicAdd(c + nx, t10);
                atomicAdd(c + nx + 1, t11);
            }
        }
        s00 = s01 = s10 = s11 = t00 = t01 = t10 = t11 = 0.f;
    };
    for (int k = r.ks; k <= r.ke; ++k) {
        const float fk = (float)k;
        const float fx = fmaf(fk, r.dfx, r.fx0), fy = fmaf(fk, r.dfy, r.fy0);
        const float xf = floorf(fx), yf = floorf(fy);
        if (!(xf >= 0.0f && xf + 1.0f < (float)nx && yf >= 0.0f && yf + 1.0f < (float)nx)) continue;
        const float xw = fx - xf, yw = fy - yf;
        int zi = iv;
        float zw = 0.0f;
        if (CONE) {
            const float fz = fmaf(fk, r.dfz, r.fz0);
            const float zf = floorf(fz);
            if (!(zf >= 0.0f && zf + 1.0f < (float)p.nz)) continue;
            zi = (int)zf;
            zw = fz - zf;
        }
        const int off = zi * plane + (int)yf * nx + (int)xf;
        if (off != cell) {
            flush();
            cell = off;
        }
        const float wl = CONE ? (1.0f - zw) * yv : yv;
        const float w00 = (1.0f - xw) * (1.0f - yw), w01 = xw * (1.0f - yw);
        const float w10 = (1.0f - xw) * yw, w11 = xw * yw;
        s00 += w00 * wl;
        s01 += w01 * wl;
        s10 += w10 * wl;
        s11 += w11 * wl;
        if (CONE) {
            const float wh = zw * yv;
            t00 += w00 * wh;
            t01 += w01 * wh;
            t10 += w10 * wh;
            t11 += w11 * wh;
        }
    }
    flush();
}

// Exact transpose of fp_kernel: every in-volume sample scatters its trilinear weights
// times the ray value into the volume.  As in the projector, the samples of one cell are
// taken together: a corner's weights summed over n equally spaced samples with midpoint m
// are n [u v w (m) + s^2 (du dv w + du dw v + dv dw u)(m)], s^2 = (n^2 - 1) / 12, for the
// corner's linear weights u, v, w along the axes.
//
// A ray that crosses into the next cell along x or y is done with the face it leaves
// behind: that face's corners are reduced, the ones it shares with the next cell stay in
// registers.  A crossing along z (rare) does the same with the corners left behind, any
// other change of cell reduces all.  Without CELLS the corners are added to the volume one
// by one.  CELLS, cone beam: the faces' sums go to two buffers in the workspace, 16 bytes
// per voxel each: XF(z, y, x) holds the face {y, y+1} x {z, z+1} at x, YF(z, y, x) the face
// {x, x+1} x {z, z+1} at y, both ordered (lo, lo) (hi, lo) (lo, hi) (hi, hi) with z last:
// one 16-byte reduction a face, two of 8 bytes in XF for a crossing along z;
// adjoint_gather_kernel then sums each voxel's entries of the faces that contain it.
// CELLS, fan beam: the 4 corner sums of a cell are one 16-byte reduction anyway (two edges
// of 8 bytes cost more: a reduction of 8 bytes takes the L2 as long as one of 16).
//
// 250^2 x 45, 501 x 47 x 181 views: 2.5 ms, sample by sample with both 16-byte groups of a
// cell reduced at every change of cell 4.6 ms.  The reductions bound it: the L2 is at 78 % of
// its peak (16 bytes for each of some 6e8 crossings), and neither more warps nor fewer
// instructions (16 selects less per cell: 2 %) nor an XF with y first, whose entries of
// neighbouring rays share a sector (0 %), bring much more.  Without CELLS, ms before /
// after: 123x123x51, 300 views 7.95 / 5.16, step 0.5 6.06 / 5.05; fan beam 300^2 x 4, 360
// views 2.35 / 1.40.  Blocks of 8 rows of rays (4 cost the scalar additions 2 to 10 %); of 4
// for cone beam with CELLS (grad above 2 %, 512^2 x 64 4 %), where the grid allows it.
// Where a cell holds few samples, fp_adjoint_samples_kernel below (adjoint_by_samples).
template <bool CONE, bool CELLS>
__global__ void __launch_bounds__(256)
fp_adjoint_kernel(FpParams p, const float* __restrict__ angles, const float* __restrict__ u_arr,
                  const float* __restrict__ v_arr, const float* __restrict__ czv, const float* __restrict__ pa,
                  const float* __restrict__ pxs, const float* __restrict__ sgm, const float* __restrict__ mask,
                  float* __restrict__ out) {
    const int iu = blockIdx.x * blockDim.x + threadIdx.x;
    const int iv = blockIdx.z * blockDim.y + threadIdx.y;
    const int j = blockIdx.y;
    if (iu >= p.nu || iv >= p.nv) return;
    const int64_t oidx = ((int64_t)iv * p.views + j) * p.nu + iu;
    if (mask && mask[oidx] != 1.0f) return;
    const float yv = sgm[oidx] * p.stepvd;
    if (yv == 0.0f) return;
    Ray r;
    if (!setup_ray(p, iu, iv, j, angles, u_arr, v_arr, czv, pa, pxs, true, r)) return;
    if (!(fabsf(yv) <= 3.4e38f)) {  // an infinite value: corners are not what others leave of it
        adjoint_ray_samples<CONE, CELLS, CONE>(p, r, iv, yv, out);
        return;
    }
    if (r.dfx < 0.0f) {
        if (r.dfy < 0.0f)
            adjoint_ray_z<CONE, CELLS, true, true>(p, r, iv, yv, out);
        else
            adjoint_ray_z<CONE, CELLS, true, false>(p, r, iv, yv, out);
    } else {
        if (r.dfy < 0.0f)
            adjoint_ray_z<CONE, CELLS, false, true>(p, r, iv, yv, out);
        else
            adjoint_ray_z<CONE, CELLS, false, false>(p, r, iv, yv, out);
    }
}

// The adjoint sample by sample, for rays with few cells or about a sample per cell.  In the
// workspace each cell has its own 32 bytes: in faces, which neighbouring cells share, many rays on a
// small volume wait for each other's additions (42x42x2, 793 views, step 0.5 84 us, now 66).
template <bool CONE, bool CELLS>
__global__ void __launch_bounds__(256)
fp_adjoint_samples_kernel(FpParams p, const float* __restrict__ angles, const float* __restrict__ u_arr,
                          const float* __restrict__ v_arr, const float* __restrict__ czv, const float* __restrict__ pa,
                          const float* __restrict__ pxs, const float* __restrict__ sgm, const float* __restrict__ mask,
                          float* __restrict__ out) {
    const int iu = blockIdx.x * blockDim.x + threadIdx.x;
    const int iv = blockIdx.z * blockDim.y + threadIdx.y;
    const int j = blockIdx.y;
    if (iu >= p.nu || iv >= p.nv) return;
    const int64_t oidx = ((int64_t)iv * p.views + j) * p.nu + iu;
    if (mask && mask[oidx] != 1.0f) return;
    const float yv = sgm[oidx] * p.stepvd;
    if (yv == 0.0f) return;
    Ray r;
    if (!setup_ray(p, iu, iv, j, angles, u_arr, v_arr, czv, pa, pxs, true, r)) return;
    adjoint_ray_samples<CONE, CELLS, false>(p, r, iv, yv, out);
}

// vol[z][y][x] += its entries of the cells that contain it (8 sums each in cone beam, 4 in fan
// beam), or with FACES of the faces (buffers XF and YF above), in a fixed order.
template <bool CONE, bool FACES>
__global__ void __launch_bounds__(256)
adjoint_gather_kernel(int nx, int nz, const float* __restrict__ cells, float* __restrict__ vol) {
    const int x = blockIdx.x * blockDim.x + threadIdx.x;
    const int y = blockIdx.y * blockDim.y + threadIdx.y;
    const int z = blockIdx.z;
    if (x >= nx || y >= nx || z >= nz) return;
    const int64_t plane = (int64_t)nx * nx;
    const int64_t v = z * plane + (int64_t)y * nx + x;
    float acc = 0.0f;
    if constexpr (FACES) {
        const float* yfaces = cells + (int64_t)nz * plane * 4;
#pragma unroll
        for (int dz = 0; dz < 2; ++dz) {
            if (z - dz < 0) continue;
#pragma unroll
            for (int d = 0; d < 2; ++d) {
                const int64_t c = v - dz * plane;
                if (y - d >= 0) acc += __ldg(cells + (c - (int64_t)d * nx) * 4 + dz * 2 + d);
                if (x - d >= 0) acc += __ldg(yfaces + (c - d) * 4 + dz * 2 + d);
            }
        }
    } else {
        constexpr int C = CONE ? 8 : 4;
#pragma unroll
        for (int dz = 0; dz < C / 4; ++dz) {
            if (z - dz < 0) continue;
#pragma unroll
            for (int dy = 0; dy < 2; ++dy) {
                if (y - dy < 0) continue;
#pragma unroll
                for (int dx = 0; dx < 2; ++dx) {
                    if (x - dx < 0) continue;
                    acc += __ldg(cells + (v - dz * plane - (int64_t)dy * nx - dx) * C + dz * 4 + dy * 2 + dx);
                }
            }
        }
    }
    vol[v] += acc;
}

// Effective ray map, run_mgfbp_iterative_recon_IRN_CGLS.py:749-833.
__global__ void __launch_bounds__(256)
emap_kernel(FpParams p, const float* __restrict__ angles, const float* __restrict__ u_arr,
            const float* __restrict__ v_arr, const float* __restrict__ czv, const float* __restrict__ pa,
            const float* __restrict__ pxs, float* __restrict__ mask) {
    const int iu = blockIdx.x * blockDim.x + threadIdx.x;
    const int iv = blockIdx.z * blockDim.y + threadIdx.y;
    const int j = blockIdx.y;
    if (iu >= p.nu || iv >= p.nv) return;
    const int64_t oidx = ((int64_t)iv * p.views + j) * p.nu + iu;
    float m = 1.0f;
    Ray r;
    if (p.cone && setup_ray(p, iu, iv, j, angles, u_arr, v_arr, czv, pa, pxs, false, r)) {
        const float h = (float)p.nx / 2.0f;
        for (int k = r.ks; k <= r.ke; ++k) {
            const float fk = (float)k;
            const float xf = floorf(fmaf(fk, r.dfx, r.fx0));
            const float yf = floorf(fmaf(fk, r.dfy, r.fy0));
            if (!(xf >= 0.0f && xf + 1.0f < (float)p.nx && yf >= 0.0f && yf + 1.0f < (float)p.nx)) continue;
            if ((xf - h) * (xf - h) + (yf - h) * (yf - h) < h * h) {
                const float zf = floorf(fmaf(fk, r.dfz, r.fz0));
                if (zf < 0.0f || zf + 1.0f >= (float)p.nz) {
                    m = 0.0f;
                    break;
                }
            }
        }
    }
    mask[oidx] = m;
}

// Number of in-volume trilinear samples (the forward projector's algorithmic work).
__global__ void __launch_bounds__(256)
fp_count_kernel(FpParams p, const float* __restrict__ angles, const float* __restrict__ u_arr,
                const float* __restrict__ v_arr, const float* __restrict__ czv, const float* __restrict__ pa,
                const float* __restrict__ pxs, const float* __restrict__ mask, unsigned long long* __restrict__ count) {
    const int iu = blockIdx.x * blockDim.x + threadIdx.x;
    const int iv = blockIdx.z * blockDim.y + threadIdx.y;
    const int j = blockIdx.y;
    unsigned long long c = 0;
    Ray r;
    if (iu < p.nu && iv < p.nv && !(mask && mask[((int64_t)iv * p.views + j) * p.nu + iu] != 1.0f) &&
        setup_ray(p, iu, iv, j, angles, u_arr, v_arr, czv, pa, pxs, true, r)) {
        for (int k = r.ks; k <= r.ke; ++k) {
            const float fk = (float)k;
            const float xf = floorf(fmaf(fk, r.dfx, r.fx0)), yf = floorf(fmaf(fk, r.dfy, r.fy0));
            if (!(xf >= 0.0f && xf + 1.0f < (float)p.nx && yf >= 0.0f && yf + 1.0f < (float)p.nx)) continue;
            if (p.cone) {
                const float zf = floorf(fmaf(fk, r.dfz, r.fz0));
                if (!(zf >= 0.0f && zf + 1.0f < (float)p.nz)) continue;
            }
            ++c;
        }
    }
    // warp-aggregate, one atomic per warp
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) c += __shfl_down_sync(0xffffffffu, c, o);
    if ((threadIdx.x & 31) == 0 && c) atomicAdd(count, c);
}

__device__ __forceinline__ uint64_t splitmix64(uint64_t x) {
    x += 0x9E3779B97F4A7C15ull;
    x = (x ^ (x >> 30)) * 0xBF58476D1CE4E5B9ull;
    x = (x ^ (x >> 27)) * 0x94D049BB133111EBull;
    return x ^ (x >> 31);
}

// Oversample binning + Gaussian-approximated photon noise, run_mgfpj_v3.py:368-391.
__global__ void bin_noise_kernel(int64_t n_out, int nu, int bin, float photons, uint64_t seed,
                                 const float* __restrict__ in, float* __restrict__ out) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n_out; i += (int64_t)gridDim.x * blockDim.x) {
        const int64_t rowv = i / nu;
        const int c = (int)(i % nu);
        const float* src = in + rowv * (int64_t)nu * bin + (int64_t)c * bin;
        float s = 0.0f;
        for (int b = 0; b < bin; ++b) s += src[b];
        float val = s / (float)bin;
        if (photons > 0.0f) {
            uint64_t h1 = splitmix64(seed ^ (uint64_t)(2 * i));
            uint64_t h2 = splitmix64(seed ^ (uint64_t)(2 * i + 1) ^ 0x5851F42D4C957F2Dull);
            float u1 = ((h1 >> 40) + 1.0f) * (1.0f / 16777217.0f);
            float u2 = (h2 >> 40) * (1.0f / 16777216.0f);
            float g = sqrtf(-2.0f * logf(u1)) * cospif(2.0f * u2);
            float t = photons * expf(-val);
            t = t + g * sqrtf(t);
            if (t <= 0.0f) t = 1e-6f;
            val = logf(photons / t);
        }
        out[i] = val;
    }
}

// Exact line integrals of rotated ellipsoids along the forward projector's rays.
__global__ void __launch_bounds__(256)
ellipsoid_kernel(FpParams p, const float* __restrict__ angles, const float* __restrict__ u_arr,
                 const float* __restrict__ v_arr, const float* __restrict__ ell, int n_ell,
                 float* __restrict__ sgm) {
    const int iu = blockIdx.x * blockDim.x + threadIdx.x;
    const int iv = blockIdx.z * blockDim.y + threadIdx.y;
    const int j = blockIdx.y;
    if (iu >= p.nu || iv >= p.nv) return;
    float sb, cb;
    sincosf(angles[j], &sb, &cb);
    const float zj = p.zpv * (float)j;
    const float uval = u_arr[iu];
    float dx, dy;
    if (p.curved) {
        float sg, cg;
        sincosf((-uval) / p.sdd, &sg, &cg);
        dx = -p.sdd * cg + p.sid;
        dy = -p.sdd * sg;
    } else {
        dx = -(p.sdd - p.sid);
        dy = uval;
    }
    const float ex = dx - p.sid, ey = dy, ez = v_arr[iv];
    const float dist = sqrtf(ex * ex + ey * ey + ez * ez);
    const double ux = ex / dist, uy = ey / dist, uz = ez / dist;
    // source and direction in the object frame (object rotated by +beta)
    const double Ox = p.sid * (double)cb, Oy = p.sid * (double)sb, Oz = zj;
    const double Dx = ux * cb - uy * sb, Dy = uy * cb + ux * sb, Dz = uz;
    double total = 0.0;
    for (int e = 0; e < n_ell; ++e) {
        const float* E = ell + 10 * e;
        const double cph = cos((double)E[6]), sph = sin((double)E[6]);
        const double qx = Ox - E[0], qy = Oy - E[1], qz = Oz - E[2];
        const double px_ = (qx * cph + qy * sph) / E[3], py_ = (-qx * sph + qy * cph) / E[4], pz_ = qz / E[5];
        const double dx_ = (Dx * cph + Dy * sph) / E[3], dy_ = (-Dx * sph + Dy * cph) / E[4], dz_ = Dz / E[5];
        const double a = dx_ * dx_ + dy_ * dy_ + dz_ * dz_;
        const double b = px_ * dx_ + py_ * dy_ + pz_ * dz_;
        const double c = px_ * px_ + py_ * py_ + pz_ * pz_ - 1.0;
        const double disc = b * b - a * c;
        if (disc > 0.0) total += E[9] * 2.0 * sqrt(disc) / a;
    }
    sgm[((int64_t)iv * p.views + j) * p.nu + iu] = (float)total;
}

// Elements per row of the gather copies: from 128 columns, 3 more than a multiple of 8,
// so that the same column of neighbouring rows lies in different 16-byte L1 banks
// (unpadded / 3 more, by cells: 512x512x256, 1080 views 181.8 / 171.9 ms; 128x128x64, 270
// views 0.819 / 0.800 ms; 1 to 7 more are within 0.7 %).  Narrower volumes and those whose
// padded copy would reach 2^31 elements are not padded.
inline int copy_pitch(const mct_geom* g) {
    const int pitch = ((g->nx + 7) & ~7) + 3;
    return g->nx >= 128 && (int64_t)g->nz * g->nx * pitch < ((int64_t)1 << 31) ? pitch : g->nx;
}
// Whether float32 quads are walked in windows (fan beam always is: its warps span more cells).
inline bool walk_in_windows(const mct_geom* g) { return g->nx >= 256; }
// Samples of a ray per cell: its cell crossings per voxel length are 1.33 on average over a scan.
inline double samples_per_cell(const mct_geom* g) {
    const double step = g->fp_step * std::sqrt(2.0 + ((double)g->pz / g->px) * ((double)g->pz / g->px));
    return 1.0 / (1.33 * step);
}
// Scans whose neighbouring views cross nearly the same cells.
inline bool long_scan(const mct_geom* g) { return g->views >= 256 || g->views >= g->nx; }
// Whether a ray is walked by samples: few samples per cell.  us, by samples / by cells (what
// the walk by samples was before the walk by cells came):
//   bf16 256x256x64, 360 views, step 0.3 (1.4 samples per cell) 3220 / 3310, 0.5 (0.9) 2100 / 2950;
//   float16, which pays more per load: 32x32x23, 35 views, 0.3 23.2 / 30.8 (27.0), 170x170x19, 37
//     views 90.6 / 108.5 (94.5); from 256 columns 0.3 is even, 0.5 2330 / 3190;
//   float32 123x123x51, 686 views, 0.3 1320 / 1261, 0.4 (1.1) 1106 / 1193, 0.5 974 / 1119;
//     224x224x64, 120 views, 0.4 901 / 897, 0.5 795 / 841; without copies 81x81x3, 171 views,
//     0.5 27.5 / 32.3 (26.8), 54x54x36, 23 views, 1.2 14.5 / 17.9 (16.4);
//   fan beam 491 columns, 147 views, 0.5 (1.1) 194 / 223 (207), 253 columns, 52 views, 1.2
//     43.7 / 49.1 (45.3); step 0.3 (1.8) costs samples 1.5 to 1.9 times as much.
//   16-bit between the two: bf16 81x81x3, 158 views (1.53) 25 / 38 (33), 459x459x10, 288 views
//     (1.63) 2093 / 2170, 412x412x94, 376 views (1.63) 16920 / 16140; float16 187x187x10, 59 views
//     (1.53) 109 / 123 (134), 96x96x53 (1.63) 932 / 858.
// With windows, from 256 columns on, float32 with copies: short scans stay by cells (512x512x64, 90
// views, 0.5 3567 / 3252) until a cell holds few samples (509x509x185, 125 views, 1.3 (0.33) 7640 /
// 8940 (8230)); long ones go by samples (319x319x109, 617 views, 0.5 13570 / 14380 (13964); 277x277x74,
// 439 views, 1.0 (0.43) 4185 / 4780 (4189); 426 columns, 0.7 (0.6) 15725 / 15290).  Without copies
// 362x362x161, 284 views, 0.5 49.1 / 56.6 (56.8) ms, 402x402x15, 346 views 4.25 / 4.54 (5.49), 0.8
// 458x458x52, 306 views 6.57 / 6.57 (8.45).
inline bool walk_by_samples(const mct_geom* g, int32_t dtype, bool copies) {
    const bool cone = (g->flags & MCT_CONE) != 0, wide = walk_in_windows(g);
    const double n = samples_per_cell(g);
    if (dtype == MCT_F32 && cone && wide) return n < (copies && !long_scan(g) ? 0.4 : 1.2);
    return n < (dtype == MCT_BF16 ? 1.65 : dtype == MCT_F16 && !wide ? 1.55 : 1.2);
}
// Whether the adjoint goes by samples; figures by samples / by cells.
// A thread pays for a walk by cells before its first sample, so grids that leave the GPU
// waiting go by samples where a cell holds about one: 66x66x2, 55 views of 2 x 123, step 1.2,
// without a workspace 7.8 / 13.6 us; 90x90x4, 73 views of 4 x 174, step 0.5, with one 36 / 42 us.
// Fan beam with a workspace: the reductions are the same either way (445^2 x 2, 179 views, step
// 0.5 417 / 425 us, 0.3 492 / 449).
// Otherwise it is the faces that the walk by cells saves, which pays until a cell holds half a
// sample.  Without a workspace 123x123x51, 300 views, step 0.7 5.7 / 5.1 ms, 1.0 3.97 / 4.02, 1.5 2.71
// / 2.81; fan beam 300^2 x 4, 360 views, 1.0 1.49 / 1.33, 1.5 0.98 / 0.97.  With one 51x51x19, 95 views,
// 0.8 31 / 46 us; 55x55x10, 227 views, 0.5 143 / 88 us; 150x150x8, 265 views, 0.8 447 / 347 us;
// 316x316x17, 69 views, 1.0 (0.43 samples) 964 / 796 us; 62x62x2, 561 views, 1.3 (0.33) 46 / 56 us.
inline bool adjoint_by_samples(const mct_geom* g, bool cells) {
    const bool cone = (g->flags & MCT_CONE) != 0;
    const double n = samples_per_cell(g);
    const int64_t rays = sgm_elems(*g);
    if ((!cone && cells) || rays < 60000) return n < (rays < 4000 ? 1.6 : 1.2);
    return cone && n < (g->nx < 64 ? 0.6 : cells ? 0.4 : 0.45);
}
inline size_t copy_elems(const mct_geom* g) { return (size_t)g->nz * g->nx * copy_pitch(g); }

int make_params(const mct_geom* g, FpParams& p, const char* who) {
    MCT_TRY(check_geom(g, who));
    MCT_TRY(check_whole_scan(g, who));
    p = ray_params(g);
    MCT_REQUIRE(p.K >= 0, "%s: negative step count", who);
    MCT_REQUIRE(g->views <= 65535, "%s: at most 65535 views per launch", who);
    MCT_REQUIRE(p.cone || g->nz >= g->nv, "%s: fan beam needs one image slice per detector row", who);
    MCT_REQUIRE(!p.cone || g->pz > 0.0f, "%s: cone beam needs a positive voxel height", who);
    MCT_REQUIRE(g->px > 0.0f, "%s: pixel size must be positive", who);
    MCT_REQUIRE((int64_t)g->nz * g->nx * g->nx < ((int64_t)1 << 31), "%s: volume must have fewer than 2^31 voxels", who);
    return MCT_OK;
}

}  // namespace
}  // namespace mct

using namespace mct;

extern "C" {

size_t mct_fp_workspace_size(const mct_geom* g) {
    if (!g || g->nx < 1 || g->nz < 1) return 0;
    const size_t n = (size_t)g->nz * g->nx * g->nx;
    // cone beam: two float32 quad copies (16 bytes per voxel each); fan beam: one
    // transposed copy
    return (g->flags & MCT_CONE) ? 2 * copy_elems(g) * sizeof(Quad16) : n * sizeof(float);
}

size_t mct_fp_storage_workspace_size(const mct_geom* g, int32_t dtype) {
    if (!g || g->nx < 1 || g->nz < 1) return 0;
    if (dtype == MCT_F32) return mct_fp_workspace_size(g);
    if (!(g->flags & MCT_CONE) || (dtype != MCT_BF16 && dtype != MCT_F16)) return 0;
    // two 16-bit cell copies (+16 bytes for the float16 scale's source maximum)
    return 2 * copy_elems(g) * sizeof(uint4) + (dtype == MCT_F16 ? 16 : 0);
}

}  // extern "C"

namespace {
// The projector's launches with a float32 or bf16 volume (TIN); the bf16 volume is read
// only by the copy kernels, so it needs cone beam and a workspace.
template <typename TIN>
int fp_storage_impl(const mct_geom* g, const mct_tables* t, const TIN* vol_in, const float* mask, float* sgm,
                    void* workspace, int32_t dtype, void* stream) {
    const float* vol = reinterpret_cast<const float*>(vol_in);  // read as float32 only when TIN is float
    constexpr bool kIn32 = std::is_same<TIN, float>::value;
    FpParams p;
    MCT_TRY(make_params(g, p, "mct_fp"));
    MCT_REQUIRE(t && t->angles && t->u && t->v && vol && sgm, "mct_fp: NULL buffer");
    MCT_REQUIRE(kIn32 || (p.cone && workspace), "mct_fp: a bf16 volume needs cone beam and a workspace");
    MCT_REQUIRE(!p.pmat || (t->pmat_a && t->pmat_xs), "mct_fp: projection-matrix tables missing");
    MCT_REQUIRE(workspace != (void*)vol, "mct_fp: workspace aliases the volume");
    MCT_REQUIRE(((uintptr_t)workspace & 15) == 0, "mct_fp: workspace must be 16-byte aligned");
    MCT_REQUIRE(dtype == MCT_F32 || dtype == MCT_BF16 || dtype == MCT_F16,
                "mct_fp: dtype must be MCT_F32, MCT_BF16 or MCT_F16");
    MCT_REQUIRE(dtype == MCT_F32 || (p.cone && workspace), "mct_fp: 16-bit storage needs cone beam and a workspace");
    cudaStream_t s = as_stream(stream);
    if (g->nx < 2 || (p.cone && g->nz < 2)) {
        // no trilinear stencil fits inside the volume: every ray sums nothing, as in the
        // reference (its inside test fails for every sample)
        cudaError_t e = cudaMemsetAsync(sgm, 0, (size_t)sgm_elems(*g) * sizeof(float), s);
        if (e != cudaSuccess) {
            set_error("mct_fp: %s", cudaGetErrorString(e));
            return MCT_E_CUDA;
        }
        return MCT_OK;
    }
    dim3 tb(32, 8), tg((g->nx + 31) / 32, (g->nx + 31) / 32, g->nz);
    // Ray tiles: 16 detector columns x 16 consecutive views of one row, warps of 2^wcs
    // columns.  The rays of neighbouring views cross nearly the same cells, the more so the
    // closer the views, so scans of at least 256 views, or of a view per image column, take
    // warps of 4 columns x 8 views and others 16 columns x 2 views.  float32, ms with 4 / 16
    // columns per warp: 512x512x256, 1080 views 159.0 / 168.7; 512x512x64: 180 views 8.68 /
    // 8.28, 90 views 5.23 / 4.86, 60 views 3.74 / 3.48; 224x224x64, 300 views 2.04 / 2.14;
    // 128x128x64, 270 views 0.698 / 0.741; 123x123x51: 140 views 0.325 / 0.335, 90 views 0.241
    // / 0.240; 100x100x40, 200 views 0.228 / 0.245; 64^3, 180 views 0.158 / 0.169.  16-bit
    // cells take 4 views x 4 rows: bf16 512x512x128, 90 views 7.60 ms against 7.73 with 16
    // views; 256x256x64, 360 views 3.457 against 3.480.  Fan beam: warps of 8 columns x 4
    // views (512^2, 720 views, 4 / 8 / 16 columns: 0.604 / 0.596 / 0.595; 128^2 x
    // 16, 360 views 0.327 / 0.324 / 0.339; one row of 32 columns x 8 rows, 7 of them idle for one
    // slice: 0.664), of 16 x 2 where the views are far apart and there are slices enough (243^2 x
    // 65, 46 views, step 0.8 0.420 / 0.368; 258^2 x 4, 67 views, step 0.1 0.124 / 0.114).  By samples, blocks of 128 rays, 16 columns x 8 views, in warps of 4 (long
    // scans) or 8 columns: 170x170x19, 37 views, float16 90.6 us against 97.7 with 4 views x 4
    // rows; 68x68x18, 224 views, bf16 13 % less, fan beam 246 columns, 134 views 53.9 us against
    // 60.4; only wide long scans keep 16 views (float32 388 columns, 885 views 26.6 / 27.3 ms).
    // Where the tile leaves a fifth of its rays outside the scan, 8 or 4 views x 2 or 4 rows
    // (fan beam 210 columns x 16 rows, 23 views 200 -> 153 us).
    // With copies, 4 rows are taken in turn per view group: neighbouring rows' rays
    // cross nearly the same cells, and the outer rows' slab (up to ~50 planes) does not fit
    // L2 across all views.  Otherwise row tiles are only grouped where the grid needs it.
    const bool copies = p.cone && workspace, by_samples = walk_by_samples(g, dtype, copies);
    // Wide float32 volumes without copies, or by samples with far apart views, take 4 views x 4 rows
    // in warps of 16 columns.  By samples, with 16 views / so: without copies 362x362x161, 284 views,
    // step 0.5 65.8 / 49.1 ms, 458x458x52, 306 views, 0.8 7.40 / 6.57; with copies 509x509x185, 125
    // views, 1.3 8.12 / 7.64.  By cells without copies 298x298x35, 536 views, 0.1 6.97 / 6.98.
    const bool wide32 = dtype == MCT_F32 && p.cone && walk_in_windows(g);
    const bool small_tile = by_samples && !wide32 && g->nv <= 65535;
    const bool row_tile = wide32 && (!copies || (by_samples && !long_scan(g)));
    p.ls = small_tile ? 7 : 8;
    p.vshift = small_tile ? 3 : (copies && dtype != MCT_F32) || row_tile ? 2 : 4;
    if (p.cone) p.wcs = row_tile ? 4 : long_scan(g) ? 2 : by_samples ? 3 : 4;
    else p.wcs = g->nv >= 4 && 2 * g->views < g->nx ? 4 : 3;
    if (!small_tile) {
        auto rays = [&](int vs) {  // of the tiles of 2^vs views, in and outside the scan
            const int64_t v = (1 << vs) - 1, r = (1 << (4 - vs)) - 1;
            return ((g->views + v) & ~v) * ((g->nv + r) & ~r);
        };
        int best = 4;
        for (int vs = 3; vs >= 2; --vs)
            if (rays(vs) < rays(best)) best = vs;
        if (rays(p.vshift) * 4 > rays(best) * 5) p.vshift = best;
    }
    const int row_bits = p.ls - 4 - p.vshift;
    p.rs = copies ? (row_bits < 2 ? 2 - row_bits : 0) : (g->nv > 65535 ? 3 : 0);
    if (copies) p.pitch = copy_pitch(g);
    const int vb = 1 << p.vshift, rb = 1 << (row_bits + p.rs);
    dim3 block(32, 1 << (p.ls - 5)), grid((g->nu + 15) / 16, ((g->views + vb - 1) / vb) << p.rs, (g->nv + rb - 1) / rb);
    const size_t n = copy_elems(g);
    if (copies && dtype == MCT_BF16) {
        uint4* cx = static_cast<uint4*>(workspace);
        uint4* cy = cx + n;
        cell16_kernel<false><<<tg, tb, 0, s>>>(g->nx, g->nz, p.pitch, vol_in, cx, cy, nullptr);
        MCT_TRY(launched("cell16_kernel"));
        auto go = by_samples ? fp_kernel<true, true, uint4, kSamples> : fp_kernel<true, true, uint4, kCells>;
        go<<<grid, block, 0, s>>>(p, t->angles, t->u, t->v, t->cz, t->pmat_a, t->pmat_xs, vol, nullptr, cx, cy, mask, sgm,
                                  nullptr);
    } else if (copies && dtype == MCT_F16) {
        uint4* cx = static_cast<uint4*>(workspace);
        uint4* cy = cx + n;
        uint32_t* vmax = reinterpret_cast<uint32_t*>(cy + n);
        cudaError_t e = cudaMemsetAsync(vmax, 0, sizeof(uint32_t), s);
        if (e != cudaSuccess) {
            set_error("mct_fp: %s", cudaGetErrorString(e));
            return MCT_E_CUDA;
        }
        const int64_t voxels = vol_elems(*g), blocks = (voxels + 255) / 256;
        vol_absmax_kernel<<<(int)(blocks < 152 * 32 ? blocks : 152 * 32), 256, 0, s>>>(voxels, vol_in, vmax);
        MCT_TRY(launched("vol_absmax_kernel"));
        cell16_kernel<true><<<tg, tb, 0, s>>>(g->nx, g->nz, p.pitch, vol_in, cx, cy, vmax);
        MCT_TRY(launched("cell16_kernel"));
        auto go = by_samples ? fp_kernel<true, true, h16x8, kSamples> : fp_kernel<true, true, h16x8, kCells>;
        go<<<grid, block, 0, s>>>(p, t->angles, t->u, t->v, t->cz, t->pmat_a, t->pmat_xs, vol, nullptr,
                                  reinterpret_cast<const h16x8*>(cx), reinterpret_cast<const h16x8*>(cy), mask, sgm, vmax);
    } else if (copies) {
        Quad16* cx = static_cast<Quad16*>(workspace);
        Quad16* cy = cx + n;
        quad32_kernel<<<tg, tb, 0, s>>>(g->nx, g->nz, p.pitch, vol_in, reinterpret_cast<float4*>(cx),
                                        reinterpret_cast<float4*>(cy));
        MCT_TRY(launched("quad32_kernel"));
        auto go = by_samples           ? fp_kernel<true, true, Quad16, kSamples>
                  : walk_in_windows(g) ? fp_kernel<true, true, Quad16, kWindows>
                                       : fp_kernel<true, true, Quad16, kCells>;
        go<<<grid, block, 0, s>>>(p, t->angles, t->u, t->v, t->cz, t->pmat_a, t->pmat_xs, vol, nullptr, cx, cy, mask, sgm,
                                  nullptr);
    } else if constexpr (kIn32) {
        float* vt = static_cast<float*>(workspace);
        if (vt) {
            transpose_xy_kernel<<<tg, tb, 0, s>>>(g->nx, g->nz, vol, vt);
            MCT_TRY(launched("transpose_xy_kernel"));
        }
        auto go = p.cone ? (by_samples ? fp_kernel<true, false, float2, kSamples> : fp_kernel<true, false, float2, kCells>)
                         : (by_samples ? fp_kernel<false, false, float2, kSamples> : fp_kernel<false, false, float2, kWindows>);
        go<<<grid, block, 0, s>>>(p, t->angles, t->u, t->v, t->cz, t->pmat_a, t->pmat_xs, vol, vt, nullptr, nullptr, mask, sgm,
                                  nullptr);
    }
    return launched("fp_kernel");
}
}  // namespace

extern "C" {

int mct_fp_storage(const mct_geom* g, const mct_tables* t, const float* vol, const float* mask, float* sgm,
                   void* workspace, int32_t dtype, void* stream) {
    return fp_storage_impl<float>(g, t, vol, mask, sgm, workspace, dtype, stream);
}

int mct_fp_storage_in(const mct_geom* g, const mct_tables* t, const void* vol, int32_t vol_dtype, const float* mask,
                      float* sgm, void* workspace, int32_t dtype, void* stream) {
    MCT_REQUIRE(vol_dtype == MCT_F32 || vol_dtype == MCT_BF16, "mct_fp_storage_in: vol_dtype must be MCT_F32 or MCT_BF16");
    if (vol_dtype == MCT_F32)
        return fp_storage_impl<float>(g, t, static_cast<const float*>(vol), mask, sgm, workspace, dtype, stream);
    return fp_storage_impl<__nv_bfloat16>(g, t, static_cast<const __nv_bfloat16*>(vol), mask, sgm, workspace, dtype,
                                          stream);
}

int mct_fp(const mct_geom* g, const mct_tables* t, const float* vol, const float* mask, float* sgm, void* workspace,
           void* stream) {
    return mct_fp_storage(g, t, vol, mask, sgm, workspace, MCT_F32, stream);
}

int mct_fp_adjoint(const mct_geom* g, const mct_tables* t, const float* sgm, const float* mask, float* vol,
                   void* stream) {
    FpParams p;
    MCT_TRY(make_params(g, p, "mct_fp_adjoint"));
    MCT_REQUIRE(t && t->angles && t->u && t->v && vol && sgm, "mct_fp_adjoint: NULL buffer");
    MCT_REQUIRE(!p.pmat || (t->pmat_a && t->pmat_xs), "mct_fp_adjoint: projection-matrix tables missing");
    if (p.cone && g->nz < 2) return MCT_OK;  // no cell, so mct_fp sums nothing: its transpose adds nothing
    dim3 block(32, 8), grid((g->nu + 31) / 32, g->views, (g->nv + 7) / 8);
    const bool by_samples = adjoint_by_samples(g, false);
    auto go = p.cone ? (by_samples ? fp_adjoint_samples_kernel<true, false> : fp_adjoint_kernel<true, false>)
                     : (by_samples ? fp_adjoint_samples_kernel<false, false> : fp_adjoint_kernel<false, false>);
    go<<<grid, block, 0, as_stream(stream)>>>(p, t->angles, t->u, t->v, t->cz, t->pmat_a, t->pmat_xs, sgm, mask, vol);
    return launched("fp_adjoint_kernel");
}

size_t mct_fp_adjoint_workspace_size(const mct_geom* g) {
    if (!g || g->nx < 1 || g->nz < 1) return 0;
    return (size_t)g->nz * g->nx * g->nx * ((g->flags & MCT_CONE) ? 32 : 16);
}

int mct_fp_adjoint_cells(const mct_geom* g, const mct_tables* t, const float* sgm, const float* mask, float* vol,
                         void* workspace, void* stream) {
    FpParams p;
    MCT_TRY(make_params(g, p, "mct_fp_adjoint_cells"));
    MCT_REQUIRE(t && t->angles && t->u && t->v && vol && sgm && workspace, "mct_fp_adjoint_cells: NULL buffer");
    MCT_REQUIRE(!p.pmat || (t->pmat_a && t->pmat_xs), "mct_fp_adjoint_cells: projection-matrix tables missing");
    MCT_REQUIRE(((uintptr_t)workspace & 15) == 0, "mct_fp_adjoint_cells: workspace must be 16-byte aligned");
    MCT_REQUIRE(g->nx <= 65535 * 8 && g->nz <= 65535, "mct_fp_adjoint_cells: at most 524280 x 524280 x 65535 voxels");
    if (p.cone && g->nz < 2) return MCT_OK;  // as in mct_fp_adjoint
    cudaStream_t s = as_stream(stream);
    float* cells = static_cast<float*>(workspace);
    MCT_REQUIRE(cudaMemsetAsync(cells, 0, mct_fp_adjoint_workspace_size(g), s) == cudaSuccess,
                "mct_fp_adjoint_cells: clearing the workspace failed");
    const bool by_samples = adjoint_by_samples(g, true);
    const int rows = p.cone && !by_samples && g->nv <= 4 * 65535 ? 4 : 8;
    dim3 block(32, rows), grid((g->nu + 31) / 32, g->views, (g->nv + rows - 1) / rows);
    auto go = p.cone ? (by_samples ? fp_adjoint_samples_kernel<true, true> : fp_adjoint_kernel<true, true>)
                     : (by_samples ? fp_adjoint_samples_kernel<false, true> : fp_adjoint_kernel<false, true>);
    go<<<grid, block, 0, s>>>(p, t->angles, t->u, t->v, t->cz, t->pmat_a, t->pmat_xs, sgm, mask, cells);
    MCT_TRY(launched("fp_adjoint_kernel"));
    dim3 gb(32, 8), gg((g->nx + 31) / 32, (g->nx + 7) / 8, g->nz);
    auto gather = !p.cone ? adjoint_gather_kernel<false, false>
                  : by_samples ? adjoint_gather_kernel<true, false>
                               : adjoint_gather_kernel<true, true>;
    gather<<<gg, gb, 0, s>>>(g->nx, g->nz, cells, vol);
    return launched("adjoint_gather_kernel");
}

int mct_fp_count_samples(const mct_geom* g, const mct_tables* t, const float* mask, uint64_t* count, void* stream) {
    FpParams p;
    MCT_TRY(make_params(g, p, "mct_fp_count_samples"));
    MCT_REQUIRE(t && t->angles && t->u && t->v && count, "mct_fp_count_samples: NULL buffer");
    MCT_REQUIRE(!p.pmat || (t->pmat_a && t->pmat_xs), "mct_fp_count_samples: projection-matrix tables missing");
    cudaError_t e = cudaMemsetAsync(count, 0, sizeof(uint64_t), as_stream(stream));
    if (e != cudaSuccess) {
        set_error("mct_fp_count_samples: %s", cudaGetErrorString(e));
        return MCT_E_CUDA;
    }
    dim3 block(32, 8), grid((g->nu + 31) / 32, g->views, (g->nv + 7) / 8);
    fp_count_kernel<<<grid, block, 0, as_stream(stream)>>>(p, t->angles, t->u, t->v, t->cz, t->pmat_a, t->pmat_xs, mask,
                                                           (unsigned long long*)count);
    return launched("fp_count_kernel");
}

int mct_effective_map(const mct_geom* g, const mct_tables* t, float* mask, void* stream) {
    FpParams p;
    MCT_TRY(make_params(g, p, "mct_effective_map"));
    MCT_REQUIRE(t && t->angles && t->u && t->v && mask, "mct_effective_map: NULL buffer");
    MCT_REQUIRE(!p.pmat || (t->pmat_a && t->pmat_xs), "mct_effective_map: projection-matrix tables missing");
    dim3 block(32, 8), grid((g->nu + 31) / 32, g->views, (g->nv + 7) / 8);
    emap_kernel<<<grid, block, 0, as_stream(stream)>>>(p, t->angles, t->u, t->v, t->cz, t->pmat_a, t->pmat_xs, mask);
    return launched("emap_kernel");
}

int mct_bin_noise(const mct_geom* g, const float* in, int32_t bin, float photons, uint64_t seed, float* out,
                  void* stream) {
    MCT_TRY(check_geom(g, "mct_bin_noise"));
    MCT_REQUIRE(in && out && bin >= 1, "mct_bin_noise: bad arguments");
    MCT_REQUIRE(bin == 1 || in != out, "mct_bin_noise: binning cannot run in place");
    int64_t n = sgm_elems(*g);
    int64_t blocks = (n + 255) / 256;
    bin_noise_kernel<<<(int)(blocks < 152 * 64 ? (blocks < 1 ? 1 : blocks) : 152 * 64), 256, 0, as_stream(stream)>>>(
        n, g->nu, bin, photons, seed, in, out);
    return launched("bin_noise_kernel");
}

int mct_project_ellipsoids(const mct_geom* g, const mct_tables* t, const float* ell, int32_t n_ell, float* sgm,
                           void* stream) {
    FpParams p;
    MCT_TRY(make_params(g, p, "mct_project_ellipsoids"));
    MCT_REQUIRE(t && t->angles && t->u && t->v && ell && sgm && n_ell >= 0, "mct_project_ellipsoids: bad arguments");
    dim3 block(32, 8), grid((g->nu + 31) / 32, g->views, (g->nv + 7) / 8);
    ellipsoid_kernel<<<grid, block, 0, as_stream(stream)>>>(p, t->angles, t->u, t->v, ell, n_ell, sgm);
    return launched("ellipsoid_kernel");
}

}  // extern "C"
