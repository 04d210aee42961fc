// Pixel-driven FDK / fan-beam backprojection (run_mgfbp.py:1062-1187).
//
// Design (sm_103a):
//   * one thread owns one (x, y) column and ZC consecutive slices, accumulating every
//     view in registers (the reference does a global read-modify-write per view);
//   * the filtered sinogram is pre-packed so that the 2x2 bilinear stencil of a
//     detector position is ONE 16-byte (f32) or 8-byte (bf16) load;
//   * per-view cos/sin/weight tables (and projection matrices) live in shared memory;
//   * the slices of a column share x and y (z runs along the image's i_z axis in the
//     axial view mode and along i_y in the coronal and sagittal ones, whose columns
//     the kernel takes over (i_x, i_z)), so u, the distance weight and the
//     magnification are evaluated once per (column, view) and v is an affine
//     function of the slice index.
// Voxels that project outside the detector in any view are written as 0, as in the
// reference (the view loop "breaks" with the voxel set to 0).  In the cone-beam
// path an off-detector row index is redirected to the packed operand's NaN row, so the
// voxel's sum becomes NaN and is written as 0 without any per-slice bookkeeping (a
// voxel whose sum is NaN because the sinogram itself holds NaN is written as 0 too,
// where the reference would return NaN).
#include <cmath>
#include <type_traits>

#include "common.cuh"
#include "fan.cuh"

namespace mct {
namespace {

// Blocks of two warps: with 8 warps (32 x 8 columns) a small volume's 256 blocks left a third
// of the SMs half empty, and the warps of a block waited for each other at every chunk of
// views.  128x128x64 / 180 views, FDK: 284 -> 275 us; 333x333x101 / 500 views, curved 5.03 ->
// 4.72 ms; 512x512x256 / 1080 views 49.3 -> 46.6 ms; 256^3 / 360 views coronal, bf16 4.07 ms
// both (one warp: 4.19 ms there, the others as with two; four warps 278 us, 4.82, 47.7 ms).
constexpr int BP_TX = 8, BP_TY = 8, BP_ZC = 16, BP_VCHUNK = 256;
constexpr int BP_WX = 4;  // columns along x per warp (32 / BP_WX along y)
static_assert(BP_TX % BP_WX == 0 && BP_TY % (32 / BP_WX) == 0, "warps tile the block");
// Minimum resident blocks per SM, i.e. a register budget of 65536 / (64 * minb) per
// thread.  The axial kernel needs enough registers to issue all BP_ZC stencil gathers
// of a view before their arithmetic (that hides the gather latency): measured at
// 512x512x256 / 1080 views, float32 stencils run fastest with 128 registers (8
// blocks), bf16 stencils with 80 (12 blocks); 16-bit stencils of a curved detector spill
// there (512x512x128 / 360 views, FDK: 15.9 ms with 12 blocks, 8.4 with 8).  The general
// modes use 8, columns of 8 slices 10 (12 with 16-bit stencils).
template <int MODE, typename QT, bool CURVED, int ZC>
constexpr int bp_min_blocks() {
    if (ZC == 8 && (sizeof(QT) == 16 || CURVED)) return 10;
    return (MODE == 0 || MODE == 2) && sizeof(QT) == 8 && !CURVED ? 12 : 8;
}

struct BpParams {
    int nx, nz, nu, nv, views, cone, curved;
    // the kernel's index frame: a thread owns column (ix, iy) with ix in [0, nx), iy in
    // [0, ncb), and slices iz in [0, nsl) at vol[iz * ss + iy * sb + ix].  Axial: (iy, iz)
    // are the image's (i_y, i_z); coronal and sagittal: the image's (i_z, i_y), so that
    // the slice axis is the one along z and x, y stay fixed per column
    int ncb, nsl;
    int64_t sb, ss;
    int view_begin, views_total, accumulate;  // view-chunked FBP (scan index of view 0, scan size)
    float sid, sdd, img_rot;
    float u0, inv_ustep;   // uidx = (u - u0) * inv_ustep
    float v0, kv;          // vidx = (mag*z - v0) * kv, kv = sign(v_step)/dv
    float div;             // redundancy factor
    // voxel centre of (ix, iy, iz) of the kernel's frame = P + ix*EX + iy*EY + iz*EZ (rotated)
    float px_x, px_y, px_z;  // EX
    float py_x, py_y, py_z;  // EY
    float pz_x, pz_y, pz_z;  // EZ
    float o_x, o_y, o_z;     // P
};

// View j's entry of the tables: {cos b', sin b', weight, 0} with b' = b - img_rot and weight =
// delta-beta (run_mgfbp.py:1107-1111) x the redundancy factor x the float16 unscale.
__device__ __forceinline__ float4 view_entry(const BpParams& p, const float* __restrict__ angles, int j, float unscale) {
    const int jg = p.view_begin + j;  // scan index (angles is the whole scan's table)
    const int vt = p.views_total;
    float s, c;
    sincosf(angles[jg] - p.img_rot, &s, &c);
    const float db = (jg == vt - 1) ? fabsf(angles[vt - 1] - angles[0]) / (vt - 1) : fabsf(angles[jg + 1] - angles[jg]);
    return make_float4(c, s, db * p.div * unscale, 0.0f);
}

// Per-view table of a chunk of nvc views starting at jc.
__device__ __forceinline__ void fill_view_table(const BpParams& p, const float* __restrict__ angles, float4* tab,
                                                int jc, int nvc, int tid, int nthreads, float unscale) {
    for (int q = tid; q < nvc; q += nthreads) tab[q] = view_entry(p, angles, jc + q, unscale);
}

// MODE 0: cone beam in any view mode; flat or curved detector, no projection matrix
//         (u hoisted per column of the kernel's frame); MODE 2: the same for detectors of
//         more than 2^22 rows
// MODE 1: fan beam in the coronal or sagittal view mode (per-voxel u)
// MODE 3: projection matrix geometry in any view mode (per-column matrix rows)
template <int MODE, bool CONE, typename QT, typename PT, bool CURVED = false, int ZC = BP_ZC>
__global__ void __launch_bounds__(BP_TX* BP_TY, bp_min_blocks<MODE, QT, CURVED, ZC>())
fdk_bp_kernel(BpParams p, const float* __restrict__ angles, const float* __restrict__ pmat,
              const void* __restrict__ packed, float* __restrict__ vol, const uint32_t* __restrict__ f16_max) {
    // views per chunk of the shared tables; with projection matrices the chunk's 3x4
    // matrices are staged too (12 floats a view), in chunks of a quarter the size
    constexpr int VCH = MODE == 3 ? BP_VCHUNK / 4 : BP_VCHUNK;
    __shared__ float4 tab[VCH];  // {cos b, sin b, dbeta*div, unused}
    __shared__ __align__(16) float pms[MODE == 3 ? 12 * VCH : 4];
    const int tid = threadIdx.y * BP_TX + threadIdx.x;
    // A warp is 4 columns along x x 8 along y of the block's 8 x 8: for one view its
    // columns project onto fewer detector columns than a row of 32 (about 4|sin| + 8|cos|
    // + 1 against 32|sin| + 1), so each gather touches fewer L1 lines.  At 512x512x256 /
    // 1080 views: 52.19 -> 50.22 ms (float32), 49.07 -> 47.17 ms (bf16); warps of 16 x 2
    // 51.62 / 48.50, 8 x 4 50.78 / 47.70 (blocks of 32 x 8; in today's 8 x 8, 8 x 4 costs 1 %).
    const int warp = tid >> 5, lane = tid & 31;
    const int ix = blockIdx.x * BP_TX + (warp % (BP_TX / BP_WX)) * BP_WX + (lane % BP_WX);
    const int iy = blockIdx.y * BP_TY + (warp / (BP_TX / BP_WX)) * (32 / BP_WX) + lane / BP_WX;
    const int zb = blockIdx.z * ZC;
    const bool active = ix < p.nx && iy < p.ncb;
    const int nq = p.nu - 1;  // packed columns; packed rows per view: nv (cone: row nv-1 is NaN)

    // voxel centres of the ZC slices of this column: c_k = c0 + k * dc
    const float c0x = p.o_x + ix * p.px_x + iy * p.py_x + zb * p.pz_x;
    const float c0y = p.o_y + ix * p.px_y + iy * p.py_y + zb * p.pz_y;
    const float c0z = p.o_z + ix * p.px_z + iy * p.py_z + zb * p.pz_z;

    float acc[ZC];
#pragma unroll
    for (int k = 0; k < ZC; ++k) acc[k] = 0.0f;
    uint32_t dead = 0;  // bit k: slice zb+k projected off the detector in some view

    // float16 operands hold values scaled by 2^e: fold 2^-e (exact) into the view weight
    const float unscale = IsF16<QT>::value ? ldexpf(1.0f, -f16_scale_exp(*f16_max)) : 1.0f;
    for (int jc = 0; jc < p.views; jc += VCH) {
        const int nvc = min(VCH, p.views - jc);
        __syncthreads();
        fill_view_table(p, angles, tab, jc, nvc, tid, BP_TX * BP_TY, unscale);
        if (MODE == 3) {
            const float* src = pmat + 12 * (int64_t)(p.view_begin + jc);
            for (int q = tid; q < 12 * nvc; q += BP_TX * BP_TY) pms[q] = __ldg(src + q);
        }
        __syncthreads();
        if (!active || dead == 0xffffffffu) continue;

        if constexpr (MODE == 0 || MODE == 2) {
            // Cone beam: everything but the row is shared by the column's slices.  Views are
            // software-pipelined: the next view's geometry (a chain of about 35 dependent
            // instructions) is computed between the issue of this view's gathers and their
            // use, in one basic block: the reciprocal has no branch, and a column that leaves
            // the detector goes on with a clamped index to the end of its run of kViewRun
            // views.  512x512x256 / 1080 views, FDK: float32 53.7 -> 49.2 ms; 256^3 / 360
            // views coronal, bf16: 4.55 -> 4.08 ms; 333x333x101 / 500 views, curved 6.42 ->
            // 5.30 ms (float32 bit-identical; the bf16 volume moved by 2e-7, single voxels by up to
            // 8e-5 of the range).  L1 wavefronts bind now (82 % for float32).
            static_assert(CONE && ZC % 2 == 0, "cone-beam modes, slices in pairs");
            struct View {
                const char* base;  // the view's cell (row 0, column floor(u))
                float ru, w, vA, vB;  // column fraction, weight; row of slice k = vA + k vB
            };
            const float umax = (float)(p.nu - 1);
            bool off = false;
            auto geometry = [&](int q) {
                const float4 tb = tab[q];
                const float cb = tb.x, sb = tb.y;
                const float L = p.sid - c0x * cb - c0y * sb;
                const float t = -c0x * sb + c0y * cb;
                const float rL = reciprocal(L);  // for the magnification and the flat distance weight
                const float mag = p.sdd * rL;
                // products rounded on their own: a detector index that fuses them differs by an
                // ulp, and voxels at the detector's edge would change sides
                const float u = CURVED ? __fmul_rn(p.sdd, atan2f(t, L)) : __fmul_rn(mag, t);
                const float ui = (u - p.u0) * p.inv_ustep;
                off |= !(ui >= 0.0f && ui + 1.0f <= umax);  // NaN counts as off-detector
                const float uf = floorf(ui);
                const int uc = min(max((int)uf, 0), p.nu - 2);
                const float dw = CURVED ? 1.0f / (L * L + t * t) : rL * rL;
                View v;
                v.ru = ui - uf;
                v.w = (p.sid * dw) * tb.z;
                v.vA = (mag * c0z - p.v0) * p.kv;
                v.vB = (mag * p.pz_z) * p.kv;
                v.base = static_cast<const char*>(packed) + ((int64_t)(jc + q) * p.nv * nq + uc) * (int64_t)sizeof(QT);
                return v;
            };
            // rows outside [0, nv-2] (negative ones wrap around) read the NaN row nv-1
            const unsigned nan_row = (unsigned)(p.nv - 1);
            const uint32_t stride = (uint32_t)(nq * sizeof(QT));
            View cur = geometry(0);
            for (int q0 = 0; q0 < nvc && !off; q0 += kViewRun) {
                const int q1 = min(q0 + kViewRun, nvc);
                for (int q = q0; q < q1; ++q) {
                    const float2 ru2 = make_float2(cur.ru, cur.ru);
                    float2 lo[ZC], hi[ZC];
                    float rv[ZC];
                    auto load = [&](int k, unsigned row) {
                        Quad<QT>::load(reinterpret_cast<const QT*>(cur.base + (uint64_t)min(row, nan_row) * stride), lo[k],
                                       hi[k]);
                    };
                    // floor by adding M = 1.5 * 2^23 rounded down, on the FMA pipe: exact for
                    // rows below 2^22 (MODE 2: taller detectors, on the conversion unit); any
                    // other value leaves the difference to M's bits above nan_row.  float32
                    // takes slices in pairs (f32x2), 16 bits one by one: 49.2 / 49.4 ms and
                    // 4.14 / 4.08 ms at the sizes above.
                    const float M = 12582912.0f;
                    const unsigned MB = 0x4B400000u;  // M's bits
                    if constexpr (MODE == 2) {
#pragma unroll
                        for (int k = 0; k < ZC; ++k) {
                            const float vi = fmaf((float)k, cur.vB, cur.vA);
                            const float vf = floorf(vi);
                            rv[k] = vi - vf;
                            load(k, (unsigned)(int)vf);
                        }
                    } else if constexpr (sizeof(QT) == 16) {
                        const float2 vA2 = make_float2(cur.vA, cur.vA), vB2 = make_float2(cur.vB, cur.vB);
#pragma unroll
                        for (int k = 0; k < ZC; k += 2) {
                            const float2 vi = __ffma2_rn(make_float2((float)k, (float)(k + 1)), vB2, vA2);
                            const float2 m = __fadd2_rd(vi, make_float2(M, M));
                            const float2 fl = __fadd2_rn(m, make_float2(-M, -M));
                            const float2 f = __fadd2_rn(vi, make_float2(-fl.x, -fl.y));
                            rv[k] = f.x;
                            rv[k + 1] = f.y;
                            load(k, __float_as_uint(m.x) - MB);
                            load(k + 1, __float_as_uint(m.y) - MB);
                        }
                    } else {
#pragma unroll
                        for (int k = 0; k < ZC; ++k) {
                            const float vi = fmaf((float)k, cur.vB, cur.vA);
                            const float m = __fadd_rd(vi, M);
                            rv[k] = vi - (m - M);
                            load(k, __float_as_uint(m) - MB);
                        }
                    }
                    const View next = geometry(min(q + 1, nvc - 1));
                    const float w = cur.w;
#pragma unroll
                    for (int k = 0; k < ZC; ++k) {
                        const float2 s2 = __ffma2_rn(ru2, hi[k], lo[k]);
                        acc[k] = fmaf(w, fmaf(rv[k], s2.y, s2.x), acc[k]);
                    }
                    cur = next;
                }
            }
            if (off) dead = 0xffffffffu;
        } else for (int q = 0; q < nvc; ++q) {
            const int j = jc + q;
            const float4 tb = tab[q];
            const float cb = tb.x, sb = tb.y;
            if (MODE == 3) {
                // Projection matrices: in the kernel's frame x and y are fixed per column, so
                // the matrix rows are affine in the slice index and the distance weight does
                // not depend on z.  An untilted trajectory has no z term in the u and depth
                // rows (P2 = P10 = 0 up to rounding left by the matrix processing): when
                // 16 |B| < 2^-26 |A| for both, fmaf(k, B, A) rounds to A for every slice, so
                // u and the magnification are the column's (as in MODE 0) and taking them
                // once gives exactly the per-slice result.
                const float4* P = reinterpret_cast<const float4*>(pms + 12 * q);  // the view's matrix, staged
                const float4 r0 = P[0], r1 = P[1], r2 = P[2];
                const float P0 = r0.x, P1 = r0.y, P2 = r0.z, P3 = r0.w;
                const float P4 = r1.x, P5 = r1.y, P6 = r1.z, P7 = r1.w;
                const float P8 = r2.x, P9 = r2.y, P10 = r2.z, P11 = r2.w;
                const float dz = p.pz_z;
                const float Au = P0 * c0x + P1 * c0y + P2 * c0z + P3, Bu = P2 * dz;
                const float Av = P4 * c0x + P5 * c0y + P6 * c0z + P7, Bv = P6 * dz;
                const float Aw = P8 * c0x + P9 * c0y + P10 * c0z + P11, Bw = P10 * dz;
                const float L = p.sid - c0x * cb - c0y * sb;
                const float t = -c0x * sb + c0y * cb;
                const float dw = p.curved ? 1.0f / (L * L + t * t) : 1.0f / (L * L);
                const float w = (p.sid * dw) * tb.z;
                const unsigned nan_row = (unsigned)(p.nv - 1);  // rows outside [0, nv-2] read the NaN row
                const QT* view = reinterpret_cast<const QT*>(packed) + (int64_t)j * p.nv * nq;
                const float tiny = 0x1p-26f / (float)ZC;
                if (fabsf(Bu) <= tiny * fabsf(Au) && fabsf(Bw) <= tiny * fabsf(Aw)) {
                    const float mag = 1.0f / Aw;
                    const float ui = Au * mag;
                    if (!(ui >= 0.0f && ui + 1.0f <= (float)(p.nu - 1))) {  // NaN counts as off-detector
                        dead = 0xffffffffu;
                        break;
                    }
                    const float uf = floorf(ui);
                    const float ru = ui - uf;
                    const QT* base = view + (int)uf;
                    const float2 ru2 = make_float2(ru, ru);
#pragma unroll
                    for (int k = 0; k < ZC; ++k) {
                        const float vi = fmaf((float)k, Bv, Av) * mag;  // as in the per-slice branch
                        const float vf = floorf(vi);
                        const unsigned vr = min((unsigned)(int)vf, nan_row);
                        const float rv = vi - vf;
                        float2 lo, hi;
                        Quad<QT>::load(base + vr * (unsigned)nq, lo, hi);
                        const float2 s2 = __ffma2_rn(ru2, hi, lo);
                        acc[k] = fmaf(w, fmaf(rv, s2.y, s2.x), acc[k]);
                    }
                } else {
#pragma unroll
                    for (int k = 0; k < ZC; ++k) {
                        if ((dead >> k) & 1u) continue;
                        const float fk = (float)k;
                        const float mag = 1.0f / fmaf(fk, Bw, Aw);
                        const float ui = fmaf(fk, Bu, Au) * mag;
                        if (!(ui >= 0.0f && ui + 1.0f <= (float)(p.nu - 1))) {
                            dead |= 1u << k;
                            continue;
                        }
                        const float uf = floorf(ui);
                        const float ru = ui - uf;
                        const float vi = fmaf(fk, Bv, Av) * mag;
                        const float vf = floorf(vi);
                        const unsigned vr = min((unsigned)(int)vf, nan_row);
                        const float rv = vi - vf;
                        float2 lo, hi;
                        Quad<QT>::load(view + vr * (unsigned)nq + (int)uf, lo, hi);
                        const float2 s2 = __ffma2_rn(make_float2(ru, ru), hi, lo);
                        acc[k] = fmaf(w, fmaf(rv, s2.y, s2.x), acc[k]);
                    }
                }
            } else {
                // MODE 1 (fan beam, coronal or sagittal view mode): the voxel moves by
                // (pz_x, pz_y) per slice, so L and t are affine in k; slice k reads
                // detector row zb + k
                static_assert(MODE != 1 || !CONE, "cone beam takes MODE 0 or 3 in every view mode");
                const float L0 = p.sid - c0x * cb - c0y * sb, dL = -(p.pz_x * cb + p.pz_y * sb);
                const float t0 = -c0x * sb + c0y * cb, dt = -p.pz_x * sb + p.pz_y * cb;
#pragma unroll
                for (int k = 0; k < ZC; ++k) {
                    if (zb + k >= p.nsl || (dead >> k) & 1u) continue;
                    const float L = fmaf((float)k, dL, L0);
                    const float t = fmaf((float)k, dt, t0);
                    const float rL = 1.0f / L;  // one reciprocal for the magnification and the flat distance weight
                    const float mag = p.sdd * rL;
                    const float u = p.curved ? p.sdd * atan2f(t, L) : mag * t;
                    const float ui = (u - p.u0) * p.inv_ustep;
                    if (!(ui >= 0.0f && ui + 1.0f <= (float)(p.nu - 1))) {
                        dead |= 1u << k;
                        continue;
                    }
                    const float uf = floorf(ui);
                    const float ru = ui - uf;
                    const int uc = (int)uf;
                    const float dw = p.curved ? 1.0f / (L * L + t * t) : rL * rL;
                    const float w = (p.sid * dw) * tb.z;
                    const float2 pr = Pair<PT>::load(reinterpret_cast<const PT*>(packed) + ((int64_t)j * p.nv + zb + k) * nq + uc);
                    acc[k] = fmaf(w, fmaf(ru, pr.y, pr.x), acc[k]);
                }
            }
        }
    }
    if (!active) return;
    float* out = vol + (int64_t)zb * p.ss + (int64_t)iy * p.sb + ix;
#pragma unroll
    for (int k = 0; k < ZC; ++k) {
        if (zb + k < p.nsl) {
            const bool off_detector = ((dead >> k) & 1u) || acc[k] != acc[k];
            if (p.accumulate)  // a voxel off the detector in any chunk stays NaN until mct_fdk_bp_finish
                out[(int64_t)k * p.ss] = off_detector ? __int_as_float(0x7fffffff) : out[(int64_t)k * p.ss] + acc[k];
            else
                out[(int64_t)k * p.ss] = off_detector ? 0.0f : acc[k];
        }
    }
}

__global__ void nan_to_zero_kernel(int64_t n, float* __restrict__ v) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        if (v[i] != v[i]) v[i] = 0.0f;
}

// Axial fan beam (one detector row per slice, run_mgfbp.py:1183-1187).  With one slice
// every voxel x view update pays for its own geometry, so instructions bound it.  A thread
// takes one or two pairs of pixels above each other and every operation that allows it is one
// packed f32x2 instruction for the pair: position, reciprocal step, detector index, floor,
// weight.  The floor adds M = 1.5 * 2^23 rounded down, a column's smallest and largest index
// are kept instead of a test per view (a view that sees it off the detector has its index
// clamped and the column's result is discarded; a NaN index makes the sum NaN), and the
// table holds each cosine and sine twice, as operand pairs.
//
// A 2D image has few pixels, so the views of a column are split over FB_G threads: block
// (32 x-pixels, FB_G view groups) for 2 or 4 image rows and ZC slices (1 for a single slice,
// else 8), thread g taking views g, g + FB_G, ...  The group sums are added in a fixed order
// through shared memory (deterministic).
//
// 57.6 -> 19 instructions per update; now latency at half occupancy, issue 61 % and the packed
// operations' half of the FMA pipe (63 %) share the limit.  ms, one pixel a thread with scalar
// arithmetic / now: FBP 256^2 x 720 views 0.133 / 0.086; 1024^2 x 1440 views, bf16 2.65 / 1.21;
// helical, 140 slices of 512^2 x 720 views 48.9 / 24.1; 512^2 x 8, 720 views 1.14 / 0.67.
constexpr int FB_G = 8, FB_VCHUNK = 512;
// Pairs of rows per thread and views unrolled.  One slice, 1 pair x 2 / 1 x 4 / 2 x 2 / 2 x 3 /
// 4 x 1: helical FBP, 140 slices of 512^2 x 720 views 26.6 / 26.8 / 25.2 / 24.1 / 24.9 ms;
// 1024^2 x 1440 views, bf16 1.33 / 1.22 / 1.24 / 1.21 / 1.17 ms.  8 slices and curved detectors
// (two arc tangents a pair) take 1 x 2: 512^2 x 8, 720 views 0.668 ms against 0.747 with 2 x 3;
// curved 512^2 0.419 against 0.474.  (Left to itself the compiler
// takes 48 registers and spills: 256^2 0.092 ms against 0.086.)
template <int ZC, bool CURVED>
struct FanShape {
    static constexpr int R = ZC == 1 && !CURVED ? 2 : 1, U = ZC == 1 && !CURVED ? 3 : 2;
    static constexpr int B = ZC == 8 && !CURVED ? 3 : 2;  // blocks per SM, by the register budget
};
template <int ZC, bool CURVED, typename PT>
__global__ void __launch_bounds__(32 * FB_G, FanShape<ZC, CURVED>::B)
fdk_bp_fan_kernel(BpParams p, const float* __restrict__ angles, const void* __restrict__ packed,
                  float* __restrict__ vol, const uint32_t* __restrict__ f16_max) {
    constexpr int R = FanShape<ZC, CURVED>::R, NP = 2 * R;  // image rows of a block
    __shared__ float4 tab[FB_VCHUNK];   // {cos b, cos b, sin b, sin b}
    __shared__ float2 tabw[FB_VCHUNK];  // sid x weight, twice
    __shared__ float part[FB_G][NP][ZC][32];
    __shared__ int off_g[FB_G][NP][32];
    const int tx = threadIdx.x, g = threadIdx.y;
    const int ix = blockIdx.x * 32 + tx;
    const int iy0 = blockIdx.y * NP;
    const int zb = blockIdx.z * ZC;
    const int tid = g * 32 + tx;
    const bool active = ix < p.nx;
    const int nq = p.nu - 1;
    // pixel centres (x, y) of the pairs; rows below the image are computed and not stored
    float2 x2[R], y2[R], nx2[R], ny2[R];
#pragma unroll
    for (int r = 0; r < R; ++r) {
        float x[2], y[2];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int iy = iy0 + 2 * r + h;
            x[h] = p.o_x + ix * p.px_x + iy * p.py_x;
            y[h] = p.o_y + ix * p.px_y + iy * p.py_y;
        }
        x2[r] = make_float2(x[0], x[1]);
        y2[r] = make_float2(y[0], y[1]);
        nx2[r] = make_float2(-x[0], -x[1]);
        ny2[r] = make_float2(-y[0], -y[1]);
    }
    float2 acc[R][ZC], lo[R], hi[R];  // sums; smallest and largest index of the pair's pixels
#pragma unroll
    for (int r = 0; r < R; ++r) {
        lo[r] = make_float2(3.0e38f, 3.0e38f);
        hi[r] = make_float2(-3.0e38f, -3.0e38f);
#pragma unroll
        for (int k = 0; k < ZC; ++k) acc[r][k] = make_float2(0.0f, 0.0f);
    }
    const float unscale = IsF16<PT>::value ? ldexpf(1.0f, -f16_scale_exp(*f16_max)) : 1.0f;
    auto two = [](float a) { return make_float2(a, a); };
    const float M = 12582912.0f;
    const unsigned MB = 0x4B400000u;  // M's bits
    const unsigned last = (unsigned)(p.nu - 2);
    // the warp's pixels are inside the detector in every view: no test, no clamp
    bool in = true;
#pragma unroll
    for (int r = 0; r < R; ++r)
        in = in && fan_pair_inside<CURVED>(x2[r].x, y2[r].x, x2[r].y, y2[r].y, p.sid, p.sdd, p.u0, p.inv_ustep, p.nu);
    const bool inside = __all_sync(0xffffffffu, in);
    if (inside) {  // no index was recorded: any valid one
#pragma unroll
        for (int r = 0; r < R; ++r) lo[r] = hi[r] = make_float2(0.0f, 0.0f);
    }
    for (int jc = 0; jc < p.views; jc += FB_VCHUNK) {
        const int nvc = min(FB_VCHUNK, p.views - jc);
        bool angles_ok = true;  // an angle that is no finite number has NaN indices: its views are tested
        __syncthreads();
        for (int q = tid; q < nvc; q += 32 * FB_G) {
            const float4 e = view_entry(p, angles, jc + q, unscale);
            tab[q] = make_float4(e.x, e.x, e.y, e.y);
            tabw[q] = two(p.sid * e.z);
            angles_ok = angles_ok && fabsf(e.x) <= 1.0f && fabsf(e.y) <= 1.0f;
        }
        angles_ok = __syncthreads_and(angles_ok);
        if (!active) continue;
        auto views = [&](auto inside_tag) {
            constexpr bool kInside = decltype(inside_tag)::value;
            // with the column index taken from the bits of M + floor, M's bits are in the base
            const char* base = static_cast<const char*>(packed) + ((int64_t)(jc + g) * p.nv + zb) * nq * (int64_t)sizeof(PT) -
                               (kInside ? (int64_t)MB * (int64_t)sizeof(PT) : 0);
            const int64_t step = (int64_t)FB_G * p.nv * nq * (int64_t)sizeof(PT);
            constexpr int kViewUnroll = FanShape<ZC, CURVED>::U;
#pragma unroll kViewUnroll
            for (int q = g; q < nvc; q += FB_G, base += step) {
                const float4 tb = tab[q];
                const float2 cb = make_float2(tb.x, tb.y), sb = make_float2(tb.z, tb.w), sw = tabw[q];
#pragma unroll
                for (int r = 0; r < R; ++r) {
                    const float2 L = __ffma2_rn(ny2[r], sb, __ffma2_rn(nx2[r], cb, two(p.sid)));
                    const float2 t = __ffma2_rn(y2[r], cb, __fmul2_rn(nx2[r], sb));
                    const float2 rL = reciprocal2(L);
                    // u rounded on its own (an FMA with 0: a packed product would be fused with
                    // the subtraction below, and columns at the detector's edge change sides)
                    const float2 u = CURVED ? __ffma2_rn(two(p.sdd), make_float2(atan2f(t.x, L.x), atan2f(t.y, L.y)), two(0.0f))
                                            : __ffma2_rn(__fmul2_rn(two(p.sdd), rL), t, two(0.0f));
                    const float2 ui = __fmul2_rn(__fadd2_rn(u, two(-p.u0)), two(p.inv_ustep));
                    const float2 m = __fadd2_rd(ui, two(M));
                    const float2 uf = __fadd2_rn(m, two(-M));
                    const float2 ru = __fadd2_rn(ui, make_float2(-uf.x, -uf.y));
                    unsigned c0 = __float_as_uint(m.x), c1 = __float_as_uint(m.y);
                    if (!kInside) {
                        lo[r] = make_float2(fminf(lo[r].x, ui.x), fminf(lo[r].y, ui.y));
                        hi[r] = make_float2(fmaxf(hi[r].x, ui.x), fmaxf(hi[r].y, ui.y));
                        c0 = min(c0 - MB, last);
                        c1 = min(c1 - MB, last);
                    }
                    const float2 dw = CURVED ? reciprocal2(__ffma2_rn(L, L, __fmul2_rn(t, t))) : __fmul2_rn(rL, rL);
                    const float2 w = __fmul2_rn(dw, sw);
                    const char* b0 = base + (uint64_t)c0 * (uint32_t)sizeof(PT);
                    const char* b1 = base + (uint64_t)c1 * (uint32_t)sizeof(PT);
#pragma unroll
                    for (int k = 0; k < ZC; ++k) {
                        if (ZC == 1 || zb + k < p.nz) {
                            const float2 p0 = Pair<PT>::load(reinterpret_cast<const PT*>(b0) + (int64_t)k * nq);
                            const float2 p1 = Pair<PT>::load(reinterpret_cast<const PT*>(b1) + (int64_t)k * nq);
                            acc[r][k] = __ffma2_rn(w, make_float2(fmaf(ru.x, p0.y, p0.x), fmaf(ru.y, p1.y, p1.x)), acc[r][k]);
                        }
                    }
                }
            }
        };
        if (inside && angles_ok) views(std::true_type{});
        else views(std::false_type{});
    }
    const float umax = (float)(p.nu - 1);
    auto off = [&](float a, float b) { return !(a >= 0.0f && b + 1.0f <= umax); };
#pragma unroll
    for (int r = 0; r < R; ++r) {
        off_g[g][2 * r][tx] = off(lo[r].x, hi[r].x);
        off_g[g][2 * r + 1][tx] = off(lo[r].y, hi[r].y);
#pragma unroll
        for (int k = 0; k < ZC; ++k) {
            part[g][2 * r][k][tx] = acc[r][k].x;
            part[g][2 * r + 1][k][tx] = acc[r][k].y;
        }
    }
    __syncthreads();
    if (!active) return;
    // the groups share the block's rows and slices out among them
    const int groups = min(FB_G, p.views);  // groups beyond the number of views saw none
    for (int o = g; o < NP * ZC; o += FB_G) {
        const int row = o / ZC, k = o % ZC;
        if (iy0 + row >= p.nx || zb + k >= p.nz) continue;
        float sum = 0.0f;
        int any_off = 0;
        for (int h = 0; h < groups; ++h) {
            sum += part[h][row][k][tx];
            any_off |= off_g[h][row][tx];
        }
        const bool off_detector = any_off || sum != sum;
        float* out = vol + (int64_t)(zb + k) * p.nx * p.nx + (int64_t)(iy0 + row) * p.nx + ix;
        if (p.accumulate)  // a voxel off the detector in any chunk stays NaN until mct_fdk_bp_finish
            *out = off_detector ? __int_as_float(0x7fffffff) : *out + sum;
        else
            *out = off_detector ? 0.0f : sum;
    }
}

template <int ZC, bool CURVED>
void launch_bp_fan(const BpParams& p, const mct_geom* g, cudaStream_t s, const float* angles, const void* packed,
                   int dtype, float* vol, const uint32_t* f16_max) {
    constexpr int rows = 2 * FanShape<ZC, CURVED>::R;
    dim3 grid((g->nx + 31) / 32, (g->nx + rows - 1) / rows, (g->nz + ZC - 1) / ZC), block(32, FB_G);
    if (dtype == MCT_BF16)
        fdk_bp_fan_kernel<ZC, CURVED, uint32_t><<<grid, block, 0, s>>>(p, angles, packed, vol, nullptr);
    else if (dtype == MCT_F16)
        fdk_bp_fan_kernel<ZC, CURVED, h16x2><<<grid, block, 0, s>>>(p, angles, packed, vol, f16_max);
    else
        fdk_bp_fan_kernel<ZC, CURVED, float2><<<grid, block, 0, s>>>(p, angles, packed, vol, nullptr);
}

template <int MODE, bool CONE, bool CURVED = false, int ZC = BP_ZC>
void launch_bp(const BpParams& p, dim3 grid, dim3 block, cudaStream_t s, const float* angles, const float* pmat,
               const void* packed, int dtype, float* vol, const uint32_t* f16_max) {
    if (dtype == MCT_BF16)
        fdk_bp_kernel<MODE, CONE, uint2, uint32_t, CURVED, ZC><<<grid, block, 0, s>>>(p, angles, pmat, packed, vol, nullptr);
    else if (dtype == MCT_F16)
        fdk_bp_kernel<MODE, CONE, h16x4, h16x2, CURVED, ZC><<<grid, block, 0, s>>>(p, angles, pmat, packed, vol, f16_max);
    else
        fdk_bp_kernel<MODE, CONE, float4, float2, CURVED, ZC><<<grid, block, 0, s>>>(p, angles, pmat, packed, vol, nullptr);
}

}  // namespace
}  // namespace mct

using namespace mct;

extern "C" int mct_fdk_bp(const mct_geom* g, const mct_tables* t, const void* packed, int32_t dtype, float* vol,
                          void* stream) {
    MCT_TRY(check_geom(g, "mct_fdk_bp"));
    MCT_REQUIRE(t && t->angles && packed && vol, "mct_fdk_bp: NULL buffer");
    MCT_REQUIRE(dtype == MCT_F32 || dtype == MCT_BF16 || dtype == MCT_F16,
                "mct_fdk_bp: dtype must be MCT_F32, MCT_BF16 or MCT_F16");
    const bool cone = (g->flags & MCT_CONE) != 0;
    const bool pm = (g->flags & MCT_PMATRIX) != 0;
    MCT_REQUIRE(!pm || (cone && t->pmatrix), "mct_fdk_bp: projection matrices need cone beam and the table");
    MCT_REQUIRE(!cone || g->nv >= 2, "mct_fdk_bp: cone beam needs at least 2 detector rows");
    MCT_REQUIRE(cone || g->nz <= g->nv, "mct_fdk_bp: fan beam needs nz <= detector rows");
    MCT_REQUIRE(g->u_step != 0.0f, "mct_fdk_bp: zero detector spacing");
    MCT_REQUIRE((int64_t)g->nv * (g->nu - 1) < ((int64_t)1 << 31), "mct_fdk_bp: detector too large");
    BpParams p{};
    p.nx = g->nx; p.nz = g->nz; p.nu = g->nu; p.nv = g->nv; p.views = g->views;
    p.view_begin = g->view_begin;
    p.views_total = g->views_total > 0 ? g->views_total : g->views;
    p.accumulate = (g->flags & MCT_ACCUMULATE) != 0;
    p.cone = cone; p.curved = (g->flags & MCT_CURVED) != 0;
    p.sid = g->sid; p.sdd = g->sdd; p.img_rot = g->img_rot;
    p.u0 = g->u0; p.inv_ustep = (float)(1.0 / (double)g->u_step);
    p.v0 = g->v0;
    if (cone && !pm) {
        MCT_REQUIRE(g->v_step != 0.0f && g->dv != 0.0f, "mct_fdk_bp: zero row spacing");
        p.kv = (float)((g->v_step > 0 ? 1.0 : -1.0) / (double)g->dv);
    }
    p.div = (float)div_factor(*g);
    // voxel coordinates, run_mgfbp.py:1090-1104, as an affine map of (ix, iy, iz)
    const double nx = g->nx, nz = g->nz, px = g->px, pz = g->pz;
    const double cr = std::cos((double)g->img_rot), sr = std::sin((double)g->img_rot);
    double ax[3] = {0, 0, 0}, ay[3] = {0, 0, 0}, az[3] = {0, 0, 0}, a0[3] = {0, 0, 0};  // (xa, ya, z) per unit index
    if (g->view_mode == 1) {
        ax[0] = px; a0[0] = -px * (nx - 1) / 2.0 + g->cx;
        ay[1] = -px; a0[1] = px * (nx - 1) / 2.0 + g->cy;
        az[2] = pz; a0[2] = -(nz - 1) / 2.0 * pz + g->cz;
    } else if (g->view_mode == 2) {
        ax[0] = px; a0[0] = -px * (nx - 1) / 2.0 + g->cx;
        ay[2] = -px; a0[2] = px * (nx - 1) / 2.0 + g->cz;
        az[1] = -pz; a0[1] = (nz - 1) / 2.0 * pz + g->cy;
    } else {
        ay[2] = -px; a0[2] = px * (nx - 1) / 2.0 + g->cz;
        ax[1] = -px; a0[1] = px * (nx - 1) / 2.0 + g->cy;
        az[0] = pz; a0[0] = -(nz - 1) / 2.0 * pz + g->cx;
    }
    auto rot = [&](const double* a, float& x, float& y, float& z) {
        x = (float)(a[0] * cr + a[1] * sr);
        y = (float)(-a[0] * sr + a[1] * cr);
        z = (float)a[2];
    };
    // The kernel's frame.  In the coronal and sagittal view modes the image's i_y axis is
    // the one along z and its i_x, i_z axes lie in the (x, y) plane, so with cone beam the
    // kernel takes (i_x, i_z) as the column and i_y as the slice axis: x and y are then
    // fixed per column, as in the axial mode, and the same hoisted kernels apply (u, the
    // weight and the truncation test once per column and view, v affine in the slice).
    const int64_t plane = (int64_t)g->nx * g->nx;
    const bool permuted = cone && g->view_mode != 1;
    rot(ax, p.px_x, p.px_y, p.px_z);
    rot(permuted ? az : ay, p.py_x, p.py_y, p.py_z);
    rot(permuted ? ay : az, p.pz_x, p.pz_y, p.pz_z);
    rot(a0, p.o_x, p.o_y, p.o_z);
    p.ncb = permuted ? g->nz : g->nx;
    p.nsl = permuted ? g->nx : g->nz;
    p.sb = permuted ? plane : g->nx;
    p.ss = permuted ? g->nx : plane;
    dim3 block(BP_TX, BP_TY);
    dim3 grid((g->nx + BP_TX - 1) / BP_TX, (p.ncb + BP_TY - 1) / BP_TY, (p.nsl + BP_ZC - 1) / BP_ZC);
    const bool slices8 = cone && !pm && g->nv <= (1 << 22) &&
                         columns_of_8((int64_t)grid.x * grid.y * grid.z, p.nsl, p.curved);
    if (slices8) grid.z = (unsigned)((p.nsl + 7) / 8);
    MCT_REQUIRE(grid.y <= 65535 && grid.z <= 65535, "mct_fdk_bp: volume too large for the launch grid");
    cudaStream_t s = as_stream(stream);
    const uint32_t* fm = dtype == MCT_F16 ? f16_trailer(g, packed) : nullptr;
    if (pm) launch_bp<3, true>(p, grid, block, s, t->angles, t->pmatrix, packed, dtype, vol, fm);
    else if (cone && g->nv > (1 << 22) && p.curved)
        launch_bp<2, true, true>(p, grid, block, s, t->angles, nullptr, packed, dtype, vol, fm);
    else if (cone && g->nv > (1 << 22))
        launch_bp<2, true>(p, grid, block, s, t->angles, nullptr, packed, dtype, vol, fm);
    else if (slices8 && p.curved)
        launch_bp<0, true, true, 8>(p, grid, block, s, t->angles, nullptr, packed, dtype, vol, fm);
    else if (slices8) launch_bp<0, true, false, 8>(p, grid, block, s, t->angles, nullptr, packed, dtype, vol, fm);
    else if (cone && p.curved) launch_bp<0, true, true>(p, grid, block, s, t->angles, nullptr, packed, dtype, vol, fm);
    else if (cone) launch_bp<0, true>(p, grid, block, s, t->angles, nullptr, packed, dtype, vol, fm);
    else if (g->view_mode == 1 && g->nu <= (1 << 22)) {  // column indices exact in the float floor
        MCT_REQUIRE(g->nx <= 65535, "mct_fdk_bp: fan beam images are at most 65535 pixels wide");
        if (g->nz == 1 && p.curved) launch_bp_fan<1, true>(p, g, s, t->angles, packed, dtype, vol, fm);
        else if (g->nz == 1) launch_bp_fan<1, false>(p, g, s, t->angles, packed, dtype, vol, fm);
        else if (p.curved) launch_bp_fan<8, true>(p, g, s, t->angles, packed, dtype, vol, fm);
        else launch_bp_fan<8, false>(p, g, s, t->angles, packed, dtype, vol, fm);
    }
    else launch_bp<1, false>(p, grid, block, s, t->angles, nullptr, packed, dtype, vol, fm);
    return launched("fdk_bp_kernel");
}

extern "C" int mct_fdk_bp_finish(const mct_geom* g, float* vol, void* stream) {
    MCT_REQUIRE(g && vol && g->nx >= 1 && g->nz >= 1, "mct_fdk_bp_finish: bad arguments");
    const int64_t n = (int64_t)g->nz * g->nx * g->nx;
    const int64_t blocks = (n + 255) / 256;
    nan_to_zero_kernel<<<(int)(blocks < 152 * 32 ? blocks : 152 * 32), 256, 0, as_stream(stream)>>>(n, vol);
    return launched("nan_to_zero_kernel");
}
