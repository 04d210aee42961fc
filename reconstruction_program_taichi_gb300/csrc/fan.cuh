// Which fan-beam pixels need no detector test (fdk_bp_fan_kernel), also compiled for the host
// (the tests check the rule there).
#pragma once
#include <cmath>

#define MCT_HD __host__ __device__ __forceinline__

namespace mct {
namespace {

// Scans whose index computation cannot overflow or lose a column to rounding, so that the rule
// below can hold: positive, finite distances and a detector whose indices float32 holds to
// 2^-8.  For others every pixel is tested.
MCT_HD bool fan_scan_bounded(float sid, float sdd, float u0, float inv_ustep, int nu) {
    const float big = 1e15f;  // products of any three stay finite
    return sid >= 1.0f / big && sid <= big && fabsf(sdd) <= big && fabsf(u0) <= big && fabsf(inv_ustep) <= big && nu <= 65536;
}

// A pixel at distance rho from the axis is seen at most asin(rho / sid) off the central ray:
// whether that stays a column inside the detector for both pixels of a pair, so that in every
// view floor(index) lies in [0, nu - 2].  The column is for rounding, which the distance to the
// source, at least 0.05 sid, amplifies to at most half of one.
template <bool CURVED>
MCT_HD bool fan_pair_inside(float xa, float ya, float xb, float yb, float sid, float sdd, float u0, float inv_ustep,
                            int nu) {
    const float inv_sid = 1.0f / sid;
    const float ax = xa * inv_sid, ay = ya * inv_sid, bx = xb * inv_sid, by = yb * inv_sid;
    const float a2 = ax * ax + ay * ay, b2 = bx * bx + by * by, q2 = fmaxf(a2, b2);  // (rho / sid)^2
    const float reach = CURVED ? sdd * asinf(sqrtf(q2)) : sdd * sqrtf(q2 / (1.0f - q2));
    const float i0 = (-reach - u0) * inv_ustep, i1 = (reach - u0) * inv_ustep;
    return fan_scan_bounded(sid, sdd, u0, inv_ustep, nu) && a2 <= 0.9f && b2 <= 0.9f && fminf(i0, i1) >= 1.0f &&
           fmaxf(i0, i1) <= (float)(nu - 3);
}

}  // namespace
}  // namespace mct
