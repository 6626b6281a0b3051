// Conservative FP32 rejection of far pairs in the broad phases. Positions are
// taken relative to a point of their instance and rounded to FP32; a pair is
// called far only when a direction separates its two hulls by more than `lim`
// (the support-function bound, which holds for every direction: the one tried
// joins the pair's approximately closest points, by the usual clamped solution of
// their two linear equations). Callers add kFarMargin times
// the instance's extent to lim, well above the rounding of the coordinates
// (1e-7 of it) and of the products (1e-6), so that no pair that the FP64 tests
// accept is rejected. NaN and degenerate pairs are never called far.
#pragma once
#include "common.cuh"

namespace idp {

constexpr float kFarMargin = 4e-6f;

__device__ __forceinline__ F3 ldf(const float4* __restrict__ p, int v) {
    const float4 a = __ldg(p + v);
    return {a.x, a.y, a.z};
}

// hull of a (na points) against hull of b, relative to a common origin, along n
__device__ __forceinline__ bool separated(F3 n, float hi_a, float lo_b, float lim) {
    const float nn = sqn(n), gap = lo_b - hi_a;
    return gap > 0.0f && gap * gap > lim * lim * nn;
}

// point p against triangle (a, b, c)
__device__ __forceinline__ bool far_point_triangle(F3 p, F3 a, F3 b, F3 c, float lim) {
    const F3 ab = b - a, ac = c - a, ap = p - a;
    // approximately closest point a + s ab + t ac
    const float d1 = dot(ab, ap), d2 = dot(ac, ap), aa = sqn(ab), bb = dot(ab, ac), cc = sqn(ac);
    const float det = aa * cc - bb * bb;
    if (!(det > 1e-7f * aa * cc)) return false;
    float s = (cc * d1 - bb * d2) / det, t = (aa * d2 - bb * d1) / det;
    if (!(s >= 0.0f && t >= 0.0f && s + t <= 1.0f)) {
        // outside: the nearest of the three edges
        const float s0 = fminf(fmaxf(d1 / aa, 0.0f), 1.0f), t0 = fminf(fmaxf(d2 / cc, 0.0f), 1.0f);
        const F3 bc = c - b, bp = p - b;
        const float w = fminf(fmaxf(dot(bc, bp) / sqn(bc), 0.0f), 1.0f);
        const float q0 = sqn(ap - s0 * ab), q1 = sqn(ap - t0 * ac), q2 = sqn(bp - w * bc);
        if (q0 <= q1 && q0 <= q2) { s = s0; t = 0.0f; }
        else if (q1 <= q2) { s = 0.0f; t = t0; }
        else { s = 1.0f - w; t = w; }
    }
    const F3 n = ap - (s * ab + t * ac);  // from the triangle to the point
    return separated(n, fmaxf(0.0f, fmaxf(dot(n, ab), dot(n, ac))), dot(n, ap), lim);
}

// segment (a0, a1) against segment (b0, b1)
__device__ __forceinline__ bool far_segments(F3 a0, F3 a1, F3 b0, F3 b1, float lim) {
    const F3 u = a1 - a0, v = b1 - b0, r = a0 - b0;
    const float a = sqn(u), e = sqn(v), f = dot(v, r), c = dot(u, r), b = dot(u, v);
    const float den = a * e - b * b;
    if (!(a > 0.0f && e > 0.0f)) return false;
    float s = den > 1e-6f * a * e ? fminf(fmaxf((b * f - c * e) / den, 0.0f), 1.0f) : 0.0f;
    float t = (b * s + f) / e;
    t = fminf(fmaxf(t, 0.0f), 1.0f);
    s = fminf(fmaxf((b * t - c) / a, 0.0f), 1.0f);
    const F3 n = (r + s * u) - t * v;  // from b to a
    const float na = dot(n, r);
    return separated(n, fmaxf(0.0f, dot(n, v)), fminf(na, na + dot(n, u)), lim);
}

}  // namespace idp
