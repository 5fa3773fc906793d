// Thresholds and small helpers shared by the compositing kernels and the index kernels.
#pragma once

#include "common.cuh"

namespace splatad {

constexpr float kAlphaMax = 0.999f;
constexpr float kAlphaMin = 1.f / 255.f;
constexpr float kTStop = 1e-4f;

// Exactly fmodf((a - b + 180), 360) - 180 with the reference's final fix-up, but without the
// fmodf call whenever |a - b + 180| stays within one turn of [0, 360).
__device__ __forceinline__ float angle_difference(float a, float b) {
    const float x = a - b + 180.f;
    float r;
    if (fabsf(x) < 360.f) r = x;
    else if (x >= 360.f && x < 720.f) r = x - 360.f;
    else r = fmodf(x, 360.f);
    const float d = r - 180.f;
    return d < -180.f ? d + 360.f : d;
}

// Whether a Gaussian can reach alpha >= 1/255 at a sample whose offset from its (possibly shifted) mean
// lies in a box: alpha = min(0.999, opacity * exp(-sigma)) < 1/255 needs sigma > ln(255 * opacity), and
// sigma(dx, dy) = 0.5 (a dx^2 + c dy^2) + b dx dy is bounded from below over the box. For a positive
// definite conic the minimum is zero when the box holds the centre; otherwise it lies on an edge that
// faces the centre - at the minimiser the way to the centre leaves the box - and there are at most two
// of those, each a clamped 1-D parabola. Decided with a margin far above the float32 rounding of either
// side; anything doubtful (a conic that is not positive definite, NaNs) may reach every sample. Skipping
// what cannot reach a sample changes nothing there.
struct BoxTest {
    float a, b, c, slope_x, slope_y, s_max;
    bool never, always;
    __device__ __forceinline__ BoxTest(float a_, float b_, float c_, float opacity) : a(a_), b(b_), c(c_) {
        never = opacity * 1.0001f < kAlphaMin;             // exp(-sigma) <= 1 wherever sigma >= 0
        always = !(a > 1e-20f && c > 1e-20f && a * c - b * b > 0.f);
        s_max = __logf(255.f * opacity) * 1.001f + 1e-3f;
        slope_x = __fdividef(-b, c);                       // minimiser over dy on an edge dx = X: slope_x * X
        slope_y = __fdividef(-b, a);
    }
    // The least sigma in a box of numbers, of a positive definite conic, but for rounding.
    __device__ __forceinline__ float nearest(float dx_lo, float dx_hi, float dy_lo, float dy_hi) const {
        const float X = fminf(fmaxf(0.f, dx_lo), dx_hi), Y = fminf(fmaxf(0.f, dy_lo), dy_hi);
        const float y = fminf(fmaxf(slope_x * X, dy_lo), dy_hi);
        const float x = fminf(fmaxf(slope_y * Y, dx_lo), dx_hi);
        const float s_x = 0.5f * (a * X * X + c * y * y) + b * X * y;
        const float s_y = 0.5f * (a * x * x + c * Y * Y) + b * x * Y;
        return fminf(s_x, s_y);
    }
    // It less a margin; -INF where there is no telling.
    __device__ __forceinline__ float lowest(float dx_lo, float dx_hi, float dy_lo, float dy_hi) const {
        if (always || !(dx_lo <= dx_hi && dy_lo <= dy_hi)) return -INFINITY;   // NaN offsets
        return nearest(dx_lo, dx_hi, dy_lo, dy_hi) * 0.999f - 1e-3f;
    }
    __device__ __forceinline__ bool misses(float dx_lo, float dx_hi, float dy_lo, float dy_hi) const {
        if (never) return true;
        if (always || !(dx_lo <= dx_hi && dy_lo <= dy_hi)) return false;   // NaN offsets
        return nearest(dx_lo, dx_hi, dy_lo, dy_hi) * 0.999f - 1e-3f > s_max;
    }
};

// 1 / x of two values in [1 - kAlphaMax, 1]: one Newton-Raphson step on the hardware's approximation (which is off
// by up to one unit in the last place) gives the correctly rounded quotient for every float in that range
// (splatad_debug_check_reciprocals compares all 83.7 million of them) at half the instructions of a division.
__device__ __forceinline__ float2 reciprocal_pair(float2 x) {
    float2 r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r.x) : "f"(x.x));
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r.y) : "f"(x.y));
    return __ffma2_rn(r, __ffma2_rn(make_float2(-x.x, -x.y), r, make_float2(1.f, 1.f)), r);
}

struct TileRange { int32_t start, end; };

__device__ __forceinline__ TileRange tile_range(const int32_t *__restrict__ offsets, uint32_t tile,
                                                uint32_t n_tiles_total, int64_t n_isects) {
    TileRange r;
    r.start = offsets[tile];
    // n_isects < 0: the caller's offsets carry one more entry, the total, written on the device
    r.end = (tile + 1 == n_tiles_total && n_isects >= 0) ? (int32_t)n_isects : offsets[tile + 1];
    return r;
}

} // namespace splatad
