// Front-to-back alpha compositing of the depth-sorted per-tile Gaussian lists, to camera
// pixels (rasterize_to_pixels) and to lidar points (rasterize_to_points), forward and
// backward. FP32 on the CUDA cores; there is no dense contraction in this path.
//
// A camera warp draws a patch of a tile by itself; a lidar CTA works on one patch with all its warps, or on one for each of
// them. Either walks the tile's list in batches staged into shared memory, and stops as soon as every sample is
// saturated. An entry is staged only if it can reach alpha >= 1/255 somewhere in one of the patches (an exact,
// conservative bound of the quadratic form over the patch's box) and looked at only by the warps it
// can reach: the bounding rectangles behind the tile lists are loose. The backward pass starts at the
// last list position any of the patch's samples consumed instead of the end of the list.
//
// Semantics follow the reference kernels
//   pixels fwd  gsplat/cuda/csrc/rasterization.cu:1360-1518     bwd 2833-3089
//   points fwd  gsplat/cuda/csrc/rasterization.cu:2021-2219     bwd 3728-4054
//   angle wrap  gsplat/cuda/csrc/utils.cuh:552-555
// Thresholds kept: alpha cap 0.999, alpha < 1/255 skipped, sigma < 0 skipped, a pixel stops
// (exclusively) when T*(1-alpha) <= 1e-4, median depth where T crosses 0.5, points with
// range <= 0 are not rendered.
#include <type_traits>

#include "common.cuh"
#include "composite_common.cuh"

namespace splatad {

// Infinities and NaNs become zeros.
__device__ __forceinline__ float finite_or_zero(float v) { return fabsf(v) < INFINITY ? v : 0.f; }
__device__ __forceinline__ float4 finite_or_zero(float4 v) {
    return make_float4(finite_or_zero(v.x), finite_or_zero(v.y), finite_or_zero(v.z), finite_or_zero(v.w));
}

// Copies row g of a [*, n] float table to dst (one thread per row), zero-padded to a multiple of
// four floats: 16-byte loads when the rows are 16-byte aligned.
template <bool kFinite = false>
__device__ __forceinline__ void stage_row(float *__restrict__ dst, const float *__restrict__ table,
                                          size_t g, uint32_t n, bool vec) {
    const float *src = table + g * n;
    if (vec) {
        for (uint32_t k = 0; k < n; k += 4) {
            const float4 v = __ldg(reinterpret_cast<const float4 *>(src + k));
            *reinterpret_cast<float4 *>(dst + k) = kFinite ? finite_or_zero(v) : v;
        }
    } else if (kFinite) {
        for (uint32_t k = 0; k < n; k += 4)
            *reinterpret_cast<float4 *>(dst + k) = finite_or_zero(make_float4(
                __ldg(src + k), k + 1 < n ? __ldg(src + k + 1) : 0.f, k + 2 < n ? __ldg(src + k + 2) : 0.f, k + 3 < n ? __ldg(src + k + 3) : 0.f));
    } else {
        const uint32_t npad = (n + 3u) & ~3u;
        for (uint32_t k = 0; k < npad; ++k) dst[k] = k < n ? __ldg(src + k) : 0.f;
    }
}

// acc += row * w over a staged row of exactly CDIM floats (zero behind the channels in use).
template <int CDIM>
__device__ __forceinline__ void axpy_staged_full(float (&acc)[CDIM], const float *__restrict__ row, float w) {
    const float4 *r4 = reinterpret_cast<const float4 *>(row);
    const float2 w2 = make_float2(w, w);
#pragma unroll
    for (int k4 = 0; k4 < CDIM / 4; ++k4) {
        const float4 v = r4[k4];
        // two channels per instruction: the packed multiply-add rounds each half like fmaf does
        const float2 lo = __ffma2_rn(make_float2(v.x, v.y), w2, make_float2(acc[4 * k4 + 0], acc[4 * k4 + 1]));
        const float2 hi = __ffma2_rn(make_float2(v.z, v.w), w2, make_float2(acc[4 * k4 + 2], acc[4 * k4 + 3]));
        acc[4 * k4 + 0] = lo.x; acc[4 * k4 + 1] = lo.y;
        acc[4 * k4 + 2] = hi.x; acc[4 * k4 + 3] = hi.y;
    }
}

// ---------------------------------------------------------------------------------------
// Camera tiles. A lane draws PX pixels next to each other in a row, so that everything that depends on
// the Gaussian and the row alone is worked out once per lane, and the per-pixel arithmetic runs on
// pairs of pixels (packed FP32: two results per issued instruction). A warp covers a compact patch of
// the tile - 8 x 8 pixels of a 16 x 16 tile with PX = 2, 16 x 8 with PX = 4, all of it with PX = 8.
// ---------------------------------------------------------------------------------------
constexpr float kExpectedMin = 1e-10f;   // alphas below it do not divide (gsplat/rendering.py:423-430)
constexpr float kLog2E = 1.4426950408889634f, kLn2 = 0.6931471805599453f;

template <int PX>
struct TilePixels {
    uint32_t x, y;   // of the thread's first pixel, within the tile
};

// threads of a CTA: whole rows of ceil(tile_size / PX) threads, rounded up to whole warps by the caller
template <int PX>
__host__ __device__ inline uint32_t tile_threads(uint32_t tile_size) {
    return tile_size * ((tile_size + PX - 1) / PX);
}

template <int PX>
__device__ __forceinline__ TilePixels<PX> tile_pixels(uint32_t tile_size, uint32_t tr) {
    TilePixels<PX> p;
    if (PX == 2 && tile_size == 16u) {   // 8 x 8 patches
        const uint32_t w = tr >> 5, l = tr & 31u;
        p.x = (w & 1u) * 8u + (l & 3u) * 2u;
        p.y = (w >> 1) * 8u + (l >> 2);
    } else {
        const uint32_t per_row = (tile_size + PX - 1) / PX;
        p.y = tr / per_row;
        p.x = (tr - p.y * per_row) * PX;
    }
    return p;
}

// Pixel centres of a warp's patch.
struct PatchBox { float x0, x1, y0, y1; };

// The box of the calling warp's patch, in every lane; an empty patch gets an empty box (nothing is visible in it).
__device__ __forceinline__ PatchBox warp_box(float px, float py, uint32_t n_inside) {
    PatchBox b = {3.0e38f, -3.0e38f, 3.0e38f, -3.0e38f};
    if (n_inside) b = {px, px + (float)(n_inside - 1), py, py};
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
        b.x0 = fminf(b.x0, __shfl_xor_sync(0xffffffffu, b.x0, off));
        b.x1 = fmaxf(b.x1, __shfl_xor_sync(0xffffffffu, b.x1, off));
        b.y0 = fminf(b.y0, __shfl_xor_sync(0xffffffffu, b.y0, off));
        b.y1 = fmaxf(b.y1, __shfl_xor_sync(0xffffffffu, b.y1, off));
    }
    return b;
}

// A list entry as its staging lane sees it.
struct PixelEntry {
    float4 A, B;       // mean, its velocity | conic, opacity
};

__device__ __forceinline__ PixelEntry load_pixel_entry(int32_t g, const float2 *__restrict__ means2d,
                                                       const float *__restrict__ conics,
                                                       const float *__restrict__ opacities,
                                                       const float2 *__restrict__ pix_vels) {
    PixelEntry e;
    const float2 xy = __ldg(means2d + g), v = __ldg(pix_vels + g);
    e.A = make_float4(xy.x, xy.y, v.x, v.y);
    e.B = make_float4(__ldg(conics + 3 * (size_t)g), __ldg(conics + 3 * (size_t)g + 1),
                      __ldg(conics + 3 * (size_t)g + 2), __ldg(opacities + g));
    return e;
}

constexpr uint32_t kSeenEntry = 1u, kCarefulEntry = 2u, kOddEntry = 4u, kFullEntry = 8u;

// What a warp has to know about an entry: whether it can reach the warp's patch (kSeenEntry; 0: it need not look at it),
// whether its alphas need looking at one by one (kCarefulEntry: a sigma that could come out negative, an alpha above the
// cap), and whether it is one for odd_pixels_fwd() (kOddEntry). The alphas of the others need no test but the one
// against 1/255: with ac - b^2 >= 1e-5 ac the form a dx^2 + 2 b dx dy + c dy^2 is at least 5e-6 (a dx^2 + c dy^2), ten times
// what its rounding can take away, and an opacity within the cap keeps every alpha there. The mean moves with the
// row's shutter time; roll_lo / roll_hi bound it over the tile.
template <bool kMarkOdd>
__device__ __forceinline__ uint32_t patch_sees(const PixelEntry &e, const PatchBox &box, float roll_lo, float roll_hi) {
    const BoxTest test(e.B.x, e.B.y, e.B.z, e.B.w);
    if (test.never) return 0u;
    const float mx_a = e.A.x + roll_lo * e.A.z, mx_b = e.A.x + roll_hi * e.A.z;
    const float my_a = e.A.y + roll_lo * e.A.w, my_b = e.A.y + roll_hi * e.A.w;
    const float mx_lo = fminf(mx_a, mx_b), mx_hi = fmaxf(mx_a, mx_b);
    const float my_lo = fminf(my_a, my_b), my_hi = fmaxf(my_a, my_b);
    uint32_t seen = 0u;
    if (kMarkOdd) {   // a NaN somewhere, an opacity without bound, a conic too flat or too steep
        const bool plain = fabsf(e.B.x) > 1e-30f && fabsf(e.B.x) + fabsf(e.B.y) + fabsf(e.B.z) < 1e30f;
        if (!plain || !(mx_lo <= mx_hi) || !(my_lo <= my_hi) || !(test.s_max < 1e30f)) seen = kOddEntry;
    }
    const float ac = e.B.x * e.B.z;
    const bool sized = e.B.x > 1e-15f && e.B.z > 1e-15f && e.B.x < 1e15f && e.B.z < 1e15f;   // nothing under- or overflows
    if (!(sized && ac - e.B.y * e.B.y >= 1e-5f * ac && e.B.w <= kAlphaMax)) seen |= kCarefulEntry;
    if (box.x0 <= box.x1 && !test.misses(mx_lo - box.x1, mx_hi - box.x0, my_lo - box.y1, my_hi - box.y0)) seen |= kSeenEntry;
    else seen &= kOddEntry;
    return seen;
}

// The same, and whether every pixel of the patch blends the entry and needs no other care (kFullEntry): sigma is convex, so that the
// corners of the box bound it from above, and with ac - b^2 >= 0.05 ac its terms are at most forty times itself, which leaves their
// rounding a tenth of the margin. `most` bounds the alphas in the patch, by the least sigma where that holds, else by the opacity. (One
// function for both, the other kernels are 1 % slower; the bounds in one of their own, these are 3 %.)
template <bool kMarkOdd>
__device__ __forceinline__ uint32_t patch_covered(const PixelEntry &e, const PatchBox &box, float roll_lo, float roll_hi, float &most) {
    const BoxTest test(e.B.x, e.B.y, e.B.z, e.B.w);
    if (test.never) return 0u;
    const float mx_a = e.A.x + roll_lo * e.A.z, mx_b = e.A.x + roll_hi * e.A.z;
    const float my_a = e.A.y + roll_lo * e.A.w, my_b = e.A.y + roll_hi * e.A.w;
    const float mx_lo = fminf(mx_a, mx_b), mx_hi = fmaxf(mx_a, mx_b);
    const float my_lo = fminf(my_a, my_b), my_hi = fmaxf(my_a, my_b);
    uint32_t seen = 0u;
    if (kMarkOdd) {   // a NaN somewhere, an opacity without bound, a conic too flat or too steep
        const bool plain = fabsf(e.B.x) > 1e-30f && fabsf(e.B.x) + fabsf(e.B.y) + fabsf(e.B.z) < 1e30f;
        if (!plain || !(mx_lo <= mx_hi) || !(my_lo <= my_hi) || !(test.s_max < 1e30f)) seen = kOddEntry;
    }
    const float ac = e.B.x * e.B.z, det = ac - e.B.y * e.B.y;
    const bool sized = e.B.x > 1e-15f && e.B.z > 1e-15f && e.B.x < 1e15f && e.B.z < 1e15f;   // nothing under- or overflows
    if (!(sized && det >= 1e-5f * ac && e.B.w <= kAlphaMax)) seen |= kCarefulEntry;
    const float x0 = mx_lo - box.x1, x1 = mx_hi - box.x0, y0 = my_lo - box.y1, y1 = my_hi - box.y0;
    const float lowest = test.lowest(x0, x1, y0, y1);
    if (!(box.x0 <= box.x1) || lowest > test.s_max) return seen & kOddEntry;
    most = fminf(kAlphaMax, det >= 0.05f * ac ? e.B.w * __expf(-lowest) : e.B.w);
    const float xx = 0.5f * e.B.x * fmaxf(x0 * x0, x1 * x1), yy = 0.5f * e.B.z * fmaxf(y0 * y0, y1 * y1);
    const float xy = fmaxf(fmaxf(e.B.y * x0 * y0, e.B.y * x0 * y1), fmaxf(e.B.y * x1 * y0, e.B.y * x1 * y1));
    if (seen == 0u && det >= 0.05f * ac && xx + yy + xy <= __logf(255.f * e.B.w) * 0.999f - 4e-3f) seen = kFullEntry;
    return seen | kSeenEntry;
}

// The staged form: exp(-sigma) = 2^(a dx^2 + b dx dy + c dy^2) with the conic scaled once per entry.
__device__ __forceinline__ float4 scaled_conic(float4 B) {
    return make_float4(-0.5f * kLog2E * B.x, -kLog2E * B.y, -0.5f * kLog2E * B.z, B.w);
}

__device__ __forceinline__ float exp2_approx(float x) {
    float r;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}

__device__ __forceinline__ float lg2_approx(float x) {
    float r;
    asm("lg2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}

// The lane of a one-warp block, in a register that stays: read from its special register inside a loop it takes twenty cycles.
__device__ __forceinline__ uint32_t lane_index() {
    uint32_t lane;
    asm volatile("mov.u32 %0, %%tid.x;" : "=r"(lane));
    return lane;
}

// exponents of a pair of pixels in one row: dx of the two, the row's b * dy and c * dy * dy
__device__ __forceinline__ float2 pair_power(float a, float2 dx, float bdy, float cdy2) {
    const float2 t = __ffma2_rn(make_float2(a, a), dx, make_float2(bdy, bdy));
    return __ffma2_rn(t, dx, make_float2(cdy2, cdy2));
}

// ---------------------------------------------------------------------------------------
// Values that are not finite. The kernels below let every pixel of a warp take every entry that one of them
// blends, with weight zero where it is not blended - and zero times an infinity is a NaN. A pixel that comes out
// with one is worked out again by itself, and its last id marked: the backward kernel leaves the tiles that hold
// a mark, or a cotangent that is not finite, to a pass in which a pixel takes nothing from an entry that it does
// not blend. A NaN in an entry's geometry or opacity makes its alpha the largest there is wherever sigma is not
// negative; the kernels' comparisons drop it, and theirs is also a conic so flat that it reaches the column a pixel
// moves to when it stops (see kPixelGone): a warp that meets such an entry works all of its pixels out again.
// Both out of line and from nothing but the kernels' own arguments, so that the kernels hold nothing for
// them. What no pixel of a backward patch blends must not reach it either: there a value that is not finite becomes zero when
// its row is staged (13 channels 673 -> 676 us, 32 channels 1862 -> 1869; a vote for every entry costs 1 to 4 %, careful entries
// that leave the loop 3 %).
// ---------------------------------------------------------------------------------------
constexpr int32_t kOddPixel = INT32_MIN;   // in a last id: the pixel blended something that is not finite

__device__ __forceinline__ int32_t last_position(int32_t last_id) { return last_id & INT32_MAX; }

struct PixelTask {
    uint32_t C, W, H, tile_size, tile_w, tile_h, channels;
    int64_t n_isects;
    const float2 *means2d, *pix_vels;
    const float *conics, *opacities, *colors, *rs_time, *backgrounds;
    const int32_t *offsets, *flatten_ids;
};

// Where a pixel of the calling thread lies; `pix` is its place in the images.
struct TaskPixel {
    bool inside;
    float x, y, roll;
    size_t pix;
    const float *bg;
};

template <int PX>
__device__ __forceinline__ TaskPixel task_pixel(const PixelTask &a, uint32_t gtile, uint32_t tr, uint32_t k) {
    const uint32_t per_cam = a.tile_w * a.tile_h, cam = gtile / per_cam, tile = gtile - cam * per_cam;
    const uint32_t ty = tile / a.tile_w, tx = tile - ty * a.tile_w;
    const TilePixels<PX> tp = tile_pixels<PX>(a.tile_size, tr);
    const uint32_t i = ty * a.tile_size + tp.y, j = tx * a.tile_size + tp.x + k;
    TaskPixel p;
    p.inside = tp.y < a.tile_size && tp.x + k < a.tile_size && i < a.H && j < a.W;
    p.x = (float)j + 0.5f;
    p.y = (float)i + 0.5f;
    p.roll = a.rs_time[cam] * ((p.y - 0.5f) / (float)(a.H - 1) - 0.5f);
    p.pix = ((size_t)cam * a.H + i) * a.W + j;
    p.bg = a.backgrounds ? a.backgrounds + (size_t)cam * a.channels : nullptr;
    return p;
}

struct PixelAlpha {
    float4 B;              // scaled conic, opacity
    float dx, dy, vis, alpha;
    bool blends;
};

__device__ __forceinline__ PixelAlpha pixel_alpha(const PixelTask &a, int32_t g, const TaskPixel &p) {
    const PixelEntry e = load_pixel_entry(g, a.means2d, a.conics, a.opacities, a.pix_vels);
    PixelAlpha r;
    r.B = scaled_conic(e.B);
    r.dx = e.A.x + p.roll * e.A.z - p.x;
    r.dy = e.A.y + p.roll * e.A.w - p.y;
    const float power = fmaf(fmaf(r.B.x, r.dx, r.B.y * r.dy), r.dx, r.B.z * r.dy * r.dy);
    r.vis = exp2_approx(power);
    r.alpha = r.B.w * r.vis;
    r.blends = !(power > 0.f) && !(r.alpha < kAlphaMin);   // a NaN is blended, with the capped alpha
    return r;
}

template <int PX>
__device__ __noinline__ void odd_pixels_fwd(const PixelTask &a, uint32_t gtile, uint32_t tr, float *colors_out, float *alphas, int32_t *last_ids, bool expected,
                                            float *expected_depths) {
    const TileRange range = tile_range(a.offsets, gtile, a.C * a.tile_w * a.tile_h, a.n_isects);
    for (uint32_t h = 0; h < (uint32_t)PX; ++h) {
        const TaskPixel p = task_pixel<PX>(a, gtile, tr, h);
        if (!p.inside) continue;
        float *color = colors_out + p.pix * a.channels, T = 1.f;
        int32_t pos = 0;
        for (uint32_t k = 0; k < a.channels; ++k) color[k] = 0.f;
        for (int32_t idx = range.start; idx < range.end; ++idx) {
            const int32_t g = a.flatten_ids[idx];
            const PixelAlpha e = pixel_alpha(a, g, p);
            if (!e.blends) continue;
            const float alpha = fminf(kAlphaMax, e.alpha), next_T = T * (1.f - alpha), vis = alpha * T;
            if (next_T <= kTStop) break;
            for (uint32_t k = 0; k < a.channels; ++k) color[k] = fmaf(a.colors[(size_t)g * a.channels + k], vis, color[k]);
            pos = idx;
            T = next_T;
        }
        alphas[p.pix] = 1.f - T;
        last_ids[p.pix] = pos | kOddPixel;
        for (uint32_t k = 0; p.bg != nullptr && k < a.channels; ++k) color[k] += T * p.bg[k];
        if (expected) color[a.channels - 1] /= fmaxf(1.f - T, kExpectedMin);
        if (expected_depths != nullptr) expected_depths[p.pix] = color[a.channels - 1];
    }
}

struct PixelGrads {
    const float *alphas, *v_colors_in, *v_alphas, *expected;
    const int32_t *last_ids;
    float *means2d, *means2d_abs, *conics, *colors, *opacities, *pix_vels;
};

__device__ __forceinline__ void add_warp_total(float *to, float v) {
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
    if ((threadIdx.x & 31u) == 0u && v != 0.f) atomicAdd(to, v);
}

// By whole warps.
template <int PX>
__device__ __noinline__ void odd_pixels_bwd(const PixelTask &a, uint32_t gtile, uint32_t tr, const PixelGrads &grad) {
    const TileRange range = tile_range(a.offsets, gtile, a.C * a.tile_w * a.tile_h, a.n_isects);
    const uint32_t n = a.channels;
    for (uint32_t h = 0; h < (uint32_t)PX; ++h) {
        const TaskPixel p = task_pixel<PX>(a, gtile, tr, h);
        const int32_t last = p.inside ? min(range.end - 1, last_position(grad.last_ids[p.pix])) : -1;
        const float *v_out = grad.v_colors_in + p.pix * n;
        float T = 1.f, behind = 0.f, divisor = 1.f;
        if (last >= 0) {
            const float alpha = grad.alphas[p.pix];
            float v_a = grad.v_alphas[p.pix], bg_dot = 0.f;
            T = 1.f - alpha;
            if (grad.expected != nullptr) {
                divisor = fmaxf(alpha, kExpectedMin);
                if (alpha >= kExpectedMin) v_a -= v_out[n - 1] * grad.expected[p.pix] / divisor;
            }
            for (uint32_t k = 0; p.bg != nullptr && k < n; ++k) bg_dot += p.bg[k] * (k + 1 == n ? v_out[k] / divisor : v_out[k]);
            behind = -T * (v_a - bg_dot);
        }
        for (int32_t idx = __reduce_max_sync(0xffffffffu, last); idx >= range.start; --idx) {
            const size_t g = (size_t)a.flatten_ids[idx];
            const PixelAlpha e = pixel_alpha(a, (int32_t)g, p);
            const bool ok = e.blends && idx <= last;
            if (!__any_sync(0xffffffffu, ok)) continue;
            float fac = 0.f, v_alpha = 0.f;
            if (ok) {
                const float alpha = fminf(kAlphaMax, e.alpha), ra = 1.f / (1.f - alpha);
                T *= ra;
                fac = alpha * T;
                float dot = 0.f;
                for (uint32_t k = 0; k < n; ++k) dot = fmaf(a.colors[g * n + k], k + 1 == n ? v_out[k] / divisor : v_out[k], dot);
                v_alpha = fmaf(T, dot, -ra * behind);
                behind = fmaf(fac, dot, behind);
            }
            for (uint32_t k = 0; k < n; ++k)
                add_warp_total(grad.colors + g * n + k, ok ? fac * (k + 1 == n ? v_out[k] / divisor : v_out[k]) : 0.f);
            // a capped alpha passes no gradient on to the geometry
            float v = 0.f, wx = 0.f, wy = 0.f, q0 = 0.f, q1 = 0.f, q2 = 0.f, vx = 0.f, vy = 0.f;
            if (ok && e.alpha <= kAlphaMax) {
                v = e.vis * v_alpha;
                const float w = -e.B.w * v;   // dL/dsigma
                q0 = 0.5f * w * e.dx * e.dx;
                q1 = w * e.dx * e.dy;
                q2 = 0.5f * w * e.dy * e.dy;
                wx = kLn2 * e.B.w * v * (2.f * e.B.x * e.dx + e.B.y * e.dy);
                wy = kLn2 * e.B.w * v * (e.B.y * e.dx + 2.f * e.B.z * e.dy);
                vx = wx * p.roll;
                vy = wy * p.roll;
            }
            add_warp_total(grad.conics + 3 * g, q0);
            add_warp_total(grad.conics + 3 * g + 1, q1);
            add_warp_total(grad.conics + 3 * g + 2, q2);
            add_warp_total(grad.means2d + 2 * g, wx);
            add_warp_total(grad.means2d + 2 * g + 1, wy);
            add_warp_total(grad.pix_vels + 2 * g, vx);
            add_warp_total(grad.pix_vels + 2 * g + 1, vy);
            add_warp_total(grad.opacities + g, v);
            if (grad.means2d_abs != nullptr) {
                add_warp_total(grad.means2d_abs + 2 * g, fabsf(wx));
                add_warp_total(grad.means2d_abs + 2 * g + 1, fabsf(wy));
            }
        }
    }
}

// A row of n floats to shared memory, zeros behind them: all loads are on their way before the first is waited for.
template <int CDIM, bool kFinite = false>
__device__ __forceinline__ void stage_whole_row(float4 *dst, const float *__restrict__ src, uint32_t n, bool vec) {
#pragma unroll
    for (int k = 0; k < CDIM; k += 4) {
        float4 w = make_float4(0.f, 0.f, 0.f, 0.f);
        if (vec) {
            if ((uint32_t)k < n) w = __ldg(reinterpret_cast<const float4 *>(src + k));
        } else {
            if ((uint32_t)k < n) w.x = __ldg(src + k);
            if ((uint32_t)k + 1u < n) w.y = __ldg(src + k + 1);
            if ((uint32_t)k + 2u < n) w.z = __ldg(src + k + 2);
            if ((uint32_t)k + 3u < n) w.w = __ldg(src + k + 3);
        }
        dst[k / 4] = kFinite ? finite_or_zero(w) : w;
    }
}

__device__ __forceinline__ void async_copy(float *dst_smem, const float *src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(smem_addr(dst_smem)), "l"(__cvta_generic_to_global(src)) : "memory");
}
__device__ __forceinline__ void async_copy_16(float *dst_smem, const float *src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 16;" ::"r"(smem_addr(dst_smem)), "l"(__cvta_generic_to_global(src)) : "memory");
}
__device__ __forceinline__ void async_copy_row(float *dst_smem, const float *__restrict__ src, uint32_t n, bool vec) {
    if (vec)
        for (uint32_t k = 0; k < n; k += 4) async_copy_16(dst_smem + k, src + k);
    else
        for (uint32_t k = 0; k < n; ++k) async_copy(dst_smem + k, src + k);
}
__device__ __forceinline__ void async_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// Rows of n floats, whole 16-byte pieces, between a table and a warp's shared memory, where row r lies at r * CDIM: lane r
// names the table's row for it, `mask` the rows that are wanted. The lanes go over the rows' pieces in
// sequence, so that one access touches a few lines; a lane that copies a row by itself touches as many lines
// with every access as there are lanes. Copies to shared memory are asynchronous: none waits for the one before. Forward kernel, a lane
// per row, rows together, rows together and asynchronous: 1920 x 1080, 32 channels 727, 543, 506 us, 20 channels 396, 408, 377; 640 x 360 and 20
// channels 111 and 91 (together, asynchronous). One float at a time, of rows that are no multiple of 16 bytes, 13 channels: 297 -> 334, 25: 617 -> 643; the
// backward kernel has no registers for it (20 channels, two pixels: 950 -> 1128).
template <int CDIM, bool kStore>
__device__ __forceinline__ void copy_rows(float *rows, std::conditional_t<kStore, float, const float> *table, int32_t row_id,
                                          uint32_t mask, uint32_t n, uint32_t lane) {
    const uint32_t pieces = n / 4u, skip = 32u / pieces, rest = 32u - skip * pieces;
    uint32_t r = lane / pieces, k = lane - r * pieces;
    for (uint32_t round = 0; round < pieces; ++round) {
        const size_t id = (size_t)__shfl_sync(0xffffffffu, row_id, r);
        if ((mask >> r) & 1u) {
            auto *there = table + id * n + 4u * k;
            float *here = rows + r * CDIM + 4u * k;
            if constexpr (kStore) *reinterpret_cast<float4 *>(there) = *reinterpret_cast<const float4 *>(here);
            else async_copy_16(here, there);
        }
        r += skip;
        k += rest;
        if (k >= pieces) { k -= pieces; ++r; }
    }
}

template <int CDIM>
__device__ __forceinline__ void stage_rows(float *rows, const float *table, int32_t row_id, uint32_t mask, uint32_t n, uint32_t lane) {
    copy_rows<CDIM, false>(rows, table, row_id, mask, n, lane);
    async_wait_all();
}

// The values of a thread's PX pixels, next to each other in memory: in 16-byte pieces where they lie so. One float at a
// time every lane of a warp touches a line of its own, and 32 such loads are what 8 of these are (backward
// kernel of the 1920 x 1080 benchmark: 335 -> 312 us).
template <int M>
__device__ __forceinline__ bool in_pieces(const void *p) { return M % 4 == 0 && (reinterpret_cast<uintptr_t>(p) & 15u) == 0u; }

template <int M, typename T>
__device__ __forceinline__ void load_pieces(T (&v)[M], const T *src) {
    static_assert(sizeof(T) == 4, "");
#pragma unroll
    for (int k = 0; k + 4 <= M; k += 4) {
        const int4 w = __ldg(reinterpret_cast<const int4 *>(src + k));
        v[k] = reinterpret_cast<const T &>(w.x); v[k + 1] = reinterpret_cast<const T &>(w.y);
        v[k + 2] = reinterpret_cast<const T &>(w.z); v[k + 3] = reinterpret_cast<const T &>(w.w);
    }
}

template <int M, typename T>
__device__ __forceinline__ void store_pieces(T *dst, const T (&v)[M]) {
    static_assert(sizeof(T) == 4, "");
#pragma unroll
    for (int k = 0; k + 4 <= M; k += 4)
        *reinterpret_cast<int4 *>(dst + k) = make_int4(reinterpret_cast<const int &>(v[k]), reinterpret_cast<const int &>(v[k + 1]),
                                                       reinterpret_cast<const int &>(v[k + 2]), reinterpret_cast<const int &>(v[k + 3]));
}

// One value of each of a thread's pixels; `outside` beyond the image.
template <int PX, typename T>
__device__ __forceinline__ void load_pixels(T (&v)[PX], const T *src, uint32_t n_inside, T outside) {
    if (n_inside == (uint32_t)PX && in_pieces<PX>(src)) load_pieces<PX>(v, src);
    else
#pragma unroll
        for (int k = 0; k < PX; ++k) v[k] = (uint32_t)k < n_inside ? src[k] : outside;
}

template <int PX, typename T>
__device__ __forceinline__ void store_pixels(T *dst, const T (&v)[PX], uint32_t n_inside) {
    if (n_inside == (uint32_t)PX && in_pieces<PX>(dst)) store_pieces<PX>(dst, v);
    else
#pragma unroll
        for (int k = 0; k < PX; ++k)
            if ((uint32_t)k < n_inside) dst[k] = v[k];
}

// The channels of a thread's pixels, zeros behind those there are.
template <int CDIM, int PX, int N>
__device__ __forceinline__ bool load_whole_channels(float (&v)[PX][CDIM], const float *src, uint32_t channels) {
    if (channels != (uint32_t)N || !in_pieces<PX * N>(src)) return false;
    float flat[PX * N];
    load_pieces<PX * N>(flat, src);
#pragma unroll
    for (int k = 0; k < PX; ++k)
#pragma unroll
        for (int c = 0; c < CDIM; ++c) v[k][c] = c < N ? flat[k * N + (c < N ? c : 0)] : 0.f;
    return true;
}

template <int CDIM, int PX>
__device__ __forceinline__ void load_channels(float (&v)[PX][CDIM], const float *src, uint32_t channels, uint32_t n_inside) {
    if constexpr (CDIM == 4)
        if (n_inside == (uint32_t)PX &&
            (load_whole_channels<CDIM, PX, 4>(v, src, channels) || load_whole_channels<CDIM, PX, 3>(v, src, channels))) return;
#pragma unroll
    for (int k = 0; k < PX; ++k)
#pragma unroll
        for (int c = 0; c < CDIM; ++c) v[k][c] = (uint32_t)k < n_inside && (uint32_t)c < channels ? src[k * channels + c] : 0.f;
}

template <int CDIM, int PX, int N>
__device__ __forceinline__ bool store_whole_channels(float *dst, const float (&v)[PX][CDIM], uint32_t channels) {
    if (channels != (uint32_t)N || !in_pieces<PX * N>(dst)) return false;
    float flat[PX * N];
#pragma unroll
    for (int k = 0; k < PX; ++k)
#pragma unroll
        for (int c = 0; c < N; ++c) flat[k * N + c] = v[k][c];
    store_pieces<PX * N>(dst, flat);
    return true;
}

template <int CDIM, int PX>
__device__ __forceinline__ void store_channels(float *dst, const float (&v)[PX][CDIM], uint32_t channels, uint32_t n_inside) {
    if constexpr (CDIM == 4)
        if (n_inside == (uint32_t)PX &&
            (store_whole_channels<CDIM, PX, 4>(dst, v, channels) || store_whole_channels<CDIM, PX, 3>(dst, v, channels))) return;
#pragma unroll
    for (int k = 0; k < PX; ++k)
#pragma unroll
        for (int c = 0; c < CDIM; ++c)
            if ((uint32_t)k < n_inside && (uint32_t)c < channels) dst[k * channels + c] = v[k][c];
}

// ---------------------------------------------------------------------------------------
// Camera forward. A warp draws a patch by itself: PX pixels of a row per lane, 16 x 16 pixels of a tile with eight, 16 x 8
// with four, 8 x 8 with two; no barrier and no other warp's list position concerns it.
//
// What bounds it is instruction issue and, as more pixels share a lane, the FP32 pipe. What an entry costs whatever
// the number of pixels - loads, bits, the row's terms, the stop test - was a third of the work at two pixels, and
// where Gaussians are larger than tiles (62 of 64 pixels of an 8 x 8 patch blend an entry that is looked at in the benchmark scenes) there is nothing
// to gain from small patches. So: eight pixels; alphas tested against 1/255 only, unless the entry was marked
// (patch_sees()); no instruction spent on a sign; the transmittance updated in place by one multiply-add, which rounds once.
// A pixel that has stopped moves its column out to where every alpha vanishes; a warp leaves when all of its have.
// 1920 x 1080, 4 channels: 201 M -> 104 M warp instructions, 222 -> 147 us (two pixels 208, four 156); 16 channels, 1237 x 719:
// 180 -> 152 (1920 x 1080: 8, 13, 20 and 32 channels 303, 360, 432, 662 -> 214, 297, 377, 506; 640 x 360, two pixels: 4, 13, 20 and 32 channels 64, 84, 87, 105 -> 62, 88, 91, 101). Staging every value twice for the packed operands: 12 us slower; asynchronous copies of the next batches: 9.
// ---------------------------------------------------------------------------------------
constexpr float kPixelGone = 1e18f;   // a column no Gaussian reaches: sigma overflows, alpha is 0 (or NaN, never drawn)

// log2 of 1.01 kTStop: where the bound of the transmittances comes that low they are looked at. The bound may be off by 2e-3 of the 1.4e-2 that this
// leaves: some 2340 entries of 1/255 fit between two looks, each off by 2^-22 of lg2.approx and half of an ulp of 1 - alpha, 7e-4 in all; their sums, five additions
// a batch and one over the batches of numbers up to 14, 5e-4; and the transmittances' own product, 2e-4.
constexpr float kLowBound = -13.2733571f;

// registers per thread, by measurement (4 channels, eight pixels: 147 us at 128 registers, 163 at 112 and 96, with runs 130 at 96 (20 warps an SM), 145
// at 104 to 128 (16), 135 at 80 (24, spills); 8 channels, four
// pixels: 218 at 96, 243 at 112 and 128; 20 channels: 426 at 96, 445 at 112 and 160)
constexpr int pixels_fwd_regs(int cdim, int px, bool runs) {
    return runs ? 96 : cdim <= 4 ? (px == 8 ? 128 : px == 4 ? 80 : 64) : cdim <= 8 ? (px == 4 ? 96 : 72) : cdim <= 16 ? (px == 4 ? 128 : 96) : cdim <= 20 ? 96 : 128;
}

// kRuns: for scenes of large Gaussians, where most entries that are looked at cover their patch (84 % in the camera benchmark, 98 % in
// its rigs). Those go through in runs that test nothing: every pixel blends them, the last of a run is noted once a batch, and no
// transmittance can come below the limit before a bound of them all does - the sum of the entries' least logarithms, one scan a
// batch -, which it reaches with one entry in 15 to 45. Such an entry, one that does not cover the patch and one that needs care are
// looked at one by one. What bounds it then is the FP32 pipe, at 75 % of its rate within a run, and the batches. 1920 x 1080, 27 tiles per
// Gaussian 104 M -> 82 M warp instructions, 145 -> 130 us, 54 tiles 119 -> 95, six cameras 584 -> 445. Where few entries cover their patch it
// is slower by up to half: see covers_patches(). (Entries two by two: 5 % slower, for the registers; the next batch's entries loaded ahead: no change.)
//
// kTogether: rows in 16-byte pieces, staged by copy_rows(). A kernel of its own: with both ways in one, 1920 x 1080 and 32 channels
// take 648 us instead of 506.
template <int CDIM, int PX, bool kTogether, bool kRuns>
__global__ void __maxnreg__(pixels_fwd_regs(CDIM, PX, kRuns)) rasterize_to_pixels_fwd_kernel(
    uint32_t C, int64_t n_isects, const float2 *__restrict__ means2d,
    const float *__restrict__ conics, const float *__restrict__ colors, uint32_t channels,
    const float *__restrict__ opacities, const float2 *__restrict__ pix_vels,
    const float *__restrict__ rs_time, const float *__restrict__ backgrounds, uint32_t W,
    uint32_t H, uint32_t tile_size, uint32_t tile_w, uint32_t tile_h, uint32_t patches /* of a tile */,
    const int32_t *__restrict__ offsets, const int32_t *__restrict__ flatten_ids,
    float *__restrict__ render_colors, float *__restrict__ render_alphas,
    int32_t *__restrict__ last_ids, uint32_t expected /* divide the last channel by the alpha */,
    float *__restrict__ expected_depths /* optional: and keep it for the backward pass */) {
    chain_enter();
    static_assert(PX % 2 == 0, "pixels are handled in pairs");
    constexpr int P2 = PX / 2;
    __shared__ float4 sA[32];                // x, y, vx, vy
    __shared__ float4 sB[32];                // scaled conic, minus the opacity
    __shared__ float4 sCol[32 * CDIM / 4];   // zeros behind the channels
    const bool vec = (channels % 4u == 0u) && ((reinterpret_cast<uintptr_t>(colors) & 15u) == 0u);

    const uint32_t tiles_per_cam = tile_w * tile_h;
    const uint32_t gtile = blockIdx.x / patches, cam = gtile / tiles_per_cam;
    const uint32_t tile = gtile - cam * tiles_per_cam;
    const uint32_t ty = tile / tile_w, tx = tile - ty * tile_w;
    uint32_t lane = threadIdx.x;
    if constexpr (kRuns) lane = lane_index();
    const uint32_t tr = (blockIdx.x - gtile * patches) * 32u + lane;
    const TilePixels<PX> tp = tile_pixels<PX>(tile_size, tr);
    const uint32_t i = ty * tile_size + tp.y, j = tx * tile_size + tp.x;
    uint32_t n_inside = 0;   // pixels of this thread inside the tile and the image
    if (tp.y < tile_size && i < H && j < W) n_inside = min(min((uint32_t)PX, tile_size - tp.x), W - j);
    const float px0 = (float)j + 0.5f, py = (float)i + 0.5f;
    const float rs = rs_time[cam];
    const float roll = rs * ((py - 0.5f) / (float)(H - 1) - 0.5f);
    // shutter times of the tile's first and last row
    const float roll_a = rs * ((float)(ty * tile_size) / (float)(H - 1) - 0.5f);
    const float roll_b = rs * ((float)(min((ty + 1) * tile_size, H) - 1) / (float)(H - 1) - 0.5f);
    const float roll_lo = fminf(roll_a, roll_b), roll_hi = fmaxf(roll_a, roll_b);
    const PatchBox box = warp_box(px0, py, n_inside);

    const TileRange range = tile_range(offsets, gtile, C * tiles_per_cam, n_isects);

    float2 npx[P2], T[P2], out[CDIM][P2];   // minus the columns; transmittances; minus the colours, by channel
    int32_t pos[PX];                        // list position of the last entry blended
#pragma unroll
    for (int q = 0; q < P2; ++q) {
        npx[q] = make_float2(n_inside > 2u * q ? -(px0 + (float)(2 * q)) : -kPixelGone,
                             n_inside > 2u * q + 1u ? -(px0 + (float)(2 * q + 1)) : -kPixelGone);
        T[q] = make_float2(1.f, 1.f);
#pragma unroll
        for (int c = 0; c < CDIM; ++c) out[c][q] = make_float2(0.f, 0.f);
    }
#pragma unroll
    for (int k = 0; k < PX; ++k) pos[k] = 0;
    if (kTogether)
        for (uint32_t k = channels; k < (uint32_t)CDIM; ++k) reinterpret_cast<float *>(sCol)[lane * CDIM + k] = 0.f;
    uint32_t odd = 0u;   // kOddEntry: the warp was to blend one
    bool done = __all_sync(0xffffffffu, n_inside == 0);

    int32_t next_id = 0;
    if (range.start + (int32_t)lane < range.end) next_id = flatten_ids[range.start + lane];
    if constexpr (kRuns) {
        float bound = 0.f;   // log2 of a transmittance that no pixel that still blends is below, the same in every lane
        constexpr int kEntry = 2 + CDIM / 4;
        __shared__ float4 sEntry[32 * kEntry];   // x, y, vx, vy | scaled conic, minus the opacity | channels, zeros behind them
        __shared__ float sT[PX][32];        // transmittances of the pixels that have stopped
        __shared__ int32_t sLast[PX][32];   // list positions of the last entries blended
        __shared__ int32_t sIdx[32];        // list positions
        int32_t *sl = &sLast[0][lane];      // 32 apart for the lane's pixels
#pragma unroll
        for (int k = 0; k < PX; ++k) sl[32 * k] = 0;
        for (int32_t start = range.start; start < range.end && !done; start += 32) {
            const int32_t idx = start + (int32_t)lane;
            const int32_t g = next_id;
            uint32_t seen = 0u;
            float most = 0.f;
            PixelEntry e;
            if (idx < range.end) {
                e = load_pixel_entry(g, means2d, conics, opacities, pix_vels);
                if (idx + 32 < range.end) next_id = flatten_ids[idx + 32];   // on its way meanwhile
                seen = patch_covered<true>(e, box, roll_lo, roll_hi, most);
            }
            // The entries to be looked at move up to the front; n of them, bit t of the masks for the one in place t
            const uint32_t kept = __ballot_sync(0xffffffffu, seen != 0u), n = __popc(kept);
            const uint32_t place = __popc(kept & ((1u << lane) - 1u));
            const uint32_t full = __reduce_or_sync(0xffffffffu, (seen & kFullEntry) ? 1u << place : 0u);
            const uint32_t careful = __reduce_or_sync(0xffffffffu, (seen & (kCarefulEntry | kOddEntry)) ? 1u << place : 0u);
            odd |= seen & kOddEntry;
            // what the entries up to this lane's leave of a transmittance, at least
            float left = seen ? lg2_approx(1.f - most) : 0.f;
#pragma unroll
            for (int off = 1; off < 32; off <<= 1) {
                const float o = __shfl_up_sync(0xffffffffu, left, off);
                if ((int)lane >= off) left += o;
            }
            __syncwarp();   // the batch before has been read
            if (seen) {
                float4 *entry = sEntry + place * kEntry;
                entry[0] = e.A;
                entry[1] = scaled_conic(make_float4(e.B.x, e.B.y, e.B.z, -e.B.w));
                sIdx[place] = idx;
                stage_whole_row<CDIM>(entry + 2, colors + (size_t)g * channels, channels, CDIM < 20 && vec);
            }
            __syncwarp();
            // minus the alphas of entry t
            const auto evaluate = [&](uint32_t t, float2 (&w)[P2]) {
                const float4 A = sEntry[t * kEntry], B = sEntry[t * kEntry + 1];
                const float mx = A.x + roll * A.z, dy = A.y + roll * A.w - py;
                const float bdy = B.y * dy, cdy2 = B.z * dy * dy;
#pragma unroll
                for (int q = 0; q < P2; ++q) {
                    const float2 pw = pair_power(B.x, __fadd2_rn(make_float2(mx, mx), npx[q]), bdy, cdy2);
                    w[q] = __fmul2_rn(make_float2(B.w, B.w), make_float2(exp2_approx(pw.x), exp2_approx(pw.y)));
                }
            };
            const auto drop_small = [&](float2 (&w)[P2]) {
#pragma unroll
                for (int q = 0; q < P2; ++q) w[q] = make_float2(w[q].x <= -kAlphaMin ? w[q].x : 0.f, w[q].y <= -kAlphaMin ? w[q].y : 0.f);
            };
            const auto pass = [&](float2 (&w)[P2]) {   // to minus the weights
#pragma unroll
                for (int q = 0; q < P2; ++q) {
                    const float2 alpha = w[q];
                    w[q] = __fmul2_rn(alpha, T[q]);
                    T[q] = __ffma2_rn(alpha, T[q], T[q]);
                }
            };
            const auto blend = [&](uint32_t t, const float2 (&w)[P2]) {
#pragma unroll
                for (int c = 0; c < CDIM; c += 4) {
                    const float4 c4 = sEntry[t * kEntry + 2 + c / 4];
#pragma unroll
                    for (int q = 0; q < P2; ++q) {
                        out[c][q] = __ffma2_rn(make_float2(c4.x, c4.x), w[q], out[c][q]);
                        out[c + 1][q] = __ffma2_rn(make_float2(c4.y, c4.y), w[q], out[c + 1][q]);
                        out[c + 2][q] = __ffma2_rn(make_float2(c4.z, c4.z), w[q], out[c + 2][q]);
                        out[c + 3][q] = __ffma2_rn(make_float2(c4.w, c4.w), w[q], out[c + 3][q]);
                    }
                }
            };
            const auto note = [&](uint32_t t, const float2 (&w)[P2]) {
                const int32_t at = sIdx[t];
#pragma unroll
                for (int k = 0; k < PX; ++k)
                    if ((k & 1 ? w[k / 2].y : w[k / 2].x) != 0.f) sl[32 * k] = at;
            };
            // the last of some full entries, as the last one blended of pixel k
            const auto note_full = [&](int k, uint32_t entries) {
                if (entries) sl[32 * k] = max(sl[32 * k], sIdx[31 - __clz(entries)]);
            };
            float passed = 0.f;   // log2 of what the entries before t leave
            for (uint32_t t = 0; t < n;) {
                // T stays above the limit, so only a blended entry can take a pixel below it: the first that might, by the bound
                const uint32_t below = __ballot_sync(0xffffffffu, seen && place >= t && bound + (left - passed) <= kLowBound);
                const uint32_t cross = below ? __popc(kept & ((below & (0u - below)) - 1u)) : n;
                const uint32_t stop = min(cross, (careful >> t) ? t + (uint32_t)__ffs(careful >> t) - 1u : n);
                while (t < stop) {
                    const uint32_t rest = ~full >> t, end = min(stop, rest ? t + (uint32_t)__ffs(rest) - 1u : n);
#pragma unroll 2
                    for (; t < end; ++t) {
                        float2 w[P2];
                        evaluate(t, w);
                        pass(w);
                        blend(t, w);
                    }
                    if (t >= stop) break;
                    float2 w[P2];
                    evaluate(t, w);
                    drop_small(w);
                    pass(w);
                    note(t, w);
                    blend(t, w);
                    ++t;
                }
                if (t >= n) break;
                float2 w[P2];
                evaluate(t, w);
                if ((careful >> t) & 1u) {
                    const float4 A = sEntry[t * kEntry], B = sEntry[t * kEntry + 1];
                    const float mx = A.x + roll * A.z, dy = A.y + roll * A.w - py;
                    const float bdy = B.y * dy, cdy2 = B.z * dy * dy;
#pragma unroll
                    for (int q = 0; q < P2; ++q) {
                        const float2 pw = pair_power(B.x, __fadd2_rn(make_float2(mx, mx), npx[q]), bdy, cdy2);
                        w[q].x = pw.x <= 0.f ? fmaxf(-kAlphaMax, w[q].x) : 0.f;
                        w[q].y = pw.y <= 0.f ? fmaxf(-kAlphaMax, w[q].y) : 0.f;
                    }
                }
                drop_small(w);
                pass(w);
                float low = 1.f;
#pragma unroll
                for (int q = 0; q < P2; ++q) low = fminf(low, fminf(T[q].x, T[q].y));
                low = __uint_as_float(__reduce_min_sync(0xffffffffu, __float_as_uint(low)));
                if (low <= kTStop) {
                    bool gone = true;
#pragma unroll
                    for (int k = 0; k < PX; ++k) {
                        float &Tk = k & 1 ? T[k / 2].y : T[k / 2].x, &wk = k & 1 ? w[k / 2].y : w[k / 2].x, &column = k & 1 ? npx[k / 2].y : npx[k / 2].x;
                        if (Tk <= kTStop) {
                            sT[k][lane] = Tk - wk;
                            Tk = 1.f;
                            wk = 0.f;
                            column = -kPixelGone;
                            note_full(k, full & ((1u << t) - 1u));
                        }
                        gone = gone && column == -kPixelGone;
                    }
                    done = __all_sync(0xffffffffu, gone);
                }
                note(t, w);
                blend(t, w);
                if (done) break;
                bound = lg2_approx(low);
                passed = __shfl_sync(0xffffffffu, left, __ffs(__ballot_sync(0xffffffffu, seen && place == t)) - 1);
                ++t;
            }
            bound += __shfl_sync(0xffffffffu, left, 31) - passed;
            if (full && !done)
#pragma unroll
                for (int k = 0; k < PX; ++k)
                    if ((k & 1 ? npx[k / 2].y : npx[k / 2].x) != -kPixelGone) note_full(k, full);
        }
#pragma unroll
        for (int k = 0; k < PX; ++k) {   // pixels outside the image are gone without having drawn anything
            pos[k] = sl[32 * k];
            float &Tk = k & 1 ? T[k / 2].y : T[k / 2].x;
            if ((k & 1 ? npx[k / 2].y : npx[k / 2].x) == -kPixelGone && n_inside > (uint32_t)k) Tk = sT[k][lane];
        }
    } else {
        for (int32_t start = range.start; start < range.end && !done; start += 32) {
            const int32_t idx = start + (int32_t)lane;
            const int32_t g = next_id;
            uint32_t seen = 0u;
            PixelEntry e;
            if (idx < range.end) {
                e = load_pixel_entry(g, means2d, conics, opacities, pix_vels);
                if (idx + 32 < range.end) next_id = flatten_ids[idx + 32];   // on its way meanwhile
                seen = patch_sees<true>(e, box, roll_lo, roll_hi);
            }
            uint32_t todo = __ballot_sync(0xffffffffu, seen != 0u);
            const uint32_t careful = __ballot_sync(0xffffffffu, seen > kSeenEntry);
            odd |= seen;
            __syncwarp();   // the batch before has been read
            if (seen) {
                sA[lane] = e.A;
                sB[lane] = scaled_conic(make_float4(e.B.x, e.B.y, e.B.z, -e.B.w));
                if (!kTogether) stage_whole_row<CDIM>(sCol + lane * (CDIM / 4), colors + (size_t)g * channels, channels, CDIM < 20 && vec);
            }
            if (kTogether) stage_rows<CDIM>(reinterpret_cast<float *>(sCol), colors, g, todo, channels, lane);
            __syncwarp();
            uint32_t blended[PX];   // entries of the batch, one bit each
#pragma unroll
            for (int k = 0; k < PX; ++k) blended[k] = 0u;
            while (todo) {
                const uint32_t t = (uint32_t)__ffs(todo) - 1u, bit = 1u << t;
                todo ^= bit;
                const float4 A = sA[t], B = sB[t];
                const float mx = A.x + roll * A.z, dy = A.y + roll * A.w - py;
                const float bdy = B.y * dy, cdy2 = B.z * dy * dy;
                float2 w[P2];   // minus the alphas, then minus the weights
#pragma unroll
                for (int q = 0; q < P2; ++q) {
                    const float2 pw = pair_power(B.x, __fadd2_rn(make_float2(mx, mx), npx[q]), bdy, cdy2);
                    w[q] = __fmul2_rn(make_float2(B.w, B.w), make_float2(exp2_approx(pw.x), exp2_approx(pw.y)));
                }
                if (careful & bit) {
#pragma unroll
                    for (int q = 0; q < P2; ++q) {
                        const float2 pw = pair_power(B.x, __fadd2_rn(make_float2(mx, mx), npx[q]), bdy, cdy2);
                        w[q].x = pw.x <= 0.f ? fmaxf(-kAlphaMax, w[q].x) : 0.f;
                        w[q].y = pw.y <= 0.f ? fmaxf(-kAlphaMax, w[q].y) : 0.f;
                    }
                }
                float low = 1.f;
#pragma unroll
                for (int q = 0; q < P2; ++q) {
                    const bool ok0 = w[q].x <= -kAlphaMin, ok1 = w[q].y <= -kAlphaMin;
                    if (ok0) blended[2 * q] |= bit;
                    if (ok1) blended[2 * q + 1] |= bit;
                    const float2 alpha = make_float2(ok0 ? w[q].x : 0.f, ok1 ? w[q].y : 0.f);
                    w[q] = __fmul2_rn(alpha, T[q]);
                    T[q] = __ffma2_rn(alpha, T[q], T[q]);
                    low = fminf(low, fminf(T[q].x, T[q].y));
                }
                // T stays above the limit, so only a blended entry can take a pixel below it; few entries do
                if (__any_sync(0xffffffffu, low <= kTStop)) {
                    bool gone = true;
#pragma unroll
                    for (int q = 0; q < P2; ++q) {
                        if (T[q].x <= kTStop) { npx[q].x = -kPixelGone; T[q].x -= w[q].x; w[q].x = 0.f; blended[2 * q] &= ~bit; }
                        if (T[q].y <= kTStop) { npx[q].y = -kPixelGone; T[q].y -= w[q].y; w[q].y = 0.f; blended[2 * q + 1] &= ~bit; }
                        gone = gone && npx[q].x == -kPixelGone && npx[q].y == -kPixelGone;
                    }
                    done = __all_sync(0xffffffffu, gone);
                    if (done) todo = 0u;
                }
#pragma unroll
                for (int c = 0; c < CDIM; c += 4) {
                    const float4 c4 = sCol[t * (CDIM / 4) + c / 4];
#pragma unroll
                    for (int q = 0; q < P2; ++q) {
                        out[c][q] = __ffma2_rn(make_float2(c4.x, c4.x), w[q], out[c][q]);
                        out[c + 1][q] = __ffma2_rn(make_float2(c4.y, c4.y), w[q], out[c + 1][q]);
                        out[c + 2][q] = __ffma2_rn(make_float2(c4.z, c4.z), w[q], out[c + 2][q]);
                        out[c + 3][q] = __ffma2_rn(make_float2(c4.w, c4.w), w[q], out[c + 3][q]);
                    }
                }
            }
#pragma unroll
            for (int k = 0; k < PX; ++k)
                if (blended[k]) pos[k] = start + 31 - __clz(blended[k]);
        }
    }
    const float *bg = backgrounds ? backgrounds + (size_t)cam * channels : nullptr;
    const size_t pix = ((size_t)cam * H + i) * W + j;
    float none = 0.f;   // a NaN: see odd_pixels_fwd()
    if constexpr (CDIM == 4) {
        float alphas[PX], depths[PX], v[PX][CDIM];
#pragma unroll
        for (int h = 0; h < PX; ++h) {
            const float Tk = h & 1 ? T[h / 2].y : T[h / 2].x;
            alphas[h] = 1.f - Tk;
            depths[h] = 0.f;
#pragma unroll
            for (int k = 0; k < CDIM; ++k) {
                v[h][k] = -(h & 1 ? out[k][h / 2].y : out[k][h / 2].x);
                none = fmaf(v[h][k], 0.f, none);
                if (bg && (uint32_t)k < channels) v[h][k] += Tk * bg[k];
                if (expected && (uint32_t)k + 1u == channels) depths[h] = v[h][k] /= fmaxf(1.f - Tk, kExpectedMin);
            }
        }
        if (n_inside) {
            store_pixels<PX>(render_alphas + pix, alphas, n_inside);
            store_pixels<PX>(last_ids + pix, pos, n_inside);
            store_channels<CDIM, PX>(render_colors + pix * channels, v, channels, n_inside);
            if (expected && expected_depths != nullptr) store_pixels<PX>(expected_depths + pix, depths, n_inside);
        }
    } else {   // one pixel after the other: all at once costs the 16-channel kernel 13 us in registers
        const bool drawn_together = kTogether && (reinterpret_cast<uintptr_t>(render_colors) & 15u) == 0u;
        float4 *row = sCol + lane * (CDIM / 4);
#pragma unroll
        for (int h = 0; h < PX; ++h) {
            const float Tk = h & 1 ? T[h / 2].y : T[h / 2].x;
            const bool in = (uint32_t)h < n_inside;
            if (in) {
                render_alphas[pix + h] = 1.f - Tk;
                last_ids[pix + h] = pos[h];
            }
            if (drawn_together) __syncwarp();
#pragma unroll
            for (int k = 0; k < CDIM; k += 4) {
                float v[4];
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    v[c] = -(h & 1 ? out[k + c][h / 2].y : out[k + c][h / 2].x);
                    none = fmaf(v[c], 0.f, none);
                    if (in && (uint32_t)(k + c) < channels) {
                        if (bg) v[c] += Tk * bg[k + c];
                        if (expected && (uint32_t)(k + c) + 1u == channels) {
                            v[c] /= fmaxf(1.f - Tk, kExpectedMin);
                            if (expected_depths != nullptr) expected_depths[pix + h] = v[c];
                        }
                        if (!drawn_together) render_colors[(pix + h) * channels + k + c] = v[c];
                    }
                }
                if (drawn_together) row[k / 4] = make_float4(v[0], v[1], v[2], v[3]);
            }
            if (drawn_together) {
                const uint32_t drawn = __ballot_sync(0xffffffffu, in);
                __syncwarp();
                copy_rows<CDIM, true>(reinterpret_cast<float *>(sCol), render_colors + (size_t)cam * H * W * channels, (int32_t)(i * W + j) + h,
                                      drawn, channels, lane);
            }
        }
        __syncwarp();   // odd_pixels_fwd() may write again what other lanes wrote
    }
    if (__any_sync(0xffffffffu, odd >= kOddEntry) || none != 0.f) {
        const PixelTask task = {C, W, H, tile_size, tile_w, tile_h, channels, n_isects, means2d, pix_vels, conics, opacities,
                                colors, rs_time, backgrounds, offsets, flatten_ids};
        odd_pixels_fwd<PX>(task, gtile, tr, render_colors, render_alphas, last_ids, expected != 0u, expected_depths);
    }
}

// ---------------------------------------------------------------------------------------
// Lidar tiles. The points of a tile are cut into patches of one warp each - 8 columns x 4 beams of the
// usual 32 x 8 tile - and the warps of a tile are spread over several small CTAs: tiles differ widely in
// how many entries saturate them (41 on average in the lidar benchmark, several hundred at worst), and
// a scan of 64 tiles does not fill the machine with one CTA per tile.
// ---------------------------------------------------------------------------------------
struct PointPatch {
    uint32_t col, row;     // first point of the thread within the tile
    bool patched;          // patches are kPatchW columns wide, else points in row-major order
};

constexpr uint32_t kPatchW = 8;

// Thread `index` of the tile's threads (PX points in one beam or, in row-major order, PX in sequence).
template <int PX>
__device__ __forceinline__ PointPatch point_patch(uint32_t tile_width, uint32_t tile_height, uint32_t index) {
    constexpr uint32_t kPatchH = 32 * PX / kPatchW;
    PointPatch p;
    p.patched = tile_width % kPatchW == 0u && tile_height % kPatchH == 0u;
    if (p.patched) {
        const uint32_t patch = index >> 5, lane = index & 31u, per_row = tile_width / kPatchW;
        p.col = (patch % per_row) * kPatchW + (lane * PX) % kPatchW;
        p.row = (patch / per_row) * kPatchH + (lane * PX) / kPatchW;
    } else {
        p.row = index * PX / tile_width;   // the first of PX points in sequence
        p.col = index * PX - p.row * tile_width;
    }
    return p;
}

// Azimuths, elevations (as centre and half width) and time offsets of a warp's points.
struct PointBox { float az, az_half, el, el_half, roll_lo, roll_hi; };

struct PointExtent {
    float az0 = 3.0e38f, az1 = -3.0e38f, el0 = 3.0e38f, el1 = -3.0e38f, r0 = 3.0e38f, r1 = -3.0e38f;
    float none = 0.f;   // a NaN: a coordinate that is not finite
    template <bool kOdd = true>
    __device__ __forceinline__ void add(float az, float el, float roll) {
        az0 = fminf(az0, az); az1 = fmaxf(az1, az);
        el0 = fminf(el0, el); el1 = fmaxf(el1, el);
        r0 = fminf(r0, roll); r1 = fmaxf(r1, roll);
        if (kOdd) none = fmaf(az, 0.f, fmaf(el, 0.f, fmaf(roll, 0.f, none)));
    }
    // The box of the whole warp, in every lane; no points: a negative half width. A point with a coordinate that is not
    // finite takes every entry with the capped alpha: no offset is ruled out where the centre is not a number. (The
    // backward pass has such patches marked and works on them elsewhere.)
    template <bool kOdd = true>
    __device__ __forceinline__ PointBox warp_box() {
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) {
            az0 = fminf(az0, __shfl_xor_sync(0xffffffffu, az0, off)); az1 = fmaxf(az1, __shfl_xor_sync(0xffffffffu, az1, off));
            el0 = fminf(el0, __shfl_xor_sync(0xffffffffu, el0, off)); el1 = fmaxf(el1, __shfl_xor_sync(0xffffffffu, el1, off));
            r0 = fminf(r0, __shfl_xor_sync(0xffffffffu, r0, off)); r1 = fmaxf(r1, __shfl_xor_sync(0xffffffffu, r1, off));
        }
        if (kOdd && __any_sync(0xffffffffu, none != 0.f)) return {NAN, 0.f, 0.f, 0.f, 0.f, 0.f};
        return {0.5f * (az0 + az1), 0.5f * (az1 - az0), 0.5f * (el0 + el1), 0.5f * (el1 - el0), r0, r1};
    }
    template <bool kOdd = true>
    __device__ __forceinline__ void write_box(PointBox *box) {   // by the warp's first lane
        const PointBox b = warp_box<kOdd>();
        if ((threadIdx.x & 31u) == 0u) *box = b;
    }
};

struct PointEntry {
    float4 A, B;      // azimuth, elevation, their velocities | conic, opacity
    float4 C;         // range velocity, depth compensation (2), range
};

__device__ __forceinline__ PointEntry load_point_entry(int32_t g, const float2 *__restrict__ means2d,
                                                       const float *__restrict__ conics,
                                                       const float *__restrict__ opacities,
                                                       const float *__restrict__ pix_vels,
                                                       const float2 *__restrict__ depth_comps) {
    PointEntry e;
    const float2 xy = __ldg(means2d + g), dc = __ldg(depth_comps + g);
    const float *v = pix_vels + 3 * (size_t)g, *q = conics + 3 * (size_t)g;
    e.A = make_float4(xy.x, xy.y, __ldg(v), __ldg(v + 1));
    e.B = make_float4(__ldg(q), __ldg(q + 1), __ldg(q + 2), __ldg(opacities + g));
    e.C = make_float4(__ldg(v + 2), dc.x, dc.y, 0.f);
    return e;
}

// Offsets of a moving mean from the points of a box, [lo, hi]: a range that reaches across half a turn
// is the whole turn. The slack of a millidegree covers the rounding of the wrapped differences. Returns how far the offsets
// reach before any wrap: below half a turn none of them wraps.
__device__ __forceinline__ float angle_range(float mean, float vel, float centre, float half, float roll_lo, float roll_hi,
                                            float &lo, float &hi) {
    const float a = roll_lo * vel, b = roll_hi * vel;
    const float m = mean + 0.5f * (a + b), d = angle_difference(m, centre);
    const float reach = half + 0.5f * fabsf(b - a) + 1e-3f;
    lo = d - reach;
    hi = d + reach;
    if (lo < -180.f || hi > 180.f) { lo = -180.f; hi = 180.f; }
    return fabsf(m - centre) + reach;
}

// Bit w: the entry may contribute to a point of box w; bit 16 + w: its angles may wrap between mean and point there, or its
// alphas need looking at one by one (as kCarefulEntry for the cameras).
constexpr uint32_t kCarefulShift = 16;

// kMark: with the upper bits; kOdd: a box without a centre sees every entry
template <bool kMark, bool kOdd>
__device__ __forceinline__ uint32_t boxes_that_see(const PointEntry &e, const PointBox *s_box, uint32_t n_boxes) {
    const BoxTest test(e.B.x, e.B.y, e.B.z, e.B.w);
    if (!kOdd && test.never) return 0u;
    const float ac = e.B.x * e.B.z;
    const bool plain = e.B.x > 1e-15f && e.B.z > 1e-15f && e.B.x < 1e15f && e.B.z < 1e15f && ac - e.B.y * e.B.y >= 1e-5f * ac &&
                       e.B.w <= kAlphaMax;
    uint32_t seen = 0u;
    for (uint32_t w = 0; w < n_boxes; ++w) {
        const PointBox b = s_box[w];
        if (!(b.az_half >= 0.f)) continue;
        float x_lo, x_hi, y_lo, y_hi;
        const float x = angle_range(e.A.x, e.A.z, b.az, b.az_half, b.roll_lo, b.roll_hi, x_lo, x_hi);
        const float y = angle_range(e.A.y, e.A.w, b.el, b.el_half, b.roll_lo, b.roll_hi, y_lo, y_hi);
        if (!(kOdd && b.az != b.az) && test.misses(x_lo, x_hi, y_lo, y_hi)) continue;
        seen |= 1u << w;
        if (kMark && !(plain && x < 179.9f && y < 179.9f)) seen |= 1u << (w + kCarefulShift);
    }
    return seen;
}

// Offset of an entry from a point and its exp(-sigma); sigma decides with alpha whether it is blended. Every kernel rounds
// the steps alike - one or two values at a time, and the transmittances' factors as T * (1 - alpha) -, because the median
// range of a point is that of the entry at which its transmittance crosses a half: the last bit decides between two
// ranges that may lie far apart.
struct PointFootprint { float dx, dy, sigma, vis; };

__device__ __forceinline__ float point_sigma(const float4 &B, float dx, float dy) {
    return fmaf(__fmul_rn(B.y, dx), dy, __fmul_rn(0.5f, fmaf(__fmul_rn(B.x, dx), dx, __fmul_rn(__fmul_rn(B.z, dy), dy))));
}
__device__ __forceinline__ float2 point_sigma(float2 a, float2 b, float2 c, float2 dx, float2 dy) {
    const float2 square = __ffma2_rn(__fmul2_rn(a, dx), dx, __fmul2_rn(__fmul2_rn(c, dy), dy));
    return __ffma2_rn(__fmul2_rn(b, dx), dy, __fmul2_rn(make_float2(0.5f, 0.5f), square));
}

__device__ __forceinline__ PointFootprint point_footprint(const float4 &A, const float4 &B, float roll, float az, float el) {
    PointFootprint f;
    const float mx = fmaf(roll, A.z, A.x), my = fmaf(roll, A.w, A.y);
    f.dx = angle_difference(mx, az);
    f.dy = angle_difference(my, el);
    f.sigma = point_sigma(B, f.dx, f.dy);
    f.vis = __expf(-f.sigma);
    return f;
}

// Copies the feature row of entry g, the range behind it when it comes from its own array, then zeros.
template <int CDIM>
__device__ __forceinline__ void stage_features(float *row, const float *__restrict__ colors, size_t g, uint32_t fstride,
                                               bool vec, bool has_range, float range) {
    uint32_t filled = 0;
    if (fstride) {
        stage_row(row, colors, g, fstride, vec);
        filled = (fstride + 3u) & ~3u;
    }
    if (has_range) {
        row[fstride] = range;
        filled = max(filled, fstride + 1u);
    }
    for (uint32_t k = filled; k < (uint32_t)CDIM; ++k) row[k] = 0.f;
}

// ---------------------------------------------------------------------------------------
// Lidar forward. One point per lane; a warp looks only at the entries that can reach its patch (a ninth
// of the (point, entry) pairs of a small scan contribute, two thirds of the benchmark's) and evaluates
// two of them at a time, because what it waits for is the chain from the offsets through the exponential
// to the transmittance. (Leaving the wrap, the sign of sigma and the cap to the entries that need them, as the other
// lidar kernels do, gains nothing here: 128 x 1800 43.3 -> 44.4 us. What a scan takes hangs on what lies next to the sensor: 128 x 1800, 17
// channels 45 to 93 us over eight turns of it, backward 84 to 186; figures of that size here and below are of a turn of 37 degrees.) The rendered rows leave through shared memory: a beam's eight points
// are consecutive floats.
// ---------------------------------------------------------------------------------------
// entries per thread and batch (their loads overlap), while the shared memory of a batch stays small
constexpr uint32_t points_fwd_stage(int cdim) { return cdim <= 8 ? 2 : 1; }
// (17 channels: 128 x 1800 40 us at 80 registers, 42 at 96; 64 x 1083 64 and 56)
constexpr int points_fwd_regs(int cdim) { return cdim <= 8 ? 96 : cdim <= 20 ? 80 : 112; }

template <int CDIM>
__global__ void __maxnreg__(points_fwd_regs(CDIM)) rasterize_to_points_fwd_kernel(
    uint32_t C, int64_t n_isects, const float2 *__restrict__ means2d,
    const float *__restrict__ conics, const float *__restrict__ colors,
    const float *__restrict__ ranges /* optional: last channel comes from here */, uint32_t channels,
    const float *__restrict__ opacities, const float *__restrict__ pix_vels /* [.,3] */,
    const float2 *__restrict__ depth_comps, const float *__restrict__ backgrounds,
    const float4 *__restrict__ raster_pts, uint32_t W, uint32_t H, uint32_t tile_width,
    uint32_t tile_height, uint32_t grid_w, uint32_t grid_h, uint32_t ctas_per_tile, int compute_alpha_sum,
    float alpha_sum_threshold, const int32_t *__restrict__ offsets,
    const int32_t *__restrict__ flatten_ids, uint32_t depth_idx,
    float *__restrict__ render_colors, float *__restrict__ render_alphas,
    float *__restrict__ alpha_sum_out, int32_t *__restrict__ last_ids,
    float *__restrict__ median_depths) {
    chain_enter();
    constexpr uint32_t kStage = points_fwd_stage(CDIM);
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ PointBox s_box[8];
    __shared__ uint32_t s_warp_kept[kStage * 16];
    const uint32_t bs = blockDim.x, cap = kStage * bs;
    float4 *sA = reinterpret_cast<float4 *>(smem_raw);
    float4 *sB = sA + cap;
    float4 *sC = sB + cap;
    float *sFeat = reinterpret_cast<float *>(sC + cap);                 // [cap * CDIM]
    int32_t *sPos = reinterpret_cast<int32_t *>(sFeat + cap * CDIM);    // list position
    uint32_t *sSeen = reinterpret_cast<uint32_t *>(sPos + cap);         // warps that may see it

    const uint32_t tiles_per_cam = grid_w * grid_h;
    const uint32_t gtile = blockIdx.x / ctas_per_tile, part = blockIdx.x - gtile * ctas_per_tile;
    const uint32_t cam = gtile / tiles_per_cam;
    const uint32_t tile = gtile - cam * tiles_per_cam;
    const uint32_t ty = tile / grid_w, tx = tile - ty * grid_w;
    const uint32_t tr = threadIdx.x, lane = tr & 31u, warp = tr >> 5, n_warps = bs >> 5;
    const uint32_t index = part * bs + tr;
    const PointPatch pp = point_patch<1>(tile_width, tile_height, index);
    const uint32_t i = ty * tile_height + pp.row, j = tx * tile_width + pp.col;
    const bool in_image = index < tile_width * tile_height && i < H && j < W;
    bool inside = in_image;
    const size_t pix = ((size_t)cam * H + i) * W + j;
    float px = 0.f, py = 0.f, pz = 0.f, roll = 0.f;
    if (inside) {
        const float4 rp = raster_pts[pix];
        px = rp.x; py = rp.y; pz = rp.z; roll = rp.w;
        if (pz <= 0.f) inside = false;
    }
    PointExtent extent;
    if (inside) extent.add(px, py, roll);
    extent.write_box(s_box + warp);
    const TileRange range = tile_range(offsets, gtile, C * tiles_per_cam, n_isects);
    const uint32_t num_batches = (uint32_t)(range.end - range.start + cap - 1) / cap;

    // with a separate range array the feature rows hold channels - 1 columns; a staged row holds all CDIM
    // accumulated channels: the features, behind them the range when it comes from its own array, then
    // zeros, so that one unconditional multiply-add pass covers them
    const uint32_t fstride = ranges ? channels - 1 : channels;
    const bool vec = (fstride % 4u == 0u) && ((reinterpret_cast<uintptr_t>(colors) & 15u) == 0u);
    bool done = !inside;
    bool warp_done = __all_sync(0xffffffffu, done);
    float T = 1.f;
    int32_t cur_idx = 0;
    float depth_extra = 0.f, alpha_sum = 0.f, median = 0.f;
    const float alpha_sum_limit = pz - alpha_sum_threshold;
    float pix_out[CDIM];
#pragma unroll
    for (int k = 0; k < CDIM; ++k) pix_out[k] = 0.f;

    int32_t next_id[kStage];
#pragma unroll
    for (uint32_t q = 0; q < kStage; ++q) {
        const int32_t idx = range.start + (int32_t)(q * bs + tr);
        next_id[q] = idx < range.end ? flatten_ids[idx] : 0;
    }
    for (uint32_t b = 0; b < num_batches; ++b) {
        if (__syncthreads_and(warp_done)) break;
        const int32_t batch_start = range.start + (int32_t)(cap * b);
        PointEntry e[kStage];
        int32_t g[kStage];
        uint32_t seen[kStage], kept[kStage];
#pragma unroll
        for (uint32_t q = 0; q < kStage; ++q) {
            g[q] = next_id[q];
            const int32_t idx = batch_start + (int32_t)(q * bs + tr);
            if (idx < range.end) e[q] = load_point_entry(g[q], means2d, conics, opacities, pix_vels, depth_comps);
        }
#pragma unroll
        for (uint32_t q = 0; q < kStage; ++q) {
            const int32_t idx = batch_start + (int32_t)(q * bs + tr);
            if (idx < range.end) e[q].C.w = ranges ? __ldg(ranges + g[q]) : __ldg(colors + (size_t)g[q] * channels + depth_idx);
            if (idx + (int32_t)cap < range.end) next_id[q] = flatten_ids[idx + cap];   // on its way meanwhile
        }
        // compact the survivors to the front of the staging arrays, list order kept
#pragma unroll
        for (uint32_t q = 0; q < kStage; ++q) {
            seen[q] = batch_start + (int32_t)(q * bs + tr) < range.end ? boxes_that_see<false, true>(e[q], s_box, n_warps) : 0u;
            kept[q] = __ballot_sync(0xffffffffu, seen[q] != 0u);
            if (lane == 0) s_warp_kept[q * n_warps + warp] = __popc(kept[q]);
        }
        __syncthreads();
        uint32_t n_kept = 0, pos[kStage];
#pragma unroll
        for (uint32_t q = 0; q < kStage; ++q) {
            pos[q] = __popc(kept[q] & ((1u << lane) - 1u));
            for (uint32_t w = 0; w < n_warps; ++w) {
                if (w == warp) pos[q] += n_kept;
                n_kept += s_warp_kept[q * n_warps + w];
            }
        }
#pragma unroll
        for (uint32_t q = 0; q < kStage; ++q)
            if (seen[q]) {
                sA[pos[q]] = e[q].A;
                sB[pos[q]] = e[q].B;
                sC[pos[q]] = e[q].C;
                sPos[pos[q]] = batch_start + (int32_t)(q * bs + tr);
                sSeen[pos[q]] = seen[q];
                stage_features<CDIM>(sFeat + pos[q] * CDIM, colors, (size_t)g[q], fstride, vec, ranges != nullptr, e[q].C.w);
            }
        __syncthreads();
        if (warp_done) continue;
        const auto blend = [&](uint32_t t, const PointFootprint &f, float alpha) {
            const float next_T = T * (1.f - alpha);
            if (next_T <= kTStop) { done = true; return; }
            const float vis = alpha * T;
            const float4 Cc = sC[t];
            axpy_staged_full<CDIM>(pix_out, sFeat + t * CDIM, vis);   // the zero padding adds nothing
            const float dterm = Cc.y * f.dx + Cc.z * f.dy + Cc.x * roll;
            depth_extra += dterm * vis;
            if (T > 0.5f && next_T <= 0.5f) median = Cc.w + dterm;
            if (compute_alpha_sum && Cc.w < alpha_sum_limit) alpha_sum += alpha;
            cur_idx = sPos[t];
            T = next_T;
        };
        for (uint32_t t0 = 0; t0 < n_kept && !warp_done; t0 += 32) {
            const uint32_t mine = t0 + lane;
            uint32_t todo = __ballot_sync(0xffffffffu, mine < n_kept && ((sSeen[mine] >> warp) & 1u));
            while (todo && !(warp_done = __all_sync(0xffffffffu, done))) {
                // two entries at a time; an odd one out is evaluated twice and blended once
                const uint32_t t = t0 + (uint32_t)__ffs(todo) - 1u;
                todo &= todo - 1u;
                const bool two = todo != 0u;
                const uint32_t u = two ? t0 + (uint32_t)__ffs(todo) - 1u : t;
                todo &= todo - 1u;   // of 0: stays 0
                const float4 A0 = sA[t], B0 = sB[t], A1 = sA[u], B1 = sB[u];
                const PointFootprint f0 = point_footprint(A0, B0, roll, px, py), f1 = point_footprint(A1, B1, roll, px, py);
                const float alpha0 = fminf(kAlphaMax, B0.w * f0.vis), alpha1 = fminf(kAlphaMax, B1.w * f1.vis);
                const bool ok0 = !(f0.sigma < 0.f || alpha0 < kAlphaMin), ok1 = two && !(f1.sigma < 0.f || alpha1 < kAlphaMin);
                if (ok0 && !done) blend(t, f0, alpha0);
                if (ok1 && !done) blend(u, f1, alpha1);
            }
            warp_done = __all_sync(0xffffffffu, done);
        }
    }
    // points that are not rendered (range <= 0) produce zeros everywhere
    const float *bg = backgrounds ? backgrounds + (size_t)cam * channels : nullptr;
    __syncthreads();   // the rendered rows take the place of the feature rows
    float *rows = sFeat + warp * 32u * CDIM;
    float none = 0.f;   // a NaN: see odd_points_bwd()
#pragma unroll
    for (int k = 0; k < CDIM; ++k)
        if ((uint32_t)k < channels) {
            float v = pix_out[k];
            if ((uint32_t)k == depth_idx) v += depth_extra;
            none = fmaf(v, 0.f, none);
            if (bg) v += T * bg[k];
            v = inside ? v : 0.f;
            if (pp.patched) rows[lane * channels + k] = v;
            else if (in_image) render_colors[pix * channels + k] = v;
        }
    if (in_image) {
        render_alphas[pix] = inside ? 1.f - T : 0.f;
        last_ids[pix] = inside ? cur_idx | (none != 0.f ? kOddPixel : 0) : 0;
        median_depths[pix] = inside ? median : 0.f;
        if (alpha_sum_out != nullptr) alpha_sum_out[pix] = inside ? alpha_sum : 0.f;
    }
    if (!pp.patched) return;
    __syncwarp();
    const uint32_t i0 = __shfl_sync(0xffffffffu, i, 0), j0 = __shfl_sync(0xffffffffu, j, 0);
    const bool any = __shfl_sync(0xffffffffu, (int)(index < tile_width * tile_height), 0);
    const uint32_t n = any && j0 < W ? min(kPatchW, W - j0) * channels : 0u;
    for (uint32_t r = 0; r < 32u / kPatchW && i0 + r < H; ++r) {
        float *dst = render_colors + (((size_t)cam * H + i0 + r) * W + j0) * channels;
        const float *src = rows + r * kPatchW * channels;
        for (uint32_t k = lane; k < n; k += 32u) dst[k] = src[k];
    }
}

// ---------------------------------------------------------------------------------------
// Lidar forward for few patches: all warps of a CTA work on ONE patch, four consecutive entries each of the 32 between two
// barriers. What depends on the order - the transmittance, where a point stops, its median - stays one chain per point, with
// the same operations as above, but it is all that is left in the chain:
//   1. every warp evaluates its four entries, two per instruction, and leaves their 1 - alpha;
//   2. behind the barrier every warp multiplies its way down all 32 of them by itself - no second barrier, nothing handed
//      back -, and goes over its share again for weights, where a point stops, median, sums and features. The warps' partial
//      results are put together at the end.
// The chain runs on behind a point's stop: the transmittance never rises, so an entry is blended exactly
// if what it would leave is above the threshold. The next batch's entries are on their way while the chunks of
// one are worked through, the range terms and features of those that stay while the first chunk is evaluated: a gather
// of 32 lines holds the load unit for 32 cycles, and 256 entries with all they have took it for 2500.
// What bounds it is the issue slots of the SM that holds the patch with the longest list (75 instructions per entry kept, 350 of
// 1900 there) and, eight times, the way from a batch's gathers to its first chunk. A 32 x 512 scan, 8 channels: 43 -> 35 us (one
// warp multiplying down all 32, two barriers, everything gathered for every entry: 43; every warp leaving one product of its
// four, which rounds differently: 32).
// ---------------------------------------------------------------------------------------
constexpr uint32_t kCoopWarps = 8, kCoopShare = 4, kCoopChunk = kCoopWarps * kCoopShare;

__device__ __forceinline__ float2 half_of(const float4 &v, int h) { return h ? make_float2(v.z, v.w) : make_float2(v.x, v.y); }

template <int CDIM>
__global__ void __launch_bounds__(kCoopWarps * 32, 2) rasterize_to_points_fwd_coop_kernel(
    uint32_t C, int64_t n_isects, const float2 *__restrict__ means2d,
    const float *__restrict__ conics, const float *__restrict__ colors,
    const float *__restrict__ ranges, uint32_t channels,
    const float *__restrict__ opacities, const float *__restrict__ pix_vels /* [.,3] */,
    const float2 *__restrict__ depth_comps, const float *__restrict__ backgrounds,
    const float4 *__restrict__ raster_pts, uint32_t W, uint32_t H, uint32_t tile_width,
    uint32_t tile_height, uint32_t grid_w, uint32_t grid_h, uint32_t patches_per_tile, int compute_alpha_sum,
    float alpha_sum_threshold, const int32_t *__restrict__ offsets,
    const int32_t *__restrict__ flatten_ids, uint32_t depth_idx,
    float *__restrict__ render_colors, float *__restrict__ render_alphas,
    float *__restrict__ alpha_sum_out, int32_t *__restrict__ last_ids,
    float *__restrict__ median_depths) {
    chain_enter();
    constexpr uint32_t kThreadsC = kCoopWarps * 32;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ uint32_t s_warp_kept[2][kCoopWarps];
    __shared__ float4 sLeft[2][kCoopWarps][32];   // 1 - alpha of the warps' shares
    // by value, so that four entries in sequence are one 16-byte access: azimuth, elevation, their velocities; conic, opacity;
    // range velocity, depth compensation (2), range
    float *sE = reinterpret_cast<float *>(smem_raw);                        // [12][kThreadsC]
    float *sFeat = sE + 12 * kThreadsC;                                     // [kThreadsC * CDIM]
    int32_t *sPos = reinterpret_cast<int32_t *>(sFeat + kThreadsC * CDIM);  // list position; the sign bit: needs care

    const uint32_t tiles_per_cam = grid_w * grid_h;
    const uint32_t gtile = blockIdx.x / patches_per_tile, part = blockIdx.x - gtile * patches_per_tile;
    const uint32_t cam = gtile / tiles_per_cam;
    const uint32_t tile = gtile - cam * tiles_per_cam;
    const uint32_t ty = tile / grid_w, tx = tile - ty * grid_w;
    const uint32_t tr = threadIdx.x, lane = tr & 31u, warp = tr >> 5;
    const uint32_t index = part * 32u + lane;   // every warp holds the same points
    const PointPatch pp = point_patch<1>(tile_width, tile_height, index);
    const uint32_t i = ty * tile_height + pp.row, j = tx * tile_width + pp.col;
    const bool in_image = index < tile_width * tile_height && i < H && j < W;
    bool inside = in_image;
    const size_t pix = ((size_t)cam * H + i) * W + j;
    const TileRange range = tile_range(offsets, gtile, C * tiles_per_cam, n_isects);
    float px = 0.f, py = 0.f, pz = 0.f, roll = 0.f;
    if (inside) {
        const float4 rp = raster_pts[pix];
        px = rp.x; py = rp.y; pz = rp.z; roll = rp.w;
        if (pz <= 0.f) inside = false;
    }
    PointExtent extent;
    if (inside) extent.add(px, py, roll);
    const PointBox box = extent.warp_box();
    const uint32_t num_batches = (uint32_t)(range.end - range.start + kThreadsC - 1) / kThreadsC;
    const uint32_t fstride = ranges ? channels - 1 : channels;
    const bool vec = (fstride % 4u == 0u) && ((reinterpret_cast<uintptr_t>(colors) & 15u) == 0u);
    for (uint32_t k = channels; k < (uint32_t)CDIM; ++k) sFeat[tr * CDIM + k] = 0.f;   // no row is written there
    float T_run = inside ? 1.f : 0.f;   // the chain, the same in every warp
    // of this warp's share
    float T = 1.f, depth_extra = 0.f, alpha_sum = 0.f, median = 0.f;
    int32_t cur_idx = 0;
    const float alpha_sum_limit = pz - alpha_sum_threshold;
    float pix_out[CDIM];
#pragma unroll
    for (int k = 0; k < CDIM; ++k) pix_out[k] = 0.f;
    const float2 roll2 = make_float2(roll, roll), npx2 = make_float2(-px, -px), npy2 = make_float2(-py, -py);

    bool finished = __all_sync(0xffffffffu, !inside);   // the same in every warp
    int32_t g = 0, next_id = 0;
    PointEntry e;
    // the thread's entry of batch b, as far as the test needs it; the id of the one behind it
    const auto load_entry = [&](uint32_t b) {
        const int32_t idx = range.start + (int32_t)(kThreadsC * b + tr);
        g = next_id;
        if (idx < range.end) {
            const float2 xy = __ldg(means2d + g);
            const float *v = pix_vels + 3 * (size_t)g, *q = conics + 3 * (size_t)g;
            e.A = make_float4(xy.x, xy.y, __ldg(v), __ldg(v + 1));
            e.B = make_float4(__ldg(q), __ldg(q + 1), __ldg(q + 2), __ldg(opacities + g));
            if (idx + (int32_t)kThreadsC < range.end) next_id = flatten_ids[idx + kThreadsC];
        }
    };
    if (!finished && range.start + (int32_t)tr < range.end) next_id = flatten_ids[range.start + tr];
    if (!finished) load_entry(0);
    uint32_t buffer = 0;
    for (uint32_t b = 0; b < num_batches && !finished; ++b) {
        const int32_t idx = range.start + (int32_t)(kThreadsC * b + tr);
        const uint32_t seen = idx < range.end ? boxes_that_see<true, true>(e, &box, 1u) : 0u;
        const uint32_t kept = __ballot_sync(0xffffffffu, seen != 0u);
        if (lane == 0) s_warp_kept[b & 1u][warp] = __popc(kept);
        __syncthreads();   // the batch before has been read
        uint32_t n_kept = 0, pos = __popc(kept & ((1u << lane) - 1u));
#pragma unroll
        for (uint32_t w = 0; w < kCoopWarps; ++w) {
            if (w == warp) pos += n_kept;
            n_kept += s_warp_kept[b & 1u][w];
        }
        if (seen) {
            const float v[8] = {e.A.x, e.A.y, e.A.z, e.A.w, e.B.x, e.B.y, e.B.z, e.B.w};
#pragma unroll
            for (uint32_t k = 0; k < 8; ++k) sE[k * kThreadsC + pos] = v[k];
            sPos[pos] = seen >> kCarefulShift ? idx | INT32_MIN : idx;
            float *late = sE + 8 * kThreadsC + pos, *row = sFeat + pos * CDIM;
            const float *dc = reinterpret_cast<const float *>(depth_comps + g);
            const float *distance = ranges ? ranges + g : colors + (size_t)g * channels + depth_idx;
            async_copy(late, pix_vels + 3 * (size_t)g + 2);
            async_copy(late + kThreadsC, dc);
            async_copy(late + 2 * kThreadsC, dc + 1);
            async_copy(late + 3 * kThreadsC, distance);
            async_copy_row(row, colors + (size_t)g * fstride, fstride, vec);
            if (ranges) async_copy(row + fstride, distance);
        }
        if (b + 1 < num_batches) load_entry(b + 1);
        __syncthreads();
        for (uint32_t c0 = 0; c0 < n_kept && !finished; c0 += kCoopChunk) {
            const uint32_t t0 = c0 + warp * kCoopShare;
            const bool mine = t0 < n_kept;
            float alpha[kCoopShare];
            float2 dx[2], dy[2];
            int4 at = make_int4(0, 0, 0, 0);
            float4 left = make_float4(1.f, 1.f, 1.f, 1.f);   // 1 - alpha
            if (mine) {
                const auto four = [&](uint32_t k) { return *reinterpret_cast<const float4 *>(sE + k * kThreadsC + t0); };
                const float4 X = four(0), Y = four(1), VX = four(2), VY = four(3), Ba = four(4), Bb = four(5), Bc = four(6), Op = four(7);
                at = *reinterpret_cast<const int4 *>(sPos + t0);
                const float2 turn = make_float2(180.f, 180.f), back = make_float2(-180.f, -180.f);
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    // a difference that does not wrap, rounded as angle_difference() rounds it
                    dx[h] = __fadd2_rn(__fadd2_rn(__fadd2_rn(__ffma2_rn(roll2, half_of(VX, h), half_of(X, h)), npx2), turn), back);
                    dy[h] = __fadd2_rn(__fadd2_rn(__fadd2_rn(__ffma2_rn(roll2, half_of(VY, h), half_of(Y, h)), npy2), turn), back);
                    const float2 sigma = point_sigma(half_of(Ba, h), half_of(Bb, h), half_of(Bc, h), dx[h], dy[h]);
                    const float2 a = __fmul2_rn(half_of(Op, h), make_float2(__expf(-sigma.x), __expf(-sigma.y)));
                    alpha[2 * h] = a.x >= kAlphaMin ? a.x : 0.f;
                    alpha[2 * h + 1] = a.y >= kAlphaMin ? a.y : 0.f;
                }
                if (t0 + kCoopShare > n_kept || (at.x | at.y | at.z | at.w) < 0) {
#pragma unroll
                    for (uint32_t k = 0; k < kCoopShare; ++k) {
                        const uint32_t t = t0 + k;
                        if (t >= n_kept) { alpha[k] = 0.f; continue; }
                        if (sPos[t] >= 0) continue;
                        const float *q = sE + t;
                        const float4 A = make_float4(q[0], q[kThreadsC], q[2 * kThreadsC], q[3 * kThreadsC]);
                        const float4 B = make_float4(q[4 * kThreadsC], q[5 * kThreadsC], q[6 * kThreadsC], q[7 * kThreadsC]);
                        const PointFootprint f = point_footprint(A, B, roll, px, py);
                        const float a = fminf(kAlphaMax, B.w * f.vis), x = f.dx, y = f.dy;
                        alpha[k] = f.sigma < 0.f || a < kAlphaMin ? 0.f : a;
                        if (k & 1) { dx[k / 2].y = x; dy[k / 2].y = y; } else { dx[k / 2].x = x; dy[k / 2].x = y; }
                    }
                }
                left = make_float4(1.f - alpha[0], 1.f - alpha[1], 1.f - alpha[2], 1.f - alpha[3]);
            }
            sLeft[buffer][warp][lane] = left;
            if (c0 == 0) async_wait_all();   // the features
            __syncthreads();
            float before = T_run;
#pragma unroll
            for (uint32_t w = 0; w < kCoopWarps; ++w) {
                const float4 l = sLeft[buffer][w][lane];
                if (w == warp) before = T_run;
                T_run = T_run * l.x * l.y * l.z * l.w;
            }
            buffer ^= 1u;
            finished = __all_sync(0xffffffffu, T_run <= kTStop);
            if (!mine) continue;
            // weights; what is not blended has none, and leaves nothing else behind
            const auto four = [&](uint32_t k) { return *reinterpret_cast<const float4 *>(sE + k * kThreadsC + t0); };
            const float4 RV = four(8), DX = four(9), DY = four(10), R = four(11);
            float vis[kCoopShare];
#pragma unroll
            for (uint32_t k = 0; k < kCoopShare; ++k) {
                const auto of = [&](const float4 &v) { return k == 0 ? v.x : k == 1 ? v.y : k == 2 ? v.z : v.w; };
                const float next_T = before * of(left);
                const bool take = alpha[k] > 0.f && next_T > kTStop;
                const float x = k & 1 ? dx[k / 2].y : dx[k / 2].x, y = k & 1 ? dy[k / 2].y : dy[k / 2].x;
                const float d = fmaf(of(DX), x, fmaf(of(DY), y, of(RV) * roll));
                vis[k] = take ? alpha[k] * before : 0.f;
                depth_extra = fmaf(take ? d : 0.f, vis[k], depth_extra);
                if (take && before > 0.5f && next_T <= 0.5f) median = of(R) + d;
                if (compute_alpha_sum && take && of(R) < alpha_sum_limit) alpha_sum += alpha[k];
                if (take) cur_idx = k == 0 ? at.x : k == 1 ? at.y : k == 2 ? at.z : at.w;
                if (take) T = next_T;
                before = next_T;
            }
#pragma unroll
            for (uint32_t k = 0; k < kCoopShare; ++k)
                if (vis[k] > 0.f) axpy_staged_full<CDIM>(pix_out, sFeat + (t0 + k) * CDIM, vis[k]);   // a branch: elsewhere it would be 0 * inf
        }
    }
    cur_idx &= INT32_MAX;
    async_wait_all();
    // partial sums of the warps, added in order
    __syncthreads();
    float *parts = reinterpret_cast<float *>(smem_raw);   // [warps][32][CDIM]
#pragma unroll
    for (int k = 0; k < CDIM; k += 4)
        *reinterpret_cast<float4 *>(parts + (warp * 32 + lane) * CDIM + k) =
            make_float4(pix_out[k], pix_out[k + 1], pix_out[k + 2], pix_out[k + 3]);
    float *s_T = parts + kCoopWarps * 32 * CDIM, *s_extra = s_T + kCoopWarps * 32, *s_sum = s_extra + kCoopWarps * 32,
          *s_median = s_sum + kCoopWarps * 32;   // [warps][32] each
    int32_t *s_last = reinterpret_cast<int32_t *>(s_median + kCoopWarps * 32);
    s_T[tr] = T;
    s_extra[tr] = depth_extra;
    s_sum[tr] = alpha_sum;
    s_median[tr] = median;
    float none = fmaf(depth_extra, 0.f, 0.f);   // a NaN: see odd_points_bwd()
#pragma unroll
    for (int k = 0; k < CDIM; ++k) none = fmaf(pix_out[k], 0.f, none);
    s_last[tr] = none != 0.f ? cur_idx | kOddPixel : cur_idx;
    __syncthreads();
    // the last transmittance and the last entry are the smallest and the largest of the warps'; the median
    // was met by one warp alone
    T = s_T[lane]; depth_extra = s_extra[lane]; alpha_sum = s_sum[lane]; median = s_median[lane]; cur_idx = s_last[lane];
    int32_t mark = cur_idx & kOddPixel;
    cur_idx = last_position(cur_idx);
#pragma unroll
    for (uint32_t w = 1; w < kCoopWarps; ++w) {
        T = fminf(T, s_T[w * 32 + lane]);
        depth_extra += s_extra[w * 32 + lane];
        alpha_sum += s_sum[w * 32 + lane];
        median += s_median[w * 32 + lane];
        mark |= s_last[w * 32 + lane] & kOddPixel;
        cur_idx = max(cur_idx, last_position(s_last[w * 32 + lane]));
    }
    if (warp == 0 && in_image) {
        // points that are not rendered (range <= 0) produce zeros everywhere
        render_alphas[pix] = inside ? 1.f - T : 0.f;
        last_ids[pix] = inside ? cur_idx | mark : 0;
        median_depths[pix] = inside ? median : 0.f;
        if (alpha_sum_out != nullptr) alpha_sum_out[pix] = inside ? alpha_sum : 0.f;
    }
    const float *bg = backgrounds ? backgrounds + (size_t)cam * channels : nullptr;
    for (uint32_t k = warp; k < channels; k += kCoopWarps) {
        float v = 0.f;
#pragma unroll
        for (uint32_t w = 0; w < kCoopWarps; ++w) v += parts[(w * 32 + lane) * CDIM + k];
        if (k == depth_idx) v += depth_extra;
        if (bg) v += T * bg[k];
        if (in_image) render_colors[pix * channels + k] = inside ? v : 0.f;
    }
}

// ---------------------------------------------------------------------------------------
// Backward helpers
// ---------------------------------------------------------------------------------------
__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
    return v;
}

// Sums N <= 32 per-lane values over the warp at once: every step pairs the first half of the values a lane
// carries with the second, keeps one of each pair and swaps the other with the partner lane; an odd value
// out is summed on both sides. 12 values take 48 instructions where one butterfly per value takes 120 (and
// padding them to 16 62). sum_slot() says which value's total a lane ends up with, and which of the lanes
// that hold the same one writes it. Call with kOff = 16.
template <int N, int kOff>
__device__ __forceinline__ float warp_sum_values(const float (&v)[N], uint32_t lane) {
    constexpr int kPairs = N / 2, kNext = kPairs + (N & 1);
    const bool upper = (lane & (uint32_t)kOff) != 0u;
    float next[kNext];
    if (N & 1) next[kPairs] = v[N - 1] + __shfl_xor_sync(0xffffffffu, v[N - 1], kOff);
#pragma unroll
    for (int i = 0; i < kPairs; ++i) {
        const float send = upper ? v[i] : v[i + kPairs], keep = upper ? v[i + kPairs] : v[i];
        next[i] = keep + __shfl_xor_sync(0xffffffffu, send, kOff);
    }
    if constexpr (kOff > 1) return warp_sum_values<kNext, kOff / 2>(next, lane);
    else return next[0];
}

struct SumSlot { int value; bool writes; };

template <int N>
__device__ __forceinline__ SumSlot sum_slot(uint32_t lane) {
    // backwards through the steps: place 0 of the last one is which place of the first?
    int sizes[6] = {N, 0, 0, 0, 0, 0};
#pragma unroll
    for (int s = 0; s < 5; ++s) sizes[s + 1] = sizes[s] / 2 + (sizes[s] & 1);
    SumSlot r = {0, true};
#pragma unroll
    for (int s = 4; s >= 0; --s) {
        const int pairs = sizes[s] / 2;
        const bool upper = (lane & (16u >> s)) != 0u;
        if (r.value == pairs) { r.value = sizes[s] - 1; r.writes = r.writes && !upper; }   // the odd one out (or the only one)
        else if (upper) r.value += pairs;
    }
    return r;
}

// What a lane does with the warp total it ends up holding: which array it belongs to, and the factor
// common to all samples (times one of the entry's own, see the kernels).
struct GradSlot {
    float *base;
    uint32_t stride;
    float scale;
    bool times_factor;
    __device__ __forceinline__ void add(size_t g, float total, float factor, bool writes) const {
        const float v = total * (times_factor ? scale * factor : scale);
        if (writes && base != nullptr && v != 0.f) atomicAdd(base + g * stride, v);
    }
};

template <bool kAbs>
__device__ __forceinline__ GradSlot pixel_grad_slot(int slot, int cdim, uint32_t channels, float *v_colors,
                                                    float *v_conics, float *v_means2d, float *v_pix_vels,
                                                    float *v_opacities, float *v_means2d_abs) {
    if (slot < cdim) return {(uint32_t)slot < channels ? v_colors + slot : nullptr, channels, 1.f, false};
    switch (slot - cdim) {
        case 0: return {v_conics, 3u, -0.5f, false};
        case 1: return {v_conics + 1, 3u, -1.f, false};
        case 2: return {v_conics + 2, 3u, -0.5f, false};
        case 3: return {v_means2d, 2u, kLn2, false};
        case 4: return {v_means2d + 1, 2u, kLn2, false};
        case 5: return {v_pix_vels, 2u, kLn2, false};
        case 6: return {v_pix_vels + 1, 2u, kLn2, false};
        case 7: return {v_opacities, 1u, 1.f, true};   // by the opacity
        case 8: return {kAbs ? v_means2d_abs : nullptr, 2u, kLn2, false};
        case 9: return {kAbs ? v_means2d_abs + 1 : nullptr, 2u, kLn2, false};
        default: return {nullptr, 0u, 0.f, false};
    }
}

// ---------------------------------------------------------------------------------------
// Camera backward: back to front from the last entry any pixel of the patch consumed; patches as in the forward kernel.
//
// What bounds it is instruction issue, the FP32 pipe at half its rate, and sixteen warps an SM to hide the way from the
// exponentials through the reciprocals to the sums. The parts that do not depend on the pixel - the butterflies above all -
// were most of it with one pixel per thread; eight pixels of a row (four above four channels, two above sixteen) add their
// terms up before anything is exchanged, and as dy and the row's shutter time are common to them the geometry needs only
// the sums of v, v dx and v dx^2 (v = alpha dL/dalpha; the opacity's own derivative is the first of them by the opacity). The
// channels behind an entry enter through one number per pixel: dL/dalpha = T (c . g) - (1 / (1 - alpha)) (sum over
// the entries behind of their weight times their (c . g)), g the pixel's cotangent - a running scalar in place of a running
// colour. A pixel lies far out until its last entry comes, which takes a look at few entries of a list instead of a
// comparison per pixel and entry. The pairs are worked through in one straight line: a branch for the entries that need
// care between them costs 7 us.
// 1920 x 1080, 4 channels: 323 M -> 200 M warp instructions, 385 -> 305 us (four pixels 347); 16 channels and absolute
// gradients, 1237 x 719: 445 -> 374 (1920 x 1080 without: 4, 8, 13, 20 and 32 channels 385, 477, 827, 911, 1914 -> 305, 474, 676, 815, 1869;
// 640 x 360, two pixels: 150, 164, 155, 168, 297 -> 113, 124, 153, 160, 305). Sums through shared memory instead of butterflies: 361; asynchronous copies
// of the next batches: 9 us more. The atomics cost 14 us, the butterflies 40.
// ---------------------------------------------------------------------------------------
// The other variant of a kernel, for the cases that other registers or a skip suit better; pixels_bwd_other() chooses.
//   Four pixels per lane, up to 8 channels, splats of a few tiles: entries that no pixel blends - behind the last of
//   those they reach - are left before the sums. 1920 x 1080, 4 / 8 channels, 5.4 tiles per Gaussian 442 / 563 -> 415 / 532 us; 12.7
//   tiles 362 / 506 -> 371 / 512.
//   Two pixels, 9 to 16 channels, many tiles: 96 registers. 1920 x 1080, 2.5 and 27.5 tiles per Gaussian 442, 875 -> 404, 834; 640 x 360,
//   5.1 tiles 153 -> 158.
//   Up to sixteen channels, scenes of large Gaussians (kRunsBwd, chosen as in the forward kernel): what is staged moves up to the front, so that
// entries that cover the patch follow one another without a look at a mask, a threshold or a pixel's first entry - the place of the next one is known -,
// two at a time up to eight channels with one butterfly for their 24 or 32 sums, whose five steps are the longest chain there is. 4 channels: 200 M -> 180 M warp
// instructions, 1920 x 1080 305 -> 287 us, three cameras 366 -> 335; 8 channels 475 -> 448 and 475 -> 438; 14 channels, one at a time, 682 -> 661 and 683 -> 650. Neither more warps (96 registers, the cotangents in shared memory: 20 an SM, 344) nor fewer (one entry at a time
// with 128 registers, 16: 337) nor the order of the additions helps: at 12 warps an SM the FP32 pipe is busy 55 % of the time, the
// exponentials and reciprocals (8 cycles each) 30 %, shuffles (4 cycles an SM) 25 %.
//   Above 20 channels, few tiles: the chain of the longest list counts, so no spills, whole rows at once and the skip. 640 x 360, 32
//   channels, scales of 1, 0.6, 0.3 and 0.1: 326, 346, 244, 205 -> 303, 332, 236, 199; 1920 x 1080: 1862 -> 1999.
constexpr bool has_other_bwd(int cdim, int px) { return (px == 4 && cdim <= 8) || (px == 2 && cdim == 16) || cdim == 32; }
constexpr bool pixels_bwd_skips(int cdim, int px, bool other) { return other && cdim != 16; }

// registers per thread, by measurement (4 channels, eight pixels: 335 us at 128, 348 at 112, 361 at 144; 16 channels:
// 386 at 168, 394 at 128; 8: 483 at 96, 520 at 128; 20, four pixels: 847 at 168, 980 at 200; 32: 1950 at 128, 2075 at 160)
constexpr int kPlainBwd = 0, kOtherBwd = 1, kRunsBwd = 2;
constexpr bool has_runs_bwd(int cdim, int px) { return px == 8 || (px == 4 && cdim > 4 && cdim <= 16); }
constexpr int pixels_bwd_regs(int cdim, int px, int kind) {
    const bool other = kind == kOtherBwd;
    if (kind == kRunsBwd) return px == 4 && cdim <= 8 ? 128 : 168;
    return cdim <= 4 ? (px == 8 ? 128 : px == 4 ? 80 : 72) : cdim <= 8 ? (px == 4 ? 96 : 88) : cdim <= 16 ? (px == 4 ? 168 : other ? 96 : 104)
                     : cdim <= 20 ? 168 : other ? 168 : 128;
}

template <int CDIM, int PX, bool kAbs, int kKind>
__global__ void __maxnreg__(pixels_bwd_regs(CDIM, PX, kKind))
rasterize_to_pixels_bwd_kernel(
    uint32_t C, int64_t n_isects, const float2 *__restrict__ means2d,
    const float *__restrict__ conics, const float *__restrict__ colors, uint32_t channels,
    const float *__restrict__ opacities, const float2 *__restrict__ pix_vels,
    const float *__restrict__ rs_time, const float *__restrict__ backgrounds, uint32_t W,
    uint32_t H, uint32_t tile_size, uint32_t tile_w, uint32_t tile_h, uint32_t patches /* of a tile */,
    const int32_t *__restrict__ offsets, const int32_t *__restrict__ flatten_ids,
    const float *__restrict__ render_alphas, const int32_t *__restrict__ last_ids,
    const float *__restrict__ v_render_colors, const float *__restrict__ v_render_alphas,
    float *__restrict__ v_means2d_abs, float *__restrict__ v_means2d,
    float *__restrict__ v_conics, float *__restrict__ v_colors, float *__restrict__ v_opacities,
    float *__restrict__ v_pix_vels, const float *__restrict__ expected /* [C,H,W] last channel, where it was divided by the alpha */) {
    chain_enter();
    static_assert(PX % 2 == 0, "pixels are handled in pairs");
    constexpr int P2 = PX / 2;
    constexpr bool kOther = kKind == kOtherBwd, kRuns = kKind == kRunsBwd;
    __shared__ float4 sA[32];                // x, y, vx, vy
    __shared__ float4 sB[32];                // scaled conic, opacity
    __shared__ float4 sCol[32 * CDIM / 4];   // zeros behind the channels
    __shared__ float2 sId[32];               // Gaussian, 1 / opacity
    __shared__ int32_t sLast[PX][32];        // last list positions of the lanes' pixels

    const uint32_t tiles_per_cam = tile_w * tile_h;
    const uint32_t gtile = blockIdx.x / patches, cam = gtile / tiles_per_cam;
    const uint32_t tile = gtile - cam * tiles_per_cam;
    const uint32_t ty = tile / tile_w, tx = tile - ty * tile_w;
    uint32_t lane = threadIdx.x;
    if constexpr (kRuns) lane = lane_index();
    const uint32_t tr = (blockIdx.x - gtile * patches) * 32u + lane;
    const TilePixels<PX> tp = tile_pixels<PX>(tile_size, tr);
    const uint32_t i = ty * tile_size + tp.y, j = tx * tile_size + tp.x;
    uint32_t n_inside = 0;   // pixels of this thread inside the tile and the image
    if (tp.y < tile_size && i < H && j < W) n_inside = min(min((uint32_t)PX, tile_size - tp.x), W - j);
    const float px0 = (float)j + 0.5f, py = (float)i + 0.5f;
    const float rs = rs_time[cam];
    const float roll = rs * ((py - 0.5f) / (float)(H - 1) - 0.5f);
    // shutter times of the tile's first and last row
    const float roll_a = rs * ((float)(ty * tile_size) / (float)(H - 1) - 0.5f);
    const float roll_b = rs * ((float)(min((ty + 1) * tile_size, H) - 1) / (float)(H - 1) - 0.5f);
    const float roll_lo = fminf(roll_a, roll_b), roll_hi = fmaxf(roll_a, roll_b);
    const PatchBox box = warp_box(px0, py, n_inside);

    const TileRange range = tile_range(offsets, gtile, C * tiles_per_cam, n_isects);
    const bool vec = (channels % 4u == 0u) && ((reinterpret_cast<uintptr_t>(colors) & 15u) == 0u);

    float2 npx[P2];                  // minus the columns; far out before a pixel's last entry has come
    float2 T[P2], behind[P2];        // transmittance in front of the entry; weighted (c . g) behind it
    float2 v_out[CDIM][P2];          // cotangents of the pixels' channels
    int32_t thread_last = -1;
    float none = 0.f;                // a NaN: see odd_pixels_bwd()
    {
        const size_t pix = ((size_t)cam * H + (n_inside ? i : 0u)) * W + (n_inside ? j : 0u);
        float a_final[PX], v_a[PX], depths[PX], v[PX][CDIM];
        int32_t last[PX];
        load_pixels<PX>(a_final, render_alphas + pix, n_inside, 0.f);
        load_pixels<PX>(v_a, v_render_alphas + pix, n_inside, 0.f);
        load_pixels<PX>(last, last_ids + pix, n_inside, -1);
        load_channels<CDIM, PX>(v, v_render_colors + pix * channels, channels, n_inside);
        if (expected != nullptr) load_pixels<PX>(depths, expected + pix, n_inside, 0.f);
#pragma unroll
        for (int k = 0; k < PX; ++k) {
            const bool in = (uint32_t)k < n_inside;
            const float T_final = 1.f - a_final[k], divisor = fmaxf(a_final[k], kExpectedMin);
            thread_last = (in && last[k] < 0) ? INT32_MAX : max(thread_last, last[k]);
            sLast[k][lane] = last[k];
            float bg_dot = 0.f;
#pragma unroll
            for (int c = 0; c < CDIM; ++c) {
                if (expected != nullptr && (uint32_t)c + 1u == channels) {
                    if (in && a_final[k] >= kExpectedMin) v_a[k] -= v[k][c] * depths[k] / divisor;
                    v[k][c] /= divisor;
                }
                if (backgrounds != nullptr && (uint32_t)c < channels) bg_dot += backgrounds[(size_t)cam * channels + c] * v[k][c];
                none = fmaf(v[k][c], 0.f, none);
                if (k & 1) v_out[c][k / 2].y = v[k][c]; else v_out[c][k / 2].x = v[k][c];
            }
            // what the background and the alpha output receive through everything in front of them
            const float to_last = -T_final * (v_a[k] - bg_dot);
            none = fmaf(to_last, 0.f, none);
            if (k & 1) { T[k / 2].y = T_final; behind[k / 2].y = to_last; npx[k / 2].y = -kPixelGone; }
            else { T[k / 2].x = T_final; behind[k / 2].x = to_last; npx[k / 2].x = -kPixelGone; }
        }
    }

    // last list position consumed by any pixel of the patch
    const int32_t warp_last = __reduce_max_sync(0xffffffffu, none != 0.f ? INT32_MAX : thread_last);
    if (warp_last == INT32_MAX) {
        const PixelTask task = {C, W, H, tile_size, tile_w, tile_h, channels, n_isects, means2d, pix_vels, conics, opacities,
                                colors, rs_time, backgrounds, offsets, flatten_ids};
        const PixelGrads grads = {render_alphas, v_render_colors, v_render_alphas, expected, last_ids, v_means2d,
                                  kAbs ? v_means2d_abs : nullptr, v_conics, v_colors, v_opacities, v_pix_vels};
        odd_pixels_bwd<PX>(task, gtile, tr, grads);
        return;
    }
    const int32_t eff_end = min(range.end, warp_last + 1);

    // Where the warp total that ends up on this lane goes: colours first, then the geometry.
    constexpr int kGeo = kAbs ? 10 : 8;
    constexpr bool kSplit = CDIM + kGeo > 32;   // the geometry in a butterfly of its own
    constexpr int kSums = kSplit ? CDIM : CDIM + kGeo;
    const SumSlot mine_a = sum_slot<kSums>(lane);
    const GradSlot slot_a = pixel_grad_slot<kAbs>(mine_a.value, CDIM, channels, v_colors,
                                                  v_conics, v_means2d, v_pix_vels, v_opacities, v_means2d_abs);

    if constexpr (kRuns) {
        int32_t next_id = 0;
        if (eff_end - 1 - (int32_t)lane >= range.start) next_id = flatten_ids[eff_end - 1 - (int32_t)lane];
        constexpr uint32_t kEntry = 2 + CDIM / 4;
        __shared__ float4 sEntry[32 * kEntry];   // x, y, vx, vy | scaled conic, opacity | channels, zeros behind them
        // two entries' sums: colours and geometry of the first, then of the second
        constexpr bool kTwo = 2 * kSums <= 32;
        const SumSlot mine_two = sum_slot<kTwo ? 2 * kSums : kSums>(lane);
        const uint32_t two_entry = mine_two.value >= kSums ? 1u : 0u;
        const GradSlot slot_two = pixel_grad_slot<kAbs>(mine_two.value - (two_entry ? kSums : 0), CDIM, channels, v_colors, v_conics, v_means2d,
                                                        v_pix_vels, v_opacities, v_means2d_abs);
        int32_t event = warp_last;   // the next entry that is any pixel's last one
        for (int32_t batch_end = eff_end - 1; batch_end >= range.start; batch_end -= 32) {
            const int32_t idx = batch_end - (int32_t)lane;
            const int32_t g = next_id;
            uint32_t seen = 0u;
            float most;
            PixelEntry e;
            if (idx >= range.start) {
                e = load_pixel_entry(g, means2d, conics, opacities, pix_vels);
                if (idx - 32 >= range.start) next_id = flatten_ids[idx - 32];   // on its way meanwhile
                seen = patch_covered<false>(e, box, roll_lo, roll_hi, most);
            }
            const uint32_t kept = __ballot_sync(0xffffffffu, seen != 0u), n = __popc(kept);
            const uint32_t place = __popc(kept & ((1u << lane) - 1u));
            const uint32_t full = __reduce_or_sync(0xffffffffu, (seen & kFullEntry) ? 1u << place : 0u);
            const uint32_t careful = __reduce_or_sync(0xffffffffu, (seen & kCarefulEntry) ? 1u << place : 0u);
            __syncwarp();   // the batch before has been read
            if (seen) {
                float4 *entry = sEntry + place * kEntry;
                entry[0] = e.A;
                entry[1] = scaled_conic(e.B);
                sId[place] = make_float2(__int_as_float(g), 1.f / e.B.w);
                stage_whole_row<CDIM, true>(entry + 2, colors + (size_t)g * channels, channels, vec);
            }
            __syncwarp();
            // kCount entries in sequence, whose sums share a butterfly; kFull: they cover the patch
            const auto process = [&](uint32_t t, auto count, auto covers) {
                constexpr int kCount = decltype(count)::value;
                constexpr bool kFull = decltype(covers)::value;
                float4 A[kCount], B[kCount], col[kCount][CDIM / 4];
                float mx[kCount], dy[kCount];
                float2 alpha[kCount][P2];
                uint32_t capped = 0u;   // pixels with a capped alpha, which passes no gradient on to the geometry
#pragma unroll
                for (int h = 0; h < kCount; ++h) {
                    const float4 *entry = sEntry + (t + h) * kEntry;
                    A[h] = entry[0];
                    B[h] = entry[1];
                    mx[h] = A[h].x + roll * A[h].z;
                    dy[h] = A[h].y + roll * A[h].w - py;
                    const float bdy = B[h].y * dy[h], cdy2 = B[h].z * dy[h] * dy[h];
#pragma unroll
                    for (int q = 0; q < P2; ++q) {
                        const float2 pw = pair_power(B[h].x, __fadd2_rn(make_float2(mx[h], mx[h]), npx[q]), bdy, cdy2);
                        alpha[h][q] = __fmul2_rn(make_float2(B[h].w, B[h].w), make_float2(exp2_approx(pw.x), exp2_approx(pw.y)));
                        if (!kFull) alpha[h][q] = make_float2(alpha[h][q].x >= kAlphaMin ? alpha[h][q].x : 0.f, alpha[h][q].y >= kAlphaMin ? alpha[h][q].y : 0.f);
                    }
                    if (!kFull && ((careful >> t) & 1u)) {
#pragma unroll
                        for (int q = 0; q < P2; ++q) {
                            const float2 pw = pair_power(B[h].x, __fadd2_rn(make_float2(mx[h], mx[h]), npx[q]), bdy, cdy2);
                            if (alpha[h][q].x > kAlphaMax) capped |= 1u << (2 * q);
                            if (alpha[h][q].y > kAlphaMax) capped |= 2u << (2 * q);
                            alpha[h][q].x = pw.x <= 0.f ? fminf(kAlphaMax, alpha[h][q].x) : 0.f;
                            alpha[h][q].y = pw.y <= 0.f ? fminf(kAlphaMax, alpha[h][q].y) : 0.f;
                        }
                    }
#pragma unroll
                    for (int c = 0; c < CDIM / 4; ++c) col[h][c] = entry[2 + c];
                }
                float2 csum[kCount][CDIM], s0[kCount], s1[kCount], s2[kCount], ax[kCount], ay[kCount];
#pragma unroll
                for (int q = 0; q < P2; ++q)
#pragma unroll
                    for (int h = 0; h < kCount; ++h) {
                        const float2 ra = reciprocal_pair(__fadd2_rn(make_float2(1.f, 1.f), make_float2(-alpha[h][q].x, -alpha[h][q].y)));
                        T[q] = __fmul2_rn(T[q], ra);
                        const float2 fac = __fmul2_rn(alpha[h][q], T[q]);
                        float2 dot = make_float2(0.f, 0.f);   // (c . g) of the two pixels
#pragma unroll
                        for (int k = 0; k < CDIM; ++k) {
                            const float4 c4 = col[h][k / 4];
                            const float c = (k & 3) == 0 ? c4.x : (k & 3) == 1 ? c4.y : (k & 3) == 2 ? c4.z : c4.w;
                            dot = k == 0 ? __fmul2_rn(make_float2(c, c), v_out[k][q]) : __ffma2_rn(make_float2(c, c), v_out[k][q], dot);
                            csum[h][k] = q == 0 ? __fmul2_rn(fac, v_out[k][q]) : __ffma2_rn(fac, v_out[k][q], csum[h][k]);
                        }
                        const float2 v_alpha = __ffma2_rn(T[q], dot, __fmul2_rn(make_float2(-ra.x, -ra.y), behind[q]));
                        behind[q] = __ffma2_rn(fac, dot, behind[q]);
                        float2 v = __fmul2_rn(alpha[h][q], v_alpha);
                        if (!kFull) {
                            if (capped & (1u << (2 * q))) v.x = 0.f;
                            if (capped & (2u << (2 * q))) v.y = 0.f;
                        }
                        const float2 dx = __fadd2_rn(make_float2(mx[h], mx[h]), npx[q]), vx = __fmul2_rn(v, dx);
                        s0[h] = q == 0 ? v : __fadd2_rn(s0[h], v);
                        s1[h] = q == 0 ? vx : __fadd2_rn(s1[h], vx);
                        s2[h] = q == 0 ? __fmul2_rn(vx, dx) : __ffma2_rn(vx, dx, s2[h]);
                        if (kAbs) {   // (v first: a pixel that is far out must not meet a conic of any size)
                            const float bdy = B[h].y * dy[h], cdy = 2.f * B[h].z * dy[h];
                            const float2 gx = __ffma2_rn(make_float2(2.f * B[h].x, 2.f * B[h].x), vx, __fmul2_rn(make_float2(bdy, bdy), v));
                            const float2 gy = __ffma2_rn(make_float2(B[h].y, B[h].y), vx, __fmul2_rn(make_float2(cdy, cdy), v));
                            const float2 bx = make_float2(fabsf(gx.x), fabsf(gx.y)), by = make_float2(fabsf(gy.x), fabsf(gy.y));
                            ax[h] = q == 0 ? bx : __fadd2_rn(ax[h], bx);
                            ay[h] = q == 0 ? by : __fadd2_rn(ay[h], by);
                        }
                    }
                float sums[kCount * kSums];
#pragma unroll
                for (int h = 0; h < kCount; ++h) {
                    float *sum = sums + h * kSums;
#pragma unroll
                    for (int k = 0; k < CDIM; ++k) sum[k] = csum[h][k].x + csum[h][k].y;
                    const float m0 = s0[h].x + s0[h].y, m1 = s1[h].x + s1[h].y, my = dy[h] * m0;
                    const float gx = 2.f * B[h].x * m1 + B[h].y * my, gy = B[h].y * m1 + 2.f * B[h].z * my;
                    sum[CDIM + 0] = s2[h].x + s2[h].y;
                    sum[CDIM + 1] = dy[h] * m1;
                    sum[CDIM + 2] = dy[h] * my;
                    sum[CDIM + 3] = gx;
                    sum[CDIM + 4] = gy;
                    sum[CDIM + 5] = gx * roll;
                    sum[CDIM + 6] = gy * roll;
                    sum[CDIM + 7] = m0;
                    if (kAbs) {
                        sum[CDIM + 8] = ax[h].x + ax[h].y;
                        sum[CDIM + 9] = ay[h].x + ay[h].y;
                    }
                }
                const float2 id = sId[kCount == 1 ? t : t + two_entry];
                const float total = warp_sum_values<kCount * kSums, 16>(sums, lane);
                if (kCount == 1) slot_a.add((size_t)__float_as_int(id.x), total, id.y, mine_a.writes);
                else slot_two.add((size_t)__float_as_int(id.x), total, id.y, mine_two.writes);
            };
            // the first place at which a pixel of the warp takes part
            const auto next_event = [&](uint32_t t) {
                const uint32_t due = __ballot_sync(0xffffffffu, seen && place >= t && idx <= event);
                return due ? (uint32_t)__popc(kept & ((due & (0u - due)) - 1u)) : n;
            };
            uint32_t t = 0, t_event = next_event(0);
            while (t < n) {
                if (t == t_event) {
                    const int32_t entry = __shfl_sync(0xffffffffu, idx, __ffs(__ballot_sync(0xffffffffu, seen && place == t)) - 1);
                    int32_t next = -1;
#pragma unroll
                    for (int k = 0; k < PX; ++k) {
                        const int32_t last = sLast[k][lane];
                        if (entry <= last) {
                            if (k & 1) npx[k / 2].y = -(px0 + (float)k); else npx[k / 2].x = -(px0 + (float)k);
                        } else next = max(next, last);
                    }
                    event = __reduce_max_sync(0xffffffffu, next);
                    t_event = next_event(t + 1u);
                }
                const uint32_t rest = ~full >> t, end = min(t_event, rest ? t + (uint32_t)__ffs(rest) - 1u : n);
                if constexpr (kTwo)
                    for (; t + 1u < end; t += 2u) process(t, std::integral_constant<int, 2>(), std::true_type());
                for (; t < end;) process(t++, std::integral_constant<int, 1>(), std::true_type());
                if (t < t_event && t < n) process(t++, std::integral_constant<int, 1>(), std::false_type());
            }
        }
    } else {
        constexpr bool kSkip = pixels_bwd_skips(CDIM, PX, kOther);
        int32_t waiting = thread_last;   // position of the next entry that is a pixel's of this lane last one; -1: none
        bool pending = true;             // a lane of the warp waits for one
        int32_t next_id = 0;
        if (eff_end - 1 - (int32_t)lane >= range.start) next_id = flatten_ids[eff_end - 1 - (int32_t)lane];
        for (int32_t batch_end = eff_end - 1; batch_end >= range.start; batch_end -= 32) {
            const int32_t idx = batch_end - (int32_t)lane;
            const int32_t g = next_id;
            uint32_t seen = 0u;
            PixelEntry e;
            if (idx >= range.start) {
                e = load_pixel_entry(g, means2d, conics, opacities, pix_vels);
                if (idx - 32 >= range.start) next_id = flatten_ids[idx - 32];   // on its way meanwhile
                seen = patch_sees<false>(e, box, roll_lo, roll_hi);
            }
            uint32_t todo = __ballot_sync(0xffffffffu, seen != 0u);
            const uint32_t careful = __ballot_sync(0xffffffffu, (seen & kCarefulEntry) != 0u);
            __syncwarp();   // the batch before has been read
            if (seen) {
                sA[lane] = e.A;
                sB[lane] = scaled_conic(e.B);
                sId[lane] = make_float2(__int_as_float(g), 1.f / e.B.w);
                // A colour that is not finite is blended by no pixel of the patch - it would have left its mark there. It may lie
                // behind the last entry of some pixels and out of reach of the others, and must not meet their weights of zero.
                if (CDIM <= 16 || (CDIM == 32 && kOther)) stage_whole_row<CDIM, true>(sCol + lane * (CDIM / 4), colors + (size_t)g * channels, channels, vec);
                else {   // (20 channels: all loads of a row at once take registers, 990 -> 1130 us)
                    float *row = reinterpret_cast<float *>(sCol) + lane * CDIM;
                    stage_row<true>(row, colors, (size_t)g, channels, vec);
                    for (uint32_t k = (channels + 3u) & ~3u; k < (uint32_t)CDIM; ++k) row[k] = 0.f;
                }
            }
            __syncwarp();
            while (todo) {
                const uint32_t t = (uint32_t)__ffs(todo) - 1u, bit = 1u << t;
                todo ^= bit;
                const int32_t entry = batch_end - (int32_t)t;
                if (pending && __any_sync(0xffffffffu, entry <= waiting)) {
                    // pixels whose last entry this is, or lay behind it: they take part from here on
                    int32_t next = -1;
#pragma unroll
                    for (int k = 0; k < PX; ++k) {
                        const int32_t last = sLast[k][lane];
                        if (entry <= last) {
                            if (k & 1) npx[k / 2].y = -(px0 + (float)k); else npx[k / 2].x = -(px0 + (float)k);
                        } else next = max(next, last);
                    }
                    waiting = next;
                    pending = __any_sync(0xffffffffu, waiting >= 0);
                }
                const float4 A = sA[t], B = sB[t];
                const float mx = A.x + roll * A.z, dy = A.y + roll * A.w - py;
                const float bdy = B.y * dy, cdy2 = B.z * dy * dy;
                float4 col[CDIM / 4];
#pragma unroll
                for (int k = 0; k < CDIM / 4; ++k) col[k] = sCol[t * (CDIM / 4) + k];
                float2 alpha[P2], v[P2], csum[CDIM];
#pragma unroll
                for (int q = 0; q < P2; ++q) {
                    const float2 pw = pair_power(B.x, __fadd2_rn(make_float2(mx, mx), npx[q]), bdy, cdy2);
                    const float2 av = __fmul2_rn(make_float2(B.w, B.w), make_float2(exp2_approx(pw.x), exp2_approx(pw.y)));
                    alpha[q] = make_float2(av.x >= kAlphaMin ? av.x : 0.f, av.y >= kAlphaMin ? av.y : 0.f);
                }
                uint32_t capped = 0u;   // pixels with a capped alpha, which passes no gradient on to the geometry
                if (careful & bit) {
#pragma unroll
                    for (int q = 0; q < P2; ++q) {
                        const float2 pw = pair_power(B.x, __fadd2_rn(make_float2(mx, mx), npx[q]), bdy, cdy2);
                        if (alpha[q].x > kAlphaMax) capped |= 1u << (2 * q);
                        if (alpha[q].y > kAlphaMax) capped |= 2u << (2 * q);
                        alpha[q].x = pw.x <= 0.f ? fminf(kAlphaMax, alpha[q].x) : 0.f;
                        alpha[q].y = pw.y <= 0.f ? fminf(kAlphaMax, alpha[q].y) : 0.f;
                    }
                }
                if (kSkip) {
                    bool any = false;
#pragma unroll
                    for (int q = 0; q < P2; ++q) any = any || alpha[q].x > 0.f || alpha[q].y > 0.f;
                    if (!__any_sync(0xffffffffu, any)) continue;
                }
#pragma unroll
                for (int q = 0; q < P2; ++q) {
                    const float2 ra = reciprocal_pair(__fadd2_rn(make_float2(1.f, 1.f), make_float2(-alpha[q].x, -alpha[q].y)));
                    T[q] = __fmul2_rn(T[q], ra);
                    const float2 fac = __fmul2_rn(alpha[q], T[q]);
                    float2 dot = make_float2(0.f, 0.f);   // (c . g) of the two pixels
#pragma unroll
                    for (int k = 0; k < CDIM; ++k) {
                        const float4 c4 = col[k / 4];
                        const float c = (k & 3) == 0 ? c4.x : (k & 3) == 1 ? c4.y : (k & 3) == 2 ? c4.z : c4.w;
                        dot = k == 0 ? __fmul2_rn(make_float2(c, c), v_out[k][q]) : __ffma2_rn(make_float2(c, c), v_out[k][q], dot);
                        csum[k] = q == 0 ? __fmul2_rn(fac, v_out[k][q]) : __ffma2_rn(fac, v_out[k][q], csum[k]);
                    }
                    const float2 v_alpha = __ffma2_rn(T[q], dot, __fmul2_rn(make_float2(-ra.x, -ra.y), behind[q]));
                    behind[q] = __ffma2_rn(fac, dot, behind[q]);
                    v[q] = __fmul2_rn(alpha[q], v_alpha);
                }
                if (capped) {
#pragma unroll
                    for (int q = 0; q < P2; ++q) {
                        if (capped & (1u << (2 * q))) v[q].x = 0.f;
                        if (capped & (2u << (2 * q))) v[q].y = 0.f;
                    }
                }
                float2 s0 = make_float2(0.f, 0.f), s1 = s0, s2 = s0, ax = s0, ay = s0;
#pragma unroll
                for (int q = 0; q < P2; ++q) {
                    const float2 dx = __fadd2_rn(make_float2(mx, mx), npx[q]), vx = __fmul2_rn(v[q], dx);
                    s0 = q == 0 ? v[q] : __fadd2_rn(s0, v[q]);
                    s1 = q == 0 ? vx : __fadd2_rn(s1, vx);
                    s2 = q == 0 ? __fmul2_rn(vx, dx) : __ffma2_rn(vx, dx, s2);
                    if (kAbs) {   // (v first: a pixel that is far out must not meet a conic of any size)
                        const float2 gx = __ffma2_rn(make_float2(2.f * B.x, 2.f * B.x), vx, __fmul2_rn(make_float2(bdy, bdy), v[q]));
                        const float2 gy = __ffma2_rn(make_float2(B.y, B.y), vx, __fmul2_rn(make_float2(2.f * B.z * dy, 2.f * B.z * dy), v[q]));
                        ax = __fadd2_rn(ax, make_float2(fabsf(gx.x), fabsf(gx.y)));
                        ay = __fadd2_rn(ay, make_float2(fabsf(gy.x), fabsf(gy.y)));
                    }
                }
                // sigma's derivatives: v_sigma = -v; the factors that are the same for every
                // pixel follow when the totals are written
                float sum[CDIM + kGeo];
#pragma unroll
                for (int k = 0; k < CDIM; ++k) sum[k] = csum[k].x + csum[k].y;
                const float m0 = s0.x + s0.y, m1 = s1.x + s1.y, my = dy * m0;
                const float gx = 2.f * B.x * m1 + B.y * my, gy = B.y * m1 + 2.f * B.z * my;
                sum[CDIM + 0] = s2.x + s2.y;
                sum[CDIM + 1] = dy * m1;
                sum[CDIM + 2] = dy * my;
                sum[CDIM + 3] = gx;
                sum[CDIM + 4] = gy;
                sum[CDIM + 5] = gx * roll;
                sum[CDIM + 6] = gy * roll;
                sum[CDIM + 7] = m0;
                if (kAbs) {
                    sum[CDIM + 8] = ax.x + ax.y;
                    sum[CDIM + 9] = ay.x + ay.y;
                }
                const float2 id = sId[t];
                const size_t gg = (size_t)__float_as_int(id.x);
                float sums[kSums];
#pragma unroll
                for (int k = 0; k < kSums; ++k) sums[k] = sum[k];
                slot_a.add(gg, warp_sum_values<kSums, 16>(sums, lane), id.y, mine_a.writes);
                if (kSplit) {
                    float geo[kGeo];
#pragma unroll
                    for (int k = 0; k < kGeo; ++k) geo[k] = sum[CDIM + k];
                    const float geo_total = warp_sum_values<kGeo, 16>(geo, lane);
                    const SumSlot mine_b = sum_slot<kGeo>(lane);
                    const GradSlot slot_b = pixel_grad_slot<kAbs>(CDIM + mine_b.value, CDIM, channels, v_colors, v_conics,
                                                                  v_means2d, v_pix_vels, v_opacities, v_means2d_abs);
                    slot_b.add(gg, geo_total, id.y, mine_b.writes);
                }
            }
        }
    }
}

// ---------------------------------------------------------------------------------------
// Lidar backward: as the camera's, with two points per thread. Wraps, signs and caps only where an entry needs care, as in the
// forward kernels: 64 x 1083, 8 channels 83 -> 72 us, 17 channels 106 -> 95, 32 x 512 68 -> 58. Every point has its own elevation and time
// offset, so each term is formed per point - in pairs - before the sum over the thread's points goes into
// the warp totals. `behind` also carries the depth compensation of the range channel.
// ---------------------------------------------------------------------------------------
template <bool kAbs>
__device__ __forceinline__ GradSlot point_grad_slot(int slot, int cdim, uint32_t channels, uint32_t fstride, float *v_colors,
                                                    float *v_ranges, float *v_conics, float *v_means2d, float *v_pix_vels,
                                                    float *v_depth_comps, float *v_opacities, float *v_means2d_abs) {
    if (slot < cdim) {
        if ((uint32_t)slot < fstride) return {v_colors + slot, fstride, 1.f, false};
        return {(uint32_t)slot < channels ? v_ranges : nullptr, 1u, 1.f, false};
    }
    switch (slot - cdim) {
        case 0: return {v_conics, 3u, 0.5f, false};
        case 1: return {v_conics + 1, 3u, 1.f, false};
        case 2: return {v_conics + 2, 3u, 0.5f, false};
        case 3: return {v_means2d, 2u, 1.f, false};
        case 4: return {v_means2d + 1, 2u, 1.f, false};
        case 5: return {v_pix_vels, 3u, 1.f, false};
        case 6: return {v_pix_vels + 1, 3u, 1.f, false};
        case 7: return {v_pix_vels + 2, 3u, 1.f, false};
        case 8: return {v_depth_comps, 2u, 1.f, false};
        case 9: return {v_depth_comps + 1, 2u, 1.f, false};
        case 10: return {v_opacities, 1u, 1.f, false};
        case 11: return {kAbs ? v_means2d_abs : nullptr, 2u, 1.f, false};
        case 12: return {kAbs ? v_means2d_abs + 1 : nullptr, 2u, 1.f, false};
        default: return {nullptr, 0u, 0.f, false};
    }
}

// What odd_pixels_bwd() is to cameras: the patch of the calling warp, two points per lane, one after the other.
struct PointTask {
    uint32_t C, W, H, tile_width, tile_height, grid_w, grid_h, ctas_per_tile, channels, depth_idx;
    int64_t n_isects;
    bool alpha_sum;
    float alpha_sum_threshold;
    const float2 *means2d, *depth_comps;
    const float *pix_vels, *conics, *opacities, *colors, *ranges, *backgrounds;
    const float4 *raster_pts;
    const int32_t *offsets, *flatten_ids;
};

struct PointGrads {
    const float *alphas, *v_colors_in, *v_alphas, *v_alpha_sum;
    const int32_t *last_ids;
    float *means2d, *means2d_abs, *conics, *colors, *ranges, *opacities, *pix_vels, *depth_comps;
};

__device__ __noinline__ void odd_points_bwd(const PointTask &a, const PointGrads &grad) {
    const uint32_t n = a.channels, fstride = a.ranges ? n - 1 : n, per_cam = a.grid_w * a.grid_h;
    const uint32_t gtile = blockIdx.x / a.ctas_per_tile, part = blockIdx.x - gtile * a.ctas_per_tile, cam = gtile / per_cam;
    const uint32_t tile = gtile - cam * per_cam, ty = tile / a.grid_w, tx = tile - ty * a.grid_w;
    const TileRange tiles = tile_range(a.offsets, gtile, a.C * per_cam, a.n_isects);
    const PointPatch pp = point_patch<2>(a.tile_width, a.tile_height, part * 32u + (threadIdx.x & 31u));
    for (uint32_t h = 0; h < 2; ++h) {
        uint32_t row = pp.row, col = pp.col + h;
        if (col >= a.tile_width) { col -= a.tile_width; ++row; }
        const uint32_t i = ty * a.tile_height + row, j = tx * a.tile_width + col;
        const size_t pix = ((size_t)cam * a.H + i) * a.W + j;
        float4 pt = make_float4(0.f, 0.f, 0.f, 0.f);
        if (row < a.tile_height && i < a.H && j < a.W) pt = a.raster_pts[pix];
        int32_t last = -1;
        float T = 1.f, behind = 0.f, v_depth = 0.f, v_asum = 0.f;
        const float *v_out = grad.v_colors_in + pix * n;
        if (pt.z > 0.f) {
            last = min(tiles.end - 1, last_position(grad.last_ids[pix]));
            T = 1.f - grad.alphas[pix];
            float bg_dot = 0.f;
            for (uint32_t k = 0; a.backgrounds != nullptr && k < n; ++k) bg_dot += a.backgrounds[(size_t)cam * n + k] * v_out[k];
            behind = -T * (grad.v_alphas[pix] - bg_dot);
            v_depth = v_out[a.depth_idx];
            if (a.alpha_sum && grad.v_alpha_sum != nullptr) v_asum = grad.v_alpha_sum[pix];
        }
        for (int32_t idx = __reduce_max_sync(0xffffffffu, last); idx >= tiles.start; --idx) {
            const size_t g = (size_t)a.flatten_ids[idx];
            const PointEntry e = load_point_entry((int32_t)g, a.means2d, a.conics, a.opacities, a.pix_vels, a.depth_comps);
            const float range = a.ranges ? a.ranges[g] : a.colors[g * n + a.depth_idx];
            const PointFootprint f = point_footprint(e.A, e.B, pt.w, pt.x, pt.y);
            const float alpha = fminf(kAlphaMax, e.B.w * f.vis);
            const bool ok = idx <= last && !(f.sigma < 0.f || alpha < kAlphaMin);
            if (!__any_sync(0xffffffffu, ok)) continue;
            float fac = 0.f, v_alpha = 0.f;
            if (ok) {
                const float ra = 1.f / (1.f - alpha);
                T *= ra;
                fac = alpha * T;
                float dot = (e.C.y * f.dx + e.C.z * f.dy + e.C.x * pt.w) * v_depth;
                for (uint32_t k = 0; k < fstride; ++k) dot = fmaf(a.colors[g * fstride + k], v_out[k], dot);
                if (a.ranges) dot = fmaf(range, v_out[fstride], dot);
                v_alpha = fmaf(T, dot, -ra * behind);
                behind = fmaf(fac, dot, behind);
            }
            for (uint32_t k = 0; k < fstride; ++k) add_warp_total(grad.colors + g * fstride + k, ok ? fac * v_out[k] : 0.f);
            if (a.ranges) add_warp_total(grad.ranges + g, ok ? fac * v_out[fstride] : 0.f);
            float q0 = 0.f, q1 = 0.f, q2 = 0.f, mx = 0.f, my = 0.f, ax = 0.f, ay = 0.f, v_o = 0.f;
            float vd = 0.f, vx = 0.f, vy = 0.f, vz = 0.f, dx = 0.f, dy = 0.f;
            const auto through_sigma = [&](float v, float gx, float gy) {
                const float w = -e.B.w * v;   // dL/dsigma
                const float ux = w * (e.B.x * f.dx + e.B.y * f.dy) + gx, uy = w * (e.B.y * f.dx + e.B.z * f.dy) + gy;
                q0 += 0.5f * w * f.dx * f.dx;
                q1 += w * f.dx * f.dy;
                q2 += 0.5f * w * f.dy * f.dy;
                mx += ux;
                my += uy;
                vx = mx * pt.w;
                vy = my * pt.w;
                ax += fabsf(ux);
                ay += fabsf(uy);
                v_o += v;
            };
            if (ok && e.B.w * f.vis <= kAlphaMax) {   // a capped alpha passes no gradient on to the geometry
                vd = fac * v_depth;
                vz = vd * pt.w;
                dx = vd * f.dx;
                dy = vd * f.dy;
                through_sigma(f.vis * v_alpha, vd * e.C.y, vd * e.C.z);
            }
            if (ok && a.alpha_sum && range < pt.z - a.alpha_sum_threshold) through_sigma(f.vis * v_asum, 0.f, 0.f);
            add_warp_total(grad.conics + 3 * g, q0);
            add_warp_total(grad.conics + 3 * g + 1, q1);
            add_warp_total(grad.conics + 3 * g + 2, q2);
            add_warp_total(grad.means2d + 2 * g, mx);
            add_warp_total(grad.means2d + 2 * g + 1, my);
            add_warp_total(grad.pix_vels + 3 * g, vx);
            add_warp_total(grad.pix_vels + 3 * g + 1, vy);
            add_warp_total(grad.pix_vels + 3 * g + 2, vz);
            add_warp_total(grad.depth_comps + 2 * g, dx);
            add_warp_total(grad.depth_comps + 2 * g + 1, dy);
            add_warp_total(grad.opacities + g, v_o);
            if (grad.means2d_abs != nullptr) {
                add_warp_total(grad.means2d_abs + 2 * g, ax);
                add_warp_total(grad.means2d_abs + 2 * g + 1, ay);
            }
        }
    }
}

constexpr uint32_t kPointsBwdStage = 2;   // entries per thread and batch: their loads overlap

template <int CDIM, bool kAbs>
__global__ void __launch_bounds__(CDIM <= 8 ? 512 : 256, CDIM <= 8 || CDIM > 20 ? 1 : 2) rasterize_to_points_bwd_kernel(
    uint32_t C, int64_t n_isects, const float2 *__restrict__ means2d,
    const float *__restrict__ conics, const float *__restrict__ colors,
    const float *__restrict__ ranges, uint32_t channels,
    const float *__restrict__ opacities, const float *__restrict__ pix_vels,
    const float2 *__restrict__ depth_comps, const float *__restrict__ backgrounds,
    const float4 *__restrict__ raster_pts, uint32_t W, uint32_t H, uint32_t tile_width,
    uint32_t tile_height, uint32_t grid_w, uint32_t grid_h, uint32_t ctas_per_tile, int compute_alpha_sum,
    float alpha_sum_threshold, const int32_t *__restrict__ offsets,
    const int32_t *__restrict__ flatten_ids, uint32_t depth_idx,
    const float *__restrict__ render_alphas, const int32_t *__restrict__ last_ids,
    const float *__restrict__ v_render_colors, const float *__restrict__ v_render_alphas,
    const float *__restrict__ v_alpha_sum, float *__restrict__ v_means2d_abs,
    float *__restrict__ v_means2d, float *__restrict__ v_conics, float *__restrict__ v_colors,
    float *__restrict__ v_opacities, float *__restrict__ v_pix_vels,
    float *__restrict__ v_depth_comps, float *__restrict__ v_ranges) {
    chain_enter();
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ PointBox s_box;
    constexpr uint32_t kStage = kPointsBwdStage;
    __shared__ uint32_t s_warp_kept[kStage * 16];
    const uint32_t bs = blockDim.x, cap = kStage * bs;
    float4 *sA = reinterpret_cast<float4 *>(smem_raw);
    float4 *sB = sA + cap;
    float4 *sC = sB + cap;   // range velocity, depth compensation (2), range
    float *sRgb = reinterpret_cast<float *>(sC + cap);                 // [cap * CDIM], zeros behind the channels
    int32_t *sId = reinterpret_cast<int32_t *>(sRgb + cap * CDIM);
    int32_t *sPos = sId + cap;
    float4 *sSeg = reinterpret_cast<float4 *>(sPos + cap);   // [warps][32] what a segment does to its two points

    const uint32_t tiles_per_cam = grid_w * grid_h;
    const uint32_t gtile = blockIdx.x / ctas_per_tile, part = blockIdx.x - gtile * ctas_per_tile;
    const uint32_t cam = gtile / tiles_per_cam;
    const uint32_t tile = gtile - cam * tiles_per_cam;
    const uint32_t ty = tile / grid_w, tx = tile - ty * grid_w;
    const uint32_t tr = threadIdx.x, lane = tr & 31u, warp = tr >> 5, n_warps = bs >> 5;
    const PointPatch pp = point_patch<2>(tile_width, tile_height, part * 32u + lane);   // every warp holds the same points

    const TileRange range = tile_range(offsets, gtile, C * tiles_per_cam, n_isects);
    const uint32_t fstride = ranges ? channels - 1 : channels;
    const bool vec = (fstride % 4u == 0u) && ((reinterpret_cast<uintptr_t>(colors) & 15u) == 0u);

    float2 az, el, roll, T, behind, v_depth, v_asum, sum_limit;
    float v_out[2][CDIM];
    int32_t bin_final[2], thread_last = -1;
    float none = 0.f;   // a NaN: see odd_points_bwd()
    PointExtent extent;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        // the second point follows the first in its beam, or in the tile's row-major order
        uint32_t row = pp.row, col = pp.col + h;
        if (col >= tile_width) { col -= tile_width; ++row; }
        const uint32_t i = ty * tile_height + row, j = tx * tile_width + col;
        bool in = row < tile_height && i < H && j < W;
        const size_t pix = in ? ((size_t)cam * H + i) * W + j : 0u;
        float4 rp = make_float4(0.f, 0.f, 0.f, 0.f);
        if (in) {
            rp = raster_pts[pix];
            if (rp.z <= 0.f) in = false;
        }
        if (in) extent.add<false>(rp.x, rp.y, rp.w);
        const float T_final = in ? 1.f - render_alphas[pix] : 1.f;
        bin_final[h] = in ? last_ids[pix] : -1;
        thread_last = (in && bin_final[h] < 0) ? INT32_MAX : max(thread_last, bin_final[h]);
        float bg_dot = 0.f, vd = 0.f;
#pragma unroll
        for (int c = 0; c < CDIM; ++c) {
            v_out[h][c] = (in && (uint32_t)c < channels) ? v_render_colors[pix * channels + c] : 0.f;
            if ((uint32_t)c == depth_idx) vd = v_out[h][c];
            if (backgrounds != nullptr && (uint32_t)c < channels)
                bg_dot += backgrounds[(size_t)cam * channels + c] * v_out[h][c];
            none = fmaf(v_out[h][c], 0.f, none);
        }
        const float va = in ? v_render_alphas[pix] : 0.f;
        const float vs = (in && compute_alpha_sum && v_alpha_sum != nullptr) ? v_alpha_sum[pix] : 0.f;
        // what the background and the alpha output receive through everything in front of them
        const float last = -T_final * (va - bg_dot);
        none = fmaf(last, 0.f, fmaf(vs, 0.f, none));
        const float limit = rp.z - alpha_sum_threshold;
        if (h) { az.y = rp.x; el.y = rp.y; roll.y = rp.w; T.y = T_final; behind.y = last; v_depth.y = vd; v_asum.y = vs; sum_limit.y = limit; }
        else { az.x = rp.x; el.x = rp.y; roll.x = rp.w; T.x = T_final; behind.x = last; v_depth.x = vd; v_asum.x = vs; sum_limit.x = limit; }
    }
    if (warp == 0) extent.write_box<false>(&s_box);

    // last list position consumed by any of the patch's points
    const int32_t patch_last = __reduce_max_sync(0xffffffffu, none != 0.f ? INT32_MAX : thread_last);
    if (patch_last == INT32_MAX) {
        if (warp != 0u) return;
        const PointTask task = {C, W, H, tile_width, tile_height, grid_w, grid_h, ctas_per_tile, channels, depth_idx, n_isects,
                                compute_alpha_sum != 0, alpha_sum_threshold, means2d, depth_comps, pix_vels, conics, opacities,
                                colors, ranges, backgrounds, raster_pts, offsets, flatten_ids};
        const PointGrads grads = {render_alphas, v_render_colors, v_render_alphas, v_alpha_sum, last_ids, v_means2d,
                                  kAbs ? v_means2d_abs : nullptr, v_conics, v_colors, v_ranges, v_opacities, v_pix_vels,
                                  v_depth_comps};
        odd_points_bwd(task, grads);
        return;
    }
    const int32_t eff_end = min(range.end, patch_last + 1);
    if (eff_end <= range.start) return;
    const uint32_t num_batches = (uint32_t)(eff_end - range.start + cap - 1) / cap;

    constexpr int kGeo = kAbs ? 13 : 11;
    constexpr bool kSplit = CDIM + kGeo > 32;   // the geometry in a butterfly of its own
    constexpr int kSums = kSplit ? CDIM : CDIM + kGeo;
    const SumSlot mine_a = sum_slot<kSums>(lane);
    const GradSlot slot_a = point_grad_slot<kAbs>(mine_a.value, CDIM, channels, fstride,
                                                  v_colors, v_ranges, v_conics, v_means2d, v_pix_vels, v_depth_comps,
                                                  v_opacities, v_means2d_abs);

    int32_t next_id[kStage];
#pragma unroll
    for (uint32_t q = 0; q < kStage; ++q) {
        const int32_t idx = eff_end - 1 - (int32_t)(q * bs + tr);
        next_id[q] = idx >= range.start ? flatten_ids[idx] : 0;
    }
    for (uint32_t b = 0; b < num_batches; ++b) {
        const int32_t batch_end = eff_end - 1 - (int32_t)(cap * b);
        PointEntry e[kStage];
        int32_t g[kStage];
        uint32_t kept[kStage];
        uint32_t seen[kStage];
#pragma unroll
        for (uint32_t q = 0; q < kStage; ++q) {
            const int32_t idx = batch_end - (int32_t)(q * bs + tr), ahead = idx - (int32_t)cap;
            g[q] = next_id[q];
            if (idx >= range.start) {
                e[q] = load_point_entry(g[q], means2d, conics, opacities, pix_vels, depth_comps);
                e[q].C.w = ranges ? __ldg(ranges + g[q]) : __ldg(colors + (size_t)g[q] * channels + depth_idx);
            }
            if (ahead >= range.start) next_id[q] = flatten_ids[ahead];   // on its way meanwhile
        }
        __syncthreads();   // the batch before has been read; the box has been written
        // survivors to the front, still back to front in list order
#pragma unroll
        for (uint32_t q = 0; q < kStage; ++q) {
            seen[q] = batch_end - (int32_t)(q * bs + tr) >= range.start ? boxes_that_see<true, false>(e[q], &s_box, 1u) : 0u;
            kept[q] = __ballot_sync(0xffffffffu, seen[q] != 0u);
            if (lane == 0) s_warp_kept[q * n_warps + warp] = __popc(kept[q]);
        }
        __syncthreads();
        uint32_t n_kept = 0;
#pragma unroll
        for (uint32_t q = 0; q < kStage; ++q) {
            uint32_t pos = __popc(kept[q] & ((1u << lane) - 1u));
            for (uint32_t w = 0; w < n_warps; ++w) {
                if (w == warp) pos += n_kept;
                n_kept += s_warp_kept[q * n_warps + w];
            }
            if (seen[q]) {
                sA[pos] = e[q].A;
                sB[pos] = e[q].B;
                sC[pos] = e[q].C;
                sId[pos] = seen[q] >> kCarefulShift ? g[q] | INT32_MIN : g[q];
                sPos[pos] = batch_end - (int32_t)(q * bs + tr);
                stage_features<CDIM>(sRgb + pos * CDIM, colors, (size_t)g[q], fstride, vec, ranges != nullptr, e[q].C.w);
            }
        }
        __syncthreads();
        // The entries are cut into one segment per warp. A warp first runs its segment from T = 1 and nothing
        // behind it; those products and sums of the segments behind its own are what its second run starts
        // from, in which the gradients are formed. (One warp per patch: the only segment starts where the
        // batch before ended.)
        const uint32_t per = (n_kept + n_warps - 1) / n_warps;
        const uint32_t t_lo = min(n_kept, warp * per), t_hi = min(n_kept, t_lo + per);
        // alpha and exp(-sigma) of the entry, zeros where a point does not blend it; `open`, of an entry that needs care: zero where
        // the alpha is capped and passes no gradient on to the geometry
        const auto evaluate = [&](uint32_t t, int32_t id, float4 &B, float2 &dx, float2 &dy, float2 &vis, float2 &alpha, float2 &open) {
            const float4 A = sA[t];
            B = sB[t];
            const int32_t entry = sPos[t];
            const float2 mx = __ffma2_rn(roll, make_float2(A.z, A.z), make_float2(A.x, A.x)), my = __ffma2_rn(roll, make_float2(A.w, A.w), make_float2(A.y, A.y));
            const float2 turn = make_float2(180.f, 180.f), back = make_float2(-180.f, -180.f);
            dx = __fadd2_rn(__fadd2_rn(__fadd2_rn(mx, make_float2(-az.x, -az.y)), turn), back);
            dy = __fadd2_rn(__fadd2_rn(__fadd2_rn(my, make_float2(-el.x, -el.y)), turn), back);
            const float2 sigma = point_sigma(make_float2(B.x, B.x), make_float2(B.y, B.y), make_float2(B.z, B.z), dx, dy);
            vis = make_float2(__expf(-sigma.x), __expf(-sigma.y));
            alpha = __fmul2_rn(make_float2(B.w, B.w), vis);
            bool ok0 = alpha.x >= kAlphaMin, ok1 = alpha.y >= kAlphaMin;
            if (id < 0) {
                const PointFootprint f0 = point_footprint(A, B, roll.x, az.x, el.x), f1 = point_footprint(A, B, roll.y, az.y, el.y);
                dx = make_float2(f0.dx, f1.dx);
                dy = make_float2(f0.dy, f1.dy);
                vis = make_float2(f0.vis, f1.vis);
                open = make_float2(B.w * f0.vis <= kAlphaMax ? 1.f : 0.f, B.w * f1.vis <= kAlphaMax ? 1.f : 0.f);
                alpha = make_float2(fminf(kAlphaMax, B.w * f0.vis), fminf(kAlphaMax, B.w * f1.vis));
                ok0 = !(f0.sigma < 0.f || alpha.x < kAlphaMin);
                ok1 = !(f1.sigma < 0.f || alpha.y < kAlphaMin);
            }
            ok0 = ok0 && entry <= bin_final[0];
            ok1 = ok1 && entry <= bin_final[1];
            vis = make_float2(ok0 ? vis.x : 0.f, ok1 ? vis.y : 0.f);
            alpha = make_float2(ok0 ? alpha.x : 0.f, ok1 ? alpha.y : 0.f);
            return ok0 || ok1;
        };
        float2 T_batch = T, behind_batch = behind;
        if (n_warps > 1) {
            float2 P = make_float2(1.f, 1.f), Q = make_float2(0.f, 0.f);
            for (uint32_t t = t_lo; t < t_hi; ++t) {
                float4 B;
                float2 dx, dy, vis, alpha, open;
                const int32_t id = sId[t];
                if (!__any_sync(0xffffffffu, evaluate(t, id, B, dx, dy, vis, alpha, open))) continue;
                const float4 Cc = sC[t];
                const float2 om = __fadd2_rn(make_float2(1.f, 1.f), make_float2(-alpha.x, -alpha.y));
                P = __fmul2_rn(P, reciprocal_pair(om));
                const float2 dterm = __ffma2_rn(make_float2(Cc.x, Cc.x), roll,
                                                __ffma2_rn(make_float2(Cc.z, Cc.z), dy, __fmul2_rn(make_float2(Cc.y, Cc.y), dx)));
                float2 dot = __fmul2_rn(dterm, v_depth);
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    float2 d2 = make_float2(0.f, 0.f);
#pragma unroll
                    for (int k = 0; k < CDIM; k += 4) {
                        const float4 c4 = *reinterpret_cast<const float4 *>(sRgb + t * CDIM + k);
                        d2 = __ffma2_rn(make_float2(c4.x, c4.y), make_float2(v_out[h][k], v_out[h][k + 1]), d2);
                        d2 = __ffma2_rn(make_float2(c4.z, c4.w), make_float2(v_out[h][k + 2], v_out[h][k + 3]), d2);
                    }
                    if (h) dot.y += d2.x + d2.y; else dot.x += d2.x + d2.y;
                }
                Q = __ffma2_rn(__fmul2_rn(alpha, P), dot, Q);
            }
            sSeg[warp * 32 + lane] = make_float4(P.x, P.y, Q.x, Q.y);
            __syncthreads();
            for (uint32_t w = 0; w < n_warps; ++w) {
                if (w == warp) { T = T_batch; behind = behind_batch; }
                const float4 s = sSeg[w * 32 + lane];
                behind_batch = __ffma2_rn(T_batch, make_float2(s.z, s.w), behind_batch);
                T_batch = __fmul2_rn(T_batch, make_float2(s.x, s.y));
            }
        }
        for (uint32_t t = t_lo; t < t_hi; ++t) {
            float4 B;
            float2 dx, dy, vis, alpha, open;
            const int32_t id = sId[t];
            if (!__any_sync(0xffffffffu, evaluate(t, id, B, dx, dy, vis, alpha, open))) continue;
            const float4 Cc = sC[t];
            const float2 om = __fadd2_rn(make_float2(1.f, 1.f), make_float2(-alpha.x, -alpha.y));
            const float2 ra = reciprocal_pair(om);
            T = __fmul2_rn(T, ra);
            const float2 fac = __fmul2_rn(alpha, T);
            const float2 dterm = __ffma2_rn(make_float2(Cc.x, Cc.x), roll,
                                            __ffma2_rn(make_float2(Cc.z, Cc.z), dy, __fmul2_rn(make_float2(Cc.y, Cc.y), dx)));
            float sum[CDIM + kGeo];
            float2 dot = __fmul2_rn(dterm, v_depth);   // (c . g) of the two points, the compensated range in it
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const float *v = v_out[h];
                const float2 f2 = h ? make_float2(fac.y, fac.y) : make_float2(fac.x, fac.x);
                float2 d2 = make_float2(0.f, 0.f);
#pragma unroll
                for (int k = 0; k < CDIM; k += 4) {
                    const float4 c4 = *reinterpret_cast<const float4 *>(sRgb + t * CDIM + k);
#pragma unroll
                    for (int m = 0; m < 4; m += 2) {
                        const float2 c2 = m ? make_float2(c4.z, c4.w) : make_float2(c4.x, c4.y);
                        const float2 v2 = make_float2(v[k + m], v[k + m + 1]);
                        d2 = k + m == 0 ? __fmul2_rn(c2, v2) : __ffma2_rn(c2, v2, d2);
                        const float2 acc = h == 0 ? __fmul2_rn(f2, v2) : __ffma2_rn(f2, v2, make_float2(sum[k + m], sum[k + m + 1]));
                        sum[k + m] = acc.x; sum[k + m + 1] = acc.y;
                    }
                }
                if (h) dot.y += d2.x + d2.y; else dot.x += d2.x + d2.y;
            }
            const float2 v_alpha = __ffma2_rn(T, dot, __fmul2_rn(make_float2(-ra.x, -ra.y), behind));
            behind = __ffma2_rn(fac, dot, behind);
            // v = -dL/dsigma / opacity; the alpha sum reaches the entries in front of the point
            float2 vis_open = vis, fac_open = fac;
            if (id < 0) {
                vis_open = __fmul2_rn(vis, open);
                fac_open = __fmul2_rn(fac, open);
            }
            const float2 v_main = __fmul2_rn(vis_open, v_alpha);
            float2 v_sum = make_float2(0.f, 0.f);
            if (compute_alpha_sum) {
                const float g_depth = sRgb[t * CDIM + depth_idx];
                v_sum = __fmul2_rn(vis, make_float2(g_depth < sum_limit.x ? v_asum.x : 0.f, g_depth < sum_limit.y ? v_asum.y : 0.f));
            }
            const float2 v = __fadd2_rn(v_main, v_sum);
            const float2 w = __fmul2_rn(make_float2(-B.w, -B.w), v);                   // dL/dsigma
            const float2 vd = __fmul2_rn(fac_open, v_depth);                           // dL/d(range term)
            const float2 bx = make_float2(B.x, B.x), by = make_float2(B.y, B.y), bz = make_float2(B.z, B.z);
            const float2 sx = __ffma2_rn(bx, dx, __fmul2_rn(by, dy)), sy = __ffma2_rn(by, dx, __fmul2_rn(bz, dy));
            const float2 gx = __ffma2_rn(w, sx, __fmul2_rn(vd, make_float2(Cc.y, Cc.y)));
            const float2 gy = __ffma2_rn(w, sy, __fmul2_rn(vd, make_float2(Cc.z, Cc.z)));
            const float2 wx = __fmul2_rn(w, dx), wy = __fmul2_rn(w, dy);
            const auto both = [](float2 p, float2 q) { const float2 r = __fmul2_rn(p, q); return r.x + r.y; };
            sum[CDIM + 0] = both(wx, dx);
            sum[CDIM + 1] = both(wx, dy);
            sum[CDIM + 2] = both(wy, dy);
            sum[CDIM + 3] = gx.x + gx.y;
            sum[CDIM + 4] = gy.x + gy.y;
            sum[CDIM + 5] = both(gx, roll);
            sum[CDIM + 6] = both(gy, roll);
            sum[CDIM + 7] = both(vd, roll);
            sum[CDIM + 8] = both(vd, dx);
            sum[CDIM + 9] = both(vd, dy);
            sum[CDIM + 10] = v.x + v.y;
            if (kAbs) {
                const float2 us = __fmul2_rn(make_float2(-B.w, -B.w), v_sum);
                const float2 ux = __fmul2_rn(us, sx), uy = __fmul2_rn(us, sy);
                sum[CDIM + 11] = fabsf(gx.x - ux.x) + fabsf(ux.x) + fabsf(gx.y - ux.y) + fabsf(ux.y);
                sum[CDIM + 12] = fabsf(gy.x - uy.x) + fabsf(uy.x) + fabsf(gy.y - uy.y) + fabsf(uy.y);
            }
            const size_t gid = (size_t)(id & INT32_MAX);
            float sums[kSums];
#pragma unroll
            for (int k = 0; k < kSums; ++k) sums[k] = sum[k];
            slot_a.add(gid, warp_sum_values<kSums, 16>(sums, lane), 1.f, mine_a.writes);
            if (kSplit) {
                float geo[kGeo];
#pragma unroll
                for (int k = 0; k < kGeo; ++k) geo[k] = sum[CDIM + k];
                const float geo_total = warp_sum_values<kGeo, 16>(geo, lane);
                const SumSlot mine_b = sum_slot<kGeo>(lane);
                const GradSlot slot_b = point_grad_slot<kAbs>(CDIM + mine_b.value, CDIM, channels, fstride, v_colors,
                                                              v_ranges, v_conics, v_means2d, v_pix_vels, v_depth_comps,
                                                              v_opacities, v_means2d_abs);
                slot_b.add(gid, geo_total, 1.f, mine_b.writes);
            }
        }
        if (n_warps > 1) { T = T_batch; behind = behind_batch; }
    }
}

// ---------------------------------------------------------------------------------------
// Dispatch on the channel count
// ---------------------------------------------------------------------------------------
#define SPL_DISPATCH_CDIM(channels, CALL)                                                        \
    do {                                                                                         \
        if ((channels) <= 4) { CALL(4); }                                                        \
        else if ((channels) <= 8) { CALL(8); }                                                   \
        else if ((channels) <= 16) { CALL(16); }                                                 \
        else if ((channels) <= 20) { CALL(20); }                                                 \
        else { CALL(32); }                                                                       \
    } while (0)

// Forward kernels of many blocks start on empty SMs: 1184 blocks of a lidar, four times as many one-warp blocks of a
// camera. The line is where a frame is faster, not what the kernels have room for. Chained, their first
// blocks are placed beside the last of the colour or list kernels before them, on SMs that keep that kernel's
// large shared memory and small first-level cache for as long as one block follows another, and the gathers need
// the cache. Whole frames, us, chained and apart: with spherical harmonics 640 x 360 (3680 warps) 131.7 and 130.9, 800 x 450 (5800) 133.0
// and 124.4, 960 x 540 151 and 142, 1280 x 720 198 and 194, 1600 x 900 279 and 274, 1920 x 1080 346 and 345; plain colours 106.5 and 108.3 at 480 x 270, 1 to 3 us the
// other way from there on, the launch gap; 128 x 1800 lidar with 4 and 16 features 307 and 297, 308 and 302, 128 x 1200 within 1.
static bool fits_at_once(uint64_t blocks) { return blocks <= (uint64_t)kNumSMs * 8; }
static bool warps_fit_at_once(uint64_t warps) { return fits_at_once(warps / 4); }

// Pixels per lane of the camera kernels: more of them save instructions, fewer fill the machine and leave out more of a
// tile that a small Gaussian does not reach. So the line depends on the number of tiles and on how many of them a Gaussian
// covers - list entries per listed Gaussian, where the caller knows it (splatad_rasterize_set_spread_hint()), else the
// number of tiles alone. Measured, us with two / four / eight pixels, scenes of the camera benchmark with scales shrunk (the kernels of four
// and eight pixels in the one kernel there was before, 16 x 16 pixels with four warps: in brackets).
// Forward, 4 channels: 8160 tiles, 27.5 per Gaussian 197 / 150 / 144 (214), 12.7: 205 / 162 / 158 (220), 7.5: 187 / 156 / 175 (195), 5.4: 187 / 195 / 268
// (193), 3.8: 160 / 164 / 245 (161), 2.5: 109 / 116 / 180 (109), Gaussians all of one size, 3.5: 39 / 31 / 37 (41); 5700, 9.6: 148 / 119 / 125, 5.8: 136 / 148 / 195;
// 3510, 13: 98 / 79 / 84 (105), 6.6: 87 / 96 / 129 (92), 4.3: 105 / 132 / 191 (109); 2040, 8.9: 62 / 66 / 80 (67); 920, 5.1: 62 / 84. 8 channels: 8160, 7.5: 234 / 225
// (267), 5.4: 238 / 262 (262); 3510, 13: 112 / 104 (142), 6.6: 103 / 120 (122). 16 channels: 8160, 7.5: 343 / 312 (334), 5.4: 402 / 377 (369) and with 13 of them 350 / 352 (340), 2.5: 287 / 284 (271); 3510, 13: 162 / 146 (171), 6.6: 150 /
// 157 (152).
// Backward, 4 channels: 8160 tiles, 27.5: 493 / 347 / 305 (383), 12.7: 506 / 373 / 337 (404), 7.5: 473 / 362 / 376 (383), 5.4: 442 / 415 / 584 (422), 3.8: 365 / 385 / 569
// (414), 2.5: 229 / 268 / 410 (297); 5700, 9.6: 375 / 276 / 264; 3510, 13: 240 / 180 / 175 (194), 6.6: 208 / 207 / 274 (209), 4.3: 247 / 283 / 418 (288); 2040, 8.9: 156 /
// 143 / 167 (147), 4.8: 203 / 231 / 397 (233). 8 channels: 8160, 7.5: 582 / 490 (478), 5.4: 567 / 532 (510), 3.8: 469 / 496 (495); 3510, 6.6: 255 / 250 (241), 4.3: 269 / 328 (322).
// 16 channels: 8160, 7.5: 800 / 735 (763), 5.4: 762 / 778 (735); 3510, 6.6: 362 / 330 (334), 4.3: 363 / 449 (335). 20 channels: 8160, 7.5: 907 / 890 (834), 5.4: 884 / 942 (799).
// A tile whose rows leave lanes over takes fewer (8 x 8 tiles: 99 / 136 / 227; 24 x 24: 106 / 90 / 111).
static uint32_t tiles_of_256(uint64_t blocks, uint32_t tile_size) {
    return (uint32_t)(blocks * tile_size * tile_size / 256u < 0xffffffffull ? blocks * tile_size * tile_size / 256u : 0xffffffffull);
}
static bool covers(float spread, float line) { return !(spread > 0.f) || spread >= line; }   // 0: not known
// Tiles of 16 x 16 pixels that a square over `spread` tiles covers.
static float spread_of_16(float spread, uint32_t tile_size) {
    if (!(spread > 0.f) || tile_size == 16u) return spread;
    const float side = 1.f + (sqrtf(spread < 1.f ? 1.f : spread) - 1.f) * (float)tile_size / 16.f;
    return side * side;
}
static uint32_t pixels_that_fit(bool four, bool eight, uint32_t tile_size) {
    if (eight && tile_threads<8>(tile_size) % 32u == 0u) return 8u;
    return (four || eight) && tile_threads<4>(tile_size) >= 32u ? 4u : 2u;
}
// Sparse scenes: few list entries in all, and the longest list's chain counts; fewer pixels per lane make it shorter. Used where both numbers
// are known. 4 channels, entries in thousands, two / four / eight pixels, us, forward: 3200 tiles, 8 per Gaussian, 186: 56 / 66 / 99, 698: 62 / 64 / 76,
// 1490: 84 / 68 / 70; 3536, 12, 255: 56 / 64 / 80, 990: 80 / 70 / 78; 4753, 19, 404: 74 / 68 / 82; 8160, 28, 604: 107 / 87 / 93, 1170: 142 / 113 / 113, 2300: 177 / 138 / 131. Backward: 3200, 186: 136 / 141 /
// 211, 698: 147 / 141 / 158, 1490: 209 / 162 / 152; 3536, 255: 130 / 140 / 173, 495: 159 / 166 / 199, 990: 197 / 158 / 166, 2090: 245 / 184 / 172; 4753, 404: 174 / 154 / 176, 784: 232 / 184 / 203, 1550: 286 / 213 / 199;
// 8160, 604: 258 / 193 / 196, 1170: 348 / 256 / 238.
static bool many_entries(float spread, int64_t entries, int64_t line, float or_spread) {
    return !(spread > 0.f) || entries <= 0 || entries >= line || spread >= or_spread;
}
// Whether most entries that a camera kernel looks at cover their patches, so that runs pay (forward: eight pixels per lane, up to four channels). The
// nearest Gaussians are the ones that count: how many tiles each of them covers (near: splatad_isect_set_near_tiles(); not known, no runs). Without runs and with, us, forward, by
// near tiles: 8 (three million of 3 pixels before a sky of large ones, 7 tiles and 6790 entries on the average, 2040 tiles) 225 and 322; 18 (6 pixels) 119 and 167; 54 (sizes of
// two pixels on the average and e^1.5 around it) 143 and 145; 79 141 and 145; 113 (24 pixels) 90 and 105; 203 108 and 105; 295 (48 pixels) 80 and 87; 350 and more 0.4 to 30 % less with runs in
// all of 446 scenes, such as 404 56 and 47, 479 193 and 187, 582 259 and 237, 1039 41 and 33, 1961 195 and 155. Backward: 9 248 and 334; 26 435 and 475; 66 469 and 499; 117 221 and 227; 136 438 and
// 446; 175 and more the same or less in all of 615, 202 149 and 141, 295 168 and 148, 533 236 and 232, 637 127 and 83. Neither the mean of all Gaussians, nor that of all entries, nor the
// share of entries of large ones tells these apart: what lies far away is never composited.
// Then by tiles per Gaussian times entries per tile, where near ones are large; us without runs (the better of four and eight pixels) and with. Forward: 8160 tiles, 28 tiles per Gaussian and 74
// entries per tile (2 k) 87 and 117, 27 and 143 (4 k) 113 and 136, 16 and 682 (11 k) 162 and 158, 27 and 593 (16 k) 156 and 150, 27 and 1171 (32 k) 147 and 133, 129 and 5750 142
// and 113; 16320, 26 and 198 (5 k) 246 and 271, 92 and 1307 (120 k) 225 and 180; 10800, 19 and 357 (7 k) 195 and 211, 45 and 1414 (64 k) 170 and 142; 5700, 12 and 507 (6 k) 125 and
// 138, 20 and 1234 (25 k) 117 and 104. Fewer tiles: 3510, 13 and 564 (7 k) 78 and 91, 24 and 1066 (26 k) 78 and 80; 3600, 23 and 2296 (53 k) 85 and 78; 2040, 16 and 704 (11 k)
// 56 and 62, 18 and 3107 (55 k) 66 and 50; 1450, 79 and 3643 (288 k) 21 and 23.
// Forward, sparse scenes of large Gaussians: the chain of the longest list counts, and eight pixels make it longer. Entries in millions, 1840 tiles, 68 and 573, 1.1: 53 and 58, 67 and 1124, 2.1:
// 44 and 33; 3600, 80 and 496, 1.8: 76 and 79, 59 and 596, 2.1: 78 and 81, 42 and 1008, 3.6: 72 and 67; 7200, 81 and 162, 1.2: 111 and 119, 79 and 316, 2.3: 120 and 115; 5600, 55 and
// 269, 1.5: 114 and 122; rigs of many tiles and few entries in each gain less still: 7290, 43 and 372 (16 k), 2.7: 138 and 142, 8840, 41 and 331 (14 k), 2.9: 162 and 165,
// but 8000, 31 and 439 (13 k), 3.5: 140 and 123, 10800, 44 and 420 (19 k), 4.5: 184 and 169.
// Backward: 16320, 26 and 198 (5 k) 532 and 553; 8160, 28 and 360 (10 k) 306 without, 57 and 251 (14 k) 265 and 263, 27 and 593 (16 k) 336 and 326, 27 and 1171 314 and 298, 60
// and 791 (48 k) 271 and 250; 3600, 14 and 1354 (19 k) 174 and 162; 2040, 9 and 1546 (14 k) 132 and 118, 35 and 629 (22 k) 124 and 109, 25 and 2252 (57 k) 104 and 86; 1840, 39 and 319 (13
// k) 98 and 91; 1450, 13 and 995 (13 k) 108 and 72; 920, 9 and 3660 (34 k) 90 and 66. With 8 / 14 channels: 8160, 57 and 251 420 / 610 and 410 / 606, 60 and 791 425 / 608 and 397 / 591; 3600, 14 and 1354 250 /
// 348 and 235 / 342; 2040, 9 and 1546 173 / 227 and 158 / 220, with absolute gradients 191 / 244 and 172 / 232 (fewer tiles take two pixels per lane and no runs).
// Five to eight channels, backward: not where the warps without runs, twenty an SM, just fit at once and the sixteen with do not (1500 tiles 122 and 129,
// 1550: 1.06 to 1.15 times as fast with runs in all of eighteen scenes).
static bool covers_patches(uint64_t blocks, uint32_t tile_size, uint32_t channels, float spread, int64_t entries, float near, bool backward) {
    const uint32_t tiles = tiles_of_256(blocks, tile_size);
    const double product = (double)spread * (double)entries;   // times the tiles
    if (entries <= 0 || !(near >= (backward ? 175.f : 350.f)) || tile_threads<8>(tile_size) % 32u != 0u) return false;
    if (backward) return tiles >= (channels > 4u && channels <= 8u ? 1530u : 900u) && product >= 12500.0 * tiles;
    if (tiles < 1800u || entries < 2200000) return false;
    return product >= (tiles < 5000u ? 30000.0 : entries < 400 * (int64_t)tiles ? 17000.0 : 12500.0) * tiles;
}
// Name of a camera kernel in the profile, with what was chosen.
#define PIXELS_KERNEL_NAME(way, px, runs) \
    ((runs) ? ((px) == 8u ? way "/8,runs" : way "/4,runs") : (px) == 8u ? way "/8" : (px) == 4u ? way "/4" : way "/2")
static uint32_t pixels_per_lane_fwd(uint64_t blocks, uint32_t tile_size, uint32_t channels, float spread, int64_t entries) {
    const uint32_t tiles = tiles_of_256(blocks, tile_size);
    const float line = tiles < 6000u ? 7.f : channels <= 4 ? 3.3f : channels <= 8 ? 7.f : 5.f;
    return pixels_that_fit(tiles >= (channels <= 8 ? 2700u : 1500u) && covers(spread, line) && many_entries(spread, entries, 800000, 15.f),
                           channels <= 4 && tiles >= 6000u && covers(spread, 10.f) && many_entries(spread, entries, 1200000, INFINITY), tile_size);
}
static uint32_t pixels_per_lane_bwd(uint64_t blocks, uint32_t tile_size, uint32_t channels, float spread, int64_t entries) {
    const uint32_t tiles = tiles_of_256(blocks, tile_size);
    const float line = channels <= 4 && tiles >= 6000u ? 4.f : channels <= 8 ? 5.f : channels <= 16 ? 6.f : 7.f;
    return pixels_that_fit(tiles >= 1500u && covers(spread, line) && many_entries(spread, entries, 550000, 15.f),
                           channels <= 4 && tiles >= 3000u && covers(spread, 9.f) && many_entries(spread, entries, 1100000, INFINITY), tile_size);
}
static bool pixels_bwd_other(uint64_t blocks, uint32_t tile_size, uint32_t channels, uint32_t px, float spread) {
    const uint32_t tiles = tiles_of_256(blocks, tile_size);
    if (channels > 20) return tiles < 1500u || (tiles < 3000u && !covers(spread, 7.f));
    return px == 4 ? !covers(spread, 9.f) : tiles >= 3000u;
}

// One-shot hint of the calling thread's next camera compositing call.
static thread_local float t_spread_hint = 0.f;
static thread_local int64_t t_entries_hint = 0;
static thread_local float t_near_hint = 0.f;
struct SplatHint { float spread; int64_t entries; float near; };   // 0: not known
static SplatHint take_spread_hint(uint32_t tile_size) {
    const SplatHint hint = {spread_of_16(t_spread_hint, tile_size), t_entries_hint, spread_of_16(t_near_hint, tile_size)};
    t_spread_hint = t_near_hint = 0.f;
    t_entries_hint = 0;
    return hint;
}

// Whether all warps of a CTA share one patch in the forward pass: the shared work costs more instructions in all, so the
// patches must be too few to fill the machine. Apart and shared, us, 4 / 12 channels beside the range, by rows of Gaussians per patch: 256
// patches, 40 rows 130 / 146 and 31 / 36, 600 rows 60 / 64 and 19 / 23; 512, 40: 132 / 148 and 39 / 44, 600: 41 / 46 and 27 / 33; 1024, 40: 80 / 89 and 44 / 53, 600: 39 / 42 and
// 41 / 50. From 1184 patches on it takes sparse scenes, whose lists saturate late and are walked by few warps at their end: 1280 patches, 40
// rows 78 / 90 and 50 / 60, 100: 54 / 60 and 46 / 58, 250: 46 / 46 and 48 / 58, 600: 35 / 39 and 46 / 56; 1440, 40: 70 / 74 and 52 / 64, 100: 50 / 52 and 52 / 63. 21 channels never: 1280, 40:
// 95 and 99, 100: 64 and 96. Rows not known (0): as dense.
static bool shares_patches(uint64_t patches, uint32_t channels, uint64_t rows) {
    if (patches < kNumSMs * 8u) return true;
    return patches < kNumSMs * 10u && channels <= 20 && rows > 0 && rows < patches * (channels <= 8 ? 100u : 60u);
}

// One-shot hint of the calling thread's next lidar compositing call.
static thread_local uint64_t t_rows_hint = 0;

// Warps - segments of the list - per patch in the backward pass: every segment is run twice, which pays
// while the patches alone leave the schedulers waiting on one warp's chain. One, four and eight segments, us, 8
// channels: 400 patches 163, 71, 56, 608 121, 61, 57, 800 100, 66, 64, 1088 85, 72, 80, 1600 93, 96, 108, 2240 97, 118, 138, 2816
// 126, 136, 164 (256: eight 54, sixteen 49); 17 channels: 400 203, 91, 76, 608 152, 78, 74, 800 124, 87, 87, 1088 107, 95,
// 105, 1600 121, 128, 147, 2240 126, 152, 182 (19 channels, 792: four 74, eight 76); 21 channels: 1400 one 311, four 282, 1824 303 and 317.
// Sparse scenes gain most: 5 channels, entries per tile 430, 1430, 4300 and 8600: 1344 patches one segment 180, 102, 86, 92, four 105, 92, 86, 83; 1560: 176, 105, 90, 95
// and 107, 97, 93, 89; 1824: 168, 109, 94, 96 and 117, 107, 102, 98; 2240, 630: 171 and 167. Sixteen take
// an SM each, and only up to eight channels stay within their 128 registers.
static uint32_t point_segments(uint64_t patches, uint32_t channels, bool sparse) {
    if (channels <= 8 && patches < (uint64_t)kNumSMs * 2) return 16u;
    return patches < (uint64_t)kNumSMs * (channels <= 8 ? 6 : 5) ? 8u : patches < (uint64_t)kNumSMs * (sparse ? 14 : 11) ? 4u : 1u;
}

template <typename K>
static int set_smem(K kernel, size_t bytes, const char *what) {
    if (bytes > 32 * 1024) {   // the 48 KB default also has to hold the kernels' static shared memory
        cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
        if (e != cudaSuccess) {
            set_last_error("%s: cannot reserve %zu bytes of shared memory: %s", what, bytes,
                           cudaGetErrorString(e));
            return SPLATAD_ERR_CUDA;
        }
    }
    return SPLATAD_OK;
}

} // namespace splatad

using namespace splatad;

extern "C" int splatad_rasterize_set_rows_hint(uint64_t rows) {
    t_rows_hint = rows;
    return SPLATAD_OK;
}

extern "C" int splatad_rasterize_set_spread_hint(float tiles_per_gaussian, int64_t n_isects) {
    t_spread_hint = tiles_per_gaussian;
    t_entries_hint = n_isects;
    return SPLATAD_OK;
}

extern "C" int splatad_rasterize_set_near_hint(float tiles_per_near_gaussian) {
    t_near_hint = tiles_per_near_gaussian;
    return SPLATAD_OK;
}

extern "C" int splatad_rasterize_to_pixels_fwd(
    uint32_t C, int64_t n_isects, const float *means2d, const float *conics, const float *colors,
    uint32_t channels, const float *opacities, const float *pix_vels,
    const float *rolling_shutter_time, const float *backgrounds, uint32_t image_width,
    uint32_t image_height, uint32_t tile_size, uint32_t tile_width, uint32_t tile_height,
    const int32_t *tile_offsets, const int32_t *flatten_ids, float *render_colors,
    float *render_alphas, int32_t *last_ids, void *stream) {
    return splatad_rasterize_expected_to_pixels_fwd(C, n_isects, means2d, conics, colors, channels, opacities, pix_vels,
                                                    rolling_shutter_time, backgrounds, image_width, image_height,
                                                    tile_size, tile_width, tile_height, tile_offsets, flatten_ids, 0,
                                                    render_colors, render_alphas, last_ids, nullptr, stream);
}

extern "C" int splatad_rasterize_expected_to_pixels_fwd(
    uint32_t C, int64_t n_isects, const float *means2d, const float *conics, const float *colors,
    uint32_t channels, const float *opacities, const float *pix_vels,
    const float *rolling_shutter_time, const float *backgrounds, uint32_t image_width,
    uint32_t image_height, uint32_t tile_size, uint32_t tile_width, uint32_t tile_height,
    const int32_t *tile_offsets, const int32_t *flatten_ids, int32_t expected_last_channel, float *render_colors,
    float *render_alphas, int32_t *last_ids, float *expected_depths, void *stream) {
    const SplatHint hint = take_spread_hint(tile_size);
    SPL_REQUIRE(channels >= 1 && channels <= SPLATAD_MAX_CHANNELS, SPLATAD_ERR_CHANNELS,
                "rasterize_to_pixels_fwd: unsupported channel count %u (1..%d)", channels,
                SPLATAD_MAX_CHANNELS);
    SPL_REQUIRE(tile_size >= 1 && tile_size * tile_size <= 1024, SPLATAD_ERR_BAD_ARG,
                "rasterize_to_pixels_fwd: tile_size^2 must be <= 1024");
    SPL_REQUIRE(render_colors && render_alphas && last_ids && tile_offsets && rolling_shutter_time,
                SPLATAD_ERR_BAD_ARG, "rasterize_to_pixels_fwd: null argument");
    SPL_REQUIRE(n_isects == 0 || (means2d && conics && colors && opacities && pix_vels && flatten_ids),
                SPLATAD_ERR_BAD_ARG, "rasterize_to_pixels_fwd: null input");
    const uint32_t blocks = C * tile_width * tile_height;
    if (blocks == 0 || image_width == 0 || image_height == 0) return SPLATAD_OK;
#define CALL_PX(D, P)                                                                             \
    {                                                                                             \
        const uint32_t patches = div_up(tile_threads<P>(tile_size), 32);                          \
        const auto kernel = D >= 20 && vec ? rasterize_to_pixels_fwd_kernel<D, P, (D >= 20), false>  \
                          : runs ? rasterize_to_pixels_fwd_kernel<D, P, false, (P == 8)> : rasterize_to_pixels_fwd_kernel<D, P, false, false>; \
        SPL_REQUIRE((uint64_t)blocks * patches <= 0x7fffffffull, SPLATAD_ERR_BAD_ARG, "rasterize_to_pixels_fwd: too many tiles"); \
        launch_chained_if(warps_fit_at_once((uint64_t)blocks * patches), kernel, blocks * patches, 32, 0, \
            (cudaStream_t)stream,                                                                 \
            C, n_isects, (const float2 *)means2d, conics, colors, channels, opacities,            \
            (const float2 *)pix_vels, rolling_shutter_time, backgrounds, image_width,             \
            image_height, tile_size, tile_width, tile_height, patches, tile_offsets, flatten_ids, \
            render_colors, render_alphas, last_ids, (uint32_t)(expected_last_channel != 0),       \
            expected_last_channel ? expected_depths : nullptr);                                   \
    }
#define CALL(D)                                                                                   \
    if (D <= 4 && px == 8) CALL_PX(D, (D <= 4 ? 8 : 2)) else if (D <= 16 && px == 4) CALL_PX(D, (D <= 16 ? 4 : 2)) else CALL_PX(D, 2)
    const bool runs = channels <= 4 && covers_patches(blocks, tile_size, channels, hint.spread, hint.entries, hint.near, false);
    const uint32_t px = runs ? 8u : pixels_per_lane_fwd(blocks, tile_size, channels, hint.spread, hint.entries);
    const bool vec = channels % 4u == 0u && (reinterpret_cast<uintptr_t>(colors) & 15u) == 0u;
    {
        SPL_PROF(PIXELS_KERNEL_NAME("rasterize_to_pixels_fwd_kernel", channels <= 16u ? px : 2u, runs), (cudaStream_t)stream);
        SPL_DISPATCH_CDIM(channels, CALL);
    }
#undef CALL
#undef CALL_PX
    return check_launch("rasterize_to_pixels_fwd");
}

extern "C" int splatad_rasterize_to_pixels_bwd(
    uint32_t C, int64_t n_isects, const float *means2d, const float *conics, const float *colors,
    uint32_t channels, const float *opacities, const float *pix_vels,
    const float *rolling_shutter_time, const float *backgrounds, uint32_t image_width,
    uint32_t image_height, uint32_t tile_size, uint32_t tile_width, uint32_t tile_height,
    const int32_t *tile_offsets, const int32_t *flatten_ids, const float *render_alphas,
    const int32_t *last_ids, const float *v_render_colors, const float *v_render_alphas,
    float *v_means2d_abs, float *v_means2d, float *v_conics, float *v_colors, float *v_opacities,
    float *v_pix_vels, void *stream) {
    return splatad_rasterize_expected_to_pixels_bwd(
        C, n_isects, means2d, conics, colors, channels, opacities, pix_vels, rolling_shutter_time, backgrounds,
        image_width, image_height, tile_size, tile_width, tile_height, tile_offsets, flatten_ids, nullptr, render_alphas,
        last_ids, v_render_colors, v_render_alphas, v_means2d_abs, v_means2d, v_conics, v_colors, v_opacities,
        v_pix_vels, stream);
}

extern "C" int splatad_rasterize_expected_to_pixels_bwd(
    uint32_t C, int64_t n_isects, const float *means2d, const float *conics, const float *colors,
    uint32_t channels, const float *opacities, const float *pix_vels,
    const float *rolling_shutter_time, const float *backgrounds, uint32_t image_width,
    uint32_t image_height, uint32_t tile_size, uint32_t tile_width, uint32_t tile_height,
    const int32_t *tile_offsets, const int32_t *flatten_ids, const float *expected_depths, const float *render_alphas,
    const int32_t *last_ids, const float *v_render_colors, const float *v_render_alphas,
    float *v_means2d_abs, float *v_means2d, float *v_conics, float *v_colors, float *v_opacities,
    float *v_pix_vels, void *stream) {
    const SplatHint hint = take_spread_hint(tile_size);
    SPL_REQUIRE(channels >= 1 && channels <= SPLATAD_MAX_CHANNELS, SPLATAD_ERR_CHANNELS,
                "rasterize_to_pixels_bwd: unsupported channel count %u (1..%d)", channels,
                SPLATAD_MAX_CHANNELS);
    SPL_REQUIRE(tile_size >= 1 && tile_size * tile_size <= 1024, SPLATAD_ERR_BAD_ARG,
                "rasterize_to_pixels_bwd: tile_size^2 must be <= 1024");
    const uint32_t blocks = C * tile_width * tile_height;
    if (blocks == 0 || n_isects == 0 || image_width == 0 || image_height == 0) return SPLATAD_OK;
    SPL_REQUIRE(means2d && conics && colors && opacities && pix_vels && flatten_ids &&
                    tile_offsets && render_alphas && last_ids && v_render_colors &&
                    v_render_alphas && v_means2d && v_conics && v_colors && v_opacities &&
                    v_pix_vels && rolling_shutter_time,
                SPLATAD_ERR_BAD_ARG, "rasterize_to_pixels_bwd: null argument");
    // (a limit from one thread per pixel, which these kernels do not have; callers count on the error, and frames.cpp asks the same
    // before it renders)
    const uint32_t samples = ((tile_size * tile_size + 31) / 32) * 32;
    SPL_REQUIRE(samples <= 512 || channels <= 16, SPLATAD_ERR_BAD_ARG,
                "rasterize_to_pixels_bwd: a tile of %u pixels (%u threads at one per pixel) with %u channels is more "
                "than the backward pass takes: use a smaller tile or at most 16 channels per call",
                tile_size * tile_size, samples, channels);
#define CALL_PX(D, P, A)                                                                          \
    {                                                                                             \
        const auto kernel = has_runs_bwd(D, P) && runs ? rasterize_to_pixels_bwd_kernel<D, P, A, (has_runs_bwd(D, P) ? kRunsBwd : kPlainBwd)> \
                          : has_other_bwd(D, P) && other ? rasterize_to_pixels_bwd_kernel<D, P, A, (has_other_bwd(D, P) ? kOtherBwd : kPlainBwd)> \
                                                         : rasterize_to_pixels_bwd_kernel<D, P, A, kPlainBwd>; \
        const uint32_t patches = div_up(tile_threads<P>(tile_size), 32);                          \
        SPL_REQUIRE((uint64_t)blocks * patches <= 0x7fffffffull, SPLATAD_ERR_BAD_ARG, "rasterize_to_pixels_bwd: too many tiles"); \
        launch_chained(kernel, blocks * patches, 32, 0, (cudaStream_t)stream,                     \
            C, n_isects, (const float2 *)means2d, conics, colors, channels, opacities,            \
            (const float2 *)pix_vels, rolling_shutter_time, backgrounds, image_width,             \
            image_height, tile_size, tile_width, tile_height, patches, tile_offsets, flatten_ids, \
            render_alphas, last_ids, v_render_colors, v_render_alphas, v_means2d_abs, v_means2d,  \
            v_conics, v_colors, v_opacities, v_pix_vels, expected_depths);                        \
    }
#define CALL_ABS(D, A)                                                                            \
    if (D <= 4 && px == 8) CALL_PX(D, (D <= 4 ? 8 : 2), A) else if (D <= 20 && px == 4) CALL_PX(D, (D <= 20 ? 4 : 2), A) else CALL_PX(D, 2, A)
#define CALL(D)                                                                                   \
    if (v_means2d_abs) CALL_ABS(D, true) else CALL_ABS(D, false)
    const bool runs = covers_patches(blocks, tile_size, channels, hint.spread, hint.entries, hint.near, true);
    const uint32_t px = runs && channels <= 4 ? 8u : pixels_per_lane_bwd(blocks, tile_size, channels, hint.spread, hint.entries);
    const bool other = pixels_bwd_other(blocks, tile_size, channels, px, hint.spread);
    {
        SPL_PROF(PIXELS_KERNEL_NAME("rasterize_to_pixels_bwd_kernel", channels <= 20u ? px : 2u,
                                    runs && (px == 8u || (px == 4u && channels > 4u && channels <= 16u))), (cudaStream_t)stream);
        SPL_DISPATCH_CDIM(channels, CALL);
    }
#undef CALL
#undef CALL_ABS
#undef CALL_PX
    return check_launch("rasterize_to_pixels_bwd");
}

extern "C" int splatad_rasterize_to_points_fwd(
    uint32_t C, int64_t n_isects, const float *means2d, const float *conics,
    const float *lidar_features, const float *gaussian_ranges, uint32_t channels,
    const float *opacities,
    const float *pix_vels, const float *depth_compensations, const float *backgrounds,
    const float *raster_pts, uint32_t image_width, uint32_t image_height, uint32_t tile_width,
    uint32_t tile_height, uint32_t tile_grid_width, uint32_t tile_grid_height,
    int32_t compute_alpha_sum_until_points, float alpha_sum_threshold,
    const int32_t *tile_offsets, const int32_t *flatten_ids, uint32_t depth_channel_idx,
    float *render_features, float *render_alphas, float *alpha_sum_until_points,
    int32_t *last_ids, float *median_depths, void *stream) {
    const uint64_t rows = t_rows_hint;
    t_rows_hint = 0;
    SPL_REQUIRE(channels >= 1 && channels <= SPLATAD_MAX_CHANNELS, SPLATAD_ERR_CHANNELS,
                "rasterize_to_points_fwd: unsupported channel count %u (1..%d)", channels,
                SPLATAD_MAX_CHANNELS);
    SPL_REQUIRE(depth_channel_idx < channels, SPLATAD_ERR_BAD_ARG,
                "rasterize_to_points_fwd: depth channel out of range");
    SPL_REQUIRE(!gaussian_ranges || depth_channel_idx == channels - 1, SPLATAD_ERR_BAD_ARG,
                "rasterize_to_points_fwd: a separate range array is the last channel");
    SPL_REQUIRE(tile_width >= 1 && tile_height >= 1 && tile_width * tile_height <= 1024,
                SPLATAD_ERR_BAD_ARG, "rasterize_to_points_fwd: tile must have <= 1024 points");
    SPL_REQUIRE(render_features && render_alphas && last_ids && median_depths && tile_offsets &&
                    raster_pts,
                SPLATAD_ERR_BAD_ARG, "rasterize_to_points_fwd: null argument");
    SPL_REQUIRE(!compute_alpha_sum_until_points || alpha_sum_until_points, SPLATAD_ERR_BAD_ARG,
                "rasterize_to_points_fwd: alpha-sum output missing");
    SPL_REQUIRE(n_isects == 0 || (means2d && conics && opacities && pix_vels &&
                                  depth_compensations && flatten_ids &&
                                  (lidar_features || (gaussian_ranges && channels == 1))),
                SPLATAD_ERR_BAD_ARG, "rasterize_to_points_fwd: null input");
    const uint32_t blocks = C * tile_grid_width * tile_grid_height;
    if (blocks == 0 || image_width == 0 || image_height == 0) return SPLATAD_OK;
    const uint32_t warps = div_up(tile_width * tile_height, 32);
    const bool coop = shares_patches((uint64_t)blocks * warps, channels, rows);
    // two warps per CTA otherwise: a CTA ends with its slowest warp
    const uint32_t per_cta = min(2u, warps), parts = coop ? warps : div_up(warps, per_cta), bs = coop ? kCoopWarps * 32 : 32 * per_cta;
    SPL_REQUIRE((uint64_t)blocks * parts <= 0x7fffffffull, SPLATAD_ERR_BAD_ARG, "rasterize_to_points_fwd: too many tiles");
#define CALL(D)                                                                                   \
    {                                                                                             \
        auto kernel = coop ? rasterize_to_points_fwd_coop_kernel<D> : rasterize_to_points_fwd_kernel<D>; \
        const size_t smem = (size_t)(coop ? 1 : points_fwd_stage(D)) * bs *                       \
                                (3 * sizeof(float4) + 2 * sizeof(int32_t) + D * sizeof(float));   \
        int rc = set_smem(kernel, smem, "rasterize_to_points_fwd");                               \
        if (rc != SPLATAD_OK) return rc;                                                          \
        launch_chained_if(fits_at_once((uint64_t)blocks * parts), kernel, blocks * parts, bs, smem, \
            (cudaStream_t)stream,                                                                 \
            C, n_isects, (const float2 *)means2d, conics, lidar_features, gaussian_ranges,        \
            channels, opacities,                                                                  \
            pix_vels, (const float2 *)depth_compensations, backgrounds,                           \
            (const float4 *)raster_pts, image_width, image_height, tile_width, tile_height,       \
            tile_grid_width, tile_grid_height, parts, compute_alpha_sum_until_points,             \
            alpha_sum_threshold, tile_offsets, flatten_ids, depth_channel_idx, render_features,   \
            render_alphas, alpha_sum_until_points, last_ids, median_depths);                      \
    }
    {
        SPL_PROF("rasterize_to_points_fwd_kernel", (cudaStream_t)stream);
        SPL_DISPATCH_CDIM(channels, CALL);
    }
#undef CALL
    return check_launch("rasterize_to_points_fwd");
}

extern "C" int splatad_rasterize_to_points_bwd(
    uint32_t C, int64_t n_isects, const float *means2d, const float *conics,
    const float *lidar_features, const float *gaussian_ranges, uint32_t channels,
    const float *opacities,
    const float *pix_vels, const float *depth_compensations, const float *backgrounds,
    const float *raster_pts, uint32_t image_width, uint32_t image_height, uint32_t tile_width,
    uint32_t tile_height, uint32_t tile_grid_width, uint32_t tile_grid_height,
    int32_t compute_alpha_sum_until_points, float alpha_sum_threshold,
    const int32_t *tile_offsets, const int32_t *flatten_ids, uint32_t depth_channel_idx,
    const float *render_alphas, const int32_t *last_ids, const float *v_render_features,
    const float *v_render_alphas, const float *v_alpha_sum_until_points, float *v_means2d_abs,
    float *v_means2d, float *v_conics, float *v_features, float *v_opacities, float *v_pix_vels,
    float *v_depth_compensations, float *v_gaussian_ranges, void *stream) {
    SPL_REQUIRE(channels >= 1 && channels <= SPLATAD_MAX_CHANNELS, SPLATAD_ERR_CHANNELS,
                "rasterize_to_points_bwd: unsupported channel count %u (1..%d)", channels,
                SPLATAD_MAX_CHANNELS);
    SPL_REQUIRE(depth_channel_idx < channels, SPLATAD_ERR_BAD_ARG,
                "rasterize_to_points_bwd: depth channel out of range");
    SPL_REQUIRE(tile_width >= 1 && tile_height >= 1 && tile_width * tile_height <= 1024,
                SPLATAD_ERR_BAD_ARG, "rasterize_to_points_bwd: tile must have <= 1024 points");
    const uint32_t blocks = C * tile_grid_width * tile_grid_height;
    if (blocks == 0 || n_isects == 0 || image_width == 0 || image_height == 0) return SPLATAD_OK;
    SPL_REQUIRE(means2d && conics && opacities && pix_vels &&
                    depth_compensations && flatten_ids && tile_offsets && raster_pts &&
                    render_alphas && last_ids && v_render_features && v_render_alphas &&
                    v_means2d && v_conics && v_opacities && v_pix_vels && v_depth_compensations,
                SPLATAD_ERR_BAD_ARG, "rasterize_to_points_bwd: null argument");
    SPL_REQUIRE((lidar_features && v_features) || (gaussian_ranges && channels == 1), SPLATAD_ERR_BAD_ARG,
                "rasterize_to_points_bwd: features / v_features missing");
    SPL_REQUIRE(!gaussian_ranges || (v_gaussian_ranges && depth_channel_idx == channels - 1),
                SPLATAD_ERR_BAD_ARG, "rasterize_to_points_bwd: range array needs v_gaussian_ranges");
    const uint32_t samples = ((tile_width * tile_height + 31) / 32) * 32;
    SPL_REQUIRE(samples <= 512 || channels <= 16, SPLATAD_ERR_BAD_ARG,
                "rasterize_to_points_bwd: a tile of %u points (%u threads at one per point) with %u channels is more "
                "than the backward pass takes: use a smaller tile or at most 16 channels per call",
                tile_width * tile_height, samples, channels);
    const uint32_t parts = div_up(tile_width * tile_height, 64), bs = 32 * point_segments((uint64_t)blocks * parts, channels, n_isects > 0 && n_isects < (int64_t)blocks * 1000);
    SPL_REQUIRE((uint64_t)blocks * parts <= 0x7fffffffull, SPLATAD_ERR_BAD_ARG, "rasterize_to_points_bwd: too many tiles");
#define CALL_ABS(D, A)                                                                            \
    {                                                                                             \
        auto kernel = rasterize_to_points_bwd_kernel<D, A>;                                       \
        const size_t smem = (size_t)bs * (sizeof(float4) + kPointsBwdStage *                      \
                                          (3 * sizeof(float4) + 2 * sizeof(int32_t) + D * sizeof(float))); \
        int rc = set_smem(kernel, smem, "rasterize_to_points_bwd");                               \
        if (rc != SPLATAD_OK) return rc;                                                          \
        launch_chained(kernel, blocks * parts, bs, smem, (cudaStream_t)stream,                    \
            C, n_isects, (const float2 *)means2d, conics, lidar_features, gaussian_ranges,        \
            channels, opacities,                                                                  \
            pix_vels, (const float2 *)depth_compensations, backgrounds,                           \
            (const float4 *)raster_pts, image_width, image_height, tile_width, tile_height,       \
            tile_grid_width, tile_grid_height, parts, compute_alpha_sum_until_points,             \
            alpha_sum_threshold, tile_offsets, flatten_ids, depth_channel_idx, render_alphas,     \
            last_ids, v_render_features, v_render_alphas, v_alpha_sum_until_points,               \
            v_means2d_abs, v_means2d, v_conics, v_features, v_opacities, v_pix_vels,              \
            v_depth_compensations, v_gaussian_ranges);                                            \
    }
#define CALL(D)                                                                                   \
    if (v_means2d_abs) CALL_ABS(D, true) else CALL_ABS(D, false)
    {
        SPL_PROF("rasterize_to_points_bwd_kernel", (cudaStream_t)stream);
        SPL_DISPATCH_CDIM(channels, CALL);
    }
#undef CALL
#undef CALL_ABS
    return check_launch("rasterize_to_points_bwd");
}
