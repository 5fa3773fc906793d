// Per-row opacities and colours of the projected Gaussians: what the compositing kernels read for every
// (sensor, Gaussian) row, gathered from the per-Gaussian parameters in one pass - opacities times the
// antialiasing compensation, colours with the depth behind them - and the matching VJPs. In the reference
// these are chains of torch gathers, products and concatenations (gsplat/rendering.py:325-343, 383-384).
// Bound by memory: every row is read and written once.
#include "common.cuh"

namespace splatad {

__global__ void __launch_bounds__(kThreads)
opacity_rows_fwd_kernel(uint32_t n, uint32_t N, const int64_t *__restrict__ ids, const float *__restrict__ opacities,
                        const float *__restrict__ comps, float *__restrict__ out) {
    chain_enter();
    const uint32_t i = blockIdx.x * kThreads + threadIdx.x;
    if (i >= n) return;
    const uint32_t g = ids ? (uint32_t)ids[i] : i < N ? i : i % N;
    const float o = __ldg(opacities + g);
    out[i] = comps ? o * comps[i] : o;
}

__global__ void __launch_bounds__(kThreads)
opacity_rows_bwd_kernel(uint32_t n, uint32_t N, const int64_t *__restrict__ ids, const float *__restrict__ opacities,
                        const float *__restrict__ comps, const float *__restrict__ v_rows,
                        float *__restrict__ v_opacities, float *__restrict__ v_comps) {
    chain_enter();
    const uint32_t i = blockIdx.x * kThreads + threadIdx.x;
    if (i >= n) return;
    const uint32_t g = ids ? (uint32_t)ids[i] : i < N ? i : i % N;
    const float v = v_rows[i];
    if (v_opacities != nullptr && v != 0.f) atomicAdd(v_opacities + g, comps ? v * comps[i] : v);
    if (v_comps != nullptr) v_comps[i] = v * __ldg(opacities + g);
}

// row of the colour table behind projected row i
__device__ __forceinline__ size_t color_row(uint32_t i, uint32_t N, const int64_t *camera_ids, const int64_t *gaussian_ids,
                                            uint32_t per_camera) {
    if (gaussian_ids == nullptr) return per_camera || i < N ? i : i % N;
    return (per_camera ? (size_t)camera_ids[i] * N : 0u) + (size_t)gaussian_ids[i];
}

// Rows of a block of the colour kernels: its elements are numbered in 32 bits and split into row and channel by
// a multiplication: a 64-bit division per element was what bound these kernels (211 k rows of 14 channels: 14
// -> 10 us forward and backward; 500 k packed rows of 20: 24 -> 18 and 20 -> 8).
constexpr uint32_t kColorRows = 64;

static_assert(kColorRows == 64, "the bound on the width below");

struct ByWidth {
    uint32_t width, magic;   // ceil(2^32 / width): exact while element * width < 2^32; 0 for 1 and for wider rows
    __host__ explicit ByWidth(uint32_t w) : width(w), magic(64ull * w * w < 1ull << 32 ? 0xffffffffu / w + 1u : 0u) {}
    __device__ __forceinline__ uint32_t row(uint32_t e) const { return magic != 0u ? __umulhi(e, magic) : e / width; }
};

__global__ void __launch_bounds__(kThreads)
color_rows_fwd_kernel(uint32_t n, uint32_t N, uint32_t D, ByWidth by, const int64_t *__restrict__ camera_ids,
                      const int64_t *__restrict__ gaussian_ids, uint32_t per_camera, const float *__restrict__ colors,
                      const float *__restrict__ depths, float *__restrict__ out) {
    chain_enter();
    const uint32_t i0 = blockIdx.x * kColorRows, elements = min(kColorRows, n - i0) * by.width;
    float *dst = out + (size_t)i0 * by.width;
#pragma unroll 4
    for (uint32_t e = threadIdx.x; e < elements; e += kThreads) {
        const uint32_t r = by.row(e), k = e - r * by.width, i = i0 + r;
        dst[e] = k < D ? __ldg(colors + color_row(i, N, camera_ids, gaussian_ids, per_camera) * D + k) : depths[i];
    }
}

// v_colors is added to; v_depths takes what the last channel holds, plus `add` where there is one.
__global__ void __launch_bounds__(kThreads)
color_rows_bwd_kernel(uint32_t n, uint32_t N, uint32_t D, ByWidth by, const int64_t *__restrict__ camera_ids,
                      const int64_t *__restrict__ gaussian_ids, uint32_t per_camera, const float *__restrict__ v_rows,
                      float *__restrict__ v_colors, const float *__restrict__ add, float *__restrict__ v_depths) {
    chain_enter();
    const uint32_t i0 = blockIdx.x * kColorRows, elements = min(kColorRows, n - i0) * by.width;
    const float *src = v_rows + (size_t)i0 * by.width;
#pragma unroll 4
    for (uint32_t e = threadIdx.x; e < elements; e += kThreads) {
        const uint32_t r = by.row(e), k = e - r * by.width, i = i0 + r;
        const float v = src[e];
        if (v_colors != nullptr && k < D && v != 0.f)
            atomicAdd(v_colors + color_row(i, N, camera_ids, gaussian_ids, per_camera) * D + k, v);
        if (v_depths != nullptr && k + 1u == by.width) v_depths[i] = add ? add[i] + v : v;
    }
}

// The depth channel alone: the colours' gradients took another way.
__global__ void __launch_bounds__(kThreads)
last_channel_kernel(uint32_t n, uint32_t width, const float *__restrict__ v_rows, const float *__restrict__ add,
                    float *__restrict__ out) {
    chain_enter();
    const uint32_t i = blockIdx.x * kThreads + threadIdx.x;
    if (i >= n) return;
    const float v = v_rows[(size_t)i * width + width - 1];
    out[i] = add ? add[i] + v : v;
}

} // namespace splatad

using namespace splatad;

extern "C" int splatad_opacity_rows_fwd(uint32_t n, uint32_t N, const int64_t *gaussian_ids, const float *opacities,
                                        const float *compensations, float *rows, void *stream) {
    if (n == 0) return SPLATAD_OK;
    SPL_REQUIRE(N > 0 && opacities && rows, SPLATAD_ERR_BAD_ARG, "opacity_rows_fwd: null argument");
    SPL_PROF("opacity_rows_fwd_kernel", (cudaStream_t)stream);
    launch_chained(opacity_rows_fwd_kernel, div_up(n, kThreads), kThreads, 0, (cudaStream_t)stream, n, N, gaussian_ids, opacities,
                                                                                       compensations, rows);
    return check_launch("opacity_rows_fwd");
}

extern "C" int splatad_opacity_rows_bwd(uint32_t n, uint32_t N, const int64_t *gaussian_ids, const float *opacities,
                                        const float *compensations, const float *v_rows, float *v_opacities,
                                        float *v_compensations, void *stream) {
    if (n == 0 || (!v_opacities && !v_compensations)) return SPLATAD_OK;
    SPL_REQUIRE(N > 0 && (opacities || !v_compensations) && v_rows, SPLATAD_ERR_BAD_ARG, "opacity_rows_bwd: null argument");
    SPL_PROF("opacity_rows_bwd_kernel", (cudaStream_t)stream);
    launch_chained(opacity_rows_bwd_kernel, div_up(n, kThreads), kThreads, 0, (cudaStream_t)stream,
        n, N, gaussian_ids, opacities, compensations, v_rows, v_opacities, v_compensations);
    return check_launch("opacity_rows_bwd");
}

extern "C" int splatad_color_rows_fwd(uint32_t n, uint32_t N, uint32_t D, const int64_t *camera_ids,
                                      const int64_t *gaussian_ids, uint32_t colors_per_camera, const float *colors,
                                      const float *depths, float *rows, void *stream) {
    const uint32_t width = D + (depths ? 1u : 0u);
    if (n == 0 || width == 0) return SPLATAD_OK;
    SPL_REQUIRE(N > 0 && (colors || D == 0) && rows && (!gaussian_ids || camera_ids || !colors_per_camera),
                SPLATAD_ERR_BAD_ARG, "color_rows_fwd: null argument");
    SPL_PROF("color_rows_fwd_kernel", (cudaStream_t)stream);
    launch_chained(color_rows_fwd_kernel, div_up(n, kColorRows), kThreads, 0, (cudaStream_t)stream,
        n, N, D, ByWidth(width), camera_ids, gaussian_ids, colors_per_camera, colors, depths, rows);
    return check_launch("color_rows_fwd");
}

extern "C" int splatad_color_rows_bwd(uint32_t n, uint32_t N, uint32_t D, uint32_t width, const int64_t *camera_ids,
                                      const int64_t *gaussian_ids, uint32_t colors_per_camera, const float *v_rows,
                                      float *v_colors, const float *v_depths_in, float *v_depths, void *stream) {
    if (n == 0) return SPLATAD_OK;
    SPL_REQUIRE(N > 0 && v_rows && width >= D && (!gaussian_ids || camera_ids || !colors_per_camera), SPLATAD_ERR_BAD_ARG,
                "color_rows_bwd: bad argument");
    SPL_PROF("color_rows_bwd_kernel", (cudaStream_t)stream);
    if (v_colors != nullptr && D > 0)
        launch_chained(color_rows_bwd_kernel, div_up(n, kColorRows), kThreads, 0, (cudaStream_t)stream, n, N, D, ByWidth(width),
                       camera_ids, gaussian_ids, colors_per_camera, v_rows, v_colors, v_depths_in, v_depths);
    else if (v_depths != nullptr)
        launch_chained(last_channel_kernel, div_up(n, kThreads), kThreads, 0, (cudaStream_t)stream, n, width, v_rows, v_depths_in, v_depths);
    return check_launch("color_rows_bwd");
}
