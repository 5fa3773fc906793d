// Tile intersection: per-Gaussian tile rectangles, intersection counts, and the depth-ordered
// per-tile Gaussian lists (isect_ids / flatten_ids / isect_offsets).
//
// What the reference does (gsplat/cuda/csrc/rasterization.cu:15-216 camera, 287-529 lidar,
// 218-285 offsets): count tiles per Gaussian, cumsum, emit one 64-bit key
// (sensor | tile | depth bits) per intersection in flatten-index order, then a stable LSD
// radix sort of 12-byte pairs over 43-46 key bits, then a boundary scan for the offsets.
//
// What this file does instead, with bit-identical results: because a stable sort of the
// emitted keys orders each tile's list by (depth bits, flatten index), the same lists are
// obtained by ordering the *visible elements* by (sensor, depth bits, flatten index) with depth
// buckets - at most C*N 8-byte pairs, L2 resident - and splitting their rectangles stably by blocks of
// tiles and then by tile (the block split below). Offsets fall out of the split.
//
// Depths too crowded for the buckets are ordered by radix passes and then grouped by sensor, for the same split.
// Grids beyond the block split's tables take the radix split: the elements ordered by depth alone, (sensor*n_tiles + tile, flatten index) pairs emitted in that order,
// and a stable radix split of those 8-byte pairs by the compact tile key (ceil(bits/8) passes), the last
// pass writing the 64-bit isect_ids and int32 flatten_ids directly; offsets by a binary search per tile.
//
// All kernels read problem sizes from device memory, so the whole sequence can be enqueued without a
// host round trip; the only device->host traffic is the (n_isects, n_visible, status) triple.
#include "common.cuh"

#include <algorithm>

namespace splatad {

constexpr int kSortThreads = 256;
constexpr int kSortWarps = kSortThreads / 32;
constexpr int kItemsPerLane = 8;
constexpr int kWarpItems = 32 * kItemsPerLane;           // 256
constexpr int kTileItems = kSortWarps * kWarpItems;      // 2048
constexpr int kSortGrid = 4 * kNumSMs;                   // 592 persistent blocks
constexpr int kRadixBins = 256;
static_assert(kSortThreads == kRadixBins, "one thread per radix bin");
static_assert(kSortGrid <= 1024, "row scan and emit scan use one thread per sort block");

// counters[] slots (int64 each)
// The first CNT_SLOTS are what the plan copies to the host; the rest is device-side state.
enum { CNT_NISECT = 0, CNT_NVIS = 1, CNT_STATUS = 2, CNT_TICKET = 3, CNT_SLOTS = 4,
       CNT_DMIN = 4, CNT_DMAX = 5,   // depth range of the listed elements (float bit patterns)
       CNT_BLO = 6, CNT_BHI = 7,     // depth range the buckets span when the caller gave one (BHI < BLO: none)
       CNT_DEV_SLOTS = 8 };
enum { ST_OVERFLOW_CAPACITY = 1, ST_OVERFLOW_INT32 = 2, ST_DEPTH_BUCKETS = 4 };

// ---------------------------------------------------------------------------------------
// Block-wide exclusive scan for any blockDim.x that is a multiple of 32 (<= 1024).
// ---------------------------------------------------------------------------------------
__device__ __forceinline__ uint32_t block_excl_scan(uint32_t v, uint32_t *warp_tot /*[33]*/,
                                                    uint32_t &total) {
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint32_t nwarps = blockDim.x >> 5;
    uint32_t inc = v;
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
        uint32_t o = __shfl_up_sync(0xffffffffu, inc, off);
        if (lane >= (uint32_t)off) inc += o;
    }
    if (lane == 31) warp_tot[warp] = inc;
    __syncthreads();
    if (warp == 0) {
        uint32_t w = (lane < nwarps) ? warp_tot[lane] : 0u;
        uint32_t winc = w;
#pragma unroll
        for (int off = 1; off < 32; off <<= 1) {
            uint32_t o = __shfl_up_sync(0xffffffffu, winc, off);
            if (lane >= (uint32_t)off) winc += o;
        }
        warp_tot[lane] = winc - w;   // exclusive warp offsets
        if (lane == 31) warp_tot[32] = winc;
    }
    __syncthreads();
    const uint32_t res = warp_tot[warp] + inc - v;
    total = warp_tot[32];
    __syncthreads();
    return res;
}

// ---------------------------------------------------------------------------------------
// Tile rectangles
// ---------------------------------------------------------------------------------------
struct Rect { int32_t x0, x1, y0, y1; };   // x: [x0, x1), y: [y0, y1)

struct CamGrid { uint32_t tile_size, tile_width, tile_height; };

__device__ __forceinline__ uint32_t clamp_tile(float v, uint32_t hi) {
    // float -> uint32 conversion that saturates negatives (and NaN) to 0, then min(hi)
    if (!(v > 0.f)) return 0u;
    if (v >= (float)hi) return hi;
    return (uint32_t)v;
}

__device__ __forceinline__ Rect cam_rect(float2 mean, int2 radius, CamGrid g) {
    const float ts = (float)g.tile_size;
    const float ex = (float)radius.x / ts, ey = (float)radius.y / ts;
    const float tx = mean.x / ts, ty = mean.y / ts;
    Rect r;
    r.x0 = (int32_t)clamp_tile(floorf(tx - ex), g.tile_width);
    r.y0 = (int32_t)clamp_tile(floorf(ty - ey), g.tile_height);
    r.x1 = (int32_t)clamp_tile(ceilf(tx + ex), g.tile_width);
    r.y1 = (int32_t)clamp_tile(ceilf(ty + ey), g.tile_height);
    return r;
}

struct LidarGrid {
    const float *elev_boundaries;   // [n_tiles_elev + 1], global or shared
    float tile_azim_res, min_azim;
    uint32_t n_tiles_azim, n_tiles_elev;
};

// Number of leading entries of the ascending array b[0 .. n) that are < v.
__device__ __forceinline__ int32_t lower_bound_f(const float *__restrict__ b, int32_t n, float v) {
    int32_t lo = 0, hi = n;
    while (lo < hi) {
        const int32_t m = (lo + hi) >> 1;
        if (b[m] < v) lo = m + 1; else hi = m;
    }
    return lo;
}

__device__ __forceinline__ Rect lidar_rect(float2 mean, float2 radius, const LidarGrid &g) {
    const float el_lo = mean.y - radius.y, el_hi = mean.y + radius.y;
    const float azim = mean.x - g.min_azim;
    const float az_lo = azim - radius.x, az_hi = azim + radius.x;
    const float azim_max = (float)g.n_tiles_azim * g.tile_azim_res;
    float t_lo, t_hi;
    if (az_lo >= 0.f) t_lo = az_lo / g.tile_azim_res;
    else t_lo = (fmodf(az_lo + 360.f, 360.f) - azim_max) / g.tile_azim_res;
    if (az_hi <= 360.f) t_hi = az_hi / g.tile_azim_res;
    else t_hi = (float)g.n_tiles_azim + fmodf(az_hi + 360.f, 360.f) / g.tile_azim_res;
    Rect r;
    r.x0 = (int32_t)floorf(t_lo);
    r.x1 = (int32_t)ceilf(t_hi);
    // first boundary not below the lower edge (minus one), first boundary not below the upper
    // edge: the reference walks the ascending boundaries one by one, a bisection finds the same
    // indices (a NaN edge compares false everywhere and leaves both at 0, as there)
    const int32_t ne = (int32_t)g.n_tiles_elev;
    const int32_t i = lower_bound_f(g.elev_boundaries, ne + 1, el_lo);
    r.y0 = max(i - 1, 0);
    r.y1 = min(max(i, lower_bound_f(g.elev_boundaries, ne + 1, el_hi)), ne);
    return r;
}

__device__ __forceinline__ int32_t rect_count(const Rect &r) {
    return (r.y1 - r.y0) * (r.x1 - r.x0);
}

constexpr int kMaxElevSmem = 1024;

template <bool kLidar>
struct GridArgs {
    CamGrid cam;
    LidarGrid lidar;
    const void *radii;      // int2 (camera) or float2 (lidar)
    const float2 *means2d;
};

template <bool kLidar>
__device__ __forceinline__ bool elem_rect(const GridArgs<kLidar> &a, uint32_t idx, Rect &r) {
    if (kLidar) {
        const float2 rad = reinterpret_cast<const float2 *>(a.radii)[idx];
        if (!(rad.x > 0.f)) return false;
        r = lidar_rect(a.means2d[idx], rad, a.lidar);
    } else {
        const int2 rad = reinterpret_cast<const int2 *>(a.radii)[idx];
        if (rad.x <= 0) return false;
        r = cam_rect(a.means2d[idx], rad, a.cam);
    }
    return true;
}

// Copies the elevation boundaries to shared memory when they fit and repoints the grid.
template <bool kLidar>
__device__ __forceinline__ void stage_boundaries(GridArgs<kLidar> &a, float *sb) {
    if (kLidar) {
        const uint32_t nb = a.lidar.n_tiles_elev + 1;
        if (nb <= kMaxElevSmem) {
            for (uint32_t i = threadIdx.x; i < nb; i += blockDim.x) sb[i] = a.lidar.elev_boundaries[i];
            __syncthreads();
            a.lidar.elev_boundaries = sb;
        }
    }
}

// ---------------------------------------------------------------------------------------
// Depth order by buckets. The visible elements are ordered by (depth bits, flatten index) - what a
// stable radix sort of the depth bits from flatten order gives - in four short kernels instead of
// twelve. The depth range [dmin, dmax] of the listed elements comes with the rectangle count; an
// element's bucket is its depth's position in that range, in 262144 equal steps of depth (equal
// steps of the bit pattern would crowd the far half of the range into a few buckets): a weakly
// monotone function of the depth, so buckets are ordered like the keys. Count per bucket (global
// atomics), scan, scatter into bucket order with an atomic cursor per bucket (arbitrary order
// inside a bucket), then every element finds its rank inside its bucket by counting the bucket's
// elements that precede it in (bits, flatten index) order and is written to its final place: one
// thread per element, neighbours share their bucket. For a million depths between 0.3 and 113 m a
// bucket holds 4 elements on average and 17 where they are densest. Elements of a bucket with more than kBucketMax entries
// (depths that agree to within half a millimetre by the thousand) are passed through unordered and reported
// with status bit ST_DEPTH_BUCKETS: the caller repeats the plan with the radix sort (sort = 2).
// ---------------------------------------------------------------------------------------
constexpr uint32_t kDepthBucketsMax = 262144, kDepthBucketsMin = 8192;
constexpr uint32_t kBucketMax = 1024;

// One bucket per element, rounded up to a power of two within the limits above: a frame of 20,000
// Gaussians scans 32,768 buckets, not 262,144 (bucket scan 13 -> 5 us).
__host__ __device__ inline uint32_t depth_bucket_count(uint64_t total) {
    uint32_t n = kDepthBucketsMin;
    while (n < kDepthBucketsMax && n < total) n *= 2;
    return n;
}

// How the elements are grouped before their depths order them: by sensor for the block split (every
// sensor then owns `per` consecutive buckets and its entries are consecutive), not at all otherwise.
struct BucketLayout {
    const int64_t *camera_ids;   // packed: sensor of each row, else nullptr
    uint32_t N;                  // Gaussians per sensor ([C, N] layout)
    uint32_t groups;             // sensors, or 1
    uint32_t per;                // buckets per group
    __device__ __forceinline__ uint32_t group(uint32_t idx) const {
        if (groups == 1u) return 0u;
        return camera_ids ? (uint32_t)__ldg(camera_ids + idx) : idx / N;
    }
};

struct DepthBuckets {
    float dmin, scale;
    uint32_t per;
    __device__ __forceinline__ uint32_t operator()(uint32_t bits) const {
        const float d = __uint_as_float(bits);
        if (!(d == d)) return per - 1;             // NaN patterns sort behind +infinity
        const float x = (d - dmin) * scale;        // weakly monotone in d for finite dmin, scale >= 0
        if (!(x > 0.f)) return 0u;                 // depths below a range given by the caller
        return x >= (float)(per - 1) ? per - 1 : (uint32_t)x;
    }
};

// The buckets span the range the caller gave for this frame (its last frame's, widened: depths
// outside it fall into the end buckets, which keeps the bucket index monotone in depth, and the
// ranks inside a bucket go by the full key) or, without one, the measured range of this frame.
__device__ __forceinline__ DepthBuckets depth_buckets(const int64_t *counters, uint32_t per) {
    const bool given = (uint32_t)counters[CNT_BHI] >= (uint32_t)counters[CNT_BLO];
    const uint32_t lo = (uint32_t)counters[given ? CNT_BLO : CNT_DMIN];
    const uint32_t hi = min((uint32_t)counters[given ? CNT_BHI : CNT_DMAX], 0x7f800000u);   // a NaN maximum counts as +infinity
    DepthBuckets b;
    b.per = per;
    b.dmin = __uint_as_float(min(lo, hi));
    const float range = __uint_as_float(hi) - b.dmin;
    b.scale = (range > 0.f) ? (float)(per - 1) / range : 0.f;   // infinite range: scale 0, one bucket
    return b;
}

// {count, sequence number, status bits} for a polling host, stored by whichever kernel knows them first
// into mapped pinned memory: count and status, a system-wide fence, then the sequence number.
__device__ __forceinline__ void tell_host(volatile int64_t *early_host, int64_t seq, int64_t n_isects,
                                          int64_t status, int64_t depth_range = 0) {
    early_host[0] = n_isects;
    early_host[2] = status;
    early_host[3] = depth_range;   // dmin bits | dmax bits << 32 of the listed elements, 0: not known here
    __threadfence_system();
    early_host[1] = seq;   // on its way at the latest when the kernel ends
}

// tiles_per_gauss[idx] for every (sensor, Gaussian) / packed row. With `rect` the rectangle is also
// stored for the block split, packed into two words per element ({x0 | width << 16, y0 | height << 16},
// the first column wrapped into the row; used only when the geometry is within its limits), and the
// total is added to *n_isects.
constexpr int kCountThreads = 1024;   // few, large blocks: every block ends with a handful of same-address atomics

template <bool kLidar>
__global__ void __launch_bounds__(kCountThreads)
isect_count_kernel(GridArgs<kLidar> a, uint32_t total, int32_t *__restrict__ tiles_per_gauss,
                   BucketLayout layout, uint2 *__restrict__ rect, int64_t *__restrict__ n_isects,
                   int64_t *__restrict__ ticket /* with early_host: a zeroed counter */,
                   volatile int64_t *early_host /* optional, host-mapped: {count, sequence number, status} */,
                   int64_t early_seq,
                   const uint32_t *__restrict__ depth_bits /* optional: depth range of the listed elements */,
                   int64_t *__restrict__ counters /* with depth_bits: CNT_DMIN / CNT_DMAX / CNT_NVIS */,
                   uint32_t *__restrict__ bcount /* optional, with a given bucket range: the bucket counts */) {
    chain_enter();
    DepthBuckets bucket{0.f, 0.f, 1u};
    if (bcount != nullptr) bucket = depth_buckets(counters, layout.per);
    __shared__ float sb[kLidar ? kMaxElevSmem : 1];
    __shared__ unsigned long long wsum[kCountThreads / 32];
    stage_boundaries<kLidar>(a, sb);
    unsigned long long sum = 0;
    uint32_t dmin = 0xffffffffu, dmax = 0u, nvis = 0u;
    for (uint32_t idx = blockIdx.x * blockDim.x + threadIdx.x; idx < total;
         idx += gridDim.x * blockDim.x) {
        Rect r;
        int32_t cnt = 0;
        uint2 packed = make_uint2(0u, 0u);
        if (elem_rect<kLidar>(a, idx, r)) {
            cnt = rect_count(r);
            if (rect != nullptr && cnt > 0) {
                int32_t x0 = r.x0;
                if (kLidar) {
                    const int32_t n = (int32_t)a.lidar.n_tiles_azim;
                    if (x0 < 0 || x0 >= n) {
                        x0 %= n;
                        if (x0 < 0) x0 += n;
                    }
                }
                packed = make_uint2((uint32_t)x0 | ((uint32_t)(r.x1 - r.x0) << 16),
                                    (uint32_t)r.y0 | ((uint32_t)(r.y1 - r.y0) << 16));
            }
        }
        tiles_per_gauss[idx] = cnt;
        if (rect != nullptr) rect[idx] = packed;
        sum += (unsigned long long)(cnt > 0 ? cnt : 0);
        if (depth_bits != nullptr && cnt > 0) {
            const uint32_t d = __ldg(depth_bits + idx);
            dmin = min(dmin, d);
            dmax = max(dmax, d);
            ++nvis;
            if (bcount != nullptr) atomicAdd(&bcount[layout.group(idx) * layout.per + bucket(d)], 1u);
        }
    }
    if (depth_bits != nullptr) {
        __shared__ uint32_t s_rng[3];
        if (threadIdx.x == 0) { s_rng[0] = 0xffffffffu; s_rng[1] = 0u; s_rng[2] = 0u; }
        __syncthreads();
        dmin = __reduce_min_sync(0xffffffffu, dmin);
        dmax = __reduce_max_sync(0xffffffffu, dmax);
        nvis = __reduce_add_sync(0xffffffffu, nvis);
        if ((threadIdx.x & 31) == 0 && nvis) {
            atomicMin(&s_rng[0], dmin);
            atomicMax(&s_rng[1], dmax);
            atomicAdd(&s_rng[2], nvis);
        }
        __syncthreads();
        if (threadIdx.x == 0 && s_rng[2]) {
            atomicMin(reinterpret_cast<unsigned int *>(counters + CNT_DMIN), s_rng[0]);
            atomicMax(reinterpret_cast<unsigned int *>(counters + CNT_DMAX), s_rng[1]);
            atomicAdd(reinterpret_cast<unsigned long long *>(counters + CNT_NVIS), (unsigned long long)s_rng[2]);
        }
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, off);
    if ((threadIdx.x & 31) == 0) wsum[threadIdx.x >> 5] = sum;
    __syncthreads();
    if (threadIdx.x == 0) {
        unsigned long long t = 0;
        for (uint32_t w = 0; w < blockDim.x / 32; ++w) t += wsum[w];
        if (t) atomicAdd((unsigned long long *)n_isects, t);
        if (early_host != nullptr) {
            // the block that finishes last hands the total straight to the host (a store to mapped
            // pinned memory): nobody waits on anybody, and no copy sits between this kernel and the next
            __threadfence();
            if (atomicAdd((unsigned long long *)ticket, 1ull) + 1ull == (unsigned long long)gridDim.x) {
                __threadfence();
                const unsigned long long total_isects = atomicAdd((unsigned long long *)n_isects, 0ull);
                *ticket = 0;
                tell_host(early_host, early_seq, (int64_t)total_isects, 0);
            }
        }
    }
}

// ---------------------------------------------------------------------------------------
// Radix sort passes (stable LSD, up to 8 bits per pass) on (uint32 key, uint32 value) pairs.
// Each of the kSortGrid blocks owns a contiguous run of 2048-item tiles.
//   upsweep:   per-block digit histogram            -> hist[digit][block]
//   rowscan:   exclusive scan of each digit's row   -> hist (in place), digit_totals
//   downsweep: stable rank + scatter (through shared memory so global writes are runs)
// Source of a pass is either a pair buffer with a device-side count, or (kGen) the implicit
// list idx = 0..total-1 with key = depth bits, value = idx, restricted to tiles_per_gauss>0.
// ---------------------------------------------------------------------------------------
struct PassSrc {
    const uint32_t *keys;            // pair source
    const uint32_t *vals;
    const int64_t *n_ptr;            // device count (pair source)
    const uint32_t *depth_bits;      // gen source
    const int32_t *tiles_per_gauss;  // gen source
    uint32_t total;                  // gen source length
    uint32_t n_cap;                  // pair source: upper bound on the count (buffer size); 0 = none
};

template <bool kGen>
__device__ __forceinline__ uint32_t src_count(const PassSrc &s) {
    if (kGen) return s.total;
    int64_t n = *s.n_ptr;
    if (s.n_cap != 0 && n > (int64_t)s.n_cap) n = (int64_t)s.n_cap;
    return (uint32_t)n;
}

__device__ __forceinline__ void block_range(uint32_t n, uint32_t &lo, uint32_t &hi) {
    const uint32_t tiles = (n + kTileItems - 1) / kTileItems;
    const uint32_t per = (tiles + gridDim.x - 1) / gridDim.x;
    const uint64_t l = (uint64_t)blockIdx.x * per * kTileItems;
    const uint64_t h = l + (uint64_t)per * kTileItems;
    lo = (uint32_t)(l < n ? l : n);
    hi = (uint32_t)(h < n ? h : n);
}

// Adds one key to the warp-private digit histogram (order is irrelevant for a histogram, so
// plain shared-memory atomics are used; a warp whose 32 keys share one digit - typical for the
// high tile-key digit - does a single add instead of a 32-way serialised atomic).
__device__ __forceinline__ void hist_add(uint32_t *wh_row, bool valid, uint32_t key, int shift,
                                         uint32_t mask, uint32_t lane) {
    const uint32_t digit = valid ? ((key >> shift) & mask) : 0xffffffffu;
    const uint32_t d0 = __shfl_sync(0xffffffffu, digit, 0);
    if (__all_sync(0xffffffffu, digit == d0)) {
        if (lane == 0 && valid) wh_row[d0] += 32u;
        __syncwarp();
    } else if (valid) {
        atomicAdd(&wh_row[digit], 1u);
    }
}

template <bool kGen>
__global__ void __launch_bounds__(kSortThreads)
radix_upsweep_kernel(PassSrc s, int shift, uint32_t mask, uint32_t *__restrict__ hist) {
    chain_enter();
    __shared__ uint32_t wh[kSortWarps][kRadixBins];
    for (uint32_t i = threadIdx.x; i < kSortWarps * kRadixBins; i += blockDim.x) (&wh[0][0])[i] = 0u;
    __syncthreads();
    const uint32_t n = src_count<kGen>(s);
    uint32_t lo, hi;
    block_range(n, lo, hi);   // lo is a multiple of 4096
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint32_t *row = wh[warp];
    const uint32_t *kp = kGen ? s.depth_bits : s.keys;
    const bool aligned = (reinterpret_cast<uintptr_t>(kp) & 15u) == 0 &&
                         (!kGen || (reinterpret_cast<uintptr_t>(s.tiles_per_gauss) & 15u) == 0);
    constexpr uint32_t kStep = kSortThreads * 8;   // two 128-bit loads per thread and iteration
    uint32_t base = lo;
    if (aligned) {
        for (; base + kStep <= hi; base += kStep) {
            const uint32_t i0 = base + threadIdx.x * 4, i1 = i0 + kSortThreads * 4;
            const uint4 k0 = __ldg(reinterpret_cast<const uint4 *>(kp + i0));
            const uint4 k1 = __ldg(reinterpret_cast<const uint4 *>(kp + i1));
            int4 c0 = make_int4(1, 1, 1, 1), c1 = c0;
            if (kGen) {
                c0 = __ldg(reinterpret_cast<const int4 *>(s.tiles_per_gauss + i0));
                c1 = __ldg(reinterpret_cast<const int4 *>(s.tiles_per_gauss + i1));
            }
            hist_add(row, c0.x > 0, k0.x, shift, mask, lane);
            hist_add(row, c0.y > 0, k0.y, shift, mask, lane);
            hist_add(row, c0.z > 0, k0.z, shift, mask, lane);
            hist_add(row, c0.w > 0, k0.w, shift, mask, lane);
            hist_add(row, c1.x > 0, k1.x, shift, mask, lane);
            hist_add(row, c1.y > 0, k1.y, shift, mask, lane);
            hist_add(row, c1.z > 0, k1.z, shift, mask, lane);
            hist_add(row, c1.w > 0, k1.w, shift, mask, lane);
        }
    }
    for (; base < hi; base += kSortThreads) {
        const uint32_t i = base + threadIdx.x;
        bool valid = i < hi;
        uint32_t key = 0;
        if (valid) {
            if (kGen) valid = s.tiles_per_gauss[i] > 0;
            if (valid) key = kp[i];
        }
        hist_add(row, valid, key, shift, mask, lane);
    }
    __syncthreads();
    for (uint32_t d = threadIdx.x; d < kRadixBins; d += blockDim.x) {
        uint32_t sum = 0;
#pragma unroll
        for (int w = 0; w < kSortWarps; ++w) sum += wh[w][d];
        hist[(size_t)d * gridDim.x + blockIdx.x] = sum;
    }
}

// One block per digit; blockDim.x >= grid size of the sort kernels (multiple of 32).
__global__ void radix_rowscan_kernel(uint32_t *__restrict__ hist, uint32_t nblocks,
                                     uint32_t *__restrict__ digit_totals) {
    chain_enter();
    __shared__ uint32_t wt[33];
    const uint32_t d = blockIdx.x;
    const uint32_t b = threadIdx.x;
    uint32_t v = (b < nblocks) ? hist[(size_t)d * nblocks + b] : 0u;
    uint32_t total;
    const uint32_t ex = block_excl_scan(v, wt, total);
    if (b < nblocks) hist[(size_t)d * nblocks + b] = ex;
    if (b == 0) digit_totals[d] = total;
}

struct FinalOut {
    int64_t *isect_ids;          // [capacity]
    int32_t *flatten_ids;        // [capacity]
    const uint32_t *depth_bits;  // [total elems]
    uint32_t n_tiles;            // tiles per sensor
    uint32_t tile_n_bits;
    int64_t capacity;
};

template <bool kGen, bool kFinal>
__global__ void __launch_bounds__(kSortThreads)
radix_downsweep_kernel(PassSrc s, int shift, int nbits, uint32_t mask, const uint32_t *__restrict__ hist,
                       const uint32_t *__restrict__ digit_totals, uint32_t *__restrict__ keys_out,
                       uint32_t *__restrict__ vals_out, FinalOut fin,
                       int64_t *__restrict__ n_out /* optional: total valid count */) {
    chain_enter();
    __shared__ uint32_t wh[kSortWarps][kRadixBins];
    __shared__ uint32_t digit_base[kRadixBins];
    __shared__ uint32_t tile_excl[kRadixBins];
    __shared__ uint32_t tile_cnt[kRadixBins];
    __shared__ uint32_t wt[33];
    __shared__ uint32_t st_keys[kTileItems];
    __shared__ uint32_t st_vals[kTileItems];

    const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    {
        uint32_t tot;
        const uint32_t dt = digit_totals[tid];
        const uint32_t ex = block_excl_scan(dt, wt, tot);
        digit_base[tid] = ex + hist[(size_t)tid * gridDim.x + blockIdx.x];
        if (n_out != nullptr && blockIdx.x == 0 && tid == 0) *n_out = (int64_t)tot;
    }
    __syncthreads();

    const uint32_t n = src_count<kGen>(s);
    uint32_t lo, hi;
    block_range(n, lo, hi);

    for (uint32_t tile_lo = lo; tile_lo < hi; tile_lo += kTileItems) {
        for (uint32_t i = tid; i < kSortWarps * kRadixBins; i += kSortThreads) (&wh[0][0])[i] = 0u;
        __syncthreads();

        uint32_t keys[kItemsPerLane], vals[kItemsPerLane];
        uint16_t ranks[kItemsPerLane];
        uint32_t validmask = 0;
        const uint32_t wbase = tile_lo + warp * kWarpItems + lane;
#pragma unroll
        for (int r = 0; r < kItemsPerLane; ++r) {
            const uint32_t i = wbase + r * 32;
            bool valid = i < hi;
            uint32_t key = 0, val = 0;
            if (valid) {
                if (kGen) {
                    valid = s.tiles_per_gauss[i] > 0;
                    if (valid) { key = s.depth_bits[i]; val = i; }
                } else {
                    key = s.keys[i];
                    val = s.vals[i];
                }
            }
            keys[r] = key; vals[r] = val;
            if (valid) validmask |= (1u << r);
        }
#pragma unroll
        for (int r = 0; r < kItemsPerLane; ++r) {
            const bool valid = (validmask >> r) & 1u;
            const uint32_t digit = valid ? ((keys[r] >> shift) & mask) : kRadixBins;
            // lanes with the same digit: one ballot per digit bit (cheaper than match.any when
            // a warp holds many distinct digits)
            uint32_t peers = __ballot_sync(0xffffffffu, valid);
            for (int b = 0; b < nbits; ++b) {
                const uint32_t bal = __ballot_sync(0xffffffffu, (digit >> b) & 1u);
                peers &= ((digit >> b) & 1u) ? bal : ~bal;
            }
            if (!valid) peers = 1u << lane;
            const uint32_t leader = (uint32_t)(__ffs(peers) - 1);
            uint32_t old = 0;
            if (valid && lane == leader) {
                old = wh[warp][digit];
                wh[warp][digit] = old + __popc(peers);
            }
            old = __shfl_sync(0xffffffffu, old, leader);
            ranks[r] = (uint16_t)(old + __popc(peers & ((1u << lane) - 1u)));
            __syncwarp();
        }
        __syncthreads();
        // per digit: exclusive offsets of the warps, tile count, then exclusive scan over digits
        {
            uint32_t run = 0;
#pragma unroll
            for (int w = 0; w < kSortWarps; ++w) {
                const uint32_t c = wh[w][tid];
                wh[w][tid] = run;
                run += c;
            }
            tile_cnt[tid] = run;
            uint32_t tot;
            tile_excl[tid] = block_excl_scan(run, wt, tot);
        }
        __syncthreads();
#pragma unroll
        for (int r = 0; r < kItemsPerLane; ++r) {
            if ((validmask >> r) & 1u) {
                const uint32_t digit = (keys[r] >> shift) & mask;
                const uint32_t pos = tile_excl[digit] + wh[warp][digit] + ranks[r];
                st_keys[pos] = keys[r];
                st_vals[pos] = vals[r];
            }
        }
        __syncthreads();
        const uint32_t tile_n = tile_excl[kRadixBins - 1] + tile_cnt[kRadixBins - 1];
        for (uint32_t j = tid; j < tile_n; j += kSortThreads) {
            const uint32_t k = st_keys[j];
            const uint32_t v = st_vals[j];
            const uint32_t digit = (k >> shift) & mask;
            const uint32_t gpos = digit_base[digit] + (j - tile_excl[digit]);
            if (kFinal) {
                if ((int64_t)gpos < fin.capacity) {
                    const uint32_t cid = k / fin.n_tiles;
                    const uint32_t tile = k - cid * fin.n_tiles;
                    const int64_t id = ((int64_t)cid << (32 + fin.tile_n_bits)) |
                                       ((int64_t)tile << 32) | (int64_t)fin.depth_bits[v];
                    fin.isect_ids[gpos] = id;
                    fin.flatten_ids[gpos] = (int32_t)v;
                }
            } else {
                keys_out[gpos] = k;
                vals_out[gpos] = v;
            }
        }
        __syncthreads();
        digit_base[tid] += tile_cnt[tid];
        __syncthreads();
    }
}

__global__ void __launch_bounds__(kThreads)
depth_bucket_count_kernel(const uint32_t *__restrict__ depth_bits, const int32_t *__restrict__ tiles_per_gauss,
                          uint32_t total, BucketLayout layout, const int64_t *__restrict__ counters,
                          uint32_t *__restrict__ bcount) {
    chain_enter();
    const DepthBuckets bucket = depth_buckets(counters, layout.per);
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < total; i += gridDim.x * blockDim.x)
        if (tiles_per_gauss[i] > 0)
            atomicAdd(&bcount[layout.group(i) * layout.per + bucket(__ldg(depth_bits + i))], 1u);
}

// Blocks of 1024 threads, one bucket per thread: starts within the block's 1024 buckets, counts
// back to zero (they become the scatter's cursors), the block's total. The block that finishes
// last turns the block totals into block offsets (a bucket's start = bstart[b] + boff[b >> 10]), sets
// the status bit for oversized buckets and - for a grouped order -
// notes where every group's entries and its chunks of `chunk` entries start.
__global__ void __launch_bounds__(1024)
depth_bucket_scan_kernel(uint32_t *__restrict__ bcount, uint32_t *__restrict__ bstart, uint32_t *__restrict__ boff,
                         int64_t *__restrict__ counters, uint32_t groups, uint32_t per, uint32_t chunk, uint32_t *__restrict__ group_start,
                         uint32_t *__restrict__ group_chunk /* both [groups + 1]; nullptr: not asked for */) {
    chain_enter();
    __shared__ uint32_t wt[33];
    __shared__ bool s_last;
    const uint32_t n_scan = gridDim.x;
    const uint32_t b = blockIdx.x * 1024 + threadIdx.x;
    const uint32_t c = bcount[b];
    bcount[b] = 0u;
    uint32_t total;
    bstart[b] = block_excl_scan(c, wt, total);
    const bool big = __syncthreads_or(c > kBucketMax);
    if (threadIdx.x == 0) {
        boff[n_scan + 1 + blockIdx.x] = total;
        if (big) atomicOr((unsigned long long *)&counters[CNT_STATUS], (unsigned long long)ST_DEPTH_BUCKETS);
        __threadfence();
        s_last = atomicAdd((unsigned long long *)&counters[CNT_TICKET], 1ull) + 1ull == (unsigned long long)gridDim.x;
    }
    __syncthreads();
    if (!s_last) return;
    __threadfence();
    if (threadIdx.x < 32) {
        // the block totals: kScanPerLane consecutive ones per lane
        constexpr uint32_t kScanPerLane = kDepthBucketsMax / 1024 / 32;
        const volatile uint32_t *tot = boff + n_scan + 1;
        uint32_t v[kScanPerLane], sum = 0;
#pragma unroll
        for (uint32_t k = 0; k < kScanPerLane; ++k) {
            const uint32_t i = kScanPerLane * threadIdx.x + k;
            v[k] = i < n_scan ? tot[i] : 0u;
            sum += v[k];
        }
        uint32_t inc = sum;
#pragma unroll
        for (int off = 1; off < 32; off <<= 1) {
            const uint32_t o = __shfl_up_sync(0xffffffffu, inc, off);
            if (threadIdx.x >= (uint32_t)off) inc += o;
        }
        uint32_t run = inc - sum;
#pragma unroll
        for (uint32_t k = 0; k < kScanPerLane; ++k) {
            const uint32_t i = kScanPerLane * threadIdx.x + k;
            if (i < n_scan) boff[i] = run;
            run += v[k];
        }
        if (threadIdx.x == 31) {
            boff[n_scan] = inc;
            counters[CNT_TICKET] = 0;
            __threadfence();
        }
    }
    if (group_start == nullptr) return;
    __syncthreads();
    const uint32_t n = boff[n_scan];
    uint32_t chunks = 0;
    for (uint32_t g0 = 0; g0 < groups; g0 += 1024) {
        const uint32_t g = g0 + threadIdx.x;
        uint32_t lo = 0, mine = 0;
        if (g < groups) {
            const uint32_t first = g * per, next = first + per;   // next <= buckets
            lo = __ldcg(bstart + first) + boff[first >> 10];
            const uint32_t hi = (next >> 10) < n_scan ? __ldcg(bstart + next) + boff[next >> 10] : n;
            mine = (hi - lo + chunk - 1) / chunk;
        }
        uint32_t round;
        const uint32_t ex = block_excl_scan(mine, wt, round);
        if (g < groups) {
            group_start[g] = lo;
            group_chunk[g] = chunks + ex;
        }
        chunks += round;
    }
    if (threadIdx.x == 0) {
        group_start[groups] = n;
        group_chunk[groups] = chunks;
    }
}

__global__ void __launch_bounds__(kThreads)
depth_bucket_scatter_kernel(const uint32_t *__restrict__ depth_bits, const int32_t *__restrict__ tiles_per_gauss,
                            uint32_t total, BucketLayout layout, const int64_t *__restrict__ counters,
                            volatile int64_t *early_host /* optional: the polling host's words */, int64_t early_seq,
                            volatile int64_t *listed_host /* optional, with early_host: elements listed */,
                            const uint32_t *__restrict__ bstart, const uint32_t *__restrict__ boff,
                            uint32_t *__restrict__ bcursor, uint2 *__restrict__ pairs /* {bits, flatten index} */) {
    chain_enter();
    // All the host wants to know is there since the bucket scan. Telling it takes a fence over the host link, which
    // would be the end of that kernel's last block; here the other blocks' work covers it (20,000 Gaussians: 4 us).
    if (early_host != nullptr && blockIdx.x == gridDim.x - 1 && threadIdx.x == blockDim.x - 1) {
        if (listed_host != nullptr) *listed_host = counters[CNT_NVIS];
        tell_host(early_host, early_seq, counters[CNT_NISECT], counters[CNT_STATUS],
                  (int64_t)(((unsigned long long)(uint32_t)counters[CNT_DMAX] << 32) |
                            (unsigned long long)(uint32_t)counters[CNT_DMIN]));
    }
    const DepthBuckets bucket = depth_buckets(counters, layout.per);
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < total; i += gridDim.x * blockDim.x) {
        if (tiles_per_gauss[i] <= 0) continue;
        const uint32_t d = __ldg(depth_bits + i);
        const uint32_t b = layout.group(i) * layout.per + bucket(d);
        const uint32_t pos = bstart[b] + boff[b >> 10] + atomicAdd(&bcursor[b], 1u);
        pairs[pos] = make_uint2(d, i);
    }
}

// One thread per scattered element: its rank among the elements of its bucket in (bits, flatten
// index) order, by counting, and the move to its final place. Neighbouring threads hold neighbouring
// elements, almost always of the same bucket: the loads of the loop are broadcasts.
__global__ void __launch_bounds__(kThreads)
depth_bucket_rank_kernel(BucketLayout layout, uint32_t n_buckets, const int64_t *__restrict__ counters,
                         const uint32_t *__restrict__ bstart, const uint32_t *__restrict__ boff,
                         const uint2 *__restrict__ pairs, const uint2 *__restrict__ rect,
                         uint2 *__restrict__ sorted_pair /* with rect: {depth bits, flatten index} */,
                         uint2 *__restrict__ sorted_rect, uint32_t *__restrict__ order /* without rect */) {
    chain_enter();
    const DepthBuckets bucket = depth_buckets(counters, layout.per);
    const uint32_t n = boff[n_buckets >> 10];
    for (uint32_t p = blockIdx.x * blockDim.x + threadIdx.x; p < n; p += gridDim.x * blockDim.x) {
        const uint2 mine = __ldg(pairs + p);
        const uint32_t key = mine.x, val = mine.y;
        const uint32_t b = layout.group(val) * layout.per + bucket(key);
        const uint32_t lo = bstart[b] + boff[b >> 10];
        const uint32_t hi = ((b + 1) & 1023u) ? bstart[b + 1] + boff[b >> 10] : boff[(b + 1) >> 10];   // boff ends with n
        uint32_t rank = p - lo;                      // crowded bucket: passed through as it is
        if (hi - lo <= kBucketMax) {
            rank = 0;
            const unsigned long long me = ((unsigned long long)key << 32) | val;
#pragma unroll 4
            for (uint32_t j = lo; j < hi; ++j) {
                const uint2 o = __ldg(pairs + j);
                rank += ((((unsigned long long)o.x << 32) | o.y) < me) ? 1u : 0u;
            }
        }
        if (rect != nullptr) {
            sorted_pair[lo + rank] = mine;
            sorted_rect[lo + rank] = __ldg(rect + val);
        } else {
            order[lo + rank] = val;
        }
    }
}

// ---------------------------------------------------------------------------------------
// The block split's input from a depth order of radix passes: the entries of all sensors lie in one sequence by
// depth, so with several sensors further passes - stable, by the sensor - group them, and the sorted sensors say where
// each one's begin. Without this, crowded depths had to take the radix split over (tile, entry) pairs: a
// million Gaussians, fifty of them seven kilometres away, 591 us a lidar frame and 332 with it.
// ---------------------------------------------------------------------------------------
__global__ void __launch_bounds__(kThreads)
entry_sensors_kernel(BucketLayout layout, const int64_t *__restrict__ n_entries, const uint32_t *__restrict__ order,
                     uint32_t *__restrict__ keys) {
    chain_enter();
    const uint32_t n = (uint32_t)*n_entries;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) keys[i] = layout.group(order[i]);
}

// First entry and first chunk of every group; `keys` ascending (not looked at for one group). One block.
__global__ void __launch_bounds__(1024)
group_starts_kernel(const int64_t *__restrict__ n_entries, const uint32_t *__restrict__ keys, uint32_t groups, uint32_t chunk,
                    uint32_t *__restrict__ group_start, uint32_t *__restrict__ group_chunk /* both [groups + 1] */) {
    chain_enter();
    __shared__ uint32_t wt[33];
    const uint32_t n = (uint32_t)*n_entries;
    const auto first_of = [&](uint32_t g) {
        if (g == 0u) return 0u;
        uint32_t lo = 0, hi = n;
        while (lo < hi && g < groups) {
            const uint32_t m = (lo + hi) >> 1;
            if (keys[m] < g) lo = m + 1; else hi = m;
        }
        return g < groups ? lo : n;
    };
    uint32_t chunks = 0;
    for (uint32_t g0 = 0; g0 < groups; g0 += 1024) {
        const uint32_t g = g0 + threadIdx.x;
        uint32_t lo = 0, mine = 0;
        if (g < groups) {
            lo = first_of(g);
            mine = (first_of(g + 1) - lo + chunk - 1) / chunk;
        }
        uint32_t round;
        const uint32_t ex = block_excl_scan(mine, wt, round);
        if (g < groups) {
            group_start[g] = lo;
            group_chunk[g] = chunks + ex;
        }
        chunks += round;
    }
    if (threadIdx.x == 0) {
        group_start[groups] = n;
        group_chunk[groups] = chunks;
    }
}

__global__ void __launch_bounds__(kThreads)
gather_entries_kernel(const int64_t *__restrict__ n_entries, const uint32_t *__restrict__ order,
                      const uint32_t *__restrict__ depth_bits, const uint2 *__restrict__ rect,
                      uint2 *__restrict__ sorted_pair /* {depth bits, flatten index} */, uint2 *__restrict__ sorted_rect) {
    chain_enter();
    const uint32_t n = (uint32_t)*n_entries;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const uint32_t v = order[i];
        sorted_pair[i] = make_uint2(__ldg(depth_bits + v), v);
        sorted_rect[i] = __ldg(rect + v);
    }
}

// ---------------------------------------------------------------------------------------
// Emission of (compact tile key, flatten index) pairs in depth order.
// ---------------------------------------------------------------------------------------
struct EmitArgs {
    const uint32_t *order;           // [n_vis] flatten indices in depth order, or nullptr = identity
    const int64_t *n_order_ptr;      // device count of `order` (ignored for identity)
    uint32_t total;                  // identity length
    const int32_t *tiles_per_gauss;  // [total]
    const int64_t *camera_ids;       // packed: sensor of each row, else nullptr
    uint32_t N;                      // Gaussians per sensor ([C, N] layout)
    uint32_t n_tiles;                // tiles per sensor
    uint32_t tile_n_bits;
    const uint32_t *depth_bits;
    int64_t capacity;
};

__device__ __forceinline__ void emit_range(const EmitArgs &e, uint32_t &lo, uint32_t &hi) {
    const uint32_t n = e.order ? (uint32_t)(*e.n_order_ptr) : e.total;
    const uint32_t chunks = (n + kThreads - 1) / kThreads;
    const uint32_t per = (chunks + gridDim.x - 1) / gridDim.x;
    const uint64_t l = (uint64_t)blockIdx.x * per * kThreads;
    const uint64_t h = l + (uint64_t)per * kThreads;
    lo = (uint32_t)(l < n ? l : n);
    hi = (uint32_t)(h < n ? h : n);
}

__global__ void __launch_bounds__(kThreads)
emit_blocksum_kernel(EmitArgs e, unsigned long long *__restrict__ block_sums) {
    __shared__ unsigned long long ws[kThreads / 32];
    uint32_t lo, hi;
    emit_range(e, lo, hi);
    unsigned long long sum = 0;
    for (uint32_t p = lo + threadIdx.x; p < hi; p += kThreads) {
        const uint32_t idx = e.order ? e.order[p] : p;
        const int32_t c = e.tiles_per_gauss[idx];
        sum += (unsigned long long)(c > 0 ? c : 0);
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, off);
    if ((threadIdx.x & 31) == 0) ws[threadIdx.x >> 5] = sum;
    __syncthreads();
    if (threadIdx.x == 0) {
        unsigned long long t = 0;
        for (int w = 0; w < kThreads / 32; ++w) t += ws[w];
        block_sums[blockIdx.x] = t;
    }
}

// Single block (1024 threads): exclusive scan of the per-block sums; writes n_isects and the
// status word.
__global__ void __launch_bounds__(1024)
emit_scan_kernel(const unsigned long long *__restrict__ block_sums, uint32_t nblocks,
                 unsigned long long *__restrict__ block_offs, int64_t *__restrict__ counters) {
    __shared__ unsigned long long part[1024];
    const uint32_t t = threadIdx.x;
    const unsigned long long v = (t < nblocks) ? block_sums[t] : 0ull;
    part[t] = v;
    __syncthreads();
    for (uint32_t off = 1; off < 1024; off <<= 1) {
        const unsigned long long o = (t >= off) ? part[t - off] : 0ull;
        __syncthreads();
        part[t] += o;
        __syncthreads();
    }
    if (t < nblocks) block_offs[t] = part[t] - v;
    if (t == 1023) {
        const unsigned long long run = part[1023];
        counters[CNT_NISECT] = (int64_t)run;
        if (run > 0x7fffffffull) counters[CNT_STATUS] |= ST_OVERFLOW_INT32;
    }
}

// Exclusive offset of every entry of the emission order: eoff[p] = number of intersections
// emitted before entry p. Same block ranges as emit_blocksum_kernel.
__global__ void __launch_bounds__(kThreads)
emit_offsets_kernel(EmitArgs e, const unsigned long long *__restrict__ block_offs,
                    uint32_t *__restrict__ eoff) {
    __shared__ uint32_t wt[33];
    uint32_t lo, hi;
    emit_range(e, lo, hi);
    uint32_t running = (uint32_t)block_offs[blockIdx.x];
    for (uint32_t base = lo; base < hi; base += kThreads) {
        const uint32_t p = base + threadIdx.x;
        uint32_t cnt = 0;
        if (p < hi) {
            const uint32_t idx = e.order ? e.order[p] : p;
            const int32_t c = e.tiles_per_gauss[idx];
            cnt = (uint32_t)(c > 0 ? c : 0);
        }
        uint32_t chunk_total;
        const uint32_t ex = block_excl_scan(cnt, wt, chunk_total);
        if (p < hi) eoff[p] = running + ex;
        running += chunk_total;
    }
}

constexpr uint32_t kEmitPerThread = 16;
constexpr uint32_t kEmitUnit = kThreads * kEmitPerThread;   // 4096 intersections per work unit
constexpr uint32_t kEmitEntries = 1024;                     // entries staged per sub-chunk
constexpr uint32_t kEmitUnitsPerBatch = 64;                 // unit windows searched at once

// last p in [lo, hi] with eoff[p] <= q (eoff is non-decreasing, eoff[lo] <= q)
__device__ __forceinline__ uint32_t find_entry(const uint32_t *__restrict__ eoff, uint32_t lo,
                                               uint32_t hi, uint32_t q) {
    while (lo < hi) {
        const uint32_t m = (lo + hi + 1) >> 1;
        if (__ldg(eoff + m) <= q) lo = m; else hi = m - 1;
    }
    return lo;
}

// Writes the intersections in emission order, balanced by OUTPUT position: depth-sorted
// Gaussians have wildly different tile counts (the nearest ones cover thousands of tiles), so
// work is split into units of kEmitUnit consecutive outputs. The entries overlapping a unit are
// staged in shared memory (rectangle computed once per entry), every entry marks the first output
// it owns, and a prefix-max over the unit tells each output which entry it belongs to.
template <bool kLidar, bool kDirect64>
__global__ void __launch_bounds__(kThreads)
emit_kernel(GridArgs<kLidar> a, EmitArgs e, const uint32_t *__restrict__ eoff,
            const int64_t *__restrict__ counters_in, uint32_t *__restrict__ keys_out,
            uint32_t *__restrict__ vals_out, int64_t *__restrict__ ids64_out,
            int32_t *__restrict__ flat_out, int64_t *__restrict__ counters) {
    __shared__ float sb[kLidar ? kMaxElevSmem : 1];
    __shared__ uint32_t s_off[kEmitEntries + 1];
    __shared__ int4 s_rect[kEmitEntries];           // x0, width, y0, sensor
    __shared__ uint32_t s_idx[kEmitEntries];
    __shared__ uint32_t owner[kThreads * (kEmitPerThread + 1)];   // padded: 17 words per thread
    __shared__ uint32_t s_win[2 * kEmitUnitsPerBatch];
    __shared__ uint32_t wmax[kThreads / 32];
    stage_boundaries<kLidar>(a, sb);
    const uint32_t n_entries = e.order ? (uint32_t)(*e.n_order_ptr) : e.total;
    const int64_t m_total = counters_in[CNT_NISECT];
    int64_t m64 = m_total;
    bool overflow = false;
    if (m64 > e.capacity) { m64 = e.capacity; overflow = true; }
    const uint32_t M = (uint32_t)m64;
    if (n_entries == 0 || M == 0) return;
    const uint32_t n_units = (M + kEmitUnit - 1) / kEmitUnit;
    const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;

    for (uint32_t u0 = blockIdx.x; u0 < n_units; u0 += gridDim.x * kEmitUnitsPerBatch) {
        // entry windows of this block's next units, searched in parallel
        __syncthreads();
        if (tid < 2 * kEmitUnitsPerBatch) {
            const uint32_t u = u0 + (tid >> 1) * gridDim.x;
            if (u < n_units) {
                const uint32_t q_lo = u * kEmitUnit;
                const uint32_t q_last = min(M, q_lo + kEmitUnit) - 1;
                s_win[tid] = find_entry(eoff, 0, n_entries - 1, (tid & 1) ? q_last : q_lo);
            }
        }
        __syncthreads();
        for (uint32_t b = 0; b < kEmitUnitsPerBatch; ++b) {
            const uint32_t u = u0 + b * gridDim.x;
            if (u >= n_units) break;
            const uint32_t q_lo = u * kEmitUnit;
            const uint32_t q_hi = min(M, q_lo + kEmitUnit);   // exclusive
            const uint32_t p_lo = s_win[2 * b], p_hi = s_win[2 * b + 1];
            for (uint32_t c_lo = p_lo; c_lo <= p_hi; c_lo += kEmitEntries) {
                const uint32_t c_hi = min(p_hi, c_lo + kEmitEntries - 1);
                const uint32_t n_e = c_hi - c_lo + 1;
                __syncthreads();
                for (uint32_t i = tid; i < n_e; i += kThreads) {
                    const uint32_t p = c_lo + i;
                    const uint32_t idx = e.order ? __ldg(e.order + p) : p;
                    Rect r;
                    int4 packed = make_int4(0, 0, 0, 0);
                    if (elem_rect<kLidar>(a, idx, r)) {
                        packed.x = r.x0;
                        packed.y = r.x1 - r.x0;
                        packed.z = r.y0;
                        packed.w = (int32_t)(e.camera_ids ? (uint32_t)e.camera_ids[idx] : idx / e.N);
                    }
                    s_off[i] = __ldg(eoff + p);
                    s_rect[i] = packed;
                    s_idx[i] = idx;
                }
                if (tid == 0)
                    s_off[n_e] = (c_hi + 1 < n_entries) ? __ldg(eoff + c_hi + 1)
                                                        : (uint32_t)min(m_total, (int64_t)0xffffffffll);
                for (uint32_t i = tid; i < kThreads * (kEmitPerThread + 1); i += kThreads) owner[i] = 0u;
                __syncthreads();
                // outputs of this unit covered by the staged entries
                const uint32_t o_lo = max(q_lo, s_off[0]);
                const uint32_t o_hi = min(q_hi, s_off[n_e]);
                for (uint32_t i = tid; i < n_e; i += kThreads) {
                    const uint32_t s0 = s_off[i], s1 = s_off[i + 1];
                    if (s1 > s0 && s1 > o_lo && s0 < o_hi) {
                        const uint32_t j = max(s0, o_lo) - o_lo;
                        owner[j + j / kEmitPerThread] = i + 1;
                    }
                }
                __syncthreads();
                // inclusive prefix-max over owner: per-thread segment, then across threads
                uint32_t run = 0;
                uint32_t *seg = owner + tid * (kEmitPerThread + 1);
#pragma unroll
                for (uint32_t k = 0; k < kEmitPerThread; ++k) {
                    run = max(run, seg[k]);
                    seg[k] = run;
                }
                uint32_t inc = run;
#pragma unroll
                for (int off = 1; off < 32; off <<= 1) {
                    const uint32_t o = __shfl_up_sync(0xffffffffu, inc, off);
                    if (lane >= (uint32_t)off) inc = max(inc, o);
                }
                if (lane == 31) wmax[warp] = inc;
                __syncthreads();
                uint32_t prefix = __shfl_up_sync(0xffffffffu, inc, 1);
                if (lane == 0) prefix = 0;
                for (uint32_t w = 0; w < warp; ++w) prefix = max(prefix, wmax[w]);
#pragma unroll
                for (uint32_t k = 0; k < kEmitPerThread; ++k) seg[k] = max(seg[k], prefix);
                __syncthreads();
                // coalesced emission
                const uint32_t n_out = o_hi > o_lo ? o_hi - o_lo : 0u;
                for (uint32_t j = tid; j < n_out; j += kThreads) {
                    const uint32_t own = owner[j + j / kEmitPerThread];
                    if (own == 0) continue;   // cannot happen: every output has an owner
                    const uint32_t i = own - 1;
                    const int4 r = s_rect[i];
                    const uint32_t q = o_lo + j;
                    const uint32_t k = q - s_off[i];
                    const uint32_t w = (uint32_t)r.y;
                    const uint32_t dy = k / w;
                    const uint32_t dx = k - dy * w;
                    const int32_t ty = r.z + (int32_t)dy;
                    int32_t tx = r.x + (int32_t)dx;
                    uint32_t tile;
                    if (kLidar) {
                        const int32_t na = (int32_t)a.lidar.n_tiles_azim;
                        tx %= na;
                        if (tx < 0) tx += na;
                        tile = (uint32_t)ty * a.lidar.n_tiles_azim + (uint32_t)tx;
                    } else {
                        tile = (uint32_t)ty * a.cam.tile_width + (uint32_t)tx;
                    }
                    const uint32_t idx = s_idx[i];
                    if (kDirect64) {
                        ids64_out[q] = ((int64_t)(uint32_t)r.w << (32 + e.tile_n_bits)) |
                                       ((int64_t)tile << 32) | (int64_t)e.depth_bits[idx];
                        flat_out[q] = (int32_t)idx;
                    } else {
                        keys_out[q] = (uint32_t)r.w * e.n_tiles + tile;
                        vals_out[q] = idx;
                    }
                }
            }
        }
    }
    if (overflow && blockIdx.x == 0 && threadIdx.x == 0)
        atomicOr((unsigned long long *)&counters[CNT_STATUS], (unsigned long long)ST_OVERFLOW_CAPACITY);
}

// ---------------------------------------------------------------------------------------
// Block split (sorted output, any number of sensors): builds the per-tile lists of a sensor from its
// depth-ordered rectangles without ever writing the emission out, in two stable steps.
//
//   A. blocks: the tile grid is cut into blocks of 4 x 8 tiles. Every depth-ordered entry appends one
//              record - the 32-bit mask of the block's tiles it covers and its place in the depth order
//              - to the list of each block it touches (2.3 records per entry for the lidar benchmark,
//              3.1 for the camera's, against 5.9 and 5.2 for whole tile rows). A CTA takes
//              512 consecutive entries; its warps mark their lanes' blocks in one word per (warp,
//              block), so that an entry's rank in a block's list is a population count.
//   B. tiles:  a CTA takes a unit of a block's records, every warp 32 at a time, one record per lane. A
//              32 x 32 bit transpose of the masks gives every lane the records that cover ITS tile: that
//              is the count, and, a second time, the order in which the unit's entries are written.
//
// Walking the row runs of a rectangle output by output, which this replaces, took 6 warp instructions per
// 32 outputs' lane, and the radix passes over (tile, entry) pairs that grids of more than 128 tile rows took
// before move 44 B per intersection (14 of the 17 ms of six cameras' frame). What bounds it now is the 12 B
// of every list entry, written at 4.9 TB/s where the lists are long (a fill: 7.5).
// Positions are exclusive sums over (earlier tiles, earlier units, earlier CTAs, lower lanes), all of
// them plain scans: the result is the same for any scheduling, and no block waits for another.
// ---------------------------------------------------------------------------------------
constexpr uint32_t kBlkW = 4, kBlkH = 8;                   // tiles per block: one per lane
static_assert(kBlkW * kBlkH == 32, "one lane per tile of a block");
constexpr uint32_t kBlkThreads = 512, kBlkWarps = kBlkThreads / 32;   // step A: one entry per thread
// Step B: a CTA takes a unit of 512 consecutive records of a block, or of 1024 where the lists are so long that they leave the cache as they
// are written: figures at tile_scatter_kernel, whose CTAs go with it, six or two an SM.
constexpr uint32_t kBlkUnitMin = 512, kBlkUnitMax = 1024;
constexpr uint64_t kBlkLongLists = (480ull << 20) / 12, kBlkCachedLists = (126ull << 20) / 12;   // entries
constexpr uint32_t kBlkWords = 2;                          // writing: 32-record groups per warp
constexpr uint32_t kBlkCountThreads = 128;                 // counting
constexpr uint32_t kBlkMaxPerSensor = 1024;                // blocks per sensor (32768 tiles)
constexpr uint32_t kBlkMaxPerRow = 256;                    // block columns: shared-memory tables of step A
constexpr uint32_t kBlkRows = 2;                           // block rows per CTA of step A's scatter
constexpr uint32_t kBlkMaxBlocks = 16384;                  // blocks over all sensors
constexpr uint32_t kBlkMaxSensors = 4096;
constexpr uint32_t kBlkMaxExtent = 8192;                   // tiles per row / rows: the packed rectangle's 16-bit fields
constexpr uint32_t kBlkGridB = 16 * kNumSMs;               // persistent grid of step B: counting

struct BlkArgs {
    // entries in (sensor, depth bits, flatten index) order
    const uint2 *rect;            // {x0 | width << 16, y0 | height << 16}
    const uint2 *pair;            // {depth bits, flatten index}
    const uint32_t *sensor_start; // [C + 1] first entry of every sensor
    const uint32_t *sensor_cta;   // [C + 1] first step-A CTA of every sensor
    const int64_t *counters;      // CNT_NISECT
    int64_t capacity;
    uint32_t C, n_tiles;          // sensors, tiles per sensor
    uint32_t width, height;       // tile grid of a sensor
    uint32_t bx, by, blocks;      // blocks per row, per column, per sensor
    uint32_t tile_n_bits;
    uint32_t unit;                // records per step-B unit
    // workspace
    uint32_t total, ctas;         // elements (>= entries), step-A CTAs launched
    uint32_t *table;              // [blocks][ctas] records per (block, step-A CTA); scanned in place
    uint32_t *rec_start;          // [C * blocks + 1] first record of every block (totals before the scan)
    uint32_t *unit_start;         // [C * blocks + 1] first step-B unit of every block
    uint2 *rec;                   // [capacity] {tiles covered, entry}
    uint32_t *unit_cnt;           // [units][32] list entries per (unit, tile); scanned per block in place
    uint4 *unit_info;             // [units] {block, first record, end}
    uint32_t *tile_base;          // [C * n_tiles] totals, then first list position of every tile
    float *near;                  // [1] tiles that a near entry covers, where asked for
    volatile int64_t *near_host;  // who asks: sequence << 32 | the float's bits; may be null
    uint32_t near_sequence;
    float near_least;             // list entries squared per element listed from which on it is told
    uint32_t near_shift, near_step;   // 512s of each sensor that is looked at (log2), and every how manieth sensor is
};

// More intersections than output slots: the split is skipped altogether (the record arrays are sized
// by the capacity) and only the status bit is raised.
__device__ __forceinline__ bool blk_overflow(const BlkArgs &a) { return a.counters[CNT_NISECT] > a.capacity; }

// last i in [0, n) with start[i] <= v (start ascending, start[0] <= v), by one warp: 32 probes per round
__device__ __forceinline__ uint32_t warp_find(const uint32_t *__restrict__ start, uint32_t n, uint32_t v,
                                              uint32_t lane) {
    uint32_t lo = 0;
    while (n > 1) {
        const uint32_t step = (n + 31) / 32;
        const uint32_t at = lane * step;
        const uint32_t m = __ballot_sync(0xffffffffu, at < n && __ldg(start + lo + at) <= v);
        const uint32_t k = 31u - __clz(m | 1u);
        lo += k * step;
        n = min(step, n - k * step);
    }
    return lo;
}

struct BlkCta { uint32_t sensor, first, n; bool live; };

// Which entries a step-A CTA takes: every sensor's are cut into chunks of kBlkThreads.
__device__ __forceinline__ BlkCta blk_cta(const BlkArgs &a) {
    BlkCta c{};
    if (a.C == 1) {   // nothing to look up but the number of entries
        const uint32_t n = __ldg(a.sensor_start + 1);
        c.first = blockIdx.x * kBlkThreads;
        c.live = c.first < n;
        c.n = c.live ? min(kBlkThreads, n - c.first) : 0u;
        return c;
    }
    if (blockIdx.x >= a.sensor_cta[a.C]) return c;
    c.sensor = warp_find(a.sensor_cta, a.C, blockIdx.x, threadIdx.x & 31);
    c.first = a.sensor_start[c.sensor] + (blockIdx.x - a.sensor_cta[c.sensor]) * kBlkThreads;
    c.n = min(kBlkThreads, a.sensor_start[c.sensor + 1] - c.first);
    c.live = true;
    return c;
}

// rectangle of the thread's entry, loaded before anything says whether there is one
__device__ __forceinline__ uint2 blk_load_rect(const BlkArgs &a, uint32_t entry) {
    return __ldg(a.rect + min(entry, a.total - 1));
}

// A rectangle as the blocks it touches. Columns may run on past the last tile column to the first
// (lidar grids) and, for Gaussians next to the sensor, cover the turn more than once: `layers` runs
// of at most one turn each, every one inside the one before.
struct BlkRect {
    uint32_t x0, w, y0, h;   // w may exceed the grid's width
    uint32_t sx, nx, sy, ny; // first block column, columns touched (wrapping), first block row, rows
    uint32_t layers;
};

__device__ __forceinline__ BlkRect blk_rect(const BlkArgs &a, uint2 r, bool live) {
    BlkRect b;
    b.x0 = r.x & 0xffffu; b.w = live ? r.x >> 16 : 0u;
    b.y0 = r.y & 0xffffu; b.h = live ? r.y >> 16 : 0u;
    b.layers = 1; b.nx = 0; b.ny = 0; b.sx = b.x0 / kBlkW; b.sy = b.y0 / kBlkH;
    if (b.w == 0u || b.h == 0u) return b;
    b.ny = (b.y0 + b.h - 1) / kBlkH - b.sy + 1;
    const uint32_t end = b.x0 + b.w;
    if (end <= a.width) {
        b.nx = (end - 1) / kBlkW - b.sx + 1;
    } else {
        const uint32_t over = min(end - a.width, b.x0);   // columns [0, over) after the wrap
        const uint32_t tail = over ? (over - 1) / kBlkW + 1 : 0u;
        b.nx = min(a.bx, a.bx - b.sx + tail);
        b.layers = (b.w + a.width - 1) / a.width;
    }
    return b;
}

// columns [lo, hi) of the grid as bits of block column s (lo, hi may lie outside the block)
__device__ __forceinline__ uint32_t blk_span(uint32_t lo, uint32_t hi, uint32_t first, uint32_t n) {
    const int32_t l = max((int32_t)(lo - first), 0), h = min((int32_t)(hi - first), (int32_t)n);
    return h > l ? (1u << h) - (1u << l) : 0u;
}

// The mask over a block's 32 tiles (bit y * 4 + x) of one layer of a rectangle is the product of the
// two: its rows as bits four apart, its columns as a nibble.
__device__ __forceinline__ uint32_t blk_row_bits(const BlkRect &b, uint32_t r) {
    const uint32_t rows = blk_span(b.y0, b.y0 + b.h, r * kBlkH, kBlkH);
    uint32_t m = (rows | (rows << 12)) & 0x000f000fu;
    m = (m | (m << 6)) & 0x03030303u;
    return (m | (m << 3)) & 0x11111111u;
}

__device__ __forceinline__ uint32_t blk_col_bits(const BlkArgs &a, const BlkRect &b, uint32_t s, uint32_t layer) {
    const uint32_t end = b.x0 + min(b.w - layer * a.width, a.width);
    uint32_t cols = blk_span(b.x0, min(end, a.width), s * kBlkW, kBlkW);
    if (end > a.width) cols |= blk_span(0u, end - a.width, s * kBlkW, kBlkW);
    return cols;
}

// records a rectangle leaves in a touched block of block column s: one per layer that covers part of it
__device__ __forceinline__ uint32_t blk_records(const BlkArgs &a, const BlkRect &b, uint32_t s) {
    uint32_t n = 1;
    for (uint32_t j = 1; j < b.layers; ++j) n += blk_col_bits(a, b, s, j) ? 1u : 0u;
    return n;
}

// ---- step A -----------------------------------------------------------------------------
// block columns of a rectangle in block row r
__device__ __forceinline__ uint32_t blk_row_cols(const BlkRect &b, uint32_t r) {
    return (r - b.sy) < b.ny ? b.nx : 0u;
}

// The mean number of tiles that one of the nearest Gaussians covers: of the first 4096 entries of one sensor, or of as many of
// up to eight together, by 512 until they make 32 list entries per tile. Most of what compositing looks at is theirs. A block that starts
// with the kernel and has little to count does it first, with one wait for all its loads (in the last block of 500 k Gaussians, which starts when the others
// end: 2 to 3 us of the frame); the kernel behind it tells the host, whose link a longer kernel covers (2 us here, 4 with a fence).
constexpr uint32_t kNearGroups = 8, kNearPerTile = 32, kNearCta = 300;
__device__ __forceinline__ void find_near(const BlkArgs &a) {
    __shared__ uint32_t s_near[kNearGroups], s_of[kNearGroups];   // tiles, entries
    const uint32_t tid = threadIdx.x, sensors = min(a.C, kNearGroups);
    if (tid < kNearGroups) s_near[tid] = 0u;
    uint2 r[kNearGroups];
#pragma unroll
    for (uint32_t g = 0; g < kNearGroups; ++g) {
        const uint32_t i = g >> a.near_shift, sensor = i < sensors ? i * a.near_step : 0u, k = g - (i << a.near_shift);
        const uint32_t lo = __ldg(a.sensor_start + sensor) + k * kBlkThreads, end = __ldg(a.sensor_start + sensor + 1);
        const uint32_t n = i < sensors && lo < end ? min(kBlkThreads, end - lo) : 0u;
        r[g] = tid < n ? __ldg(a.rect + lo + tid) : make_uint2(0u, 0u);
        if (tid == 0) s_of[g] = n;
    }
    __syncthreads();
#pragma unroll
    for (uint32_t g = 0; g < kNearGroups; ++g) {
        const uint32_t sum = __reduce_add_sync(0xffffffffu, (r[g].x >> 16) * (r[g].y >> 16));
        if ((tid & 31u) == 0u && sum) atomicAdd(&s_near[g], sum);
    }
    __syncthreads();
    if (tid != 0) return;
    float tiles = 0.f, of = 0.f;
    for (uint32_t i = 0; i < sensors; ++i) {
        uint32_t sum = 0;
        for (uint32_t g = i << a.near_shift; g < (i + 1) << a.near_shift && sum < kNearPerTile * a.n_tiles; ++g) {
            sum += s_near[g];
            of += (float)s_of[g];
        }
        tiles += (float)sum;
    }
    *a.near = of > 0.f && !blk_overflow(a) ? tiles / of : 0.f;
}

template <bool kWrap>
__global__ void __launch_bounds__(kBlkThreads, 4)
blk_count_kernel(BlkArgs a) {
    chain_enter();
    extern __shared__ uint32_t s_cnt[];   // [blocks]
    const bool overflow = blk_overflow(a);
    if (!kWrap && a.near_host != nullptr && blockIdx.x == min(gridDim.x - 1, kNearCta)) find_near(a);
    const BlkCta c = blk_cta(a);
    const uint2 rect = blk_load_rect(a, c.first + threadIdx.x);
    for (uint32_t k = threadIdx.x; k < a.blocks; k += kBlkThreads) s_cnt[k] = 0u;
    if (overflow || !c.live) return;
    __syncthreads();
    const BlkRect b = blk_rect(a, rect, threadIdx.x < c.n);
    for (uint32_t j = 0; j < b.ny; ++j) {
        uint32_t *row = s_cnt + (b.sy + j) * a.bx;
        for (uint32_t i = 0, s = b.sx; i < b.nx; ++i) {
            atomicAdd(&row[s], kWrap && b.layers > 1 ? blk_records(a, b, s) : 1u);
            if (++s == a.bx) s = 0;
        }
    }
    __syncthreads();
    for (uint32_t k = threadIdx.x; k < a.blocks; k += kBlkThreads) a.table[(size_t)k * a.ctas + blockIdx.x] = s_cnt[k];
}

// One CTA per (sensor, block): exclusive scan over the sensor's step-A CTAs, in place. The CTA that
// finishes last (a ticket, nobody waits) turns the totals into record and unit starts.
__global__ void __launch_bounds__(1024)
blk_scan_kernel(BlkArgs a, unsigned long long *__restrict__ ticket) {
    chain_enter();
    __shared__ uint32_t wt[33];
    __shared__ bool s_last;
    if (blk_overflow(a)) return;
    const uint32_t tid = threadIdx.x, sensor = blockIdx.x / a.blocks, k = blockIdx.x - sensor * a.blocks;
    const uint32_t cta0 = a.sensor_cta[sensor], n = a.sensor_cta[sensor + 1] - cta0;
    uint32_t *row = a.table + (size_t)k * a.ctas + cta0;
    uint32_t carry = 0;
    for (uint32_t i0 = 0; i0 < n; i0 += blockDim.x) {
        const uint32_t i = i0 + tid;
        const uint32_t v = i < n ? row[i] : 0u;
        uint32_t tot;
        const uint32_t ex = block_excl_scan(v, wt, tot);
        if (i < n) row[i] = carry + ex;
        carry += tot;
    }
    if (tid == 0) {
        a.rec_start[blockIdx.x] = carry;
        __threadfence();
        s_last = atomicAdd(ticket, 1ull) + 1ull == (unsigned long long)gridDim.x;
    }
    __syncthreads();
    if (!s_last) return;
    __threadfence();
    const uint32_t n_blocks = a.C * a.blocks;
    uint32_t recs = 0, units = 0;
    for (uint32_t i0 = 0; i0 < n_blocks; i0 += blockDim.x) {
        const uint32_t i = i0 + tid;
        const uint32_t v = i < n_blocks ? __ldcg(a.rec_start + i) : 0u;
        uint32_t tr, tu;
        const uint32_t er = block_excl_scan(v, wt, tr);
        const uint32_t eu = block_excl_scan((v + a.unit - 1) / a.unit, wt, tu);
        if (i < n_blocks) {
            a.rec_start[i] = recs + er;
            a.unit_start[i] = units + eu;
        }
        recs += tr;
        units += tu;
    }
    if (tid == 0) {
        a.rec_start[n_blocks] = recs;
        a.unit_start[n_blocks] = units;
        *ticket = 0ull;
    }
}

// blockIdx.x: 512 entries of a sensor, blockIdx.y: two block rows. Few rows per CTA, because the entries
// come in depth order and the nearest ones cover the whole image: the CTA that holds them walks 60 blocks
// per lane of a 1920 x 1080 grid instead of 270 (70 -> 39 us for the camera benchmark's frame).
// Bound by instruction issue and by the waits between its phases. A warp clears its own words, a column's sixteen counts are
// read before the first sum is written, and the columns of a rectangle that does not wrap are whole nibbles but for
// its two ends: camera benchmark 36 -> 27 us, six cameras 340 -> 233; lidar benchmark 41.
// kWrap: rectangles may cover the turn more than once and then leave several records in a block (a
// rectangle spans less than five turns): three more mask words per (warp, block) hold the bits of their
// lanes' surplus.
// kCtas an SM, by what the registers leave: the sixteen counts of a column take 64 with wraps, which pays where a CTA has many columns (30
// of them, 128 x 1800: 37.4 with three CTAs, 35.7 with two; 20, 96 x 1200: 29.2 and 27.1) and not where it has few (10, two sensors of
// 70 x 556: 35.3 and 41.4; 9, 64 x 1083 and 800,000 Gaussians: 18.9 and 21.0).
constexpr uint32_t kBlkManyCols = 16;

template <bool kWrap, int kCtas>
__global__ void __launch_bounds__(kBlkThreads, kCtas)
blk_scatter_kernel(BlkArgs a) {
    chain_enter();
    extern __shared__ uint32_t s_dyn[];
    const uint32_t r0 = blockIdx.y * kBlkRows, n_cols = min(kBlkRows, a.by - r0) * a.bx, plane = kBlkWarps * n_cols;
    uint32_t *s_base = s_dyn;              // [warps][rows][bx] position of the warp's first record
    uint32_t *s_mask = s_base + plane;     // (kWrap: 4 planes of) [warps][rows][bx] lanes with a record
    const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, lt = (1u << lane) - 1u;
    if (!kWrap && a.near_host != nullptr && tid == 0 && blockIdx.x == min(gridDim.x - 1, kNearCta) && blockIdx.y == 0) {
        const float n = (float)a.counters[CNT_NISECT];   // short lists: nobody waits, and the store would outlast a short kernel (1 us)
        if (n * n >= a.near_least * (float)a.counters[CNT_NVIS])
            *a.near_host = (int64_t)((uint64_t)a.near_sequence << 32 | __float_as_uint(*a.near));
    }
    const bool overflow = blk_overflow(a);
    const BlkCta c = blk_cta(a);
    const uint32_t entry = c.first + tid;
    const uint2 rect = blk_load_rect(a, entry);
    // the CTA's first record of the block of this thread: block start, earlier CTAs of the sensor
    uint32_t first = 0;
    if (tid < n_cols)
        first = __ldg(a.rec_start + c.sensor * a.blocks + r0 * a.bx + tid) +
                __ldg(a.table + (size_t)(r0 * a.bx + tid) * a.ctas + blockIdx.x);
    uint32_t *mask = s_mask + warp * n_cols;   // only this warp writes there
    for (uint32_t k = lane; k < n_cols; k += 32) mask[k] = 0u;
    if (overflow || !c.live) return;
    const BlkRect b = blk_rect(a, rect, tid < c.n);
    const bool layered = kWrap && __syncthreads_or(b.layers > 1);
    if (kWrap && layered)
        for (uint32_t q = 1; q < 4; ++q)
            for (uint32_t k = lane; k < n_cols; k += 32) mask[q * plane + k] = 0u;
    __syncwarp();
    for (uint32_t j = 0; j < kBlkRows; ++j) {
        const uint32_t n = blk_row_cols(b, r0 + j);
        uint32_t *row = mask + j * a.bx;
        for (uint32_t i = 0, s = b.sx; i < n; ++i) {
            atomicOr(&row[s], 1u << lane);
            if (kWrap && b.layers > 1) {
                const uint32_t more = blk_records(a, b, s) - 1u;
                for (uint32_t q = 0; q < 3; ++q)
                    if ((more >> q) & 1u) atomicOr(&row[(q + 1) * plane + s], 1u << lane);
            }
            if (++s == a.bx && kWrap) s = 0;
        }
    }
    __syncthreads();
    if (tid < n_cols) {
        uint32_t count[kBlkWarps];   // all of them read before the first base is written: one wait instead of sixteen
#pragma unroll
        for (uint32_t w = 0; w < kBlkWarps; ++w) count[w] = __popc(s_mask[w * n_cols + tid]);
        if (kWrap && layered) {
#pragma unroll
            for (uint32_t w = 0; w < kBlkWarps; ++w)
                for (uint32_t q = 0; q < 3; ++q) count[w] += __popc(s_mask[(q + 1) * plane + w * n_cols + tid]) << q;
        }
        uint32_t run = first;
#pragma unroll
        for (uint32_t w = 0; w < kBlkWarps; ++w) {
            s_base[w * n_cols + tid] = run;
            run += count[w];
        }
    }
    __syncthreads();
    const uint32_t cap = (uint32_t)min(a.capacity, (int64_t)0x7fffffff);
    // columns of a rectangle that does not wrap: whole nibbles but for its two ends
    const uint32_t end = b.x0 + b.w, left = (0xfu << (b.x0 & 3u)) & 0xfu, right = 0xfu >> (3u - ((end - 1u) & 3u));
    const bool straight = !kWrap || end <= a.width;
    static_assert(kBlkW == 4, "a nibble per row of a block");
    for (uint32_t j = 0; j < kBlkRows; ++j) {
        const uint32_t n = blk_row_cols(b, r0 + j);
        if (n == 0u) continue;
        const uint32_t *row = mask + j * a.bx, *base = s_base + warp * n_cols + j * a.bx;
        const uint32_t rows = blk_row_bits(b, r0 + j);
        for (uint32_t i = 0, s = b.sx; i < n; ++i) {
            uint32_t pos = base[s] + __popc(row[s] & lt);
            if (kWrap && layered)
                for (uint32_t q = 0; q < 3; ++q) pos += __popc(row[(q + 1) * plane + s] & lt) << q;
            const uint32_t cols = straight ? (i == 0u ? left : 0xfu) & (i + 1u == n ? right : 0xfu) : blk_col_bits(a, b, s, 0u);
            if (pos < cap) a.rec[pos] = make_uint2(rows * cols, entry);
            if (kWrap)
                for (uint32_t l = 1; l < b.layers; ++l) {
                    const uint32_t m = blk_col_bits(a, b, s, l);
                    if (m != 0u && ++pos < cap) a.rec[pos] = make_uint2(rows * m, entry);
                }
            if (++s == a.bx && kWrap) s = 0;
        }
    }
}

// ---- step B -----------------------------------------------------------------------------
struct BlkUnit { uint32_t block, lo, hi; };

__device__ __forceinline__ BlkUnit blk_unit(const BlkArgs &a, uint32_t u, uint32_t lane) {
    BlkUnit v;
    // blocks without records own no unit: the search ends at the last of equal starts, which has one
    v.block = warp_find(a.unit_start, a.C * a.blocks, u, lane);
    const uint32_t cap = (uint32_t)min(a.capacity, (int64_t)0x7fffffff);
    v.lo = min(cap, __ldg(a.rec_start + v.block) + (u - __ldg(a.unit_start + v.block)) * a.unit);
    v.hi = min(min(cap, __ldg(a.rec_start + v.block + 1)), v.lo + a.unit);
    return v;
}

// Tile of lane l of a block, as (sensor, x, y); tiles beyond the grid's edges are in no record.
struct BlkTile { uint32_t sensor, x, y; };

__device__ __forceinline__ BlkTile blk_tile(const BlkArgs &a, uint32_t block, uint32_t l) {
    BlkTile t;
    t.sensor = block / a.blocks;
    const uint32_t k = block - t.sensor * a.blocks, r = k / a.bx;
    t.x = (k - r * a.bx) * kBlkW + (l & (kBlkW - 1));
    t.y = r * kBlkH + l / kBlkW;
    return t;
}

// 32 x 32 bit transpose across a warp: lane l comes with row l and leaves with column l.
__device__ __forceinline__ uint32_t warp_transpose_bits(uint32_t x, uint32_t lane) {
#pragma unroll
    for (int j = 16; j >= 1; j >>= 1) {
        const uint32_t m = j == 16 ? 0x0000ffffu : j == 8 ? 0x00ff00ffu : j == 4 ? 0x0f0f0f0fu
                         : j == 2 ? 0x33333333u : 0x55555555u;
        const uint32_t y = __shfl_xor_sync(0xffffffffu, x, j);
        x = (lane & (uint32_t)j) ? ((x & ~m) | ((y & ~m) >> j)) : ((x & m) | ((y & m) << j));
    }
    return x;
}

template <uint32_t kWords>   // 32-record groups per warp
__global__ void __launch_bounds__(kBlkCountThreads)
tile_count_kernel(BlkArgs a) {
    chain_enter();
    constexpr uint32_t kWarps = kBlkCountThreads / 32;
    __shared__ uint32_t s_cnt[kWarps][32];
    if (blk_overflow(a)) return;
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint32_t n_units = a.unit_start[a.C * a.blocks];
    for (uint32_t u = blockIdx.x; u < n_units; u += gridDim.x) {
        const BlkUnit v = blk_unit(a, u, lane);
        uint32_t m[kWords], cnt = 0;
#pragma unroll
        for (uint32_t j = 0; j < kWords; ++j) {
            const uint32_t p = v.lo + 32 * (warp * kWords + j) + lane;
            m[j] = p < v.hi ? __ldg(&a.rec[p].x) : 0u;
        }
#pragma unroll
        for (uint32_t j = 0; j < kWords; ++j) cnt += __popc(warp_transpose_bits(m[j], lane));
        s_cnt[warp][lane] = cnt;
        __syncthreads();
        if (warp == 0) {
#pragma unroll
            for (uint32_t w = 1; w < kWarps; ++w) cnt += s_cnt[w][lane];
            a.unit_cnt[(size_t)u * 32 + lane] = cnt;
            if (lane == 0) a.unit_info[u] = make_uint4(v.block, v.lo, v.hi, 0u);
        }
        __syncthreads();
    }
}

// One CTA per block: exclusive scan over its units for each of the 32 tiles (one lane each), the units
// cut into one segment per warp. The CTA that finishes last scans the totals over all tiles: list starts.
template <uint32_t kFours>
__global__ void __launch_bounds__(1024)
tile_scan_kernel(BlkArgs a, unsigned long long *__restrict__ ticket, int32_t *__restrict__ offsets) {
    chain_enter();
    __shared__ uint32_t seg_sum[32][33];
    __shared__ bool s_last;
    const uint32_t tid = threadIdx.x, lane = tid & 31, seg = tid >> 5, n_seg = blockDim.x >> 5;
    const uint32_t n_tiles = a.C * a.n_tiles;
    if (blk_overflow(a)) {
        // the split is skipped for lack of room: every offset 0, so that compositing enqueued behind it
        // finds empty tiles instead of stale numbers
        if (offsets != nullptr)
            for (uint32_t t = blockIdx.x * blockDim.x + tid; t <= n_tiles; t += gridDim.x * blockDim.x) offsets[t] = 0;
        return;
    }
    const uint32_t u0 = a.unit_start[blockIdx.x], n_units = a.unit_start[blockIdx.x + 1] - u0;
    const uint32_t per = (n_units + n_seg - 1) / n_seg;
    const uint32_t lo = min(n_units, seg * per), hi = min(n_units, lo + per);
    uint32_t *col = a.unit_cnt + (size_t)u0 * 32 + lane;
    uint32_t sum = 0;
#pragma unroll 8
    for (uint32_t u = lo; u < hi; ++u) sum += col[(size_t)u * 32];
    seg_sum[seg][lane] = sum;
    __syncthreads();
    uint32_t run = 0, total = 0;
    for (uint32_t s = 0; s < n_seg; ++s) {
        const uint32_t v = seg_sum[s][lane];
        if (s < seg) run += v;
        total += v;
    }
#pragma unroll 8
    for (uint32_t u = lo; u < hi; ++u) {
        const uint32_t v = col[(size_t)u * 32];
        col[(size_t)u * 32] = run;
        run += v;
    }
    if (seg == 0) {
        const BlkTile t = blk_tile(a, blockIdx.x, lane);
        if (t.x < a.width && t.y < a.height) a.tile_base[t.sensor * a.n_tiles + t.y * a.width + t.x] = total;
        __threadfence();
        __syncwarp();
        if (lane == 0) s_last = atomicAdd(ticket, 1ull) + 1ull == (unsigned long long)gridDim.x;
    }
    __syncthreads();
    if (!s_last) return;
    __threadfence();
    // Where there are many, four times four totals per thread and round: one four behind the other, so that every access is whole lines, and the four scans
    // share their shuffles' and barriers' time - a round is a chain of some 2000 cycles (48960 tiles of six cameras: 48 rounds with one
    // four, 58 us; 12 rounds, 37; 8160 tiles 16.7 and 12.6).
    __shared__ uint32_t s_tot[kFours][33];
    const bool wide = offsets != nullptr && (reinterpret_cast<uintptr_t>(offsets) & 15u) == 0u;
    uint32_t carry = 0;
    for (uint32_t t0 = 0; t0 < n_tiles; t0 += 4 * kFours * blockDim.x) {
        uint4 v[kFours];
        uint32_t sum[kFours], at[kFours];
#pragma unroll
        for (uint32_t k = 0; k < kFours; ++k) {
            const uint32_t t = t0 + 4 * (k * blockDim.x + tid);
            v[k] = make_uint4(0u, 0u, 0u, 0u);
            if (t < n_tiles) v[k] = __ldcg(reinterpret_cast<const uint4 *>(a.tile_base + t));   // room for whole fours
            if (t + 1 >= n_tiles) v[k].y = 0u;
            if (t + 2 >= n_tiles) v[k].z = 0u;
            if (t + 3 >= n_tiles) v[k].w = 0u;
        }
#pragma unroll
        for (uint32_t k = 0; k < kFours; ++k) at[k] = sum[k] = v[k].x + v[k].y + v[k].z + v[k].w;
#pragma unroll
        for (int off = 1; off < 32; off <<= 1)
#pragma unroll
            for (uint32_t k = 0; k < kFours; ++k) {
                const uint32_t o = __shfl_up_sync(0xffffffffu, at[k], off);
                if (lane >= (uint32_t)off) at[k] += o;
            }
#pragma unroll
        for (uint32_t k = 0; k < kFours; ++k)
            if (lane == 31) s_tot[k][seg] = at[k];
        __syncthreads();
        if (seg < kFours) {   // a warp for each four: what the warps before have
            const uint32_t w = lane < n_seg ? s_tot[seg][lane] : 0u;
            uint32_t inc = w;
#pragma unroll
            for (int off = 1; off < 32; off <<= 1) {
                const uint32_t o = __shfl_up_sync(0xffffffffu, inc, off);
                if (lane >= (uint32_t)off) inc += o;
            }
            s_tot[seg][lane] = inc - w;
            if (lane == 31) s_tot[seg][32] = inc;
        }
        __syncthreads();
#pragma unroll
        for (uint32_t k = 0; k < kFours; ++k) {
            const uint32_t t = t0 + 4 * (k * blockDim.x + tid), first = carry + s_tot[k][seg] + at[k] - sum[k];
            const uint4 s = make_uint4(first, first + v[k].x, first + v[k].x + v[k].y, first + v[k].x + v[k].y + v[k].z);
            carry += s_tot[k][32];
            if (t < n_tiles) *reinterpret_cast<uint4 *>(a.tile_base + t) = s;
            if (wide && t + 3 < n_tiles) *reinterpret_cast<uint4 *>(offsets + t) = s;
            else if (offsets != nullptr) {
                if (t < n_tiles) offsets[t] = (int32_t)s.x;
                if (t + 1 < n_tiles) offsets[t + 1] = (int32_t)s.y;
                if (t + 2 < n_tiles) offsets[t + 2] = (int32_t)s.z;
                if (t + 3 < n_tiles) offsets[t + 3] = (int32_t)s.w;
            }
        }
        __syncthreads();   // the sums have been read
    }
    if (tid == 0) {
        *ticket = 0ull;
        if (offsets != nullptr) offsets[n_tiles] = (int32_t)carry;
    }
}

// A CTA leaves its unit's pairs and, by tile, the bits of its records in shared memory; behind that barrier a warp puts a tile's
// entries in order by itself - a lane takes the bits of 32 records, one scan says where its record numbers go, two bytes
// each - and writes the run: whole sectors two entries per lane, then what is left at the ends; with units of 512 half a
// warp each for two tiles at a time (one after the other: 56 us instead of 52 for the lidar benchmark, 18.8 instead of 16.8 where lists are short). (Before, each lane had a
// tile, the places were summed over the warps and the runs written after another barrier: 64 KB of places for three CTAs an
// SM. Storing straight from the lanes whose record covers a tile: 180 us for the lidar benchmark's 15.3 M entries.)
//
// What bounds it where the lists are long is how they reach the HBM, not the writing itself: with 592 CTAs of 1024 records 100 MB are
// under way, and the sectors that two units write in parts are evicted between the two, and every such half costs a read
// and about five whole sectors' time. So whole sectors leave the cache first, halves last (kStream: where the lists
// do not stay in the cache anyway), and two CTAs an SM are enough.
// Six cameras, 5.8 GB of lists: 1315 us before, 1390 with four CTAs an SM, 1250 with two, 1215 with two and that order of leaving (dram
// reads 401 -> 265 MB). Shorter lists want smaller units and more CTAs, us before, with six of 512 records and with two of 1024, by MB of lists: 109 (camera
// benchmark) 43, 37 and 49, 175 (lidar benchmark) 65, 50 and 60, 258 (three cameras) 75, 61 and 74, 350 (two lidars) 124, 92 and 107, 412 (150 k
// Gaussians, six cameras) 104, 102 and 106, 555: 140, 144 and 140, 687: 167, 180 and 158, 774: 199, 204 and 182, 1102: 271, 290 and 248, 1378: 329, 348 and 304; whole frames are
// 1 % faster with the smaller ones at 278 MB, the same at 412, 1 % slower at 555 and 5 % at 774. Four entries per lane (32-byte stores): 68 instead of 58 and
// 1430 instead of 1360, their record numbers lie in the same banks. (Whole sectors where the arrays begin on 32 bytes, as torch's do; others of
// 16 and 8 bytes' alignment are written two entries at a time all the same, anything else one by one.)
__device__ __forceinline__ uint64_t keep_in_cache() {
    uint64_t policy;
    asm volatile("createpolicy.fractional.L2::evict_last.b64 %0, 1.0;" : "=l"(policy));
    return policy;
}
__device__ __forceinline__ void store_kept(int64_t *to, uint64_t v, uint64_t policy) {
    asm volatile("st.global.L2::cache_hint.b64 [%0], %1, %2;" ::"l"(__cvta_generic_to_global(to)), "l"(v), "l"(policy) : "memory");
}
__device__ __forceinline__ void store_kept(int32_t *to, uint32_t v, uint64_t policy) {
    asm volatile("st.global.L2::cache_hint.b32 [%0], %1, %2;" ::"l"(__cvta_generic_to_global(to)), "r"(v), "l"(policy) : "memory");
}

template <uint32_t kWarps, bool kStream>
__global__ void __launch_bounds__(kWarps * 32, kWarps > 8 ? 2 : 6)
tile_scatter_kernel(BlkArgs a, int64_t *__restrict__ isect_ids, int32_t *__restrict__ flatten_ids,
                    int64_t *__restrict__ counters) {
    chain_enter();
    constexpr uint32_t kUnit = kWarps * kBlkWords * 32, kWords = kUnit / 32;   // words of a tile: its bits over the unit's records
    constexpr uint32_t kTiles = 32 / kWords, kRoom = kUnit + 8;   // tiles a warp puts in order at a time; places of one, from a multiple of eight on
    static_assert(kWords == 16 || kWords == 32, "a tile's words lie in a warp or in half of one");
    __shared__ uint2 s_pair[kUnit];
    __shared__ uint32_t s_word[32][kWords + 1];
    __shared__ __align__(16) uint16_t s_out[kWarps][kTiles * kRoom];   // record numbers in list order
    if (blk_overflow(a)) {
        if (blockIdx.x == 0 && threadIdx.x == 0)
            atomicOr((unsigned long long *)&counters[CNT_STATUS], (unsigned long long)ST_OVERFLOW_CAPACITY);
        return;
    }
    const uint64_t kept = keep_in_cache();
    const bool wide = ((reinterpret_cast<uintptr_t>(isect_ids) & 15u) | (reinterpret_cast<uintptr_t>(flatten_ids) & 7u)) == 0u;
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5, col = lane % kWords, half = lane / kWords;
    const uint32_t n_units = a.unit_start[a.C * a.blocks];
    const uint32_t cap = (uint32_t)min(a.capacity, (int64_t)0x7fffffff);
    uint4 info = make_uint4(0u, 0u, 0u, 0u);
    if (blockIdx.x < n_units) info = __ldg(a.unit_info + blockIdx.x);
    for (uint32_t u = blockIdx.x; u < n_units; u += gridDim.x) {
        const uint4 v = info;   // {block, first record, end}
        uint2 rec[kBlkWords];
#pragma unroll
        for (uint32_t j = 0; j < kBlkWords; ++j) {
            const uint32_t p = v.y + 32 * (warp * kBlkWords + j) + lane;
            rec[j] = p < v.z ? __ldg(a.rec + p) : make_uint2(0u, 0u);
        }
        if (u + gridDim.x < n_units) info = __ldg(a.unit_info + u + gridDim.x);
        const BlkTile t = blk_tile(a, v.x, lane);
        const uint32_t tile = t.y * a.width + t.x;
        uint32_t at = 0;   // lane l: list position of the unit's first entry of tile l
        if (t.x < a.width && t.y < a.height)
            at = __ldg(a.tile_base + t.sensor * a.n_tiles + tile) + __ldg(a.unit_cnt + (size_t)u * 32 + lane);
        const uint32_t high = (t.sensor << a.tile_n_bits) | tile;
        __syncthreads();   // the unit before has been written
#pragma unroll
        for (uint32_t j = 0; j < kBlkWords; ++j) {
            const uint32_t w = warp * kBlkWords + j;
            if (rec[j].x) s_pair[32 * w + lane] = __ldg(a.pair + rec[j].y);
            s_word[lane][w] = warp_transpose_bits(rec[j].x, lane);
        }
        __syncthreads();
        for (uint32_t l0 = warp * kTiles; l0 < 32; l0 += kWarps * kTiles) {
            // the lanes write down the record numbers of their words of a tile, behind those of the words before
            uint32_t m = s_word[l0 + half][col], place = __popc(m);
            const uint32_t mine = place;
#pragma unroll
            for (uint32_t off = 1; off < kWords; off <<= 1) {
                const uint32_t o = __shfl_up_sync(0xffffffffu, place, off, kWords);
                if (col >= off) place += o;
            }
            const uint32_t begin = __shfl_sync(0xffffffffu, at, l0 + half), id = __shfl_sync(0xffffffffu, high, l0 + half);
            const uint32_t end = min(begin + __shfl_sync(0xffffffffu, place, kWords - 1, kWords), cap);   // the last word's lane has the sum
            place += half * kRoom - mine + (begin & 7u);
            uint16_t *out = s_out[warp];
            const auto next = [&] {
                const uint32_t r = 32 * col + __ffs(m) - 1;
                m &= m - 1;
                return r;
            };
            if (m != 0u && (place & 1u)) out[place++] = (uint16_t)next();
            while (m & (m - 1)) {   // two at a time
                const uint32_t r = next();
                *reinterpret_cast<uint32_t *>(out + place) = r | next() << 16;
                place += 2;
            }
            if (m) out[place] = (uint16_t)next();
            __syncwarp();
            const uint16_t *src = out + half * kRoom - (begin & ~7u);   // indexed by list position
            const auto store_one = [&](uint32_t p, bool keep) {
                const uint2 e = s_pair[src[(int32_t)p]];
                if (keep) {
                    store_kept(isect_ids + p, ((uint64_t)id << 32) | e.x, kept);
                    store_kept(flatten_ids + p, e.y, kept);
                } else {
                    isect_ids[p] = (int64_t)(((uint64_t)id << 32) | e.x);
                    flatten_ids[p] = (int32_t)e.y;
                }
            };
            if (wide) {   // whole sectors first, then what is left at both ends
                const uint32_t inner = (begin + 7u) & ~7u, outer = end & ~7u;
#pragma unroll 2
                for (uint32_t p = inner + 2u * col; p < outer; p += 2u * kWords) {
                    const uint32_t r = *reinterpret_cast<const uint32_t *>(src + (int32_t)p);
                    const uint2 e = s_pair[r & 0xffffu], f = s_pair[r >> 16];
                    const uint4 ids = make_uint4(e.x, id, f.x, id);
                    const uint2 flat = make_uint2(e.y, f.y);
                    if (kStream) {
                        __stcs(reinterpret_cast<uint4 *>(isect_ids + p), ids);
                        __stcs(reinterpret_cast<uint2 *>(flatten_ids + p), flat);
                    } else {
                        *reinterpret_cast<uint4 *>(isect_ids + p) = ids;
                        *reinterpret_cast<uint2 *>(flatten_ids + p) = flat;
                    }
                }
                const uint32_t p = col < 8u ? begin + col : max(inner, outer) + col - 8u;
                if (col < 16u && p < (col < 8u ? min(inner, end) : end)) store_one(p, kStream);
            } else {
                for (uint32_t p = begin + col; p < end; p += kWords) store_one(p, false);
            }
            __syncwarp();
        }
    }
}

// ---------------------------------------------------------------------------------------
// Offsets: offsets[c, tile] = first position whose (sensor, tile) >= (c, tile).
// ---------------------------------------------------------------------------------------
__global__ void __launch_bounds__(kThreads)
offset_encode_kernel(const int64_t *__restrict__ isect_ids, const int64_t *n_ptr, int64_t n_imm,
                     uint32_t C, uint32_t n_tiles, uint32_t tile_n_bits,
                     int32_t *__restrict__ offsets) {
    const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
    const int64_t n = n_ptr ? (*n_ptr < n_imm ? *n_ptr : n_imm) : n_imm;
    if (t == C * n_tiles && n_ptr != nullptr) offsets[t] = (int32_t)n;   // fill only: the total
    if (t >= C * n_tiles) return;
    const int64_t cid = t / n_tiles, tile = t - (uint32_t)cid * n_tiles;
    const int64_t target = (cid << tile_n_bits) | tile;
    int64_t l = 0, h = n;   // first position with (id >> 32) >= target
    while (l < h) {
        const int64_t m = (l + h) >> 1;
        if ((isect_ids[m] >> 32) < target) l = m + 1; else h = m;
    }
    offsets[t] = (int32_t)l;
}

// counters back to zero (depth range: empty) and, for the bucket depth sort, its cursors
__global__ void init_counters_kernel(int64_t *counters, uint32_t *bcount, uint32_t n_buckets, uint32_t bucket_lo,
                                     uint32_t bucket_hi) {
    chain_enter();
    const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t < CNT_DEV_SLOTS)
        counters[t] = (t == CNT_DMIN) ? 0xffffffffll : (t == CNT_BLO) ? (int64_t)bucket_lo
                                                     : (t == CNT_BHI) ? (int64_t)bucket_hi : 0;
    if (bcount != nullptr)
        for (uint32_t i = t; i < n_buckets; i += gridDim.x * blockDim.x) bcount[i] = 0u;
}

// ---------------------------------------------------------------------------------------
// Host orchestration
// ---------------------------------------------------------------------------------------
static inline size_t align256(size_t x) { return (x + 255) & ~(size_t)255; }

struct PlanWs {
    int64_t *counters;
    uint32_t *hist;
    uint32_t *digit_totals;
    unsigned long long *block_sums;
    unsigned long long *block_offs;
    uint32_t *keyA, *valA, *keyB, *valB;
    uint32_t *eoff;
    uint2 *rect, *sorted_rect;   // block split: packed rectangles by flatten index, and in depth order
    uint32_t *blk_table;         // block split: records per (block, step-A CTA)
    uint32_t *group_start, *group_chunk;   // block split: first entry / first step-A CTA of every sensor
    uint32_t n_buckets;
    uint32_t *bcount, *bstart;   // bucket depth sort: counts / cursors, starts in their scan block
    uint32_t *boff;              // offsets of the scan blocks, total, block totals
    size_t bytes;
};

static PlanWs carve_plan(void *ws, uint64_t total) {
    PlanWs p;
    char *c = (char *)ws;
    size_t off = 0;
    auto take = [&](size_t b) { char *r = c ? c + off : nullptr; off += align256(b); return r; };
    p.counters = (int64_t *)take(sizeof(int64_t) * CNT_DEV_SLOTS);
    p.hist = (uint32_t *)take(sizeof(uint32_t) * kRadixBins * kSortGrid);
    p.digit_totals = (uint32_t *)take(sizeof(uint32_t) * kRadixBins);
    p.block_sums = (unsigned long long *)take(sizeof(unsigned long long) * kSortGrid);
    p.block_offs = (unsigned long long *)take(sizeof(unsigned long long) * kSortGrid);
    p.keyA = (uint32_t *)take(sizeof(uint32_t) * total);
    p.valA = (uint32_t *)take(sizeof(uint32_t) * total);
    p.keyB = (uint32_t *)take(sizeof(uint32_t) * total);
    p.valB = (uint32_t *)take(sizeof(uint32_t) * total);
    p.eoff = (uint32_t *)take(sizeof(uint32_t) * total);
    p.rect = (uint2 *)take(sizeof(uint2) * total);
    p.sorted_rect = (uint2 *)take(sizeof(uint2) * total);
    // blocks * (ceil(total / kBlkThreads) + sensors)
    p.blk_table = (uint32_t *)take(sizeof(uint32_t) * (kBlkMaxPerSensor * (total / kBlkThreads + 1) + kBlkMaxBlocks));
    p.group_start = (uint32_t *)take(sizeof(uint32_t) * (kBlkMaxSensors + 1));
    p.group_chunk = (uint32_t *)take(sizeof(uint32_t) * (kBlkMaxSensors + 1));
    p.n_buckets = depth_bucket_count(total);
    p.bcount = (uint32_t *)take(sizeof(uint32_t) * p.n_buckets);
    p.bstart = (uint32_t *)take(sizeof(uint32_t) * p.n_buckets);
    p.boff = (uint32_t *)take(sizeof(uint32_t) * (2 * (p.n_buckets / 1024) + 1));
    p.bytes = off;
    return p;
}

struct FillWs {
    uint32_t *keyA, *valA, *keyB, *valB;
    size_t bytes;
};

static FillWs carve_fill(void *ws, uint64_t cap) {
    FillWs f;
    char *c = (char *)ws;
    size_t off = 0;
    auto take = [&](size_t b) { char *r = c ? c + off : nullptr; off += align256(b); return r; };
    f.keyA = (uint32_t *)take(sizeof(uint32_t) * cap);
    f.valA = (uint32_t *)take(sizeof(uint32_t) * cap);
    f.keyB = (uint32_t *)take(sizeof(uint32_t) * cap);
    f.valB = (uint32_t *)take(sizeof(uint32_t) * cap);
    f.bytes = off;
    return f;
}

struct BlkWs {
    uint32_t *rec_start, *unit_start, *unit_cnt, *tile_base;
    uint4 *unit_info;
    uint2 *rec;
    float *near;
    size_t bytes;
};

static BlkWs carve_blocks(void *ws, uint64_t cap) {
    BlkWs w;
    char *c = (char *)ws;
    size_t off = 0;
    auto take = [&](size_t n) { char *r = c ? c + off : nullptr; off += align256(n); return r; };
    w.rec_start = (uint32_t *)take(sizeof(uint32_t) * (kBlkMaxBlocks + 1));
    w.unit_start = (uint32_t *)take(sizeof(uint32_t) * (kBlkMaxBlocks + 1));
    w.tile_base = (uint32_t *)take(sizeof(uint32_t) * kBlkMaxBlocks * 32);
    // a record stands for at least one list entry; every block rounds its records up to whole units
    w.unit_cnt = (uint32_t *)take(sizeof(uint32_t) * 32 * (cap / kBlkUnitMin + kBlkMaxBlocks));
    w.unit_info = (uint4 *)take(sizeof(uint4) * (cap / kBlkUnitMin + kBlkMaxBlocks));
    w.near = (float *)take(sizeof(float));
    w.rec = (uint2 *)take(sizeof(uint2) * cap);
    w.bytes = off;
    return w;
}

static uint32_t bit_length(uint64_t v) {
    uint32_t b = 0;
    while (v) { ++b; v >>= 1; }
    return b;
}

struct IsectGeom {
    bool lidar;
    GridArgs<false> cam;
    GridArgs<true> lid;
    uint32_t C, N, total, n_tiles, tile_n_bits;
    const int64_t *camera_ids;
    const uint32_t *depth_bits;
};

// The block split applies to sorted output within the limits of its tables (six 1920 x 1080 cameras have 1620
// blocks, a 128-beam lidar 30); larger grids take the radix split.
static bool use_blocks(const IsectGeom &g, int sort) {
    if (sort == 0 || g.C > kBlkMaxSensors) return false;
    const uint64_t width = g.lidar ? g.lid.lidar.n_tiles_azim : g.cam.cam.tile_width, height = g.n_tiles / width;
    if (width > kBlkMaxExtent || height > kBlkMaxExtent) return false;
    const uint64_t bx = (width + kBlkW - 1) / kBlkW, blocks = bx * ((height + kBlkH - 1) / kBlkH);
    return bx <= kBlkMaxPerRow && blocks <= kBlkMaxPerSensor && blocks * g.C <= kBlkMaxBlocks &&
           g.C <= depth_bucket_count(g.total);
}

static BucketLayout bucket_layout(const IsectGeom &g, bool grouped) {
    const uint32_t groups = grouped ? g.C : 1u;
    return BucketLayout{g.camera_ids, g.N, groups, depth_bucket_count(g.total) / groups};
}

// Radix passes of eight bits that group the depth order by sensor (sort = 2).
static uint32_t sensor_passes(uint32_t C) { return C == 1 ? 0u : (bit_length(C - 1) + 7) / 8; }

// Where the plan leaves the block split's {depth bits, flatten index} pairs. keyA and valA lie back to back, as do
// keyB and valB (each g.total words, 256-byte aligned): either has room for g.total pairs. The radix order is in valB
// after an even number of passes by sensor, in valA after an odd one; the pairs go to the other two.
static uint2 *plan_pairs(const PlanWs &p, const IsectGeom &g, int sort) {
    const bool second = sort == 1 || sensor_passes(g.C) % 2 == 1;
    return reinterpret_cast<uint2 *>(second ? p.keyB : p.keyA);
}

// One-shot request of the calling thread's next plan (splatad_isect_set_early_count): where the
// rectangle count kernel writes the intersection count for the host, and the number it tags it with.
static thread_local int64_t *t_early_host = nullptr;
static thread_local int64_t t_early_seq = 0;
static thread_local int64_t *t_listed_host = nullptr;
static thread_local bool t_range_given = false;
static thread_local uint32_t t_range_lo = 0, t_range_hi = 0;

// plan: counts, depth order of visible Gaussians, n_isects.
static int isect_plan(const IsectGeom &g, int32_t *tiles_per_gauss, int sort, void *workspace,
                      size_t workspace_bytes, int64_t *host_counts, cudaStream_t st) {
    PlanWs p = carve_plan(workspace, g.total);
    SPL_REQUIRE(workspace != nullptr && workspace_bytes >= p.bytes, SPLATAD_ERR_WORKSPACE,
                "isect plan: workspace too small (%zu < %zu)", workspace_bytes, p.bytes);
    const uint32_t cam_n_bits = bit_length(g.C);   // floor(log2(C)) + 1
    SPL_REQUIRE(g.tile_n_bits + cam_n_bits <= 32, SPLATAD_ERR_KEY_BITS,
                "isect: tile bits (%u) + sensor bits (%u) exceed 32", g.tile_n_bits, cam_n_bits);
    SPL_REQUIRE((uint64_t)g.C * g.n_tiles <= 0xffffffffull, SPLATAD_ERR_KEY_BITS,
                "isect: sensors * tiles does not fit 32 bits");
    // sort: 0 = flatten order, 1 = sorted, depth order by buckets, 2 = sorted, depth order by radix passes
    const bool buckets = sort == 1;
    // a depth range handed over for this plan (splatad_isect_set_depth_range_hint): the rectangle count
    // fills the buckets itself and the separate bucket count is not launched
    const bool ranged = buckets && t_range_given && t_range_lo <= t_range_hi && t_range_hi < 0x7f800000u;
    const uint32_t range_lo = ranged ? t_range_lo : 1u, range_hi = ranged ? t_range_hi : 0u;
    t_range_given = false;
    {
        SPL_PROF("init_counters_kernel", st);
        if (buckets)
            launch_chained(init_counters_kernel, p.n_buckets / 1024, 1024, 0, st, p.counters, p.bcount, p.n_buckets,
                           range_lo, range_hi);
        else
            launch_chained(init_counters_kernel, 1, 32, 0, st, p.counters, (uint32_t *)nullptr, 0u, 1u, 0u);
    }
    // the block split wants the packed rectangles and the order grouped by sensor; it needs neither the
    // emission offsets nor their block sums
    const bool blocks = use_blocks(g, sort);
    const BucketLayout layout = bucket_layout(g, blocks);
    const uint32_t cgrid = min(div_up(g.total, kCountThreads), (uint32_t)(2 * kNumSMs));
    // the intersection count is known when the rectangle count ends: a host that has asked for it (to
    // size or cut its lists) gets it from a kernel - the rectangle count itself, or the bucket scatter soon
    // behind it, which also knows whether the bucket sort applies - and need not wait for the depth
    // order. Both list constructions report it: a host left to wait for words that never came gave up
    // after 20 ms, which was 87 % of a three-camera training step (22.6 -> 3.2 ms).
    const auto on_device = [](int64_t *host) {
        void *dptr = nullptr;
        if (host != nullptr && cudaHostGetDevicePointer(&dptr, host, 0) != cudaSuccess) {
            (void)cudaGetLastError();   // not mapped for this device: the host falls back to the event
            dptr = nullptr;
        }
        return (int64_t *)dptr;
    };
    int64_t *early = on_device(t_early_host), *listed = on_device(t_listed_host);
    const int64_t seq = t_early_seq;
    t_early_host = t_listed_host = nullptr;
    {
        SPL_PROF("isect_count_kernel", st);
        uint2 *rect = blocks ? p.rect : nullptr;
        int64_t *tot = p.counters + CNT_NISECT;
        int64_t *ticket = p.counters + CNT_TICKET;
        int64_t *early_here = buckets ? nullptr : early;
        const uint32_t *db = buckets ? g.depth_bits : nullptr;
        if (g.lidar)
            launch_chained(isect_count_kernel<true>, cgrid, kCountThreads, 0, st, g.lid, g.total, tiles_per_gauss,
                           layout, rect, tot, ticket, early_here, seq, db, p.counters,
                           ranged ? p.bcount : (uint32_t *)nullptr);
        else
            launch_chained(isect_count_kernel<false>, cgrid, kCountThreads, 0, st, g.cam, g.total, tiles_per_gauss,
                           layout, rect, tot, ticket, early_here, seq, db, p.counters,
                           ranged ? p.bcount : (uint32_t *)nullptr);
    }

    EmitArgs e{};
    e.total = g.total;
    e.tiles_per_gauss = tiles_per_gauss;
    e.camera_ids = g.camera_ids;
    e.N = g.N;
    if (buckets) {
        // depth order of the visible (count > 0) elements by buckets; result in keyB / valB
        const uint32_t bgrid = div_up(g.total, kThreads);   // one element per thread: the atomics' latency needs the parallelism
        // {bits, flatten index} pairs in bucket order, and in the end
        uint2 *pairs = reinterpret_cast<uint2 *>(p.keyA);
        uint2 *sorted_pair = plan_pairs(p, g, sort);
        if (!ranged) {
            SPL_PROF("depth_bucket_count_kernel", st);
            launch_chained(depth_bucket_count_kernel, bgrid, kThreads, 0, st, g.depth_bits,
                           (const int32_t *)tiles_per_gauss, g.total, layout, (const int64_t *)p.counters, p.bcount);
        }
        {
            SPL_PROF("depth_bucket_scan_kernel", st);
            launch_chained(depth_bucket_scan_kernel, p.n_buckets / 1024, 1024, 0, st, p.bcount, p.bstart, p.boff,
                           p.counters, layout.groups, layout.per, kBlkThreads,
                           blocks ? p.group_start : (uint32_t *)nullptr, p.group_chunk);
        }
        {
            SPL_PROF("depth_bucket_scatter_kernel", st);
            launch_chained(depth_bucket_scatter_kernel, bgrid, kThreads, 0, st, g.depth_bits,
                           (const int32_t *)tiles_per_gauss, g.total, layout, (const int64_t *)p.counters,
                           (volatile int64_t *)early, seq, (volatile int64_t *)listed,
                           (const uint32_t *)p.bstart, (const uint32_t *)p.boff, p.bcount, pairs);
        }
        {
            SPL_PROF("depth_bucket_rank_kernel", st);
            launch_chained(depth_bucket_rank_kernel, bgrid, kThreads, 0, st, layout, p.n_buckets,
                           (const int64_t *)p.counters, (const uint32_t *)p.bstart, (const uint32_t *)p.boff, (const uint2 *)pairs,
                           blocks ? (const uint2 *)p.rect : (const uint2 *)nullptr, sorted_pair, p.sorted_rect, p.valB);
        }
        e.order = p.valB;
        e.n_order_ptr = p.counters + CNT_NVIS;
    } else if (sort) {
        // stable sort of the visible (count > 0) elements by depth bits: 4 passes of 8 bits
        uint32_t *ka = p.keyA, *va = p.valA, *kb = p.keyB, *vb = p.valB;
        FinalOut nofin{};
        for (int pass = 0; pass < 4; ++pass) {
            PassSrc s{};
            if (pass == 0) {
                s.depth_bits = g.depth_bits;
                s.tiles_per_gauss = tiles_per_gauss;
                s.total = g.total;
                {
                    SPL_PROF("depthsort_upsweep", st);
                    launch_chained(radix_upsweep_kernel<true>, kSortGrid, kSortThreads, 0, st, s, 0, 0xffu, p.hist);
                }
                {
                    SPL_PROF("depthsort_rowscan", st);
                    launch_chained(radix_rowscan_kernel, kRadixBins, ((kSortGrid + 31) / 32) * 32, 0, st,
                                   p.hist, (uint32_t)kSortGrid, p.digit_totals);
                }
                {
                    SPL_PROF("depthsort_downsweep", st);
                    launch_chained(radix_downsweep_kernel<true, false>, kSortGrid, kSortThreads, 0, st,
                                   s, 0, 8, 0xffu, p.hist, p.digit_totals, ka, va, nofin, p.counters + CNT_NVIS);
                }
            } else {
                s.keys = ka; s.vals = va; s.n_ptr = p.counters + CNT_NVIS;
                {
                    SPL_PROF("depthsort_upsweep", st);
                    launch_chained(radix_upsweep_kernel<false>, kSortGrid, kSortThreads, 0, st, s, 8 * pass, 0xffu, p.hist);
                }
                {
                    SPL_PROF("depthsort_rowscan", st);
                    launch_chained(radix_rowscan_kernel, kRadixBins, ((kSortGrid + 31) / 32) * 32, 0, st,
                                   p.hist, (uint32_t)kSortGrid, p.digit_totals);
                }
                {
                    SPL_PROF("depthsort_downsweep", st);
                    launch_chained(radix_downsweep_kernel<false, false>, kSortGrid, kSortThreads, 0, st,
                                   s, 8 * pass, 8, 0xffu, p.hist, p.digit_totals, kb, vb, nofin, nullptr);
                }
                uint32_t *t;
                t = ka; ka = kb; kb = t;
                t = va; va = vb; vb = t;
            }
        }
        // 4 passes: A -> (pass0 writes A) ... after pass 3 the result sits in `va`
        // pass0: gen->A ; pass1: A->B ; pass2: B->A ; pass3: A->B  => sorted order in valB
        e.order = va;
        e.n_order_ptr = p.counters + CNT_NVIS;
        if (blocks) {
            const uint32_t grid = min(div_up(g.total, kThreads), (uint32_t)(8 * kNumSMs));
            const uint32_t passes = sensor_passes(g.C);
            // ka / va hold the order (B), kb / vb are free
            if (passes) {
                SPL_PROF("entry_sensors_kernel", st);
                launch_chained(entry_sensors_kernel, grid, kThreads, 0, st, layout, e.n_order_ptr, (const uint32_t *)va, kb);
            }
            for (uint32_t pass = 0; pass < passes; ++pass) {
                // the keys lie apart from their values in the first pass: keys A, values B
                PassSrc s{};
                s.keys = pass == 0 ? kb : ka; s.vals = va; s.n_ptr = e.n_order_ptr;
                uint32_t *out_keys = pass == 0 ? ka : kb, *out_vals = vb;
                {
                    SPL_PROF("sensorsort_upsweep", st);
                    launch_chained(radix_upsweep_kernel<false>, kSortGrid, kSortThreads, 0, st, s, (int)(8 * pass), 0xffu, p.hist);
                }
                {
                    SPL_PROF("sensorsort_rowscan", st);
                    launch_chained(radix_rowscan_kernel, kRadixBins, ((kSortGrid + 31) / 32) * 32, 0, st,
                                   p.hist, (uint32_t)kSortGrid, p.digit_totals);
                }
                {
                    SPL_PROF("sensorsort_downsweep", st);
                    launch_chained(radix_downsweep_kernel<false, false>, kSortGrid, kSortThreads, 0, st,
                                   s, (int)(8 * pass), 8, 0xffu, p.hist, p.digit_totals, out_keys, out_vals, nofin, nullptr);
                }
                std::swap(va, vb);
            }
            // after one pass the sorted sensors are in B and the order in A, after two in A and B
            const uint32_t *sensors = passes == 1 ? ka : kb;
            {
                SPL_PROF("group_starts_kernel", st);
                launch_chained(group_starts_kernel, 1, 1024, 0, st, e.n_order_ptr, sensors, g.C, kBlkThreads, p.group_start,
                               p.group_chunk);
            }
            {
                SPL_PROF("gather_entries_kernel", st);
                launch_chained(gather_entries_kernel, grid, kThreads, 0, st, e.n_order_ptr, (const uint32_t *)va, g.depth_bits,
                               (const uint2 *)p.rect, plan_pairs(p, g, sort), p.sorted_rect);
            }
        }
    }
    if (!blocks) {
        {
            SPL_PROF("emit_blocksum_kernel", st);
            emit_blocksum_kernel<<<kSortGrid, kThreads, 0, st>>>(e, p.block_sums);
        }
        {
            SPL_PROF("emit_scan_kernel", st);
            emit_scan_kernel<<<1, 1024, 0, st>>>(p.block_sums, kSortGrid, p.block_offs, p.counters);
        }
        {
            SPL_PROF("emit_offsets_kernel", st);
            emit_offsets_kernel<<<kSortGrid, kThreads, 0, st>>>(e, p.block_offs, p.eoff);
        }
    }
    if (host_counts != nullptr)
        cudaMemcpyAsync(host_counts, p.counters, sizeof(int64_t) * CNT_SLOTS, cudaMemcpyDeviceToHost, st);
    return check_launch("isect plan");
}

// One-shot request of the calling thread's next fill (splatad_isect_set_near_tiles). Where no kernel is to answer it, it is
// answered here: not known.
static thread_local int64_t *t_near_host = nullptr;
static thread_local uint32_t t_near_seq = 0;
struct NearRequest {
    int64_t *host = t_near_host;
    const uint32_t sequence = t_near_seq;
    NearRequest() { t_near_host = nullptr; }
    ~NearRequest() {
        if (host != nullptr) __atomic_store_n(host, (int64_t)((uint64_t)sequence << 32), __ATOMIC_RELEASE);
    }
    int64_t *take_on_device() {   // for a kernel that answers
        void *dptr = nullptr;
        if (host != nullptr && cudaHostGetDevicePointer(&dptr, host, 0) != cudaSuccess) {
            (void)cudaGetLastError();
            return nullptr;
        }
        host = nullptr;
        return (int64_t *)dptr;
    }
};

static int isect_fill(const IsectGeom &g, NearRequest &near, const int32_t *tiles_per_gauss, int sort,
                      void *plan_workspace, void *fill_workspace, size_t fill_workspace_bytes,
                      int64_t capacity, int64_t *isect_ids, int32_t *flatten_ids,
                      int32_t *tile_offsets, int64_t *host_counts, cudaStream_t st) {
    PlanWs p = carve_plan(plan_workspace, g.total);
    SPL_REQUIRE(plan_workspace != nullptr, SPLATAD_ERR_WORKSPACE, "isect fill: null plan workspace");
    if (capacity <= 0) return SPLATAD_OK;
    SPL_REQUIRE(isect_ids && flatten_ids, SPLATAD_ERR_BAD_ARG, "isect fill: null output");

    EmitArgs e{};
    e.total = g.total;
    e.tiles_per_gauss = tiles_per_gauss;
    e.camera_ids = g.camera_ids;
    e.N = g.N;
    e.n_tiles = g.n_tiles;
    e.tile_n_bits = g.tile_n_bits;
    e.depth_bits = g.depth_bits;
    e.capacity = capacity;

    if (!sort) {
        if (g.lidar) {
            {
                SPL_PROF("emit_kernel", st);
                emit_kernel<true, true><<<kSortGrid, kThreads, 0, st>>>(
                    g.lid, e, p.eoff, p.counters, nullptr, nullptr, isect_ids, flatten_ids, p.counters);
            }
        } else {
            {
                SPL_PROF("emit_kernel", st);
                emit_kernel<false, true><<<kSortGrid, kThreads, 0, st>>>(
                    g.cam, e, p.eoff, p.counters, nullptr, nullptr, isect_ids, flatten_ids, p.counters);
            }
        }
    } else if (use_blocks(g, sort)) {
        BlkWs w = carve_blocks(fill_workspace, (uint64_t)capacity);
        SPL_REQUIRE(fill_workspace != nullptr && fill_workspace_bytes >= w.bytes,
                    SPLATAD_ERR_WORKSPACE, "isect fill: workspace too small (%zu < %zu)",
                    fill_workspace_bytes, w.bytes);
        BlkArgs a{};
        a.rect = p.sorted_rect;
        a.pair = plan_pairs(p, g, sort);
        a.sensor_start = p.group_start;
        a.sensor_cta = p.group_chunk;
        a.counters = p.counters;
        a.capacity = capacity;
        a.C = g.C;
        a.n_tiles = g.n_tiles;
        a.width = g.lidar ? g.lid.lidar.n_tiles_azim : g.cam.cam.tile_width;
        a.height = g.n_tiles / a.width;
        a.bx = div_up(a.width, kBlkW);
        a.by = div_up(a.height, kBlkH);
        a.blocks = a.bx * a.by;
        a.tile_n_bits = g.tile_n_bits;
        a.table = p.blk_table;
        a.total = g.total;
        a.rec_start = w.rec_start; a.unit_start = w.unit_start;
        a.rec = w.rec;
        a.near = w.near; a.near_host = g.lidar ? nullptr : near.take_on_device(); a.near_sequence = near.sequence;
        a.near_least = 10000.f * (float)(g.C * g.n_tiles);
        const uint32_t near_sensors = min(g.C, kNearGroups);
        a.near_shift = bit_length(kNearGroups / near_sensors) - 1;
        a.near_step = g.C / near_sensors;
        a.unit_cnt = w.unit_cnt; a.unit_info = w.unit_info; a.tile_base = w.tile_base;
        const uint32_t ctas_a = div_up(g.total, kBlkThreads) + (g.C > 1 ? g.C : 0u);
        a.ctas = ctas_a;
        const uint32_t n_blocks = a.C * a.blocks;
        a.unit = (uint64_t)capacity > kBlkLongLists ? kBlkUnitMax : kBlkUnitMin;
        const uint32_t units_max = div_up((uint64_t)capacity, a.unit) + n_blocks;
        const size_t smem_count = sizeof(uint32_t) * a.blocks;
        const size_t smem_scatter = sizeof(uint32_t) * kBlkWarps * min(kBlkRows, a.by) * a.bx * (g.lidar ? 5 : 2);
        auto count = g.lidar ? blk_count_kernel<true> : blk_count_kernel<false>;
        auto scatter = !g.lidar ? blk_scatter_kernel<false, 4>
                       : min(kBlkRows, a.by) * a.bx >= kBlkManyCols ? blk_scatter_kernel<true, 2> : blk_scatter_kernel<true, 3>;
        if (smem_scatter > 48 * 1024)
            cudaFuncSetAttribute(scatter, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_scatter);
        unsigned long long *ticket = (unsigned long long *)(p.counters + CNT_TICKET);
        {
            SPL_PROF("blk_count_kernel", st);
            launch_chained(count, ctas_a, kBlkThreads, smem_count, st, a);
        }
        {
            SPL_PROF("blk_scan_kernel", st);
            launch_chained(blk_scan_kernel, n_blocks, 1024, 0, st, a, ticket);
        }
        {
            SPL_PROF("blk_scatter_kernel", st);
            launch_chained(scatter, dim3(ctas_a, div_up(a.by, kBlkRows)), kBlkThreads, smem_scatter, st, a);
        }
        {
            SPL_PROF("tile_count_kernel", st);
            auto kernel = a.unit == kBlkUnitMax ? tile_count_kernel<kBlkUnitMax / kBlkCountThreads>
                                                : tile_count_kernel<kBlkUnitMin / kBlkCountThreads>;
            launch_chained(kernel, min(units_max, kBlkGridB), kBlkCountThreads, 0, st, a);
        }
        {
            SPL_PROF("tile_scan_kernel", st);
            const uint32_t threads = n_blocks < kNumSMs ? 1024 : 256;
            auto kernel = (uint64_t)a.C * a.n_tiles > 4 * threads ? tile_scan_kernel<4> : tile_scan_kernel<1>;
            launch_chained(kernel, n_blocks, threads, 0, st, a, ticket, tile_offsets);
            tile_offsets = nullptr;   // done
        }
        {
            SPL_PROF(a.unit == kBlkUnitMax ? "tile_scatter_kernel/1024" : "tile_scatter_kernel", st);
            constexpr uint32_t kMin = kBlkUnitMin / (32 * kBlkWords), kMax = kBlkUnitMax / (32 * kBlkWords);
            const bool longer = a.unit == kBlkUnitMax;
            auto kernel = longer ? tile_scatter_kernel<kMax, true>
                                 : (uint64_t)capacity > kBlkCachedLists ? tile_scatter_kernel<kMin, true> : tile_scatter_kernel<kMin, false>;
            const uint32_t grid = min(units_max, (longer ? 2u : 6u) * kNumSMs);
            // long lists: not placed while the scan still holds its SMs (six cameras: frame 2585 us, 2627 chained)
            launch_chained_if(!longer, kernel, grid, a.unit / kBlkWords, 0, st, a, isect_ids, flatten_ids, p.counters);
        }
    } else {
        FillWs f = carve_fill(fill_workspace, (uint64_t)capacity);
        SPL_REQUIRE(fill_workspace != nullptr && fill_workspace_bytes >= f.bytes,
                    SPLATAD_ERR_WORKSPACE, "isect fill: workspace too small (%zu < %zu)",
                    fill_workspace_bytes, f.bytes);
        // depth order left by the plan in valB (see isect_plan)
        e.order = p.valB;
        e.n_order_ptr = p.counters + CNT_NVIS;
        if (g.lidar) {
            {
                SPL_PROF("emit_kernel", st);
                emit_kernel<true, false><<<kSortGrid, kThreads, 0, st>>>(
                    g.lid, e, p.eoff, p.counters, f.keyA, f.valA, nullptr, nullptr, p.counters);
            }
        } else {
            {
                SPL_PROF("emit_kernel", st);
                emit_kernel<false, false><<<kSortGrid, kThreads, 0, st>>>(
                    g.cam, e, p.eoff, p.counters, f.keyA, f.valA, nullptr, nullptr, p.counters);
            }
        }

        const uint64_t span = (uint64_t)g.C * g.n_tiles;
        const uint32_t key_bits = max(1u, bit_length(span - 1));
        const uint32_t npass = (key_bits + 7) / 8;
        const uint32_t bits_per = (key_bits + npass - 1) / npass;
        FinalOut fin{};
        fin.isect_ids = isect_ids;
        fin.flatten_ids = flatten_ids;
        fin.depth_bits = g.depth_bits;
        fin.n_tiles = g.n_tiles;
        fin.tile_n_bits = g.tile_n_bits;
        fin.capacity = capacity;
        uint32_t *ka = f.keyA, *va = f.valA, *kb = f.keyB, *vb = f.valB;
        for (uint32_t pass = 0; pass < npass; ++pass) {
            PassSrc s{};
            s.keys = ka; s.vals = va; s.n_ptr = p.counters + CNT_NISECT;
            s.n_cap = (uint32_t)(capacity < 0x7fffffffll ? capacity : 0x7fffffffll);
            const int shift = (int)(pass * bits_per);
            const uint32_t mask = (1u << bits_per) - 1u;
            {
                SPL_PROF("tilesort_upsweep", st);
                radix_upsweep_kernel<false><<<kSortGrid, kSortThreads, 0, st>>>(s, shift, mask, p.hist);
            }
            {
                SPL_PROF("tilesort_rowscan", st);
                radix_rowscan_kernel<<<kRadixBins, ((kSortGrid + 31) / 32) * 32, 0, st>>>(
                    p.hist, kSortGrid, p.digit_totals);
            }
            if (pass + 1 == npass) {
                {
                    SPL_PROF("tilesort_downsweep", st);
                    radix_downsweep_kernel<false, true><<<kSortGrid, kSortThreads, 0, st>>>(
                        s, shift, (int)bits_per, mask, p.hist, p.digit_totals, nullptr, nullptr, fin, nullptr);
                }
            } else {
                FinalOut nofin{};
                {
                    SPL_PROF("tilesort_downsweep", st);
                    radix_downsweep_kernel<false, false><<<kSortGrid, kSortThreads, 0, st>>>(
                        s, shift, (int)bits_per, mask, p.hist, p.digit_totals, kb, vb, nofin, nullptr);
                }
                uint32_t *t;
                t = ka; ka = kb; kb = t;
                t = va; va = vb; vb = t;
            }
        }
    }
    if (sort && tile_offsets != nullptr) {
        SPL_PROF("offset_encode_kernel", st);
        const uint32_t n_ct = g.C * g.n_tiles;
        offset_encode_kernel<<<div_up(n_ct + 1, kThreads), kThreads, 0, st>>>(
            isect_ids, p.counters + CNT_NISECT, capacity, g.C, g.n_tiles, g.tile_n_bits, tile_offsets);
    }
    if (host_counts != nullptr)
        cudaMemcpyAsync(host_counts, p.counters, sizeof(int64_t) * CNT_SLOTS, cudaMemcpyDeviceToHost, st);
    return check_launch("isect fill");
}

// ---------------------------------------------------------------------------------------
// Lidar points -> tiles (what prepares `raster_pts` from a point cloud before a lidar render;
// reference: gsplat/cuda/csrc/rasterization.cu:531-833). Same sort machinery as above on
// (sensor * n_tiles + tile, point index) pairs.
// ---------------------------------------------------------------------------------------
// One pass over the tiles: most tiles, most blocks, points per lane and per step of a block.
constexpr uint32_t kPointBins = 2048, kPointBlocks = 4 * kNumSMs;
constexpr int kPointsPerLane = 4;
constexpr uint32_t kPointTile = kSortThreads * kPointsPerLane;

struct PointsWs {
    int64_t *count;
    uint32_t *hist, *digit_totals;
    uint32_t *keyA, *valA, *keyB, *valB;
    size_t bytes;
};

static PointsWs carve_points(void *ws, uint64_t total) {
    PointsWs p;
    char *c = (char *)ws;
    size_t off = 0;
    auto take = [&](size_t b) { char *r = c ? c + off : nullptr; off += align256(b); return r; };
    p.count = (int64_t *)take(sizeof(int64_t));
    // radix passes: 256 digits x kSortGrid blocks; one pass over the tiles: kPointBins x kPointBlocks at most
    const size_t blocks = std::min<uint64_t>((total + kPointTile - 1) / kPointTile, kPointBlocks);
    p.hist = (uint32_t *)take(sizeof(uint32_t) * std::max<size_t>(kRadixBins * kSortGrid, kPointBins * blocks));
    p.digit_totals = (uint32_t *)take(sizeof(uint32_t) * kPointBins);
    p.keyA = (uint32_t *)take(sizeof(uint32_t) * total);
    p.valA = (uint32_t *)take(sizeof(uint32_t) * total);
    p.keyB = (uint32_t *)take(sizeof(uint32_t) * total);
    p.valB = (uint32_t *)take(sizeof(uint32_t) * total);
    p.bytes = off;
    return p;
}

// Where the points are and which tiles they fall into.
struct PointGrid {
    const float *points;         // azimuth and elevation, `stride` floats from point to point
    uint32_t stride;
    const int64_t *camera_ids;   // packed: sensor of each point, else nullptr
    uint32_t N;                  // points per sensor ([C, N] layout)
    const float *elev_boundaries;
    float tile_azim_resolution, min_azim;
    uint32_t n_tiles_azim, n_tiles_elev;
};

__device__ __forceinline__ float2 load_point(const PointGrid &g, uint32_t idx) {
    const float *pt = g.points + (size_t)idx * g.stride;
    return make_float2(__ldg(pt), __ldg(pt + 1));
}

// Sensor and tile of a point: azimuth tile by truncation (angles outside [0, 360) wrapped with fmodf),
// elevation tile = number of the first n_tiles_elev boundaries below the point, minus one.
__device__ __forceinline__ uint2 point_tile(const PointGrid &g, const float *elev_boundaries, uint32_t idx, float2 pt) {
    const float elev = pt.y, azim = pt.x - g.min_azim;
    float tile_azim;
    if (azim >= 0.f && azim < 360.f) tile_azim = azim / g.tile_azim_resolution;
    else tile_azim = fmodf(azim + 360.f, 360.f) / g.tile_azim_resolution;
    // float -> int conversion saturates (NaN -> 0); a point cannot land beyond the last tile of
    // its row, the clamp only keeps a malformed input inside the key range
    const uint32_t tx = min((uint32_t)max((int32_t)tile_azim, 0), g.n_tiles_azim - 1);
    // (the reference walks the ascending boundaries one by one; a bisection finds the same index)
    const uint32_t ty = (uint32_t)max(lower_bound_f(elev_boundaries, (int32_t)g.n_tiles_elev, elev) - 1, 0);
    return make_uint2(g.camera_ids ? (uint32_t)g.camera_ids[idx] : idx / g.N, ty * g.n_tiles_azim + tx);
}

__global__ void __launch_bounds__(kThreads)
points_tile_kernel(uint32_t total, PointGrid g, uint32_t *__restrict__ keys, uint32_t *__restrict__ vals,
                   int64_t *__restrict__ tile_ids, int32_t *__restrict__ flatten_ids, int64_t *__restrict__ count) {
    chain_enter();
    const uint32_t idx = blockIdx.x * blockDim.x + threadIdx.x;
    if (idx == 0 && count != nullptr) *count = (int64_t)total;
    if (idx >= total) return;
    const uint2 at = point_tile(g, g.elev_boundaries, idx, load_point(g, idx));
    if (keys != nullptr) {
        keys[idx] = at.x * (g.n_tiles_azim * g.n_tiles_elev) + at.y;
        vals[idx] = idx;
    } else {
        tile_ids[idx] = ((int64_t)at.x << 32) | (int64_t)at.y;
        flatten_ids[idx] = (int32_t)idx;
    }
}

// ---------------------------------------------------------------------------------------
// Few tiles - up to kPointBins over all sensors, which is any usual scan - are sorted in one pass over the
// tiles themselves: count per (tile, block), scan, place. Three kernels where tiles, two radix passes and
// ids took eight; a scan's points are few and the launches, not the bytes, are what it costs (230 k points
// to a 128 x 1800 image: 72 -> 40 us for the whole path, the image and the offsets included).
// ---------------------------------------------------------------------------------------
__global__ void __launch_bounds__(kSortThreads)
points_count_kernel(uint32_t total, uint32_t per_block, PointGrid g, uint32_t bins, uint32_t *__restrict__ keys,
                    uint32_t *__restrict__ hist /* [bins, blocks] */) {
    chain_enter();
    __shared__ uint32_t count[kPointBins];
    __shared__ float sb[kMaxElevSmem];
    const float *boundaries = g.elev_boundaries;
    if (g.n_tiles_elev <= kMaxElevSmem) {
        for (uint32_t i = threadIdx.x; i < g.n_tiles_elev; i += kSortThreads) sb[i] = g.elev_boundaries[i];
        boundaries = sb;
    }
    for (uint32_t d = threadIdx.x; d < bins; d += kSortThreads) count[d] = 0u;
    __syncthreads();
    const uint32_t lo = blockIdx.x * per_block, hi = min(total, lo + per_block);
    for (uint32_t i0 = lo + threadIdx.x; i0 < hi; i0 += kPointTile) {
        float2 pt[kPointsPerLane];
#pragma unroll
        for (int r = 0; r < kPointsPerLane; ++r) pt[r] = load_point(g, min(i0 + r * kSortThreads, hi - 1));
#pragma unroll
        for (int r = 0; r < kPointsPerLane; ++r) {
            const uint32_t idx = i0 + r * kSortThreads;
            if (idx >= hi) continue;
            const uint2 at = point_tile(g, boundaries, idx, pt[r]);
            const uint32_t key = min(at.x * (g.n_tiles_azim * g.n_tiles_elev) + at.y, bins - 1);   // a sensor id out of range stays inside
            keys[idx] = key;
            atomicAdd(&count[key], 1u);
        }
    }
    __syncthreads();
    for (uint32_t d = threadIdx.x; d < bins; d += kSortThreads) hist[(size_t)d * gridDim.x + blockIdx.x] = count[d];
}

// One warp's share of a tile of kPointTile points is ranked by ballots, the warps' counts by a scan; the points
// go to shared memory in key order first, so that a tile's run is written by neighbouring threads.
__global__ void __launch_bounds__(kSortThreads)
points_place_kernel(uint32_t total, uint32_t per_block, uint32_t bins, uint32_t key_bits, uint32_t n_tiles,
                    const uint32_t *__restrict__ keys, const uint32_t *__restrict__ hist,
                    const uint32_t *__restrict__ bin_totals, int64_t *__restrict__ tile_ids, int32_t *__restrict__ flatten_ids) {
    chain_enter();
    extern __shared__ __align__(16) uint32_t s_dyn[];
    __shared__ uint32_t wt[33];
    __shared__ uint32_t s_vals[kPointTile];
    __shared__ uint16_t s_keys[kPointTile];
    uint32_t *base = s_dyn;                                            // [bins] next place of the bin
    uint16_t *first = reinterpret_cast<uint16_t *>(base + bins);       // [bins] the bin's first place in the tile
    uint16_t *warp_count = first + ((bins + 1) & ~1u);                 // [warps][bins]
    const uint32_t t = threadIdx.x, lane = t & 31, warp = t >> 5;
    const uint32_t each = (bins + kSortThreads - 1) / kSortThreads, d0 = t * each, d1 = min(bins, d0 + each);
    {
        uint32_t sum = 0, all;
        for (uint32_t d = d0; d < d1; ++d) sum += bin_totals[d];
        uint32_t run = block_excl_scan(sum, wt, all);
        for (uint32_t d = d0; d < d1; ++d) {
            base[d] = run + hist[(size_t)d * gridDim.x + blockIdx.x];
            run += bin_totals[d];
        }
    }
    const uint32_t lo = blockIdx.x * per_block, hi = min(total, lo + per_block);
    for (uint32_t tile_lo = lo; tile_lo < hi; tile_lo += kPointTile) {
        for (uint32_t i = t; i < kSortWarps * bins; i += kSortThreads) warp_count[i] = 0;
        __syncthreads();
        uint32_t key[kPointsPerLane];
        uint16_t rank[kPointsPerLane];
        const uint32_t w0 = tile_lo + warp * (32 * kPointsPerLane) + lane;
#pragma unroll
        for (int r = 0; r < kPointsPerLane; ++r) key[r] = w0 + r * 32 < hi ? keys[w0 + r * 32] : bins;
        uint16_t *mine = warp_count + warp * bins;
#pragma unroll
        for (int r = 0; r < kPointsPerLane; ++r) {
            const bool valid = key[r] < bins;
            uint32_t peers = __ballot_sync(0xffffffffu, valid);
            for (uint32_t b = 0; b < key_bits; ++b) {
                const uint32_t set = __ballot_sync(0xffffffffu, (key[r] >> b) & 1u);
                peers &= ((key[r] >> b) & 1u) ? set : ~set;
            }
            if (!valid) peers = 1u << lane;
            const int leader = __ffs(peers) - 1;
            uint32_t old = 0;
            if (valid && lane == (uint32_t)leader) {
                old = mine[key[r]];
                mine[key[r]] = (uint16_t)(old + __popc(peers));
            }
            old = __shfl_sync(0xffffffffu, old, leader);
            rank[r] = (uint16_t)(old + __popc(peers & ((1u << lane) - 1u)));
            __syncwarp();
        }
        __syncthreads();
        {
            uint32_t sum = 0, all;
            for (uint32_t d = d0; d < d1; ++d) {
                uint32_t run = 0;
                for (uint32_t w = 0; w < (uint32_t)kSortWarps; ++w) {
                    const uint32_t c = warp_count[w * bins + d];
                    warp_count[w * bins + d] = (uint16_t)run;
                    run += c;
                }
                first[d] = (uint16_t)run;
                sum += run;
            }
            uint32_t at = block_excl_scan(sum, wt, all);
            for (uint32_t d = d0; d < d1; ++d) {
                const uint32_t n = first[d];
                first[d] = (uint16_t)at;
                at += n;
            }
        }
        __syncthreads();
#pragma unroll
        for (int r = 0; r < kPointsPerLane; ++r)
            if (key[r] < bins) {
                const uint32_t pos = first[key[r]] + mine[key[r]] + rank[r];
                s_keys[pos] = (uint16_t)key[r];
                s_vals[pos] = w0 + r * 32;
            }
        __syncthreads();
        const uint32_t n = min(kPointTile, hi - tile_lo);
        for (uint32_t j = t; j < n; j += kSortThreads) {
            const uint32_t k = s_keys[j], at = base[k] + (j - first[k]), cid = k / n_tiles;
            tile_ids[at] = ((int64_t)cid << 32) | (int64_t)(k - cid * n_tiles);
            flatten_ids[at] = (int32_t)s_vals[j];
        }
        __syncthreads();
        // the next tile's runs follow this one's
        for (uint32_t d = d0; d < d1; ++d) base[d] += (d + 1 < bins ? first[d + 1] : n) - first[d];
        __syncthreads();
    }
}

__global__ void __launch_bounds__(kThreads)
points_ids_kernel(uint32_t total, uint32_t n_tiles, const uint32_t *__restrict__ keys,
                  const uint32_t *__restrict__ vals, int64_t *__restrict__ tile_ids,
                  int32_t *__restrict__ flatten_ids) {
    chain_enter();
    const uint32_t idx = blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= total) return;
    const uint32_t key = keys[idx];
    const uint32_t cid = key / n_tiles;
    tile_ids[idx] = ((int64_t)cid << 32) | (int64_t)(key - cid * n_tiles);
    flatten_ids[idx] = (int32_t)vals[idx];
}

// offsets[c, tile] = first position whose (sensor, tile) >= (c, tile); ids are sensor << 32 | tile. One warp
// per tile and 32 probes per round: four dependent loads for 230 k points where a bisection waits for 18
// (6.5 -> 3.5 us).
__global__ void __launch_bounds__(kThreads)
points_offset_encode_kernel(const int64_t *__restrict__ point_ids, int64_t n, uint32_t C, uint32_t n_tiles,
                            int32_t *__restrict__ offsets) {
    chain_enter();
    const uint32_t t = blockIdx.x * (kThreads / 32) + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (t >= C * n_tiles) return;
    // `lo` ids are known to lie before the tile, the next `left` are not known
    int64_t lo = 0, left = n;
    while (left > 0) {
        const int64_t step = (left + 31) / 32, at = (int64_t)lane * step;
        bool before = false;
        if (at < left) {
            const int64_t id = __ldg(point_ids + lo + at);
            before = (id >> 32) * (int64_t)n_tiles + (id & 0xffffffffll) < (int64_t)t;
        }
        // ascending ids: the probes that lie before the tile are the first `k`
        const int64_t k = __popc(__ballot_sync(0xffffffffu, before));
        if (k == 0) break;
        lo += (k - 1) * step + 1;
        left = min(left - (k - 1) * step, step) - 1;
    }
    if (lane == 0) offsets[t] = (int32_t)lo;
}

// One block per tile, one thread per pixel of the tile: the thread of rank k takes the tile's
// k-th point (if there is one) and writes it at its own pixel.
__global__ void populate_image_kernel(uint32_t C, int64_t n_points, const float *__restrict__ points,
                                      uint32_t W, uint32_t H, uint32_t tile_width, uint32_t tile_height,
                                      uint32_t grid_w, uint32_t grid_h, const int32_t *__restrict__ offsets,
                                      const int32_t *__restrict__ flatten_ids, float *__restrict__ image,
                                      uint32_t clear /* write zeros to the pixels without a point */) {
    chain_enter();
    const uint32_t tiles_per_cam = grid_w * grid_h;
    const uint32_t cam = blockIdx.x / tiles_per_cam;
    const uint32_t tile = blockIdx.x - cam * tiles_per_cam;
    const uint32_t by = tile / grid_w, bx = tile - by * grid_w;
    const uint32_t tr = threadIdx.x;
    if (tr >= tile_width * tile_height) return;
    const uint32_t i = by * tile_height + tr / tile_width;
    const uint32_t j = bx * tile_width + tr % tile_width;
    if (i >= H || j >= W) return;
    const int64_t start = offsets[blockIdx.x];
    int64_t end = (blockIdx.x + 1 == C * tiles_per_cam) ? n_points : (int64_t)offsets[blockIdx.x + 1];
    end = min(end, start + (int64_t)(tile_width * tile_height));
    const int64_t k = start + tr;
    if (k >= end && !clear) return;
    float *dst = image + (((size_t)cam * H + i) * W + j) * 5;
    float v[5] = {0.f, 0.f, 0.f, 0.f, 0.f};
    if (k < end) {
        const float *src = points + (size_t)flatten_ids[k] * 5;
#pragma unroll
        for (int c = 0; c < 5; ++c) v[c] = src[c];
    }
#pragma unroll
    for (int c = 0; c < 5; ++c) dst[c] = v[c];
}

} // namespace splatad

using namespace splatad;

// =======================================================================================
// C-ABI
// =======================================================================================
extern "C" size_t splatad_isect_plan_workspace_bytes(uint64_t total_elems) {
    return carve_plan(nullptr, total_elems).bytes;
}

extern "C" size_t splatad_isect_fill_workspace_bytes(uint64_t capacity) {
    // the larger of the radix buffers and the block split's records + tables
    const size_t a = carve_fill(nullptr, capacity).bytes;
    const size_t b = carve_blocks(nullptr, capacity).bytes;
    return a > b ? a : b;
}

static int make_cam_geom(IsectGeom &g, uint32_t C, uint32_t N, uint64_t total,
                         const float *means2d, const int32_t *radii, const float *depths,
                         const int64_t *camera_ids, uint32_t tile_size, uint32_t tile_width,
                         uint32_t tile_height) {
    SPL_REQUIRE(means2d && radii && depths, SPLATAD_ERR_BAD_ARG, "isect_tiles: null input");
    SPL_REQUIRE(C > 0 && tile_size > 0 && tile_width > 0 && tile_height > 0, SPLATAD_ERR_BAD_ARG,
                "isect_tiles: bad geometry");
    SPL_REQUIRE(total <= 0x7fffffffull, SPLATAD_ERR_BAD_ARG, "isect_tiles: too many elements");
    SPL_REQUIRE((uint64_t)tile_width * tile_height * C <= 0xffffffffull, SPLATAD_ERR_KEY_BITS,
                "isect_tiles: sensors * tiles does not fit 32 bits");
    g = IsectGeom{};
    g.lidar = false;
    g.cam.cam = CamGrid{tile_size, tile_width, tile_height};
    g.cam.radii = radii;
    g.cam.means2d = (const float2 *)means2d;
    g.C = C; g.N = N ? N : 1; g.total = (uint32_t)total;
    g.n_tiles = tile_width * tile_height;
    g.tile_n_bits = bit_length(g.n_tiles);
    g.camera_ids = camera_ids;
    g.depth_bits = (const uint32_t *)depths;
    return SPLATAD_OK;
}

static int make_lidar_geom(IsectGeom &g, uint32_t C, uint32_t N, uint64_t total,
                           const float *means2d, const float *radii, const float *depths,
                           const int64_t *camera_ids, const float *elev_boundaries,
                           uint32_t n_boundaries, float tile_azim_resolution, float min_azim) {
    SPL_REQUIRE(means2d && radii && depths && elev_boundaries, SPLATAD_ERR_BAD_ARG,
                "isect_lidar_tiles: null input");
    SPL_REQUIRE(C > 0 && n_boundaries >= 2 && tile_azim_resolution > 0.f, SPLATAD_ERR_BAD_ARG,
                "isect_lidar_tiles: bad geometry");
    SPL_REQUIRE(total <= 0x7fffffffull, SPLATAD_ERR_BAD_ARG, "isect_lidar_tiles: too many elements");
    g = IsectGeom{};
    g.lidar = true;
    g.lid.lidar.elev_boundaries = elev_boundaries;
    g.lid.lidar.tile_azim_res = tile_azim_resolution;
    g.lid.lidar.min_azim = min_azim;
    g.lid.lidar.n_tiles_azim = splatad_lidar_azimuth_tiles(tile_azim_resolution);
    g.lid.lidar.n_tiles_elev = n_boundaries - 1;
    g.lid.radii = radii;
    g.lid.means2d = (const float2 *)means2d;
    g.C = C; g.N = N ? N : 1; g.total = (uint32_t)total;
    g.n_tiles = g.lid.lidar.n_tiles_azim * g.lid.lidar.n_tiles_elev;
    g.tile_n_bits = bit_length(g.n_tiles);
    g.camera_ids = camera_ids;
    g.depth_bits = (const uint32_t *)depths;
    return SPLATAD_OK;
}

extern "C" int splatad_isect_tiles_plan(
    uint32_t C, uint32_t N, uint64_t total_elems, const float *means2d, const int32_t *radii,
    const float *depths, const int64_t *camera_ids, uint32_t tile_size, uint32_t tile_width,
    uint32_t tile_height, int32_t sort, int32_t *tiles_per_gauss, void *workspace,
    size_t workspace_bytes, int64_t *host_counts, void *stream) {
    if (total_elems == 0) {
        if (host_counts) for (int i = 0; i < CNT_SLOTS; ++i) host_counts[i] = 0;
        return SPLATAD_OK;
    }
    IsectGeom g;
    int rc = make_cam_geom(g, C, N, total_elems, means2d, radii, depths, camera_ids, tile_size,
                           tile_width, tile_height);
    if (rc != SPLATAD_OK) return rc;
    SPL_REQUIRE(tiles_per_gauss, SPLATAD_ERR_BAD_ARG, "isect_tiles_plan: null tiles_per_gauss");
    return isect_plan(g, tiles_per_gauss, sort, workspace, workspace_bytes, host_counts,
                      (cudaStream_t)stream);
}

extern "C" int splatad_isect_tiles_fill(
    uint32_t C, uint32_t N, uint64_t total_elems, const float *means2d, const int32_t *radii,
    const float *depths, const int64_t *camera_ids, uint32_t tile_size, uint32_t tile_width,
    uint32_t tile_height, int32_t sort, const int32_t *tiles_per_gauss, void *plan_workspace,
    void *fill_workspace, size_t fill_workspace_bytes, int64_t capacity, int64_t *isect_ids,
    int32_t *flatten_ids, int32_t *tile_offsets, int64_t *host_counts, void *stream) {
    NearRequest near;
    if (total_elems == 0 || capacity <= 0) return SPLATAD_OK;
    IsectGeom g;
    int rc = make_cam_geom(g, C, N, total_elems, means2d, radii, depths, camera_ids, tile_size,
                           tile_width, tile_height);
    if (rc != SPLATAD_OK) return rc;
    return isect_fill(g, near, tiles_per_gauss, sort, plan_workspace, fill_workspace,
                      fill_workspace_bytes, capacity, isect_ids, flatten_ids, tile_offsets, host_counts,
                      (cudaStream_t)stream);
}

extern "C" uint32_t splatad_lidar_azimuth_tiles(float tile_azim_resolution) {
    return tile_azim_resolution > 0.f ? (uint32_t)ceilf(360.f / tile_azim_resolution) : 0u;
}

extern "C" int splatad_isect_lidar_tiles_plan(
    uint32_t C, uint32_t N, uint64_t total_elems, const float *means2d, const float *radii,
    const float *depths, const int64_t *camera_ids, const float *elev_boundaries,
    uint32_t n_boundaries, float tile_azim_resolution, float min_azim, int32_t sort,
    int32_t *tiles_per_gauss, void *workspace, size_t workspace_bytes, int64_t *host_counts,
    void *stream) {
    if (total_elems == 0) {
        if (host_counts) for (int i = 0; i < CNT_SLOTS; ++i) host_counts[i] = 0;
        return SPLATAD_OK;
    }
    IsectGeom g;
    int rc = make_lidar_geom(g, C, N, total_elems, means2d, radii, depths, camera_ids,
                             elev_boundaries, n_boundaries, tile_azim_resolution, min_azim);
    if (rc != SPLATAD_OK) return rc;
    SPL_REQUIRE(tiles_per_gauss, SPLATAD_ERR_BAD_ARG, "isect_lidar_tiles_plan: null tiles_per_gauss");
    return isect_plan(g, tiles_per_gauss, sort, workspace, workspace_bytes, host_counts,
                      (cudaStream_t)stream);
}

extern "C" int splatad_isect_lidar_tiles_fill(
    uint32_t C, uint32_t N, uint64_t total_elems, const float *means2d, const float *radii,
    const float *depths, const int64_t *camera_ids, const float *elev_boundaries,
    uint32_t n_boundaries, float tile_azim_resolution, float min_azim, int32_t sort,
    const int32_t *tiles_per_gauss, void *plan_workspace, void *fill_workspace,
    size_t fill_workspace_bytes, int64_t capacity, int64_t *isect_ids, int32_t *flatten_ids,
    int32_t *tile_offsets, int64_t *host_counts, void *stream) {
    NearRequest near;   // (lidar lists: not known)
    if (total_elems == 0 || capacity <= 0) return SPLATAD_OK;
    IsectGeom g;
    int rc = make_lidar_geom(g, C, N, total_elems, means2d, radii, depths, camera_ids,
                             elev_boundaries, n_boundaries, tile_azim_resolution, min_azim);
    if (rc != SPLATAD_OK) return rc;
    return isect_fill(g, near, tiles_per_gauss, sort, plan_workspace, fill_workspace,
                      fill_workspace_bytes, capacity, isect_ids, flatten_ids, tile_offsets, host_counts,
                      (cudaStream_t)stream);
}

extern "C" int splatad_isect_set_early_count(int64_t *host_pair, int64_t sequence) {
    t_early_host = host_pair;
    t_early_seq = sequence;
    return SPLATAD_OK;
}

extern "C" int splatad_isect_set_listed_count(int64_t *host_word) {
    t_listed_host = host_word;
    return SPLATAD_OK;
}

extern "C" int splatad_isect_set_near_tiles(int64_t *host_word, uint32_t sequence) {
    t_near_host = host_word;
    t_near_seq = sequence;
    return SPLATAD_OK;
}

extern "C" int splatad_isect_set_depth_range_hint(uint32_t depth_lo_bits, uint32_t depth_hi_bits) {
    t_range_given = true;
    t_range_lo = depth_lo_bits;
    t_range_hi = depth_hi_bits;
    return SPLATAD_OK;
}

extern "C" int splatad_isect_offset_encode(const int64_t *isect_ids, int64_t n_isects, uint32_t C,
                                           uint32_t tile_width, uint32_t tile_height,
                                           int32_t *offsets, void *stream) {
    SPL_REQUIRE(offsets, SPLATAD_ERR_BAD_ARG, "isect_offset_encode: null output");
    const uint64_t n_tiles = (uint64_t)tile_width * tile_height;
    SPL_REQUIRE(C > 0 && n_tiles > 0 && (uint64_t)C * n_tiles <= 0x7fffffffull, SPLATAD_ERR_BAD_ARG,
                "isect_offset_encode: bad geometry");
    SPL_REQUIRE(n_isects == 0 || isect_ids, SPLATAD_ERR_BAD_ARG, "isect_offset_encode: null input");
    const uint32_t tile_n_bits = bit_length(n_tiles);
    const uint32_t total = (uint32_t)(C * n_tiles);
    {
        SPL_PROF("offset_encode_kernel", (cudaStream_t)stream);
        offset_encode_kernel<<<div_up(total, kThreads), kThreads, 0, (cudaStream_t)stream>>>(
            isect_ids, nullptr, n_isects, C, (uint32_t)n_tiles, tile_n_bits, offsets);
    }
    return check_launch("isect_offset_encode");
}

// =======================================================================================
// Lidar points -> tiles -> raster image
// =======================================================================================
extern "C" size_t splatad_map_points_workspace_bytes(uint64_t total_elems) {
    return carve_points(nullptr, total_elems).bytes;
}

extern "C" int splatad_map_points_to_lidar_tiles(
    uint32_t C, uint32_t N, uint64_t total_elems, const float *points2d, const int64_t *camera_ids,
    const float *elev_boundaries, uint32_t n_boundaries, float tile_azim_resolution, float min_azim,
    int32_t sort, void *workspace, size_t workspace_bytes, int64_t *tile_ids, int32_t *flatten_ids,
    void *stream) {
    return splatad_map_strided_points_to_lidar_tiles(C, N, total_elems, points2d, 2, camera_ids, elev_boundaries, n_boundaries,
                                                     tile_azim_resolution, min_azim, sort, workspace, workspace_bytes,
                                                     tile_ids, flatten_ids, stream);
}

extern "C" int splatad_map_strided_points_to_lidar_tiles(
    uint32_t C, uint32_t N, uint64_t total_elems, const float *points2d, uint32_t point_stride, const int64_t *camera_ids,
    const float *elev_boundaries, uint32_t n_boundaries, float tile_azim_resolution, float min_azim,
    int32_t sort, void *workspace, size_t workspace_bytes, int64_t *tile_ids, int32_t *flatten_ids,
    void *stream) {
    if (total_elems == 0) return SPLATAD_OK;
    cudaStream_t st = (cudaStream_t)stream;
    SPL_REQUIRE(points2d && elev_boundaries && tile_ids && flatten_ids, SPLATAD_ERR_BAD_ARG,
                "map_points_to_lidar_tiles: null argument");
    SPL_REQUIRE(C > 0 && n_boundaries >= 2 && tile_azim_resolution > 0.f && point_stride >= 2, SPLATAD_ERR_BAD_ARG,
                "map_points_to_lidar_tiles: bad geometry");
    SPL_REQUIRE(total_elems <= 0x7fffffffull, SPLATAD_ERR_BAD_ARG, "map_points_to_lidar_tiles: too many points");
    const uint32_t total = (uint32_t)total_elems;
    const uint32_t n_az = splatad_lidar_azimuth_tiles(tile_azim_resolution), n_el = n_boundaries - 1;
    const uint64_t span = (uint64_t)C * n_az * n_el;
    SPL_REQUIRE(span <= 0xffffffffull, SPLATAD_ERR_KEY_BITS, "map_points_to_lidar_tiles: sensors * tiles does not fit 32 bits");
    const PointGrid g = {points2d, point_stride, camera_ids, N ? N : 1, elev_boundaries, tile_azim_resolution, min_azim, n_az, n_el};
    const uint32_t grid = div_up(total, kThreads);
    if (!sort) {
        SPL_PROF("points_tile_kernel", st);
        launch_chained(points_tile_kernel, grid, kThreads, 0, st, total, g, nullptr, nullptr, tile_ids, flatten_ids, nullptr);
        return check_launch("map_points_to_lidar_tiles");
    }
    PointsWs p = carve_points(workspace, total);
    SPL_REQUIRE(workspace != nullptr && workspace_bytes >= p.bytes, SPLATAD_ERR_WORKSPACE,
                "map_points_to_lidar_tiles: workspace too small (%zu < %zu)", workspace_bytes, p.bytes);
    const uint32_t key_bits = max(1u, bit_length(span - 1));
    if (span <= kPointBins) {
        const uint32_t bins = (uint32_t)span, tiles = div_up(total, kPointTile);
        const uint32_t per_block = kPointTile * div_up(tiles, kPointBlocks), blocks = div_up(total, per_block);
        {
            SPL_PROF("points_count_kernel", st);
            launch_chained(points_count_kernel, blocks, kSortThreads, 0, st, total, per_block, g, bins, p.keyA, p.hist);
        }
        {
            SPL_PROF("points_sort_rowscan", st);
            launch_chained(radix_rowscan_kernel, bins, div_up(blocks, 32) * 32, 0, st, p.hist, blocks, p.digit_totals);
        }
        {
            SPL_PROF("points_place_kernel", st);
            const size_t smem = sizeof(uint32_t) * bins + sizeof(uint16_t) * (((bins + 1) & ~1u) + kSortWarps * bins);
            if (smem > 32 * 1024)
                cudaFuncSetAttribute(points_place_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
            launch_chained(points_place_kernel, blocks, kSortThreads, smem, st, total, per_block, bins, key_bits, n_az * n_el,
                           p.keyA, p.hist, p.digit_totals, tile_ids, flatten_ids);
        }
        return check_launch("map_points_to_lidar_tiles");
    }
    {
        SPL_PROF("points_tile_kernel", st);
        launch_chained(points_tile_kernel, grid, kThreads, 0, st, total, g, p.keyA, p.valA, nullptr, nullptr, p.count);
    }
    // stable LSD radix sort of the (key, index) pairs over the bits the keys use
    const uint32_t npass = (key_bits + 7) / 8;
    const uint32_t bits_per = (key_bits + npass - 1) / npass;
    uint32_t *ka = p.keyA, *va = p.valA, *kb = p.keyB, *vb = p.valB;
    FinalOut nofin{};
    for (uint32_t pass = 0; pass < npass; ++pass) {
        PassSrc s{};
        s.keys = ka; s.vals = va; s.n_ptr = p.count;
        s.n_cap = total;
        const int shift = (int)(pass * bits_per);
        const uint32_t mask = (1u << bits_per) - 1u;
        {
            SPL_PROF("points_sort_upsweep", st);
            launch_chained(radix_upsweep_kernel<false>, kSortGrid, kSortThreads, 0, st, s, shift, mask, p.hist);
        }
        {
            SPL_PROF("points_sort_rowscan", st);
            launch_chained(radix_rowscan_kernel, kRadixBins, ((kSortGrid + 31) / 32) * 32, 0, st, p.hist, kSortGrid,
                                                                                    p.digit_totals);
        }
        {
            SPL_PROF("points_sort_downsweep", st);
            launch_chained(radix_downsweep_kernel<false, false>, kSortGrid, kSortThreads, 0, st,
                s, shift, (int)bits_per, mask, p.hist, p.digit_totals, kb, vb, nofin, nullptr);
        }
        uint32_t *t;
        t = ka; ka = kb; kb = t;
        t = va; va = vb; vb = t;
    }
    {
        SPL_PROF("points_ids_kernel", st);
        launch_chained(points_ids_kernel, grid, kThreads, 0, st, total, n_az * n_el, ka, va, tile_ids, flatten_ids);
    }
    return check_launch("map_points_to_lidar_tiles");
}

extern "C" int splatad_points_mapping_offset_encode(const int64_t *point_ids, int64_t n_points, uint32_t C,
                                                    uint32_t tile_width, uint32_t tile_height,
                                                    int32_t *offsets, void *stream) {
    SPL_REQUIRE(offsets, SPLATAD_ERR_BAD_ARG, "points_mapping_offset_encode: null output");
    const uint64_t n_tiles = (uint64_t)tile_width * tile_height;
    SPL_REQUIRE(C > 0 && n_tiles > 0 && (uint64_t)C * n_tiles <= 0x7fffffffull, SPLATAD_ERR_BAD_ARG,
                "points_mapping_offset_encode: bad geometry");
    SPL_REQUIRE(n_points == 0 || point_ids, SPLATAD_ERR_BAD_ARG, "points_mapping_offset_encode: null input");
    const uint32_t total = (uint32_t)(C * n_tiles);
    {
        SPL_PROF("points_offset_encode_kernel", (cudaStream_t)stream);
        launch_chained(points_offset_encode_kernel, div_up(total, kThreads / 32), kThreads, 0, (cudaStream_t)stream,
            point_ids, n_points, C, (uint32_t)n_tiles, offsets);
    }
    return check_launch("points_mapping_offset_encode");
}

extern "C" int splatad_populate_image_from_points(
    uint32_t C, int64_t n_points, const float *points, uint32_t image_width, uint32_t image_height,
    uint32_t tile_width, uint32_t tile_height, uint32_t tile_grid_width, uint32_t tile_grid_height,
    const int32_t *tile_offsets, const int32_t *flatten_ids, float *image, void *stream) {
    cudaStream_t st = (cudaStream_t)stream;
    SPL_REQUIRE(image && tile_offsets, SPLATAD_ERR_BAD_ARG, "populate_image_from_points: null argument");
    SPL_REQUIRE(tile_width >= 1 && tile_height >= 1 && tile_width * tile_height <= 1024, SPLATAD_ERR_BAD_ARG,
                "populate_image_from_points: tile_width * tile_height must be in 1..1024");
    SPL_REQUIRE(n_points == 0 || (points && flatten_ids), SPLATAD_ERR_BAD_ARG,
                "populate_image_from_points: null input");
    const size_t n_pix = (size_t)C * image_height * image_width;
    if (n_pix == 0) return SPLATAD_OK;
    const uint32_t blocks = C * tile_grid_width * tile_grid_height;
    // tiles that cover the image write every pixel of it once: no pass over it before them
    const bool covered = blocks > 0 && n_points > 0 && (uint64_t)tile_grid_width * tile_width >= image_width &&
                         (uint64_t)tile_grid_height * tile_height >= image_height;
    if (!covered) cudaMemsetAsync(image, 0, n_pix * 5 * sizeof(float), st);
    if (blocks == 0 || n_points == 0) return check_launch("populate_image_from_points");
    const uint32_t bs = ((tile_width * tile_height + 31) / 32) * 32;
    {
        SPL_PROF("populate_image_kernel", st);
        launch_chained(populate_image_kernel, blocks, bs, 0, st, C, n_points, points, image_width, image_height, tile_width,
                                                    tile_height, tile_grid_width, tile_grid_height, tile_offsets,
                                                    flatten_ids, image, covered ? 1u : 0u);
    }
    return check_launch("populate_image_from_points");
}
