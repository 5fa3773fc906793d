// The host side of a frame in native code: one call allocates a frame's outputs, enqueues all of its
// kernels through the C ABI, waits for the counts the kernels store into pinned memory, cuts the lists to
// length and puts two nodes into torch's autograd graph - projection and compositing - whose backward
// passes run here as well. Same kernels, results, graph semantics and gradient slots as the individual ops
// (splatad_b200/ops.py) called in sequence (the reference's orchestration: gsplat/rendering.py:22-440,
// 443-819); what goes away is the Python between some fifteen launches, forward and backward.
// Measured on a scene small enough to be bound by it: camera training step 1168 -> 280 us, lidar
// training step with compensated opacities 753 -> 277 us, lidar frame 227 -> 81 us, camera frame 262 -> 67 us.
//
// A frame needs the counts of an earlier frame of its shape to size its lists; the caller keeps those and
// falls back to the individual ops when there are none, when a count outgrew its room, or for arguments
// that this file does not take (the functions return None for them before anything is enqueued).
#include <dlfcn.h>
#include <torch/extension.h>

#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>

#include <cstring>
#include <map>
#include <tuple>
#include <vector>

#include "../../../include/splatad_b200.h"

namespace {

using at::Tensor;
using torch::autograd::AutogradContext;
using torch::autograd::variable_list;
using OptTensor = c10::optional<Tensor>;

// ---------------------------------------------------------------------------------------------
// The CUDA library: the same image the ctypes bindings use, symbols looked up once.
// ---------------------------------------------------------------------------------------------
#define SPL_SYMBOLS(X)                                                                                                  \
    X(splatad_last_error)                                                                                               \
    X(splatad_lidar_projection_fwd) X(splatad_lidar_projection_bwd) X(splatad_projection_fwd) X(splatad_projection_bwd)  \
    X(splatad_projection_packed_workspace_bytes) X(splatad_projection_packed_count) X(splatad_projection_packed_fill)    \
    X(splatad_projection_packed_bwd) X(splatad_camera_centers) X(splatad_sh_colors_fwd) X(splatad_sh_colors_bwd)         \
    X(splatad_opacity_rows_fwd) X(splatad_opacity_rows_bwd) X(splatad_color_rows_fwd) X(splatad_color_rows_bwd)          \
    X(splatad_isect_plan_workspace_bytes) X(splatad_isect_fill_workspace_bytes) X(splatad_lidar_azimuth_tiles)           \
    X(splatad_isect_tiles_plan) X(splatad_isect_tiles_fill) X(splatad_isect_lidar_tiles_plan)                            \
    X(splatad_isect_lidar_tiles_fill) X(splatad_isect_set_early_count) X(splatad_isect_set_depth_range_hint)             \
    X(splatad_isect_set_listed_count) X(splatad_isect_set_near_tiles) X(splatad_rasterize_set_spread_hint)               \
    X(splatad_rasterize_set_near_hint) X(splatad_rasterize_set_rows_hint)                                                \
    X(splatad_rasterize_expected_to_pixels_fwd) X(splatad_rasterize_expected_to_pixels_bwd)                              \
    X(splatad_lidar_frame_fwd) X(splatad_rasterize_to_points_fwd) X(splatad_rasterize_to_points_bwd) X(splatad_map_points_workspace_bytes)          \
    X(splatad_map_strided_points_to_lidar_tiles) X(splatad_points_mapping_offset_encode) X(splatad_populate_image_from_points)

struct Lib {
#define SPL_MEMBER(name) decltype(&::name) name = nullptr;
    SPL_SYMBOLS(SPL_MEMBER)
#undef SPL_MEMBER
} lib;

void bind_library(const std::string &path) {
    void *h = dlopen(path.c_str(), RTLD_NOW | RTLD_LOCAL);
    if (h == nullptr) throw std::runtime_error(std::string("cannot load ") + path + ": " + dlerror());
#define SPL_LOOKUP(name)                                                                    \
    lib.name = reinterpret_cast<decltype(lib.name)>(dlsym(h, #name));                       \
    if (lib.name == nullptr) throw std::runtime_error(path + " lacks " #name);
    SPL_SYMBOLS(SPL_LOOKUP)
#undef SPL_LOOKUP
}

// the exception the ctypes bindings raise for the same status
void check(int rc) {
    if (rc == SPLATAD_OK) return;
    const char *msg = lib.splatad_last_error();
    if (rc == SPLATAD_ERR_BAD_ARG || rc == SPLATAD_ERR_CHANNELS) TORCH_CHECK_VALUE(false, msg);
    TORCH_CHECK(false, msg);
}

// ---------------------------------------------------------------------------------------------
// Tensors
// ---------------------------------------------------------------------------------------------
const float *F(const Tensor &t) { return t.defined() && t.numel() ? t.const_data_ptr<float>() : nullptr; }
const float *F(const OptTensor &t) { return t ? F(*t) : nullptr; }
float *M(const Tensor &t) { return t.defined() && t.numel() ? t.data_ptr<float>() : nullptr; }
int32_t *I(const Tensor &t) { return t.defined() && t.numel() ? t.data_ptr<int32_t>() : nullptr; }
int64_t *L(const Tensor &t) { return t.defined() && t.numel() ? t.data_ptr<int64_t>() : nullptr; }

// float32, dense, contiguous, on GPU `dev`: what the kernels read without a conversion. Not a tensor that stands for
// another - a dual number of forward-mode differentiation, whose tangent would be lost, or a transform's wrapper:
// the ops say what they say to those.
bool plain(const Tensor &t, c10::DeviceIndex dev) {
    return t.defined() && t.has_storage() && !t.unsafeGetTensorImpl()->is_python_dispatch() && !t._fw_grad(0).defined() && t.is_cuda() && t.get_device() == dev && t.scalar_type() == at::kFloat && t.layout() == at::kStrided &&
           t.is_contiguous() && !t.is_conj() && !t.is_neg();
}
bool plain(const OptTensor &t, c10::DeviceIndex dev) { return !t || plain(*t, dev); }

// The frame goes into the graph if any of the tensors its nodes take requires a gradient, also one that gets none.
bool wants_grad(std::initializer_list<const Tensor *> all, std::initializer_list<const OptTensor *> maybe) {
    if (!at::GradMode::is_enabled()) return false;
    for (const Tensor *t : all)
        if (t->requires_grad()) return true;
    for (const OptTensor *t : maybe)
        if (*t && (*t)->requires_grad()) return true;
    return false;
}

bool shaped(const Tensor &t, at::IntArrayRef s) { return t.sizes() == s; }
bool shaped(const OptTensor &t, at::IntArrayRef s) { return !t || t->sizes() == s; }

// The first rows of a tensor as a tensor of their own (not a view in the autograd sense: its producer is
// the node it is handed to).
Tensor alias(const Tensor &base, at::IntArrayRef sizes, int64_t offset = 0) {
    auto impl = c10::make_intrusive<c10::TensorImpl>(c10::Storage(base.storage()), base.key_set(), base.dtype());
    impl->set_storage_offset(base.storage_offset() + offset);
    impl->set_sizes_contiguous(sizes);
    return Tensor(std::move(impl));
}

Tensor head(const Tensor &t, int64_t rows) {
    if (!t.defined() || t.size(0) == rows) return t;
    std::vector<int64_t> s(t.sizes().begin(), t.sizes().end());
    s[0] = rows;
    return alias(t, s);
}

// zero-filled float32 tensors out of one buffer: one allocation and one fill for all accumulators of a
// backward pass; every one starts a multiple of 256 bytes behind the buffer's start
struct Zeros {
    std::vector<std::vector<int64_t>> shapes;
    std::vector<Tensor *> into;
    void add(Tensor &t, at::IntArrayRef shape) {
        into.push_back(&t);
        shapes.emplace_back(shape.begin(), shape.end());
    }
    void make(const at::TensorOptions &options) {
        int64_t total = 0;
        for (auto &s : shapes) total += (c10::multiply_integers(s) + 63) / 64 * 64;
        if (total == 0) total = 64;
        const Tensor buffer = at::zeros({total}, options);
        int64_t at = 0;
        for (size_t i = 0; i < into.size(); ++i) {
            *into[i] = alias(buffer, shapes[i], at);
            at += (c10::multiply_integers(shapes[i]) + 63) / 64 * 64;
        }
    }
};

// a cotangent as the kernels read it; missing: zeros of `like`'s shape
Tensor cotangent(const Tensor &g, const Tensor &like) {
    if (!g.defined()) return at::zeros_like(like);
    return (g.scalar_type() == at::kFloat ? g : g.to(at::kFloat)).contiguous();
}

// ---------------------------------------------------------------------------------------------
// Workspaces and pinned slots, per device and stream. The Python bindings take theirs from here too.
// Called with the GIL held.
// ---------------------------------------------------------------------------------------------
using StreamKey = std::pair<int, cudaStream_t>;
std::map<std::pair<std::string, StreamKey>, Tensor> workspaces;
std::map<StreamKey, std::vector<Tensor>> free_slots;
std::map<StreamKey, Tensor> still;

Tensor workspace(const char *tag, size_t bytes, c10::cuda::CUDAStream stream) {
    Tensor &t = workspaces[{tag, {stream.device_index(), stream.stream()}}];
    if (!t.defined() || (size_t)t.numel() < bytes) {
        t.reset();   // the old buffer goes back before the larger one is asked for
        // grows with headroom so that slowly growing scenes do not reallocate every frame
        const int64_t size = std::max<int64_t>((int64_t)(bytes * 1.25) + 1024, 1 << 16);
        t = at::empty({size}, at::TensorOptions().dtype(at::kByte).device(at::kCUDA, stream.device_index()));
    }
    return t;
}

// Pinned words that one frame owns until its counts have been read, stored by its kernels: [4..7] {count,
// sequence, status, depth range}, [8] the packed row count, [9] the elements listed. (The plan's own copy of its counters at its end is
// not asked for: it breaks the chain of launches, 8 us of a small frame's 120.)
struct Slot {
    StreamKey key;
    Tensor t;
    volatile int64_t *word;
    explicit Slot(c10::cuda::CUDAStream s) : key(s.device_index(), s.stream()) {
        auto &free = free_slots[key];
        if (free.empty()) {
            t = at::zeros({16}, at::TensorOptions().dtype(at::kLong)).pin_memory();
        } else {
            t = std::move(free.back());
            free.pop_back();
        }
        word = t.data_ptr<int64_t>();
    }
    ~Slot() {
        auto &free = free_slots[key];
        if (free.size() < 16) free.push_back(std::move(t));
    }
};

int64_t next_sequence() {
    static int64_t sequence = 0;
    return ++sequence;
}

// One turn of a polling loop.
inline void pause() {
#if defined(__x86_64__)
    __builtin_ia32_pause();
#elif defined(__aarch64__)
    asm volatile("yield" ::: "memory");
#endif
}

// A word that a kernel stores; what it stored before (with a fence in between) may be read behind this.
inline int64_t load_word(volatile int64_t *word) { return __atomic_load_n(const_cast<int64_t *>(word), __ATOMIC_ACQUIRE); }

// Waits until *word == value; false when the stream has drained without that.
bool wait_for(volatile int64_t *word, int64_t value, c10::cuda::CUDAStream stream) {
    for (uint32_t i = 0;; ++i) {
        if (load_word(word) == value) return true;
        if ((i & 4095u) == 4095u && stream.query()) return load_word(word) == value;
        pause();
    }
}

void release() {
    workspaces.clear();
    free_slots.clear();
    still.clear();
}

// Motion of a sensor that stands still. Per stream, like the workspaces: what replaces a smaller one, or a release,
// gives the memory back to the stream whose kernels read it.
Tensor zero_motion(int64_t C, const at::TensorOptions &options, c10::cuda::CUDAStream stream) {
    Tensor &t = still[{stream.device_index(), stream.stream()}];
    if (!t.defined() || t.numel() < 3 * C) t = at::zeros({std::max<int64_t>(3 * C, 64)}, options);
    return t;
}

// The opacities as a projection node keeps them: not at all unless a compensation's gradient needs their values, and
// where the ops multiply a copy of them, a copy - what may be edited in place behind the ops may be here.
Tensor kept_opacities(const Tensor &opacities, const Tensor &comps, bool copied) {
    return !comps.defined() ? Tensor() : copied ? opacities.detach().clone() : opacities;
}

// What came of the lists: the caller keeps the counts and decides whether the frame stands.
struct Counts {
    int64_t n_isects = 0, status = 0, depth_range = 0, listed = 0;
    // list entries per listed element, 0: not known
    float spread() const { return listed > 0 ? (float)n_isects / (float)listed : 0.f; }
};

Counts read_counts(const Slot &slot, int64_t sequence, c10::cuda::CUDAStream stream) {
    Counts c;
    if (wait_for(slot.word + 5, sequence, stream)) {
        c.n_isects = slot.word[4];
        c.status = slot.word[6];
        c.depth_range = slot.word[7];
        c.listed = slot.word[9];
    } else {
        TORCH_CHECK(false, "the frame has ended without reporting its intersection count");
    }
    return c;
}

bool usable(const Counts &c, int64_t capacity) {
    return !(c.status & 6) && c.n_isects <= 0x7fffffff && c.n_isects <= capacity;
}

// One-shot requests of this thread's next plan, disarmed again on every way out: the early count and, with
// the depth range of an earlier frame (word of the early count; 0: none), buckets that span it widened by a
// tenth on either side - the rectangle count then fills them and one kernel less is launched.
struct PlanRequests {
    PlanRequests(const Slot &slot, int64_t sequence, uint64_t last_range, bool listed) {
        if (last_range != 0) {
            const uint32_t bits[2] = {(uint32_t)last_range, (uint32_t)(last_range >> 32)};
            float lo, hi;
            memcpy(&lo, bits, 4);
            memcpy(&hi, bits + 1, 4);
            if (0.f <= lo && lo <= hi && hi < 3.0e38f) {
                const float pad = 0.1f * (hi - lo) + 1e-3f;
                lo = std::max(lo - pad, 0.f);
                hi += pad;
                uint32_t wide[2];
                memcpy(wide, &lo, 4);
                memcpy(wide + 1, &hi, 4);
                lib.splatad_isect_set_depth_range_hint(wide[0], wide[1]);
            }
        }
        slot.word[9] = 0;
        lib.splatad_isect_set_early_count(const_cast<int64_t *>(slot.word) + 4, sequence);
        if (listed) lib.splatad_isect_set_listed_count(const_cast<int64_t *>(slot.word) + 9);
    }
    ~PlanRequests() {
        lib.splatad_isect_set_early_count(nullptr, 0);
        lib.splatad_isect_set_listed_count(nullptr);
        lib.splatad_isect_set_depth_range_hint(1, 0);
    }
};

void set_absgrad(const Tensor &means2d, const Tensor &v_abs) {
    py::gil_scoped_acquire gil;
    py::cast(means2d).attr("absgrad") = py::cast(v_abs);
}

template <typename T>
c10::intrusive_ptr<T> state_of(AutogradContext *ctx) {
    return c10::static_intrusive_pointer_cast<T>(ctx->saved_data["state"].toCapsule());
}

template <typename T>
void keep_state(AutogradContext *ctx, const c10::intrusive_ptr<T> &s) {
    ctx->saved_data["state"] = c10::IValue::make_capsule(s);
}

// ---------------------------------------------------------------------------------------------
// Lidar
// ---------------------------------------------------------------------------------------------
struct LidarFrame : torch::CustomClassHolder {
    int64_t C = 0, N = 0, W = 0, H = 0, rows = 0, cols = 0, D = 0, n_isects = 0;
    uint32_t tile_w = 0, tile_h = 0;
    float eps2d = 0.f, threshold = 0.f;
    bool alpha_sum_wanted = false, absgrad = false;
    // per (sensor, Gaussian)
    Tensor radii, means2d, depths, conics, comps, pix_vels, depth_comps, opacities, tiles_per_gauss;
    Tensor isect_ids, flatten_ids, offsets;   // offsets: the total behind the last tile
    Tensor render, alphas, alpha_sum, last_ids, median;
};

struct LidarProjectionNode : torch::autograd::Function<LidarProjectionNode> {
    static variable_list forward(AutogradContext *ctx, const Tensor &means, const Tensor &quats, const Tensor &scales,
                                 const Tensor &opacities, const OptTensor &velocities, const Tensor &viewmats, const Tensor &lin,
                                 const Tensor &ang, const Tensor &rs, c10::intrusive_ptr<LidarFrame> f) {
        ctx->save_for_backward({means, quats, scales, kept_opacities(opacities, f->comps, f->C > 1), velocities.value_or(Tensor()), viewmats, lin,
                                ang, rs, f->conics, f->comps, f->radii});
        auto kept = c10::make_intrusive<LidarFrame>();   // sizes only: the outputs must not hold themselves
        kept->C = f->C; kept->N = f->N; kept->eps2d = f->eps2d;
        keep_state(ctx, kept);
        ctx->set_materialize_grads(false);
        variable_list out{f->means2d, f->depths, f->conics, f->pix_vels, f->depth_comps};
        if (f->opacities.defined()) out.push_back(f->opacities);
        return out;
    }

    static variable_list backward(AutogradContext *ctx, variable_list g) {
        const auto saved = ctx->get_saved_variables();
        const Tensor &means = saved[0], &quats = saved[1], &scales = saved[2], &opacities = saved[3], &velocities = saved[4];
        const Tensor &conics = saved[9], &comps = saved[10], &radii = saved[11];
        const auto f = state_of<LidarFrame>(ctx);
        const c10::cuda::CUDAGuard guard(means.device());
        const auto stream = c10::cuda::getCurrentCUDAStream().stream();
        const auto options = means.options().requires_grad(false);
        const int64_t C = f->C, N = f->N, n = C * N;
        const Tensor v_means2d = g[0].defined() ? cotangent(g[0], g[0]) : at::zeros({C, N, 2}, options);
        const Tensor v_depths = g[1].defined() ? cotangent(g[1], g[1]) : at::zeros({C, N}, options);
        const Tensor v_conics = cotangent(g[2], conics);
        const Tensor v_pix_vels = g[3].defined() ? cotangent(g[3], g[3]) : at::zeros({C, N, 3}, options);
        const Tensor v_dc = g[4].defined() ? cotangent(g[4], g[4]) : at::zeros({C, N, 2}, options);
        Tensor v_opacities, v_comps;
        if (g.size() > 5 && g[5].defined()) {
            const Tensor v_rows = cotangent(g[5], g[5]);
            v_opacities = at::zeros({N}, options);
            if (comps.defined()) v_comps = at::empty({C, N}, options);
            check(lib.splatad_opacity_rows_bwd((uint32_t)n, (uint32_t)N, nullptr, F(opacities), F(comps), F(v_rows),
                                               M(v_opacities), M(v_comps), stream));
        } else if (comps.defined()) {
            v_comps = at::zeros({C, N}, options);
        }
        Tensor v_means = at::empty_like(means), v_quats = at::empty_like(quats), v_scales = at::empty_like(scales);
        check(lib.splatad_lidar_projection_bwd(
            (uint32_t)C, (uint32_t)N, F(means), nullptr, F(quats), F(scales), F(velocities), F(saved[5]), F(saved[6]), F(saved[7]),
            F(saved[8]), f->eps2d, F(radii), F(conics), F(comps), F(v_means2d), F(v_depths), F(v_conics), F(v_comps),
            F(v_pix_vels), F(v_dc), M(v_means), nullptr, M(v_quats), M(v_scales), nullptr, nullptr, stream));
        variable_list out(10);
        if (ctx->needs_input_grad(0)) out[0] = std::move(v_means);
        if (ctx->needs_input_grad(1)) out[1] = std::move(v_quats);
        if (ctx->needs_input_grad(2)) out[2] = std::move(v_scales);
        if (ctx->needs_input_grad(3)) out[3] = std::move(v_opacities);
        return out;
    }
};

struct LidarCompositeNode : torch::autograd::Function<LidarCompositeNode> {
    static variable_list forward(AutogradContext *ctx, const Tensor &means2d, const Tensor &conics, const Tensor &features,
                                 const Tensor &depths, const Tensor &opacities, const Tensor &pix_vels, const Tensor &depth_comps,
                                 const Tensor &raster_pts, c10::intrusive_ptr<LidarFrame> f) {
        ctx->save_for_backward({means2d, conics, features, depths, opacities, pix_vels, depth_comps, raster_pts, f->alphas,
                                f->last_ids, f->offsets, f->flatten_ids});
        auto kept = c10::make_intrusive<LidarFrame>();
        kept->C = f->C; kept->W = f->W; kept->H = f->H; kept->rows = f->rows; kept->cols = f->cols; kept->D = f->D;
        kept->n_isects = f->n_isects;
        kept->tile_w = f->tile_w; kept->tile_h = f->tile_h; kept->threshold = f->threshold;
        kept->alpha_sum_wanted = f->alpha_sum_wanted; kept->absgrad = f->absgrad;
        keep_state(ctx, kept);
        ctx->set_materialize_grads(false);
        variable_list out{f->render, f->alphas};
        if (f->alpha_sum.defined()) out.push_back(f->alpha_sum);
        return out;
    }

    static variable_list backward(AutogradContext *ctx, variable_list g) {
        const auto saved = ctx->get_saved_variables();
        const Tensor &means2d = saved[0], &conics = saved[1], &features = saved[2], &depths = saved[3], &opacities = saved[4],
                     &pix_vels = saved[5], &depth_comps = saved[6], &alphas = saved[8];
        const auto f = state_of<LidarFrame>(ctx);
        const c10::cuda::CUDAGuard guard(means2d.device());
        const auto options = means2d.options().requires_grad(false);
        const Tensor v_render = g[0].defined() ? cotangent(g[0], g[0]) : at::zeros({f->C, f->H, f->W, f->D + 1}, options);
        const Tensor v_alphas = cotangent(g[1], alphas);
        Tensor v_sum;
        if (f->alpha_sum_wanted && g.size() > 2 && g[2].defined()) v_sum = cotangent(g[2], g[2]);
        Tensor v_means2d, v_conics, v_features, v_opacities, v_pix_vels, v_dc, v_depths, v_abs;
        Zeros zeros;
        zeros.add(v_means2d, means2d.sizes());
        zeros.add(v_conics, conics.sizes());
        zeros.add(v_features, features.sizes());
        zeros.add(v_opacities, opacities.sizes());
        zeros.add(v_pix_vels, pix_vels.sizes());
        zeros.add(v_dc, depth_comps.sizes());
        zeros.add(v_depths, depths.sizes());
        if (f->absgrad) zeros.add(v_abs, means2d.sizes());
        zeros.make(options);
        check(lib.splatad_rasterize_to_points_bwd(
            (uint32_t)f->C, f->n_isects, F(means2d), F(conics), F(features), F(depths), (uint32_t)(f->D + 1), F(opacities), F(pix_vels),
            F(depth_comps), nullptr, F(saved[7]), (uint32_t)f->W, (uint32_t)f->H, f->tile_w, f->tile_h, (uint32_t)f->cols,
            (uint32_t)f->rows, f->alpha_sum_wanted, f->threshold, I(saved[10]), I(saved[11]), (uint32_t)f->D, F(alphas), I(saved[9]),
            F(v_render), F(v_alphas), F(v_sum), M(v_abs), M(v_means2d), M(v_conics), M(v_features), M(v_opacities), M(v_pix_vels),
            M(v_dc), M(v_depths), c10::cuda::getCurrentCUDAStream().stream()));
        if (f->absgrad) set_absgrad(means2d, v_abs);
        variable_list out(9);
        out[0] = std::move(v_means2d); out[1] = std::move(v_conics); out[2] = std::move(v_features); out[3] = std::move(v_depths);
        out[4] = std::move(v_opacities); out[5] = std::move(v_pix_vels); out[6] = std::move(v_dc);
        return out;
    }
};

// Returns None when the arguments are not this function's to take, else (counts..., outputs or None).
py::object lidar_frame(const Tensor &means, const Tensor &quats, const Tensor &scales, const Tensor &opacities,
                       const Tensor &features, const OptTensor &velocities, const Tensor &viewmats, const Tensor &raster_pts,
                       const Tensor &boundaries, const OptTensor &lin, const OptTensor &ang, const OptTensor &rs, double min_az,
                       double max_az, double min_el, double max_el, double az_res, int64_t tile_w, int64_t tile_h, double near_plane,
                       double far_plane, double radius_clip, double eps2d, bool alpha_sum, double threshold, bool absgrad,
                       bool antialiased, int64_t rows, int64_t cols, int64_t capacity, uint64_t last_range) {
    if (!means.defined() || !means.is_cuda()) return py::none();
    const c10::DeviceIndex dev = means.get_device();
    for (const Tensor *t : {&means, &quats, &scales, &opacities, &features, &viewmats, &raster_pts, &boundaries})
        if (!plain(*t, dev)) return py::none();
    for (const OptTensor *t : {&velocities, &lin, &ang, &rs})
        if (!plain(*t, dev)) return py::none();
    if (means.dim() != 2 || viewmats.dim() != 3 || features.dim() != 3 || raster_pts.dim() != 4) return py::none();
    const int64_t N = means.size(0), C = viewmats.size(0), D = features.size(2), H = raster_pts.size(1), W = raster_pts.size(2);
    if (!shaped(means, {N, 3}) || !shaped(quats, {N, 4}) || !shaped(scales, {N, 3}) || !shaped(opacities, {N}) ||
        !shaped(features, {C, N, D}) || !shaped(velocities, {N, 3}) || !shaped(viewmats, {C, 4, 4}) ||
        !shaped(raster_pts, {C, H, W, 4}) || !shaped(boundaries, {rows + 1}) || !shaped(lin, {C, 3}) || !shaped(ang, {C, 3}) ||
        !shaped(rs, {C}) || C * N == 0 || C * N > 0x7fffffff || H * W == 0 || D == 0 || D + 1 > SPLATAD_MAX_CHANNELS)
        return py::none();
    if ((int64_t)lib.splatad_lidar_azimuth_tiles((float)(az_res * (double)tile_w)) != cols || cols * tile_w < W || rows * tile_h < H)
        return py::none();
    const bool grad = wants_grad({&means, &quats, &scales, &opacities, &features, &raster_pts}, {&velocities, &lin, &ang, &rs});

    const c10::cuda::CUDAGuard guard(dev);
    const auto stream = c10::cuda::getCurrentCUDAStream();
    const auto options = at::TensorOptions().dtype(at::kFloat).device(at::kCUDA, dev);
    const auto ints = options.dtype(at::kInt);
    auto f = c10::make_intrusive<LidarFrame>();
    Counts counts;
    const Tensor zeros = zero_motion(C, options, stream);
    const Tensor lin_t = lin ? *lin : alias(zeros, {C, 3}), ang_t = ang ? *ang : alias(zeros, {C, 3}), rs_t = rs ? *rs : alias(zeros, {C});
    {
        const at::NoGradGuard no_grad;
        f->C = C; f->N = N; f->W = W; f->H = H; f->rows = rows; f->cols = cols; f->D = D;
        f->tile_w = (uint32_t)tile_w; f->tile_h = (uint32_t)tile_h; f->eps2d = (float)eps2d; f->threshold = (float)threshold;
        f->alpha_sum_wanted = alpha_sum; f->absgrad = absgrad;
        f->radii = at::empty({C, N, 2}, options);
        f->means2d = at::empty({C, N, 2}, options);
        f->depths = at::empty({C, N}, options);
        f->conics = at::empty({C, N, 3}, options);
        if (antialiased) f->comps = at::empty({C, N}, options);
        f->pix_vels = at::empty({C, N, 3}, options);
        f->depth_comps = at::empty({C, N, 2}, options);
        f->tiles_per_gauss = at::empty({C, N}, ints);
        f->isect_ids = at::empty({capacity}, options.dtype(at::kLong));
        f->flatten_ids = at::empty({capacity}, ints);
        f->offsets = at::empty({C * rows * cols + 1}, ints);
        f->render = at::empty({C, H, W, D + 1}, options);
        f->alphas = at::empty({C, H, W, 1}, options);
        if (alpha_sum) f->alpha_sum = at::empty({C, H, W, 1}, options);
        f->last_ids = at::empty({C, H, W}, ints);
        f->median = at::empty({C, H, W, 1}, options);
        if (C > 1 || antialiased) f->opacities = at::empty({C, N}, options);
        const Tensor plan_ws = workspace("isect_plan", lib.splatad_isect_plan_workspace_bytes((uint64_t)(C * N)), stream);
        const Tensor fill_ws = workspace("isect_fill", lib.splatad_isect_fill_workspace_bytes((uint64_t)capacity), stream);
        Slot slot(stream);
        const int64_t sequence = next_sequence();
        const PlanRequests requests(slot, sequence, last_range, false);   // (asking costs the host a call)
        const auto opacity_rows = [&]() -> const float * {
            if (!f->opacities.defined()) return F(opacities);
            check(lib.splatad_opacity_rows_fwd((uint32_t)(C * N), (uint32_t)N, nullptr, F(opacities), F(f->comps), M(f->opacities),
                                               stream.stream()));
            return F(f->opacities);
        };
        int64_t *words = const_cast<int64_t *>(slot.word);
        if (!antialiased) {
            check(lib.splatad_lidar_frame_fwd(
                (uint32_t)C, (uint32_t)N, F(means), F(quats), F(scales), F(velocities), opacity_rows(), F(features), (uint32_t)D, F(viewmats),
                F(lin_t), F(ang_t), F(rs_t), F(raster_pts), (uint32_t)W, (uint32_t)H, F(boundaries), (uint32_t)(rows + 1), (float)az_res,
                f->tile_w, f->tile_h, (float)min_az, (float)max_az, (float)min_el, (float)max_el, (float)eps2d, (float)near_plane,
                (float)far_plane, (float)radius_clip, alpha_sum, (float)threshold, M(f->radii), M(f->means2d), M(f->depths), M(f->conics),
                M(f->pix_vels), M(f->depth_comps), I(f->tiles_per_gauss), capacity, L(f->isect_ids), I(f->flatten_ids), I(f->offsets),
                M(f->render), M(f->alphas), M(f->alpha_sum), I(f->last_ids), M(f->median), plan_ws.data_ptr(), (size_t)plan_ws.numel(),
                fill_ws.data_ptr(), (size_t)fill_ws.numel(), nullptr, words + 4, sequence, stream.stream()));
        } else {
            // the compensated opacities come between projection and compositing
            check(lib.splatad_lidar_projection_fwd(
                (uint32_t)C, (uint32_t)N, F(means), nullptr, F(quats), F(scales), F(velocities), F(viewmats), (float)min_el, (float)max_el,
                (float)min_az, (float)max_az, F(lin_t), F(ang_t), F(rs_t), (float)eps2d, (float)near_plane, (float)far_plane,
                (float)radius_clip, M(f->radii), M(f->means2d), M(f->depths), M(f->conics), M(f->comps), M(f->pix_vels),
                M(f->depth_comps), stream.stream()));
            const float *opacity = opacity_rows();
            const auto grid = [&](auto fn, auto... tail) {
                return fn((uint32_t)C, (uint32_t)N, (uint64_t)(C * N), F(f->means2d), F(f->radii), F(f->depths), nullptr, F(boundaries),
                          (uint32_t)(rows + 1), (float)(az_res * (double)tile_w), (float)min_az, 1, I(f->tiles_per_gauss), tail...);
            };
            check(grid(lib.splatad_isect_lidar_tiles_plan, plan_ws.data_ptr(), (size_t)plan_ws.numel(), (int64_t *)nullptr, stream.stream()));
            check(grid(lib.splatad_isect_lidar_tiles_fill, plan_ws.data_ptr(), fill_ws.data_ptr(), (size_t)fill_ws.numel(), capacity,
                       L(f->isect_ids), I(f->flatten_ids), I(f->offsets), (int64_t *)nullptr, stream.stream()));
            lib.splatad_rasterize_set_rows_hint((uint64_t)(C * N));
            check(lib.splatad_rasterize_to_points_fwd(
                (uint32_t)C, -1, F(f->means2d), F(f->conics), F(features), F(f->depths), (uint32_t)(D + 1), opacity, F(f->pix_vels),
                F(f->depth_comps), nullptr, F(raster_pts), (uint32_t)W, (uint32_t)H, f->tile_w, f->tile_h, (uint32_t)cols, (uint32_t)rows,
                alpha_sum, (float)threshold, I(f->offsets), I(f->flatten_ids), (uint32_t)D, M(f->render), M(f->alphas),
                M(f->alpha_sum), I(f->last_ids), M(f->median), stream.stream()));
        }
        py::gil_scoped_release no_gil;
        counts = read_counts(slot, sequence, stream);
    }
    if (!usable(counts, capacity)) return py::make_tuple(counts.n_isects, counts.status, counts.depth_range, py::none());
    f->n_isects = counts.n_isects;   // none: the lists are null pointers, which the backward pass must not ask for
    f->isect_ids = head(f->isect_ids, counts.n_isects);
    f->flatten_ids = head(f->flatten_ids, counts.n_isects);
    Tensor opacities_cn = f->opacities.defined() ? f->opacities : opacities.unsqueeze(0);
    if (grad) {
        const auto p = LidarProjectionNode::apply(means, quats, scales, opacities, velocities, viewmats, lin_t,
                                                  ang_t, rs_t, f);
        f->means2d = p[0]; f->depths = p[1]; f->conics = p[2]; f->pix_vels = p[3]; f->depth_comps = p[4];
        if (p.size() > 5) opacities_cn = p[5];
        const auto c = LidarCompositeNode::apply(p[0], p[2], features, p[1], opacities_cn, p[3], p[4], raster_pts, f);
        f->render = c[0]; f->alphas = c[1];
        if (alpha_sum) f->alpha_sum = c[2];
    }
    return py::make_tuple(
        counts.n_isects, counts.status, counts.depth_range,
        py::make_tuple(f->render, f->alphas, alpha_sum ? py::cast(f->alpha_sum) : py::none(), f->median, f->radii, f->means2d, f->depths,
                       f->conics, opacities_cn, f->pix_vels, f->tiles_per_gauss, f->isect_ids, f->flatten_ids,
                       alias(f->offsets, {C, rows, cols})));
}

// ---------------------------------------------------------------------------------------------
// Cameras
// ---------------------------------------------------------------------------------------------
struct CameraFrame : torch::CustomClassHolder {
    int64_t C = 0, N = 0, n = 0, W = 0, H = 0, tile_size = 0, tile_w = 0, tile_h = 0, channels = 0, n_isects = 0;
    std::vector<int64_t> color_sizes;
    int64_t K = 0, D = 0, sh_degree = -1;     // spherical harmonics (K coefficients) or D plain channels
    bool packed = false, per_camera = false, depth = false, expected = false, absgrad = false;
    float eps2d = 0.f, spread = 0.f, near = 0.f;   // spread, near: tiles that a listed or near Gaussian covers on the average, 0: not known
    Tensor camera_ids, gaussian_ids, radii, means2d, depths, conics, comps, pix_vels, tiles_per_gauss, campos;
    Tensor opacities, colors;                 // rows made for this frame (undefined: the parameters serve as they are)
    Tensor isect_ids, flatten_ids, offsets, render, alphas, last_ids;
    Tensor expected_depths;                   // kept for the backward pass: the render is the user's to edit
    c10::intrusive_ptr<CameraFrame> sizes() const {
        auto k = c10::make_intrusive<CameraFrame>();
        k->C = C; k->N = N; k->n = n; k->W = W; k->H = H; k->tile_size = tile_size; k->tile_w = tile_w; k->tile_h = tile_h;
        k->channels = channels; k->K = K; k->D = D; k->sh_degree = sh_degree; k->packed = packed; k->per_camera = per_camera;
        k->depth = depth; k->expected = expected; k->absgrad = absgrad; k->eps2d = eps2d; k->n_isects = n_isects;
        k->spread = spread; k->near = near;
        k->color_sizes = color_sizes;
        return k;
    }
};

struct CameraProjectionNode : torch::autograd::Function<CameraProjectionNode> {
    static variable_list forward(AutogradContext *ctx, const Tensor &means, const Tensor &quats, const Tensor &scales,
                                 const Tensor &opacities, const OptTensor &colors, const OptTensor &velocities, const Tensor &viewmats,
                                 const Tensor &Ks, const Tensor &lin, const Tensor &ang, const Tensor &rs,
                                 c10::intrusive_ptr<CameraFrame> f) {
        ctx->save_for_backward({means, quats, scales, kept_opacities(opacities, f->comps, f->packed || f->C > 1),
                                f->sh_degree >= 0 ? colors.value_or(Tensor()) : Tensor(), velocities.value_or(Tensor()), viewmats, Ks, lin,
                                ang, rs, f->conics, f->comps, f->radii, f->camera_ids, f->gaussian_ids, f->campos});
        if (colors) f->color_sizes = colors->sizes().vec();
        keep_state(ctx, f->sizes());
        ctx->set_materialize_grads(false);
        variable_list out{f->means2d, f->depths, f->conics, f->pix_vels};
        if (f->opacities.defined()) out.push_back(f->opacities);
        if (f->colors.defined()) out.push_back(f->colors);
        ctx->saved_data["opacities"] = f->opacities.defined();
        return out;
    }

    static variable_list backward(AutogradContext *ctx, variable_list g) {
        const auto saved = ctx->get_saved_variables();
        const Tensor &means = saved[0], &quats = saved[1], &scales = saved[2], &opacities = saved[3], &colors = saved[4];
        const Tensor &conics = saved[11], &comps = saved[12], &radii = saved[13], &camera_ids = saved[14], &gaussian_ids = saved[15];
        const auto f = state_of<CameraFrame>(ctx);
        const c10::cuda::CUDAGuard guard(means.device());
        const auto stream = c10::cuda::getCurrentCUDAStream().stream();
        const auto options = means.options().requires_grad(false);
        const uint32_t C = (uint32_t)f->C, N = (uint32_t)f->N, n = (uint32_t)f->n;
        const bool packed = f->packed, rows_o = ctx->saved_data["opacities"].toBool();
        const auto zeros_of = [&](int64_t per_row) {
            std::vector<int64_t> s = packed ? std::vector<int64_t>{f->n} : std::vector<int64_t>{f->C, f->N};
            if (per_row) s.push_back(per_row);
            return at::zeros(s, options);
        };
        const Tensor v_means2d = g[0].defined() ? cotangent(g[0], g[0]) : zeros_of(2);
        Tensor v_depths = g[1].defined() ? cotangent(g[1], g[1]) : Tensor();
        const Tensor v_conics = cotangent(g[2], conics);
        const Tensor v_pix_vels = g[3].defined() ? cotangent(g[3], g[3]) : zeros_of(2);
        const Tensor v_rows_o = rows_o && g[4].defined() ? cotangent(g[4], g[4]) : Tensor();
        const size_t at_colors = rows_o ? 5 : 4;
        const Tensor v_rows_c = g.size() > at_colors && g[at_colors].defined() ? cotangent(g[at_colors], g[at_colors]) : Tensor();

        // accumulated with atomics: opacities and colours always, the geometry in the packed layout
        Tensor v_means, v_quats, v_scales, v_opacities, v_colors, v_comps;
        Zeros zeros;
        if (packed) {
            zeros.add(v_means, means.sizes());
            zeros.add(v_quats, quats.sizes());
            zeros.add(v_scales, scales.sizes());
        }
        if (v_rows_o.defined()) zeros.add(v_opacities, {f->N});
        if (v_rows_c.defined() && ctx->needs_input_grad(4)) zeros.add(v_colors, f->color_sizes);
        zeros.make(options);
        if (comps.defined()) v_comps = v_rows_o.defined() ? at::empty_like(comps) : at::zeros_like(comps);
        if (v_rows_o.defined())
            check(lib.splatad_opacity_rows_bwd(n, N, L(gaussian_ids), F(opacities), F(comps), F(v_rows_o), M(v_opacities), M(v_comps),
                                               stream));
        const bool sh = f->sh_degree >= 0;
        if (v_rows_c.defined()) {
            Tensor v_total;
            if (f->depth) v_total = at::empty_like(radii.select(-1, 0), options);
            check(lib.splatad_color_rows_bwd(n, N, sh ? 0u : (uint32_t)f->D, (uint32_t)f->channels, L(camera_ids), L(gaussian_ids),
                                             f->per_camera, F(v_rows_c), sh ? nullptr : M(v_colors), F(v_depths), M(v_total), stream));
            if (f->depth) v_depths = v_total;
        }
        if (!v_depths.defined()) v_depths = zeros_of(0);
        if (packed) {
            check(lib.splatad_projection_packed_bwd(
                C, N, n, F(means), nullptr, F(quats), F(scales), F(saved[5]), F(saved[6]), F(saved[7]), (int32_t)f->W, (int32_t)f->H,
                F(saved[8]), F(saved[9]), F(saved[10]), f->eps2d, L(camera_ids), L(gaussian_ids), F(conics), F(comps), F(v_means2d),
                F(v_depths), F(v_conics), F(v_comps), F(v_pix_vels), 0, M(v_means), nullptr, M(v_quats), M(v_scales), nullptr, nullptr,
                stream));
        } else {
            v_means = at::empty_like(means); v_quats = at::empty_like(quats); v_scales = at::empty_like(scales);
            check(lib.splatad_projection_bwd(
                C, N, F(means), nullptr, F(quats), F(scales), F(saved[5]), F(saved[6]), F(saved[7]), (int32_t)f->W, (int32_t)f->H,
                F(saved[8]), F(saved[9]), F(saved[10]), f->eps2d, I(radii), F(conics), F(comps), F(v_means2d), F(v_depths), F(v_conics),
                F(v_comps), F(v_pix_vels), M(v_means), nullptr, M(v_quats), M(v_scales), nullptr, nullptr, stream));
        }
        if (sh && v_rows_c.defined())   // adds the view dependence to the gradient of the means
            check(lib.splatad_sh_colors_bwd(n, N, (uint32_t)f->K, (uint32_t)f->sh_degree, F(means), F(saved[16]), F(colors), f->per_camera,
                                            L(camera_ids), L(gaussian_ids), I(radii), (uint32_t)f->channels, F(v_rows_c), M(v_colors),
                                            M(v_means), nullptr, nullptr, stream));
        variable_list out(12);
        if (ctx->needs_input_grad(0)) out[0] = std::move(v_means);
        if (ctx->needs_input_grad(1)) out[1] = std::move(v_quats);
        if (ctx->needs_input_grad(2)) out[2] = std::move(v_scales);
        if (ctx->needs_input_grad(3)) out[3] = std::move(v_opacities);
        if (ctx->needs_input_grad(4)) out[4] = std::move(v_colors);
        return out;
    }
};

struct CameraCompositeNode : torch::autograd::Function<CameraCompositeNode> {
    static variable_list forward(AutogradContext *ctx, const Tensor &means2d, const Tensor &conics, const Tensor &colors,
                                 const Tensor &opacities, const Tensor &pix_vels, const Tensor &rs, const OptTensor &backgrounds,
                                 c10::intrusive_ptr<CameraFrame> f) {
        ctx->save_for_backward({means2d, conics, colors, opacities, pix_vels, rs, backgrounds.value_or(Tensor()), f->alphas, f->last_ids, f->offsets,
                                f->flatten_ids, f->expected_depths});
        keep_state(ctx, f->sizes());
        ctx->set_materialize_grads(false);
        return {f->render, f->alphas};
    }

    static variable_list backward(AutogradContext *ctx, variable_list g) {
        const auto saved = ctx->get_saved_variables();
        const Tensor &means2d = saved[0], &conics = saved[1], &colors = saved[2], &opacities = saved[3], &pix_vels = saved[4];
        const auto f = state_of<CameraFrame>(ctx);
        const c10::cuda::CUDAGuard guard(means2d.device());
        const auto options = means2d.options().requires_grad(false);
        const Tensor v_render = g[0].defined() ? cotangent(g[0], g[0]) : at::zeros({f->C, f->H, f->W, f->channels}, options);
        const Tensor v_alphas = cotangent(g[1], saved[7]);
        Tensor v_means2d, v_conics, v_colors, v_opacities, v_pix_vels, v_abs;
        Zeros zeros;
        zeros.add(v_means2d, means2d.sizes());
        zeros.add(v_conics, conics.sizes());
        zeros.add(v_colors, colors.sizes());
        zeros.add(v_opacities, opacities.sizes());
        zeros.add(v_pix_vels, pix_vels.sizes());
        if (f->absgrad) zeros.add(v_abs, means2d.sizes());
        zeros.make(options);
        lib.splatad_rasterize_set_spread_hint(f->spread, f->n_isects);
        lib.splatad_rasterize_set_near_hint(f->near);
        check(lib.splatad_rasterize_expected_to_pixels_bwd(
            (uint32_t)f->C, f->n_isects, F(means2d), F(conics), F(colors), (uint32_t)f->channels, F(opacities), F(pix_vels), F(saved[5]),
            F(saved[6]), (uint32_t)f->W, (uint32_t)f->H, (uint32_t)f->tile_size, (uint32_t)f->tile_w, (uint32_t)f->tile_h, I(saved[9]),
            I(saved[10]), F(saved[11]), F(saved[7]), I(saved[8]), F(v_render), F(v_alphas), M(v_abs), M(v_means2d), M(v_conics),
            M(v_colors), M(v_opacities), M(v_pix_vels), c10::cuda::getCurrentCUDAStream().stream()));
        if (f->absgrad) set_absgrad(means2d, v_abs);
        variable_list out(8);
        out[0] = std::move(v_means2d); out[1] = std::move(v_conics); out[2] = std::move(v_colors); out[3] = std::move(v_opacities);
        out[4] = std::move(v_pix_vels);
        return out;
    }
};

// mode: 0 colours, 1 colours and depth, 2 depth alone. Returns None when the arguments are not this
// function's to take, else (packed rows, counts..., outputs or None).
py::object camera_frame(const Tensor &means, const Tensor &quats, const Tensor &scales, const Tensor &opacities, const Tensor &colors,
                        const OptTensor &velocities, const Tensor &viewmats, const Tensor &Ks, int64_t W, int64_t H,
                        const OptTensor &lin, const OptTensor &ang, const OptTensor &rs, double near_plane, double far_plane,
                        double radius_clip, double eps2d, int64_t sh_degree, bool packed, int64_t tile_size, const OptTensor &backgrounds,
                        int64_t mode, bool expected, bool absgrad, bool antialiased, int64_t max_channels, int64_t row_capacity,
                        int64_t capacity, uint64_t last_range) {
    if (!means.defined() || !means.is_cuda()) return py::none();
    const c10::DeviceIndex dev = means.get_device();
    for (const Tensor *t : {&means, &quats, &scales, &opacities, &colors, &viewmats, &Ks})
        if (!plain(*t, dev)) return py::none();
    for (const OptTensor *t : {&velocities, &lin, &ang, &rs, &backgrounds})
        if (!plain(*t, dev)) return py::none();
    if (means.dim() != 2 || viewmats.dim() != 3 || (backgrounds && backgrounds->requires_grad())) return py::none();
    const int64_t N = means.size(0), C = viewmats.size(0), rows_max = packed ? row_capacity : C * N;
    const bool sh = sh_degree >= 0, per_camera = colors.dim() == (sh ? 4 : 3);
    if (!shaped(means, {N, 3}) || !shaped(quats, {N, 4}) || !shaped(scales, {N, 3}) || !shaped(opacities, {N}) ||
        !shaped(velocities, {N, 3}) || !shaped(viewmats, {C, 4, 4}) || !shaped(Ks, {C, 3, 3}) || !shaped(lin, {C, 3}) ||
        !shaped(ang, {C, 3}) || !shaped(rs, {C}) || C * N == 0 || C * N > 0x7fffffff || W <= 0 || H <= 0 || tile_size <= 0 ||
        tile_size > 32 || rows_max <= 0)
        return py::none();
    const auto cs = colors.sizes();
    if (sh) {
        if (colors.dim() != 3 + per_camera || cs.back() != 3 || (sh_degree + 1) * (sh_degree + 1) > cs[cs.size() - 2]) return py::none();
    } else if (colors.dim() != 2 + per_camera || cs.back() == 0) {
        return py::none();
    }
    if (per_camera ? (cs[0] != C || cs[1] != N) : cs[0] != N) return py::none();
    const int64_t D = sh ? 3 : cs.back(), channels = mode == 2 ? 1 : D + mode;
    if (channels > max_channels || channels > SPLATAD_MAX_CHANNELS) return py::none();
    if (backgrounds && mode != 2 && !shaped(backgrounds, {C, D})) return py::none();
    if (tile_size * tile_size > 512 && channels > 16) return py::none();   // the backward pass would refuse it
    const bool grad = wants_grad({&means, &quats, &scales, &opacities, &Ks, mode == 2 ? &means : &colors}, {&velocities, &lin, &ang, &rs});

    const c10::cuda::CUDAGuard guard(dev);
    const auto stream = c10::cuda::getCurrentCUDAStream();
    const auto options = at::TensorOptions().dtype(at::kFloat).device(at::kCUDA, dev);
    const auto ints = options.dtype(at::kInt), longs = options.dtype(at::kLong);
    const Tensor zeros = zero_motion(C, options, stream);
    const Tensor lin_t = lin ? *lin : alias(zeros, {C, 3}), ang_t = ang ? *ang : alias(zeros, {C, 3}), rs_t = rs ? *rs : alias(zeros, {C});
    auto f = c10::make_intrusive<CameraFrame>();
    const int64_t tile_w = (W + tile_size - 1) / tile_size, tile_h = (H + tile_size - 1) / tile_size;
    f->C = C; f->N = N; f->n = rows_max; f->W = W; f->H = H; f->tile_size = tile_size; f->tile_w = tile_w; f->tile_h = tile_h;
    f->channels = channels; f->K = sh ? cs[cs.size() - 2] : 0; f->D = D; f->sh_degree = sh_degree; f->packed = packed;
    f->per_camera = per_camera; f->depth = mode == 1; f->expected = expected; f->absgrad = absgrad; f->eps2d = (float)eps2d;
    Counts counts;
    int64_t nnz = rows_max;
    const bool opacity_rows = packed || C > 1 || antialiased;
    const bool color_rows = mode != 2 && (sh || packed || mode == 1 || (!per_camera && C > 1));
    Tensor bg = backgrounds && mode != 2 ? *backgrounds : Tensor();
    {
        const at::NoGradGuard no_grad;
        const auto row = [&](int64_t k) { return packed ? std::vector<int64_t>{rows_max, k} : std::vector<int64_t>{C, N, k}; };
        const auto flat = packed ? std::vector<int64_t>{rows_max} : std::vector<int64_t>{C, N};
        if (bg.defined() && mode == 1) bg = at::cat({bg, at::zeros({C, 1}, options)}, -1);
        f->radii = at::empty(row(2), ints);
        f->means2d = at::empty(row(2), options);
        f->depths = at::empty(flat, options);
        f->conics = at::empty(row(3), options);
        if (antialiased) f->comps = at::empty(flat, options);
        f->pix_vels = at::empty(row(2), options);
        Slot slot(stream);
        if (packed) {
            f->camera_ids = at::empty(flat, longs);
            f->gaussian_ids = at::empty(flat, longs);
            const size_t bytes = lib.splatad_projection_packed_workspace_bytes((uint32_t)C, (uint32_t)N);
            const Tensor ws = workspace("packed", bytes + 4 * (size_t)(C + 1), stream);
            const auto project = [&](auto fn, auto... tail) {
                return fn((uint32_t)C, (uint32_t)N, F(means), nullptr, F(quats), F(scales), F(velocities), F(viewmats), F(Ks), (int32_t)W,
                          (int32_t)H, F(lin_t), F(ang_t), F(rs_t), (float)eps2d, (float)near_plane, (float)far_plane, (float)radius_clip,
                          tail...);
            };
            slot.word[8] = -1;   // the scan stores the row count here, into host memory
            check(project(lib.splatad_projection_packed_count, ws.data_ptr(), (size_t)bytes,
                          reinterpret_cast<int32_t *>(static_cast<char *>(ws.data_ptr()) + bytes), const_cast<int64_t *>(slot.word) + 8,
                          stream.stream()));
            check(project(lib.splatad_projection_packed_fill, (const void *)ws.data_ptr(), rows_max, L(f->camera_ids), L(f->gaussian_ids),
                          I(f->radii), M(f->means2d), M(f->depths), M(f->conics), M(f->comps), M(f->pix_vels), stream.stream()));
        } else {
            check(lib.splatad_projection_fwd((uint32_t)C, (uint32_t)N, F(means), nullptr, F(quats), F(scales), F(velocities), F(viewmats),
                                             F(Ks), (int32_t)W, (int32_t)H, F(lin_t), F(ang_t), F(rs_t), (float)eps2d, (float)near_plane,
                                             (float)far_plane, (float)radius_clip, I(f->radii), M(f->means2d), M(f->depths),
                                             M(f->conics), M(f->comps), M(f->pix_vels), stream.stream()));
        }
        f->tiles_per_gauss = at::empty(flat, ints);
        f->isect_ids = at::empty({capacity}, longs);
        f->flatten_ids = at::empty({capacity}, ints);
        f->offsets = at::empty({C * tile_h * tile_w + 1}, ints);
        const Tensor plan_ws = workspace("isect_plan", lib.splatad_isect_plan_workspace_bytes((uint64_t)rows_max), stream);
        const Tensor fill_ws = workspace("isect_fill", lib.splatad_isect_fill_workspace_bytes((uint64_t)capacity), stream);
        const int64_t sequence = next_sequence();
        const auto grid = [&](auto fn, auto... tail) {
            return fn((uint32_t)C, packed ? 0u : (uint32_t)N, (uint64_t)rows_max, F(f->means2d), I(f->radii), F(f->depths), L(f->camera_ids),
                      (uint32_t)tile_size, (uint32_t)tile_w, (uint32_t)tile_h, 1, I(f->tiles_per_gauss), tail...);
        };
        {
            const PlanRequests requests(slot, sequence, last_range, true);
            check(grid(lib.splatad_isect_tiles_plan, plan_ws.data_ptr(), (size_t)plan_ws.numel(), (int64_t *)nullptr, stream.stream()));
        }
        // who may take runs: whole warps of eight pixels per lane, many tiles, forward up to four channels, backward up to sixteen
        const int64_t tiles_16 = C * tile_w * tile_h * tile_size * tile_size / 256;
        const bool ask_near = tile_size % 16 == 0 && ((tiles_16 >= 1800 && channels <= 4) || (grad && tiles_16 >= 900 && channels <= 16));
        slot.word[10] = 0;
        if (ask_near) lib.splatad_isect_set_near_tiles(const_cast<int64_t *>(slot.word) + 10, (uint32_t)sequence);
        check(grid(lib.splatad_isect_tiles_fill, plan_ws.data_ptr(), fill_ws.data_ptr(), (size_t)fill_ws.numel(), capacity,
                   L(f->isect_ids), I(f->flatten_ids), I(f->offsets), (int64_t *)nullptr, stream.stream()));
        const float *o = F(opacities), *c = mode == 2 ? F(f->depths) : F(colors);
        if (opacity_rows) {
            f->opacities = at::empty(flat, options);
            check(lib.splatad_opacity_rows_fwd((uint32_t)rows_max, (uint32_t)N, L(f->gaussian_ids), F(opacities), F(f->comps),
                                               M(f->opacities), stream.stream()));
            o = F(f->opacities);
        }
        if (color_rows) {
            f->colors = at::empty(row(channels), options);
            const float *depths = mode == 1 ? F(f->depths) : nullptr;
            if (sh) {
                f->campos = at::empty({C, 3}, options);
                check(lib.splatad_camera_centers((uint32_t)C, F(viewmats), M(f->campos), stream.stream()));
                check(lib.splatad_sh_colors_fwd((uint32_t)rows_max, (uint32_t)N, (uint32_t)f->K, (uint32_t)sh_degree, F(means), F(f->campos),
                                                F(colors), per_camera, L(f->camera_ids), L(f->gaussian_ids), I(f->radii), depths,
                                                (uint32_t)channels, M(f->colors), stream.stream()));
            } else {
                check(lib.splatad_color_rows_fwd((uint32_t)rows_max, (uint32_t)N, (uint32_t)D, L(f->camera_ids), L(f->gaussian_ids),
                                                 per_camera, F(colors), depths, M(f->colors), stream.stream()));
            }
            c = F(f->colors);
        }
        f->render = at::empty({C, H, W, channels}, options);
        f->alphas = at::empty({C, H, W, 1}, options);
        f->last_ids = at::empty({C, H, W}, ints);
        if (expected && grad) f->expected_depths = at::empty({C, H, W}, options);
        // The counts first: they choose the compositing kernel, and the lists are still being written when they arrive
        {
            py::gil_scoped_release no_gil;
            counts = read_counts(slot, sequence, stream);
            if (packed) {
                // behind the lists' count in the stream, so the rows' has arrived (or its store is about to)
                for (uint32_t i = 0; (nnz = load_word(slot.word + 8)) < 0; ++i, pause())
                    if ((i & 4095u) == 4095u && stream.query()) break;
                nnz = load_word(slot.word + 8);
            }
            // (with room to spare below what is told, and below what a kernel with runs wants)
            if (ask_near && usable(counts, capacity) &&
                (double)counts.n_isects * (double)counts.n_isects >= 11000. * (double)(C * tile_w * tile_h) * (double)std::max<int64_t>(counts.listed, 1)) {
                int64_t word;
                for (uint32_t i = 0; (uint32_t)((uint64_t)(word = load_word(slot.word + 10)) >> 32) != (uint32_t)sequence; ++i, pause())
                    if ((i & 4095u) == 4095u && stream.query()) break;
                const uint32_t bits = (uint32_t)word;
                memcpy(&f->near, &bits, 4);
            }
        }
        if (nnz <= 0 || nnz > rows_max || !usable(counts, capacity))
            return py::make_tuple(nnz, counts.n_isects, counts.status, counts.depth_range, counts.listed, py::none());
        lib.splatad_rasterize_set_spread_hint(counts.spread(), counts.n_isects);
        lib.splatad_rasterize_set_near_hint(f->near);
        check(lib.splatad_rasterize_expected_to_pixels_fwd(
            (uint32_t)C, -1, F(f->means2d), F(f->conics), c, (uint32_t)channels, o, F(f->pix_vels), F(rs_t), F(bg), (uint32_t)W, (uint32_t)H,
            (uint32_t)tile_size, (uint32_t)tile_w, (uint32_t)tile_h, I(f->offsets), I(f->flatten_ids), expected, M(f->render), M(f->alphas),
            I(f->last_ids), M(f->expected_depths), stream.stream()));
    }
    f->n = nnz;
    f->spread = counts.spread();
    if (packed && nnz < rows_max)
        for (Tensor *t : {&f->camera_ids, &f->gaussian_ids, &f->radii, &f->means2d, &f->depths, &f->conics, &f->comps, &f->pix_vels,
                          &f->tiles_per_gauss, &f->opacities, &f->colors})
            *t = head(*t, nnz);
    f->n_isects = counts.n_isects;   // none: the lists are null pointers, which the backward pass must not ask for
    f->isect_ids = head(f->isect_ids, counts.n_isects);
    f->flatten_ids = head(f->flatten_ids, counts.n_isects);
    Tensor opacities_r = f->opacities.defined() ? f->opacities : opacities.unsqueeze(0);
    if (grad) {
        const auto p = CameraProjectionNode::apply(means, quats, scales, opacities, mode == 2 ? OptTensor() : OptTensor(colors), velocities,
                                                   viewmats, Ks, lin_t, ang_t, rs_t, f);
        f->means2d = p[0]; f->depths = p[1]; f->conics = p[2]; f->pix_vels = p[3];
        if (opacity_rows) opacities_r = p[4];
        const Tensor colors_r = mode == 2 ? f->depths.unsqueeze(-1) : color_rows ? p[opacity_rows ? 5 : 4] : per_camera ? colors : colors.unsqueeze(0);
        const auto out = CameraCompositeNode::apply(p[0], p[2], colors_r, opacities_r, p[3], rs_t, bg.defined() ? OptTensor(bg) : OptTensor(), f);
        f->render = out[0]; f->alphas = out[1];
    }
    const auto opt = [](const Tensor &t) { return t.defined() ? py::cast(t) : py::object(py::none()); };
    return py::make_tuple(nnz, counts.n_isects, counts.status, counts.depth_range, counts.listed,
                          py::make_tuple(f->render, f->alphas, opt(f->camera_ids), opt(f->gaussian_ids), f->radii, f->means2d, f->depths,
                                         f->conics, opacities_r, f->pix_vels, f->tiles_per_gauss, f->isect_ids, f->flatten_ids,
                                         alias(f->offsets, {C, tile_h, tile_w})));
}

// ---------------------------------------------------------------------------------------------
// Lidar points -> tiles -> raster image. None: arguments for the Python bindings to check or convert.
// ---------------------------------------------------------------------------------------------
py::object map_points(const Tensor &points2d, const Tensor &boundaries, double tile_az, double min_az, bool sort) {
    if (!points2d.defined() || !points2d.is_cuda() || points2d.layout() != at::kStrided || points2d.dim() != 3 ||
        points2d.size(2) != 2 || points2d.numel() == 0 || points2d.is_conj() || points2d.is_neg())
        return py::none();
    const c10::DeviceIndex dev = points2d.get_device();
    const c10::cuda::CUDAGuard guard(dev);
    const at::NoGradGuard no_grad;
    if (points2d.scalar_type() != at::kFloat || !plain(boundaries, dev) || boundaries.dim() != 1) return py::none();
    const int64_t C = points2d.size(0), N = points2d.size(1), total = C * N;
    // the first two columns of a point cloud are read where they are
    int64_t stride = points2d.stride(1);
    const bool rows = points2d.stride(2) == 1 && stride >= 2 && stride < 0x7fffffff && (C == 1 || points2d.stride(0) == N * stride);
    const Tensor pts = rows ? points2d : points2d.contiguous();
    if (!rows) stride = 2;
    const auto stream = c10::cuda::getCurrentCUDAStream();
    const auto options = points2d.options().requires_grad(false);
    const Tensor ids = at::empty({total}, options.dtype(at::kLong)), flat = at::empty({total}, options.dtype(at::kInt));
    Tensor ws;
    if (sort) ws = workspace("map_points", lib.splatad_map_points_workspace_bytes((uint64_t)total), stream);
    check(lib.splatad_map_strided_points_to_lidar_tiles((uint32_t)C, (uint32_t)N, (uint64_t)total, F(pts), (uint32_t)stride, nullptr,
                                                        F(boundaries), (uint32_t)boundaries.numel(), (float)tile_az, (float)min_az,
                                                        sort, sort ? ws.data_ptr() : nullptr, sort ? (size_t)ws.numel() : 0, L(ids),
                                                        I(flat), stream.stream()));
    return py::make_tuple(ids, flat);
}

py::object encode_points(const Tensor &ids, int64_t C, int64_t tile_w, int64_t tile_h) {
    if (!ids.defined() || !ids.is_cuda() || ids.scalar_type() != at::kLong || !ids.is_contiguous() || ids.numel() == 0 ||
        C * tile_w * tile_h <= 0)
        return py::none();
    const c10::cuda::CUDAGuard guard(ids.device());
    const Tensor offsets = at::empty({C, tile_h, tile_w}, ids.options().dtype(at::kInt));
    check(lib.splatad_points_mapping_offset_encode(L(ids), ids.numel(), (uint32_t)C, (uint32_t)tile_w, (uint32_t)tile_h, I(offsets),
                                                   c10::cuda::getCurrentCUDAStream().stream()));
    return py::cast(offsets);
}

py::object populate_image(const Tensor &points, int64_t W, int64_t H, int64_t tile_w, int64_t tile_h, const Tensor &offsets,
                          const Tensor &flat) {
    if (!points.defined() || !points.is_cuda() || offsets.dim() != 3 || points.size(-1) != 5) return py::none();
    const c10::DeviceIndex dev = points.get_device();
    const auto whole = [&](const Tensor &t) {
        return t.is_cuda() && t.get_device() == dev && t.scalar_type() == at::kInt && t.is_contiguous() && t.numel() > 0;
    };
    if (!plain(points, dev) || points.numel() == 0 || !whole(offsets) || !whole(flat) || W <= 0 || H <= 0) return py::none();
    const c10::cuda::CUDAGuard guard(dev);
    const int64_t C = offsets.size(0);
    const Tensor image = at::empty({C, H, W, 5}, points.options().requires_grad(false));
    check(lib.splatad_populate_image_from_points((uint32_t)C, flat.numel(), F(points), (uint32_t)W, (uint32_t)H, (uint32_t)tile_w,
                                                 (uint32_t)tile_h, (uint32_t)offsets.size(2), (uint32_t)offsets.size(1), I(offsets),
                                                 I(flat), M(image), c10::cuda::getCurrentCUDAStream().stream()));
    return py::cast(image);
}

Tensor workspace_of(const std::string &tag, int64_t bytes, int64_t device) {
    return workspace(tag.c_str(), (size_t)bytes, c10::cuda::getCurrentCUDAStream((c10::DeviceIndex)device));
}

} // namespace

PYBIND11_MODULE(_host, m) {
    m.doc() = "Frames of splatad_b200 enqueued, waited for and differentiated in native code";
    m.def("bind_library", &bind_library);
    m.def("lidar_frame", torch::wrap_pybind_function(lidar_frame));
    m.def("camera_frame", torch::wrap_pybind_function(camera_frame));
    m.def("map_points", torch::wrap_pybind_function(map_points));
    m.def("encode_points", torch::wrap_pybind_function(encode_points));
    m.def("populate_image", torch::wrap_pybind_function(populate_image));
    m.def("workspace", torch::wrap_pybind_function(workspace_of));
    m.def("release", &release);
}
