// The library's runtime objects shared by the C ABI (capi.cpp) and the
// serving loop (server.cpp): the opaque handle types, device buffers, the
// status/error helpers, and the wave planner and enqueuer that drive the
// kernels of wavefront.cu.
#pragma once
#include <atomic>
#include <cstdint>
#include <initializer_list>
#include <memory>
#include <mutex>
#include <string>
#include <utility>
#include <vector>

#include <cuda_runtime.h>

#include "../../include/cenote_c.h"
#include "guide.h"
#include "records.h"
#include "wavefront.h"

namespace cn {

}  // namespace cn

struct cenote_context;

namespace cn {

// Record `msg` as this thread's last error and return `code`.
int32_t fail(int32_t code, const std::string& msg);
// The calling thread's last error message (cenote_last_error).
const char* last_error();

#define CN_CUDA(call)                                                                       \
    do {                                                                                    \
        cudaError_t e_ = (call);                                                            \
        if (e_ != cudaSuccess)                                                              \
            return ::cn::fail(e_ == cudaErrorMemoryAllocation ? CENOTE_E_ALLOCATION : CENOTE_E_DEVICE, \
                              std::string(#call ": ") + cudaGetErrorString(e_));            \
    } while (0)

#define CN_CHECK(cond, code, msg) \
    do {                          \
        if (!(cond)) return ::cn::fail((code), (msg)); \
    } while (0)

// Bounded wait: record `ev` on `s` and poll it until it completes or
// `timeout_ms` passes (CENOTE_E_TIMEOUT).
int32_t wait_stream(cudaStream_t s, cudaEvent_t ev, double timeout_ms);
int32_t wait_event(cudaEvent_t ev, double timeout_ms);

// Device memory to the caller's host memory on the context's stream, waited for
// as long as the work before it may take.
int32_t copy_out(cenote_context* ctx, void* host, const void* device, size_t bytes, double timeout_ms = 600000.0);

struct DeviceBuffer {
    void* ptr = nullptr;
    size_t bytes = 0;
    DeviceBuffer() = default;
    DeviceBuffer(const DeviceBuffer&) = delete;
    DeviceBuffer& operator=(const DeviceBuffer&) = delete;
    ~DeviceBuffer() { release(); }
    void release() {
        if (ptr) cudaFree(ptr);
        ptr = nullptr;
        bytes = 0;
    }
    // A refused allocation leaves the buffer empty (`bytes` 0, so that a caller
    // who keeps it by size asks again) and no error behind for the next launch.
    cudaError_t alloc(size_t n) {
        release();
        if (n == 0) n = 16;
        const cudaError_t e = cudaMalloc(&ptr, n);
        if (e != cudaSuccess) {
            ptr = nullptr;
            cudaGetLastError();
            return e;
        }
        bytes = n;
        return cudaSuccess;
    }
    template <class T>
    T* as() const {
        return static_cast<T*>(ptr);
    }
};

// Re-allocate buffers that grow together: all of them, or none is left (a
// refused one gives the others back).
inline cudaError_t alloc_together(std::initializer_list<std::pair<DeviceBuffer*, size_t>> buffers) {
    for (const auto& b : buffers) b.first->release();
    for (const auto& b : buffers) {
        const cudaError_t e = b.first->alloc(b.second);
        if (e != cudaSuccess) {
            for (const auto& x : buffers) x.first->release();
            return e;
        }
    }
    return cudaSuccess;
}

}  // namespace cn

using cn::DeviceBuffer;
using cn::DeviceScene;
using cn::LightRecord;
using cn::ShadowRay;
using cn::LaunchShape;
using cn::PathPool;
using cn::FilmTargets;
using cn::GuideRecordSink;
namespace guide = cn::guide;

struct cenote_renderer;

struct cenote_context {
    // Handles made from this context hold a reference; the context is freed
    // when cenote_context_destroy has been called and the last one is gone,
    // so destroy order never leaves a dangling pointer.
    std::atomic<int> refs{1};
    int device = 0;
    cudaStream_t stream = nullptr;
    cudaEvent_t sync_ev = nullptr;
    cudaEvent_t t0 = nullptr, t1 = nullptr;
    LaunchShape shape{};
    cn::DeviceBuffer tables;
    std::mutex mu;
    // The renderers made from this context, for give_back_pools.
    std::mutex renderers_mu;
    std::vector<cenote_renderer*> renderers;
    unsigned long long* tally_host = nullptr;  // pinned: a wave's counters come back with its last event
    // L2 persistence (this context's own set-aside; nothing outlives it).
    size_t l2_persist_max = 0, l2_window_max = 0, l2_set_aside = 0;
    uint32_t bvh_builder = CENOTE_BVH_AUTO;  // for scenes created from now on
};

struct cenote_scene {
    cenote_context* ctx = nullptr;
    DeviceScene ds{};
    std::vector<std::unique_ptr<DeviceBuffer>> buffers;
    cudaArray_t env_array = nullptr;
    cudaTextureObject_t env_tex = 0;
    cenote_camera camera{};
    std::vector<LightRecord> lights;
    uint32_t env_w = 1, env_h = 1;
    double env_power = 0.0;
    float select_prob = 0.0f;
    float prep_ms[3] = {0, 0, 0};
    uint32_t bvh_builder = CENOTE_BVH_HOST_SAH;  // the builder this scene's BVH came from
    // Every material runs the same closure code (no maps, no layers, specular
    // and metal on all or on none) and the geometry is small: a material sort
    // has nothing to group.
    bool uniform_shading = false;
    uint64_t device_bytes = 0;
    DeviceBuffer* env_marginal = nullptr;
    DeviceBuffer* env_conditional = nullptr;
    DeviceBuffer* env_cut = nullptr;
    DeviceBuffer* env_pdfs = nullptr;
    std::vector<cudaArray_t> tex_arrays;            // the bindless table's storage
    std::vector<cudaTextureObject_t> tex_objects;

    // Take ownership of memory cudaMalloc'd elsewhere (the GPU BVH build).
    DeviceBuffer* adopt(void* p, size_t bytes) {
        buffers.push_back(std::make_unique<DeviceBuffer>());
        buffers.back()->ptr = p;
        buffers.back()->bytes = bytes;
        device_bytes += bytes;
        return buffers.back().get();
    }
        DeviceBuffer* add(size_t bytes, cudaError_t* err) {
        buffers.push_back(std::make_unique<DeviceBuffer>());
        *err = buffers.back()->alloc(bytes);
        device_bytes += bytes;
        return buffers.back().get();
    }
    ~cenote_scene() {
        for (cudaTextureObject_t t : tex_objects) cudaDestroyTextureObject(t);
        for (cudaArray_t a : tex_arrays) cudaFreeArray(a);
        if (env_tex) cudaDestroyTextureObject(env_tex);
        if (env_array) cudaFreeArray(env_array);
    }
};

struct cenote_renderer {
    cenote_context* ctx = nullptr;
    uint32_t max_bounces = 8;
    uint32_t light_sampling = 0;
    uint32_t capacity_req = 0;
    uint32_t samples_per_wave = 0;
    uint32_t profiling = 0;
    std::vector<cudaEvent_t> events;
    PathPool pool{};
    DeviceBuffer ray, flux, hit, ps, q0, q1, shadows, shadow_queue, counters, tally, scratch;
    uint32_t material_sort = CENOTE_SORT_AUTO;  // CENOTE_SORT_*: see sort_mode
    uint32_t refill_idle = 0;  // 0: the kernels' default
    uint32_t top_nodes = 0;    // BVH nodes staged in shared memory by the traversal kernels
    uint32_t l2_window = 0;    // mark the BVH nodes persisting in L2 during this renderer's waves
    uint32_t per_lane_triangles = 0;  // 1: no warp triangle queue in the traversal kernels
    uint32_t trav_variant = 0;        // traversal block size and stack depth (TRAV_VARIANT_*)
    uint32_t sort_by_location = 0;    // 1: the material sort keys layer-free hits by location
    float tuned_ms_per_sample = 0.0f;
    DeviceBuffer sort_order, sort_keys, sort_bins;
    DeviceBuffer oneshot;  // a one-shot render's image
    DeviceBuffer aov, aov_guide;
    size_t pool_cap = 0, aov_cap = 0;
    // The learned guide (cenote_renderer_set_guide): per-path mixture outputs
    // and open records, the wave's training records and its sink.
    cenote_guide* guide = nullptr;
    float guide_fraction = 0.5f, guide_lr = 1e-2f;
    uint32_t guide_steps = 0;
    DeviceBuffer g_out, g_rec, g_records, g_count, g_sink;
    size_t g_cap = 0;
    // Device bytes a path of the pool takes with the denoiser guides' lanes.
    static constexpr uint64_t PATH_BYTES = 32 * 2 + 16 + 8 + 8 + sizeof(ShadowRay) + 4 + 8 + 48;
    // Waves above this many paths are taken only while memory is plentiful.
    static constexpr uint64_t PLAIN_WAVE = uint64_t(1) << 24;
    static constexpr uint32_t GUIDE_RECORDS = 1u << 20;
    static constexpr uint32_t GUIDE_BATCH = 65536;
    // The shadow walks' own stream and the events that fork it off the main
    // stream and join it back, every bounce of every wave (made on the first
    // wave; serving waves do without).
    cudaStream_t side = nullptr;
    cudaEvent_t fork = nullptr, join = nullptr;
    cudaError_t ensure_side() {
        cudaError_t e = cudaSuccess;
        if (!side) e = cudaStreamCreateWithFlags(&side, cudaStreamNonBlocking);
        if (e == cudaSuccess && !fork) e = cudaEventCreateWithFlags(&fork, cudaEventDisableTiming);
        if (e == cudaSuccess && !join) e = cudaEventCreateWithFlags(&join, cudaEventDisableTiming);
        return e;
    }

    cenote_stats stats{};
    unsigned long long tally_prev[6] = {0, 0, 0, 0, 0, 0};

    ~cenote_renderer() {
        for (cudaEvent_t e : events) cudaEventDestroy(e);
        if (side) cudaStreamDestroy(side);
        if (fork) cudaEventDestroy(fork);
        if (join) cudaEventDestroy(join);
    }
    cudaEvent_t event(size_t i) {
        while (events.size() <= i) {
            cudaEvent_t e;
            if (cudaEventCreate(&e) != cudaSuccess) return nullptr;
            events.push_back(e);
        }
        return events[i];
    }

    // The sort mode of a wave of `paths` camera paths (0: known on the device
    // only). A chosen mode holds for every wave. Without one every bounce sorts
    // (1.1x on the material chart, 1.6x on the textured terrain) but in the
    // waves whose bounces shade no faster in material order, unless a guide
    // trains on their records (which arrive in shading order); films are the
    // same bits either way where the scene has no layered materials (with
    // them, the sorted bounces split between two builds of the shading
    // kernel).
    //
    // By paths: the sort's launches cost a bounce about 10 us, its order saves
    // in proportion to the paths. Device ms unsorted / sorted of one-sample
    // frames, the chart: 60 k paths 0.61 / 0.72, 230 k 0.83 / 0.95, 300 k 0.90 /
    // 1.01, 600 k 1.19 / 1.27, 920 k 1.57 / 1.58, 1.4 M 2.08 / 2.01; the textured
    // scene: 60 k 0.26 / 0.29, 230 k 0.34 / 0.36, 300 k 0.38 / 0.39, 450 k 0.475 /
    // 0.467, 600 k 0.60 / 0.54, 1.4 M 1.30 / 0.96. The line lies below the first
    // crossing, where no measured scene gains by sorting.
    //
    // By scene: one closure class, 36 to 20,412 triangles, sorted / unsorted
    // 1.58 / 1.43 to 2.87 / 2.67 at 1 M paths, 6.04 / 5.30 to 10.3 / 9.2 at 7.4 M.
    static constexpr uint32_t SORT_MIN_PATHS = 1u << 18;
    static constexpr uint32_t UNIFORM_MAX_TRIANGLES = 1u << 15;
    uint32_t sort_mode(const cenote_scene* sc, uint32_t paths) const {
        if (material_sort != CENOTE_SORT_AUTO) return material_sort;
        if (sc->ds.has_layers || (guide && guide_steps > 0)) return CENOTE_SORT_ALL;
        if (sc->uniform_shading || (paths != 0 && paths < SORT_MIN_PATHS)) return CENOTE_SORT_NONE;
        return CENOTE_SORT_ALL;
    }

    // Free the pool and every lane sized by a wave (not the one-shot image);
    // the next wave allocates anew.
    void release_pool() {
        pool_cap = aov_cap = g_cap = 0;
        for (DeviceBuffer* b : {&ray, &flux, &hit, &ps, &q0, &q1, &shadows, &shadow_queue, &sort_order, &sort_keys,
                                &sort_bins, &aov, &aov_guide, &g_out, &g_rec})
            b->release();
    }

    cudaError_t ensure(size_t cap) {
        if (cap <= pool_cap) return cudaSuccess;
        pool_cap = 0;
        cudaError_t e = cn::alloc_together({{&ray, cap * 32},
                                            {&flux, cap * 32},
                                            {&hit, cap * 16},
                                            {&ps, cap * 8},
                                            {&q0, cap * 4},
                                            {&q1, cap * 4},
                                            {&shadows, cap * sizeof(ShadowRay)},
                                            {&shadow_queue, cap * 4},
                                            {&sort_order, cap * 4},
                                            {&sort_keys, cap * 4},
                                            {&sort_bins, cn::SORT_BINS * 4}});
        if (e != cudaSuccess) return e;
        pool.ray = ray.as<float4>();
        pool.flux = flux.as<float4>();
        pool.hit = hit.as<uint4>();
        pool.ps = ps.as<uint2>();
        pool.queue[0] = q0.as<uint32_t>();
        pool.queue[1] = q1.as<uint32_t>();
        pool.shadows = shadows.as<ShadowRay>();
        pool.shadow_queue = shadow_queue.as<uint32_t>();
        // Null here: the wave loop passes a view with all three set to the
        // bounces it sorts.
        pool.order = nullptr;
        pool.sort_keys = nullptr;
        pool.sort_bins = nullptr;
        pool.capacity = uint32_t(cap);
        pool_cap = cap;
        return cudaSuccess;
    }

    // The learned guide's lanes for waves of `paths` paths (196 bytes each; a
    // pool that unguided waves have grown is up to four times a guided wave);
    // detached without a guide.
    cudaError_t set_learned_guide(bool on, size_t paths) {
        if (on && g_cap < paths) {
            g_cap = 0;
            cudaError_t e = cn::alloc_together({{&g_out, paths * guide::OUT_ACT * 4}, {&g_rec, paths * 4}});
            if (e != cudaSuccess) return e;
            g_cap = paths;
        }
        if (on && !g_records.ptr) {
            cudaError_t e = cn::alloc_together({{&g_records, size_t(GUIDE_RECORDS) * sizeof(guide::Record)},
                                                {&g_count, 16},
                                                {&g_sink, sizeof(GuideRecordSink)}});
            if (e != cudaSuccess) return e;
        }
        pool.guide_out = on ? g_out.as<float>() : nullptr;
        pool.guide_rec = on ? g_rec.as<uint32_t>() : nullptr;
        pool.sink = on ? g_sink.as<GuideRecordSink>() : nullptr;
        return cudaSuccess;
    }

    // The guide lanes: allocated on the first wave that traces guides,
    // detached (null) for waves that do not.
    // The pool as the bounces that sort see it.
    PathPool sorted_view() const {
        PathPool p = pool;
        p.order = sort_order.as<uint32_t>();
        p.sort_keys = sort_keys.as<uint32_t>();
        p.sort_bins = sort_bins.as<uint32_t>();
        return p;
    }

        cudaError_t set_guides(bool on) {
        if (on && aov_cap < pool_cap) {
            aov_cap = 0;
            cudaError_t e = cn::alloc_together({{&aov, pool_cap * 32}, {&aov_guide, pool_cap * 16}});
            if (e != cudaSuccess) return e;
            aov_cap = pool_cap;
        }
        pool.aov = on ? aov.as<float4>() : nullptr;
        pool.aov_guide = on ? aov_guide.as<float4>() : nullptr;
        return cudaSuccess;
    }
};

struct cenote_guide {
    cenote_context* ctx = nullptr;
    DeviceBuffer params, grad, m, v, w1, w2, w3, w4, b4, err, loss;
    DeviceBuffer feats, out, save, dz4, dirs, weights;
    size_t cap = 0;
    uint32_t step = 0;
    int sms = 148;

    guide::Buffers view() {
        return {params.as<float>(), grad.as<float>(), m.as<float>(), v.as<float>(), w1.as<__nv_bfloat16>(),
                w2.as<__nv_bfloat16>(), w3.as<__nv_bfloat16>(), w4.as<__nv_bfloat16>(), b4.as<float>(),
                err.as<int>()};
    }
    guide::TrainScratch scratch(uint32_t rows) {
        return {out.as<float>(), save.as<__nv_bfloat16>(), dz4.as<__nv_bfloat16>(), loss.as<float>(), rows};
    }
    cudaError_t ensure(size_t n) {
        if (n <= cap) return cudaSuccess;
        cap = 0;
        cudaError_t e = cn::alloc_together({{&feats, n * guide::IN * 4},
                                            {&out, n * guide::OUT * 4},
                                            {&save, n * guide::ACT * 2},
                                            {&dz4, n * guide::OUT_PAD * 2},
                                            {&dirs, n * 12},
                                            {&weights, n * 4}});
        if (e == cudaSuccess) cap = n;
        return e;
    }
};

struct cenote_film {
    cenote_context* ctx = nullptr;
    uint32_t width = 0, height = 0;
    uint32_t samples = 0;
    DeviceBuffer sum, avg;
    DeviceBuffer albedo, normal, depth;  // guide sums (film.rs:95-112)
    FilmTargets targets() {
        return {sum.as<float4>(), albedo.as<float4>(), normal.as<float4>(), depth.as<float>()};
    }
};

namespace cn {
inline void free_context(cenote_context* ctx) {
    cudaSetDevice(ctx->device);
    if (ctx->stream) cudaStreamSynchronize(ctx->stream);
    ctx->tables.release();
    if (ctx->sync_ev) cudaEventDestroy(ctx->sync_ev);
    if (ctx->tally_host) cudaFreeHost(ctx->tally_host);
    if (ctx->t0) cudaEventDestroy(ctx->t0);
    if (ctx->t1) cudaEventDestroy(ctx->t1);
    if (ctx->stream) cudaStreamDestroy(ctx->stream);
    delete ctx;
}
inline void retain(cenote_context* ctx) { ctx->refs.fetch_add(1); }
inline void release(cenote_context* ctx) {
    if (ctx->refs.fetch_sub(1) == 1) free_context(ctx);
}
}  // namespace cn


namespace cn {

// Free what the context's renderers keep for their next call only because memory
// was plentiful: pools larger than a plain wave's, and the one-shot images of
// all but `busy`. True when there was any. The caller holds ctx->mu, so no wave
// of the context is in flight.
bool give_back_pools(cenote_context* ctx, const cenote_renderer* busy = nullptr);

// Allocations under ctx->mu: refused, they are tried once more if anything
// could be given back.
template <class F>
cudaError_t allocating(cenote_context* ctx, F allocations, const cenote_renderer* busy = nullptr) {
    const cudaError_t e = allocations();
    return e == cudaErrorMemoryAllocation && give_back_pools(ctx, busy) ? allocations() : e;
}

// The same for a call that makes a new object and leaves nothing behind when
// it is refused; ctx->mu is not held.
template <class F>
int32_t creating(cenote_context* ctx, F call) {
    const int32_t rc = call();
    if (rc != CENOTE_E_ALLOCATION) return rc;
    {
        std::lock_guard<std::mutex> lock(ctx->mu);
        if (!give_back_pools(ctx)) return rc;
    }
    return call();
}

// How a call splits into waves: `range` pixels per wave, `spw` samples each.
struct WavePlan {
    uint32_t range, spw;
    uint64_t need;  // paths the pool must hold
};

struct WaveCounts {
    uint32_t launches = 0, waves = 0;
    size_t events = 0;
};

// An automatic wave takes at most `most` paths where whole samples allow.
WavePlan plan_waves(const cenote_renderer* r, uint64_t pixels, uint32_t count, bool oneshot,
                    uint64_t most = uint64_t(1) << 26);

// Enqueue `count` samples from `sample0` for every pixel on `stream`, with no
// host synchronisation (so a stream capture can record it): each wave's
// samples go into the film in ascending order or, for a one-shot render,
// into `oneshot` as raw RGBA. The pool must already hold `plan.need` paths
// and the guide lanes must match `film`. `sample_offset` (device, may be
// null) is added to every sample index. Timing marks are recorded only when
// `timing` is set (never inside a capture).
cudaError_t enqueue_waves(cenote_renderer* r, const cenote_scene* sc, uint32_t width, uint32_t height,
                          uint32_t sample0, uint32_t count, uint32_t max_bounces, const WavePlan& plan,
                          const FilmTargets* film, bool film_reset, float4* oneshot, const uint32_t* sample_offset,
                          cudaStream_t stream, bool timing, bool counting, WaveCounts* wc);

// The bounces of one wave whose n0 camera paths are in the pool; `side` may be
// `stream`.
void enqueue_bounces(cenote_renderer* r, const cenote_scene* sc, const WaveParams& wp, uint32_t n0, bool guided,
                     cudaStream_t stream, cudaStream_t side, bool timing, bool counting, WaveCounts* wc);

// One multi-job wave (the serving loop): segments in device memory, their
// camera paths, the bounces, and each segment's samples into its job's film.
cudaError_t enqueue_segments(cenote_renderer* r, const cenote_scene* sc, const WaveSegment* segs, uint32_t nseg,
                             uint32_t paths, uint32_t items, const uint32_t* hdr, uint32_t max_bounces,
                             cudaStream_t stream, WaveCounts* wc);

}  // namespace cn
