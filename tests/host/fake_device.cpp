// A CUDA runtime and kernels that compute nothing, so the library's own host
// code (the C ABI, the wave planner, the pools) runs without a GPU: linked with
// its .cpp files into a library that the Python package loads in the place of
// its own. Device addresses are numbers nobody may read; every launch checks
// that the buffers it is handed are allocated and large enough for its wave.
//
// fake_* are the tests' controls and counters.
#include <chrono>
#include <cstdint>
#include <cstdlib>
#include <cstring>
#include <map>
#include <mutex>
#include <vector>

#include "runtime.h"

namespace {

std::mutex mu;
std::map<uint64_t, uint64_t> live;  // address -> bytes
uint64_t next_address = 1ull << 40, live_bytes = 0, limit = 180ull << 30, refused_size = ~0ull;
uint64_t meminfo_calls = 0, bad_launches = 0, window_free_shadows = 0, windowed_walks = 0;
uint64_t sorts = 0, waves = 0, largest_wave = 0;
int refuse_after = -1;  // this many more allocations succeed, then one is refused
cudaError_t last_error = cudaSuccess;
bool hang = false;
std::chrono::nanoseconds clock_offset{0};
std::map<uint64_t, std::vector<uint8_t>> uploads;  // what was copied to a live address
std::vector<uint8_t> streams[4];                   // the meshes' streams as the attribute kernel finds them
const void* stage = nullptr;
uint64_t late_stages = 0;
std::map<cudaStream_t, uint64_t> windows;  // stream -> bytes of its access-policy window

template <class T>
T handle() {
    static uint64_t n = 16;
    return reinterpret_cast<T>(n += 16);
}

bool holds(const void* p, uint64_t bytes) {
    auto it = live.find(reinterpret_cast<uint64_t>(p));
    return it != live.end() && it->second >= bytes;
}

void check(bool ok) {
    if (!ok) bad_launches++;
}

}  // namespace

extern "C" {

void fake_limit(uint64_t bytes) { limit = bytes; }
void fake_refuse_after(int n) { refuse_after = n; }
void fake_refuse_above(uint64_t bytes) { refused_size = bytes; }
void fake_hang(int on) { hang = on != 0; }
uint64_t fake_live_bytes() { return live_bytes; }
uint64_t fake_meminfo_calls() { return meminfo_calls; }
uint64_t fake_bad_launches() { return bad_launches; }
uint64_t fake_windowed_walks() { return windowed_walks; }
uint64_t fake_window_free_shadows() { return window_free_shadows; }
uint64_t fake_open_windows() {
    uint64_t n = 0;
    for (auto& w : windows) n += w.second != 0;
    return n;
}
uint64_t fake_late_stages() { return late_stages; }
const uint8_t* fake_stream(int k, uint64_t* bytes) {
    *bytes = streams[k].size();
    return streams[k].data();
}
uint64_t fake_sorts() { return sorts; }
uint64_t fake_waves() { return waves; }
uint64_t fake_largest_wave() { return largest_wave; }
double fake_clock_ms() { return std::chrono::duration<double, std::milli>(clock_offset).count(); }

// ---- the CUDA runtime ----------------------------------------------------------

cudaError_t cudaMalloc(void** p, size_t n) {
    std::lock_guard<std::mutex> lock(mu);
    if (refuse_after == 0 || n > refused_size || live_bytes + n > limit) {
        refuse_after = -1;
        *p = nullptr;
        return last_error = cudaErrorMemoryAllocation;
    }
    if (refuse_after > 0) refuse_after--;
    *p = reinterpret_cast<void*>(next_address);
    live[next_address] = n;
    live_bytes += n;
    next_address += (n + 4095) / 4096 * 4096;
    return cudaSuccess;
}
cudaError_t cudaFree(void* p) {
    std::lock_guard<std::mutex> lock(mu);
    auto it = live.find(reinterpret_cast<uint64_t>(p));
    if (it == live.end()) return p ? last_error = cudaErrorInvalidValue : cudaSuccess;
    live_bytes -= it->second;
    uploads.erase(uploads.lower_bound(it->first), uploads.lower_bound(it->first + it->second));
    live.erase(it);
    return cudaSuccess;
}
cudaError_t cudaMemGetInfo(size_t* free_bytes, size_t* total) {
    meminfo_calls++;
    *free_bytes = limit - live_bytes;
    *total = limit;
    return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void* dst, const void* src, size_t n, cudaMemcpyKind kind, cudaStream_t) {
    const uint8_t* p = static_cast<const uint8_t*>(src);
    if (kind == cudaMemcpyHostToDevice) uploads[reinterpret_cast<uint64_t>(dst)].assign(p, p + n);
    return cudaSuccess;
}
cudaError_t cudaMallocHost(void** p, size_t n) {
    *p = std::calloc(n, 1);
    return cudaSuccess;
}
cudaError_t cudaFreeHost(void* p) {
    std::free(p);
    return cudaSuccess;
}
cudaError_t cudaGetLastError() {
    cudaError_t e = last_error;
    last_error = cudaSuccess;
    return e;
}
const char* cudaGetErrorString(cudaError_t e) { return e == cudaErrorMemoryAllocation ? "out of memory" : "error"; }
cudaError_t cudaGetDeviceCount(int* n) {
    *n = 1;
    return cudaSuccess;
}
cudaError_t cudaGetDeviceProperties_v2(cudaDeviceProp* p, int) {
    std::memset(p, 0, sizeof *p);
    p->major = 10;
    p->persistingL2CacheMaxSize = 64 << 20;
    p->accessPolicyMaxWindowSize = 128 << 20;
    return cudaSuccess;
}
cudaError_t cudaDeviceGetStreamPriorityRange(int* least, int* greatest) {
    *least = 0;
    *greatest = -1;
    return cudaSuccess;
}
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) {
    *s = handle<cudaStream_t>();
    return cudaSuccess;
}
cudaError_t cudaStreamCreateWithPriority(cudaStream_t* s, unsigned f, int) { return cudaStreamCreateWithFlags(s, f); }
cudaError_t cudaStreamSetAttribute(cudaStream_t s, cudaStreamAttrID, const cudaStreamAttrValue* v) {
    windows[s] = v->accessPolicyWindow.num_bytes;
    return cudaSuccess;
}
cudaError_t cudaEventCreate(cudaEvent_t* e) {
    *e = handle<cudaEvent_t>();
    return cudaSuccess;
}
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { return cudaEventCreate(e); }
cudaError_t cudaEventQuery(cudaEvent_t) { return hang ? cudaErrorNotReady : cudaSuccess; }
cudaError_t cudaEventElapsedTime(float* ms, cudaEvent_t, cudaEvent_t) {
    *ms = 1.0f;
    return cudaSuccess;
}
cudaError_t cudaEventElapsedTime_v2(float* ms, cudaEvent_t a, cudaEvent_t b) { return cudaEventElapsedTime(ms, a, b); }
cudaError_t cudaMallocArray(cudaArray_t* a, const cudaChannelFormatDesc*, size_t, size_t, unsigned) {
    *a = handle<cudaArray_t>();
    return cudaSuccess;
}
cudaError_t cudaCreateTextureObject(cudaTextureObject_t* t, const cudaResourceDesc*, const cudaTextureDesc*,
                                    const cudaResourceViewDesc*) {
    *t = 1;
    return cudaSuccess;
}
cudaChannelFormatDesc cudaCreateChannelDesc(int x, int y, int z, int w, cudaChannelFormatKind f) {
    return {x, y, z, w, f};
}

}  // extern "C"

// A wait that never ends passes a tenth of a second at every look at the clock.
namespace std::chrono {
inline namespace _V2 {
steady_clock::time_point steady_clock::now() noexcept {
    if (hang) clock_offset += std::chrono::milliseconds(100);
    return steady_clock::time_point(clock_offset);
}
}  // namespace _V2
}  // namespace std::chrono

// ---- the kernels ------------------------------------------------------------------

namespace cn {

LaunchShape launch_shape(int) { return {}; }

void launch_wave_begin(const PathPool& p, const WaveParams& wp, const LaunchShape&, cudaStream_t) {
    const uint64_t n = uint64_t(wp.pixel_count) * wp.samples;
    waves++;
    largest_wave = largest_wave < n ? n : largest_wave;
    check(holds(p.ray, 32 * n) && holds(p.flux, 32 * n) && holds(p.hit, 16 * n) && holds(p.ps, 8 * n));
    check(holds(p.queue[0], 4 * n) && holds(p.queue[1], 4 * n) && holds(p.shadows, sizeof(ShadowRay) * n));
    check(holds(p.shadow_queue, 4 * n) && holds(p.counters, 4 * CTR_COUNT));
    check(n <= p.capacity);
    if (p.aov) check(holds(p.aov, 32 * n) && holds(p.aov_guide, 16 * n));
    if (p.guide_out)
        check(holds(p.guide_out, n * guide::OUT_ACT * 4) && holds(p.guide_rec, 4 * n) &&
              holds(p.sink, sizeof(GuideRecordSink)));
}
void launch_intersect(const DeviceScene&, const PathPool&, uint32_t, uint32_t, const LaunchShape&, bool,
                      cudaStream_t s) {
    if (windows[s]) windowed_walks++;
}
void launch_shadow(const DeviceScene&, const PathPool&, uint32_t, const LaunchShape&, bool, cudaStream_t s) {
    if (windows[s]) windowed_walks++;
    else window_free_shadows++;
}
void launch_material_sort(const PathPool& p, uint32_t, uint32_t n0, const LaunchShape&, cudaStream_t) {
    sorts++;
    check(holds(p.order, 4ull * n0) && holds(p.sort_keys, 4ull * n0) && holds(p.sort_bins, 4 * SORT_BINS));
}
void launch_accumulate(const PathPool&, const FilmTargets& f, uint32_t base, uint32_t count, uint32_t, uint32_t, bool,
                       cudaStream_t) {
    check(holds(f.sum, 16 * (uint64_t(base) + count)));
}
void launch_copy_rad(const PathPool&, float4* out, uint32_t base, uint32_t count, uint32_t, cudaStream_t) {
    check(holds(out, 16 * (uint64_t(base) + count)));
}
void launch_attributes(const float* positions, const float* normals, const float* uvs, const uint32_t* indices,
                       const uint32_t* first_tri, const uint64_t*, uint32_t, uint32_t n, float4* attrs, cudaStream_t) {
    check(holds(attrs, 16ull * TRI_ATTRS * n));
    stage = positions;
    const void* begin[5] = {positions, normals, uvs, indices, first_tri};
    for (int k = 0; k < 4; ++k) {
        streams[k].clear();
        uint64_t at = reinterpret_cast<uint64_t>(begin[k]);
        for (auto it = uploads.find(at); it != uploads.end() && it->first == at &&
                                         at < reinterpret_cast<uint64_t>(begin[k + 1]); it = uploads.find(at)) {
            streams[k].insert(streams[k].end(), it->second.begin(), it->second.end());
            at += it->second.size();
        }
    }
}
void launch_light_leaves(const float4*, uint32_t, const GeomRecord*, uint32_t*, cudaStream_t) {
    late_stages += holds(stage, 1);
}

namespace guide {
void launch_infer_paths(const Buffers&, const DeviceScene&, const PathPool& p, uint32_t, uint32_t n0, int,
                        cudaStream_t) {
    check(holds(p.guide_out, uint64_t(n0) * OUT_ACT * 4));
}
void launch_forward(const Buffers&, const float* feats, uint32_t rows, float* out, __nv_bfloat16*, int, cudaStream_t) {
    check(holds(feats, uint64_t(rows) * IN * 4) && holds(out, uint64_t(rows) * OUT * 4));
}
void launch_resolve_records(Record* recs, const uint32_t* count, uint32_t capacity, const float4*, cudaStream_t) {
    check(holds(recs, uint64_t(capacity) * sizeof(Record)) && holds(count, 4));
}
}  // namespace guide

}  // namespace cn
