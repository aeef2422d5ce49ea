// tr_internal.h - host-side internals shared by the C ABI translation units (tr_api.cu: one
// scene per context; tr_batch.cu: many contexts rendered in shared wavefront batches).
#pragma once
#include "transient_b200.h"

#include <cuda_runtime.h>

#include <algorithm>
#include <stdexcept>
#include <string>
#include <functional>
#include <vector>

#include "tr_guide.cuh"
#include "tr_kernels.cuh"

namespace tri {

// records msg as the thread's last error (tr_last_error) and returns s
tr_status fail(tr_status s, const std::string& msg);

// A failed CUDA call.  The runtime's own record of the error is taken back with it: the launchers report
// cudaGetLastError(), so one left behind (an allocation that did not fit) would fail the thread's next launch.
struct CudaError : std::runtime_error {
    cudaError_t code;
    CudaError(cudaError_t c, const char* what) : std::runtime_error(std::string(what) + ": " + cudaGetErrorString(c)), code(c) {
        cudaGetLastError();
    }
};

#define TR_CUDA(call)                                           \
    do {                                                        \
        cudaError_t e_ = (call);                                \
        if (e_ != cudaSuccess) throw CudaError(e_, #call);      \
    } while (0)

// Device memory of contexts, guides and batches comes from one stream-ordered pool per device
// that keeps freed memory for the next allocations (release threshold unlimited), so creating
// and destroying contexts does not map and unmap gigabytes each time; memory goes back to the
// driver only through tr_release_cached_memory or at exit.  A large render's batches come and go with
// each call; they have a pool of their own, or what other contexts keep would be carved from their blocks and the
// next large render would have to map new ones (13 to 20 ms).  That pool keeps at most kLargeWaveBytes, which
// the other gets when it finds no memory.
enum class Pool { kKept, kLarge };
cudaMemPool_t device_pool(int device, Pool which = Pool::kKept);
// pool memory of `device` reserved but not in use (free for the next allocations)
size_t pool_idle_bytes(int device, Pool which);
// cudaMallocFromPoolAsync on stream s, from the current device's pool
cudaError_t pool_malloc(void** p, size_t bytes, cudaStream_t s, Pool which = Pool::kKept);
// Gives p back to its pool: by cudaFree, which waits for the device (any stream may have used it), or in the order
// of stream s.  Both keep the count of what is in use: the pool's own goes on counting what cudaFree returned
// (and freeing in stream order after a wait for the device would end the graph captures of other threads).
void pool_free(void* p);
void pool_free_after(void* p, cudaStream_t s);

template <class T>
T* dalloc(size_t count, size_t& total, Pool which = Pool::kKept) {
    if (count == 0) count = 1;
    void* p = nullptr;
    cudaError_t e = pool_malloc(&p, count * sizeof(T), 0, which);
    if (e == cudaSuccess) e = cudaStreamSynchronize(0);     // usable from every stream
    if (e != cudaSuccess) throw CudaError(e, "device allocation");
    total += count * sizeof(T);
    return static_cast<T*>(p);
}

constexpr uint32_t kMaxBounces = 63;            // counters hold 64 depths
constexpr uint32_t kDefaultCapacity = 1u << 21; // path slots per wavefront batch
constexpr uint32_t kLargeCapacity = 1u << 23;   // of a large render's (render_region)
constexpr size_t kLargeWaveBytes = (size_t)6 << 30;  // path state a large render's batches may take
constexpr size_t kLeastFree = (size_t)2 << 30;  // device memory left for a new context's path state
#ifndef TR_WAVE_LANES
#define TR_WAVE_LANES 4
#endif
constexpr int kWaveLanes = TR_WAVE_LANES;        // wave buffer sets batches alternate between
static_assert(kWaveLanes >= 1, "a render needs a wave");
// lanes of a large render's batches (three with RGBE delivery), of those the build has
constexpr int large_lanes(bool rgbe) { return std::min(rgbe ? 3 : 2, kWaveLanes); }
// default roughness below which GGX vertices sample their BSDF instead of the learned proposal
constexpr float kGuideMinAlpha = 0.5f;
constexpr uint32_t kTrainBatch = 65536, kTrainLeast = 1024;     // samples of a training step: at most, at least

}  // namespace tri

using tri::dalloc;

struct tr_guide {
    int device = 0;
    cudaStream_t stream = nullptr;
    std::vector<void*> allocs;
    size_t bytes = 0;
    float* params = nullptr;   // FP32 master copy
    float* grads = nullptr;
    float* m1 = nullptr;
    float* m2 = nullptr;
    uint8_t* w_fwd = nullptr;  // packed BF16 tiles
    uint8_t* w_bwd = nullptr;
    // device words: [kInfer] / [kTrain] a wait of inference / of a training step timed out, [kSteps] training
    // steps applied.  Training runs beside renders that sample with the network, so each has its own word.
    enum { kInfer = 0, kTrain = 1, kSteps = 2, kWords = 3 };
    int* status = nullptr;
    float* scalars = nullptr;  // [0] weight sum, [1] loss
    uint32_t cap = 0;
    uint4* act = nullptr;
    float* scratch = nullptr;          // partial sums of a training step
    uint4* dy_bf = nullptr;
    uint4* dh = nullptr;       // BF16 hidden-layer gradients [3][n][64]
    uint32_t step = 0;                 // training steps enqueued; after one that timed out, those applied
    uint32_t spin = trg::kWaitPolls;   // mbarrier polls before a tensor-core wait times out
    template <class T>
    T* alloc(size_t n) {
        T* p = tri::dalloc<T>(n, bytes);
        allocs.push_back(p);
        return p;
    }
    void drop(void* p) {
        if (!p) return;
        tri::pool_free(p);
        allocs.erase(std::remove(allocs.begin(), allocs.end(), p), allocs.end());
    }
    trg::GuideDev dev() const {
        return trg::GuideDev{reinterpret_cast<const uint4*>(w_fwd), reinterpret_cast<const uint4*>(w_bwd),
                             params + 4 * 4096, spin};
    }
    void ensure(uint32_t n) {
        if (cap >= n) return;
        drop(act); drop(scratch); drop(dy_bf); drop(dh);
        act = dy_bf = dh = nullptr;
        scratch = nullptr;
        cap = 0;
        act = alloc<uint4>((size_t)3 * n * 8);
        scratch = alloc<float>(trg::train_scratch_floats(n));
        dy_bf = alloc<uint4>((size_t)n * 8);
        dh = alloc<uint4>((size_t)3 * n * 8);
        cap = n;
    }
};

struct tr_ctx {
    int device = 0;
    cudaStream_t stream = nullptr;
    cudaEvent_t ev0 = nullptr, ev1 = nullptr;
    size_t bytes = 0;                       // device memory held
    struct Alloc { void* p; size_t bytes; };
    std::vector<Alloc> allocs;

    // scene
    float4* d_nodes = nullptr;
    float4* d_tris = nullptr;
    float4* d_tri_ng = nullptr;
    float4* d_mats = nullptr;
    float4* d_mats2 = nullptr;
    float4* d_lights = nullptr;
    trk::SceneDev scene{};
    uint32_t nt = 0, bvh_nodes = 0, bvh_depth = 0, bvh_levels = 0;   // bvh_depth: stack entries - 1
    double bvh_ms = 0.0;

    tr_camera cam{};
    tr_film film{};
    tr_integrator integ{};

    // film
    double* d_streak = nullptr;
    double* d_steady = nullptr;
    double* d_weight = nullptr;
    double* d_bstreak = nullptr;            // per-bounce films (tr_film.bounce_films > 0)
    double* d_bsteady = nullptr;
    double* d_bweight = nullptr;
    double* d_cdepth = nullptr;             // film components (tr_film.components)
    double* d_cpos = nullptr;
    double* d_cnorm = nullptr;

    // wavefront state
    trk::Wave wave{};
    trk::Wave lane_wave[tri::kWaveLanes - 1]{};  // further lanes of batches (share wave.stats)
    uint4* lane_vrec[tri::kWaveLanes - 1]{};      // their guided-vertex records (learned proposal)
    uint32_t lane_vrec_cap[tri::kWaveLanes - 1]{};
    uint32_t guide_tag = 0;                       // last training-pool batch tag handed out
    trk::Wave lwave{};                      // light subpaths (TR_FLAG_BIDIRECTIONAL)
    trk::BidirWave bd{};
    uint32_t* d_lcounters = nullptr;
    uint32_t bd_queues = 1;                 // connection queues (two when memory allows)
    cudaEvent_t bd_free[2]{};               // a queue's rays have been traced
    // film streaming (tr_render_film)
    cudaStream_t copy_stream = nullptr;
    // shadow rays of one depth beside the closest-hit rays of the next (tr_render_region)
    cudaStream_t shadow_stream = nullptr;
    cudaStream_t lane_stream[tri::kWaveLanes - 1]{}, lane_shadow_stream[tri::kWaveLanes - 1]{};
    cudaStream_t light_stream = nullptr;    // light subpaths beside the eye walks (bidirectional)
    cudaStream_t conn_stream[2]{};          // setting up and tracing their connections
    std::vector<cudaEvent_t> dep_events;    // ordering events (no timing), reused in turn
    size_t next_dep = 0;
    float* d_stage = nullptr;               // FP32 staging of one pixel batch's rows
    size_t stage_floats = 0;
    uchar4* d_rgbe = nullptr;               // RGBE film images: [H][W][T] streak cells, then [H][W] steady
    size_t rgbe_cells = 0;
    bool film_clean = true;                 // no samples added since the film was zeroed
    int trace_grid = 0;

    // ray-batch scratch
    float* d_rays = nullptr;
    void* d_hits = nullptr;
    uint32_t ray_cap = 0;
    uint32_t* d_cursor = nullptr;

    tr_stats stats{};
    // learned proposal (tr_set_guide)
    tr_guide* guide = nullptr;
    float guide_mix = 0.5f, guide_lr = 1e-3f;
    uint32_t guide_pool = 0;
    trk::GuideWave gw{};
    uint32_t gw_capacity = 0;
    uint32_t* pool_state = nullptr;       // [0] pool fill, [1] entries with targets
    // Training pools are double-buffered: a render fills the pool in gw while the samples of the
    // previous render (pool_alt, pool_pending entries) train the proposal beside it, on the
    // guide's stream.  The render samples with a snapshot of the network (w_snap, bias_snap)
    // taken when it starts, so the training it overlaps never changes the proposal mid-render.
    struct PoolBuf { uint4* feat = nullptr; float* dir = nullptr; float* w = nullptr; uint4* meta = nullptr;
                     uint32_t* state = nullptr; };
    PoolBuf pool_alt{};
    uint32_t pool_pending = 0;
    uint4* w_snap = nullptr;              // packed forward tiles of the render's network (32 KB)
    float* bias_snap = nullptr;           // and its biases [4][64]
    cudaEvent_t ev_snap = nullptr, ev_train = nullptr;
    uint32_t guide_depth = 0xffffffffu;   // path depths whose surface vertices use the proposal
    float guide_min_alpha = tri::kGuideMinAlpha;   // GGX vertices smoother than this sample their BSDF
    float last_train_loss = 0.0f;
    uint32_t train_steps = 0;
    cudaStream_t user_stream = nullptr;   // caller's stream (tr_set_stream) or null
    int profiling = 0;                    // 0 off, 1 read out per render, 2 read out at tr_stats_get
    std::vector<cudaEvent_t> prof_events; // pool of timing events
    struct ProfMark { int kind; size_t ev; };
    std::vector<ProfMark> prof_marks;     // launches timed and not read out yet
    size_t prof_next = 0;                 // events of prof_events in use
    // read-out kernel times not yet handed to tr_stats_get: raygen, extend, shade, shadow,
    // splat, guide, then the union of the traversal intervals (milliseconds)
    double prof_sum[7] = {0, 0, 0, 0, 0, 0, 0};
    bool prof_dirty = false;              // prof_sum holds read-outs not yet published
    cudaStream_t s() const { return user_stream ? user_stream : stream; }

    template <class T>
    T* alloc(size_t n, tri::Pool which = tri::Pool::kKept) {
        const size_t before = bytes;
        T* p = tri::dalloc<T>(n, bytes, which);
        allocs.push_back({p, bytes - before});
        return p;
    }
    // gives p's memory back and forgets the address, so that it is never freed or used again: in the order of
    // the stream `after`, or at once, which waits for the device
    template <class T>
    void drop(T*& p, cudaStream_t after = nullptr) {
        if (!p) return;
        const auto it = std::find_if(allocs.begin(), allocs.end(), [&](const Alloc& a) { return a.p == p; });
        if (it != allocs.end()) {
            if (after) tri::pool_free_after(p, after);
            else tri::pool_free(p);
            bytes -= it->bytes;
            allocs.erase(it);
        }
        p = nullptr;
    }
    void release() {
        if (ev_snap) { cudaEventDestroy(ev_snap); ev_snap = nullptr; }
        if (ev_train) { cudaEventDestroy(ev_train); ev_train = nullptr; }
        for (cudaEvent_t& e : bd_free) {
            if (e) cudaEventDestroy(e);
            e = nullptr;
        }
        for (cudaEvent_t e : prof_events) cudaEventDestroy(e);
        prof_events.clear();
        for (cudaEvent_t e : dep_events) cudaEventDestroy(e);
        dep_events.clear();
        if (shadow_stream) cudaStreamDestroy(shadow_stream);
        for (int k = 0; k < tri::kWaveLanes - 1; ++k) {
            if (lane_stream[k]) cudaStreamDestroy(lane_stream[k]);
            if (lane_shadow_stream[k]) cudaStreamDestroy(lane_shadow_stream[k]);
            lane_stream[k] = lane_shadow_stream[k] = nullptr;
        }
        for (cudaStream_t& c : conn_stream) {
            if (c) cudaStreamDestroy(c);
            c = nullptr;
        }
        if (light_stream) cudaStreamDestroy(light_stream);
        shadow_stream = light_stream = nullptr;
        for (const Alloc& a : allocs) tri::pool_free(a.p);
        allocs.clear();
        if (ev0) cudaEventDestroy(ev0);
        if (ev1) cudaEventDestroy(ev1);
        if (copy_stream) cudaStreamDestroy(copy_stream);
        copy_stream = nullptr;
        if (stream) cudaStreamDestroy(stream);
        ev0 = ev1 = nullptr;
        stream = nullptr;
    }
};

namespace tri {

// Per-slot arrays of a wave of `capacity` slots with R records each, carved from one block (one
// pool allocation instead of fourteen): with w null the bytes it takes, else w's pointers into it.
size_t carve_wave(trk::Wave* w, void* block, uint32_t capacity, size_t R, bool time_sampling);
void ensure_wave(tr_ctx* x, uint32_t capacity, Pool which = Pool::kKept);
void drop_waves(tr_ctx* x, cudaStream_t after = nullptr);
void ensure_lane_wave(tr_ctx* x, int k, uint32_t capacity, Pool which);
void ensure_lane_guided(tr_ctx* x, int k, uint32_t capacity, Pool which);
void ensure_guide_pools(tr_ctx* x);
void ensure_guided(tr_ctx* x, uint32_t capacity, Pool which);
trk::Params make_params(tr_ctx* x);
trg::GuideDev guide_dev(tr_guide* g);
int* guide_err(tr_guide* g);
// waits for stream s and reports (and clears) waits that timed out in inference, in training steps or in either
tr_status guide_check(tr_guide* g, cudaStream_t s, bool infer, bool train);
// enqueues one training step of the proposal on stream s (no host synchronisation)
void train_enqueue(tr_guide* g, const uint4* x, const float* d_dirs, const float* d_weights, uint32_t n, float lr,
                   cudaStream_t s);
// trains the proposal on the pool a guided render collected (`fill` = pool_state on the device)
tr_status train_on_pool(tr_guide* g, const trk::GuideWave& gw, const uint32_t* pool_state, uint32_t pool,
                        float lr, cudaStream_t s, tr_stats& stats);

}  // namespace tri

namespace trh {
// Four-child node as the traversal reads it (128 bytes): per axis and child the box's lower and
// upper plane side by side, so one packed multiply-add gives both distances, then the child refs
// as in GpuNode.  An empty slot's planes are all at the largest float: the slab test never passes.
struct alignas(32) DevNode {
    float plane[3][4][2];
    int32_t child[4];
    int32_t pad[4];
};
static_assert(sizeof(DevNode) == 128, "node must be 128 bytes");
// Figures of a device build (its nodes and leaf order stay on the device).
struct DeviceBvh {
    uint32_t nodes = 0;          // four-child nodes
    uint32_t depth = 0;          // four-child levels on the deepest path
    uint32_t stack = 0;          // traversal stack entries a ray can need
    uint32_t binary_depth = 0;
    uint32_t leaves = 0;
    double build_ms = 0.0;
    float vlo[3], vhi[3];        // box of all vertices
};
// Binned-SAH build on the device (bvh_gpu.cu) from device-resident vertices [nv][3] and
// triangles [nt][3], collapsed to four-child nodes as build_bvh does: the nodes go to
// alloc_nodes(count), the triangle ids in leaf order to d_order [nt].  False on invalid input or
// a one-leaf scene (the host builder then builds, or reports which index or vertex is wrong).
bool build_bvh_device(const float* d_vertices, uint32_t nv, const uint32_t* d_triangles, uint32_t nt,
                      uint32_t max_leaf, cudaStream_t s, const std::function<DevNode*(size_t)>& alloc_nodes,
                      uint32_t* d_order, DeviceBvh& out);
}  // namespace trh
