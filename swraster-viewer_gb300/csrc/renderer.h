// Host runtime of the per-frame renderer: draw-list construction, device
// buffer management, exposure state (Renderer, src/renderer.rs:144-198).
#pragma once

#include <cuda_runtime.h>

#include <atomic>
#include <cstdint>
#include <deque>
#include <memory>
#include <string>
#include <vector>

#include "../../include/swr.h"
#include "internal.h"
#include "scene.h"

namespace swr {

// Grow-only device buffer.
struct DBuf {
    void* p = nullptr;
    size_t bytes = 0;
    // A graph that the caller captured holds this address and may be launched
    // at any time: a buffer that grows past it keeps it until release().
    bool in_graph = false;
    std::vector<void*> outgrown;
    cudaError_t ensure(size_t n) {
        if (n <= bytes) return cudaSuccess;
        if (p && in_graph) outgrown.push_back(p);
        else if (p) cudaFree(p);
        p = nullptr;
        bytes = 0;
        in_graph = false;
        size_t want = n + n / 4;
        cudaError_t e = cudaMalloc(&p, want);
        if (e == cudaSuccess) bytes = want;
        return e;
    }
    void release() {
        if (p) cudaFree(p);
        for (void* o : outgrown) cudaFree(o);
        outgrown.clear();
        p = nullptr;
        bytes = 0;
        in_graph = false;
    }
    template <typename T>
    T* as() const { return static_cast<T*>(p); }
};

// Pinned host staging buffer.
struct HBuf {
    void* p = nullptr;
    size_t bytes = 0;
    cudaError_t ensure(size_t n) {
        if (n <= bytes) return cudaSuccess;
        if (p) cudaFreeHost(p);
        p = nullptr;
        bytes = 0;
        size_t want = n + n / 4 + 256;
        cudaError_t e = cudaHostAlloc(&p, want, cudaHostAllocDefault);
        if (e == cudaSuccess) bytes = want;
        return e;
    }
    void release() {
        if (p) cudaFreeHost(p);
        p = nullptr;
        bytes = 0;
    }
};

// Table region layout (host staging and device copy use the same offsets).
struct TableLayout {
    // Staged from the host each frame: [0, staged). Device-written after it:
    // per node slot counts and offsets, draws, chunks.
    size_t o_dyn = 0, o_scenes = 0, o_views = 0, o_order = 0, staged = 0;
    size_t o_slots = 0, o_draws = 0, o_chunks = 0, total = 0;
};
TableLayout table_layout(uint32_t scene_cap, uint32_t view_cap, uint32_t order_cap, uint32_t draw_cap,
                         uint32_t chunk_cap);

// Byte offsets of FrameEngine::tile_block.
struct TileLayout {
    size_t o_count, o_offset, o_cursor, o_work, o_sky, o_wide, total;
    TileLayout(uint32_t stile_cap, uint32_t view_cap) {
        auto al = [](size_t x) { return (x + 255) & ~size_t(255); };
        const size_t bins = al((size_t)(stile_cap + 1) * sizeof(uint32_t));
        o_count = 0;
        o_offset = bins;
        o_cursor = 2 * bins;
        o_work = 3 * bins;
        o_sky = o_work + al((size_t)(stile_cap / 2 + 1) * sizeof(uint4));
        o_wide = o_sky + al((size_t)view_cap * 256);
        total = o_wide + 2u * kWideCap * sizeof(uint2);
    }
};

// Reusable frame engine: everything a batch of views needs on the device.
// prepare() builds the per-frame tables on the host and grows capacities;
// launch() uploads the tables with one copy and runs the frame, either as
// direct launches or by replaying a CUDA graph captured for the current
// capacities (every per-frame count is read from the device table header).
struct FrameEngine {
    int num_sms = 148;
    uint32_t sched_tile = 64;
    uint64_t bin_cap = 0, extra_cap = 0;
    uint32_t scene_cap = 0, view_cap = 0, order_cap = 0, draw_cap = 0, chunk_cap = 0, tri_cap = 0, stile_cap = 0,
             quad_cap = 0;
    uint32_t pixel_cap = 0;
    uint64_t key_cap = 0;
    uint32_t raster_grid = 0, shade_grid = 0, grid_tile = 0;
    uint32_t raster_cta_cap = 0, grid_cap = 0;  // raster CTAs per SM (0: as many as fit; batch autotuner's choice)
    bool fuse32 = false;        // 32-px tiles shade inside the raster kernel (batch autotuner's choice)
    bool grid_fused32 = false, grid_narrow = false;
    // 32-px tiles shaded apart are rasterized by CTAs of 128 threads, not 256,
    // from kNarrowTiles tiles per SM on, and from kNarrowLow on where
    // kCrowdedTris triangles (of the scenes, drawn or not) come to a tile. With
    // few tiles the kernel waits for the heaviest ones, and those take the narrow
    // CTAs longer; with many, less of a CTA waits at each round's barriers. us of
    // a frame or batch with 256 -> 128 threads at so many tiles an SM: spheres of
    // 82k triangles before a sky 12: 155 -> 177, 24: 166 -> 180, 38: 344 -> 355,
    // 54: 382 -> 378, 126: 930 -> 910, 358: 2,399 -> 2,327; of 307k 12: 202 ->
    // 243, 54: 430 -> 450, 126: 1,231 -> 1,207; pictures filled by 400k triangles
    // 13: 381 -> 379, 24: 478 -> 457, 54: 715 -> 679, 126: 1,712 -> 1,617. With
    // 128 below 44 some light ones were slower than they had been before these
    // CTAs and that culling (30k triangles in twelve views of 640x480, 25: 198,
    // 194 with 256 and 206 with 128). Crowded tiles, 256 -> 128:
    // filled pictures of 1920x1080 gain (700k triangles 459 -> 442, 1.5M 584 ->
    // 549), spheres lose (1.2M 250 -> 288). The server's batches, beside which
    // others run, take the lower line (a burst of six frames of 54k triangles 322
    // -> 307). A capped CTA count keeps 256.
    static constexpr uint32_t kNarrowTiles = 44, kNarrowLow = 12;
    static constexpr uint64_t kCrowdedTris = 176;
    // Triangles (of the scenes, drawn or not) per tile from which 16-px tiles
    // are culled. Device time of a frame without -> with culling: 1.5M at
    // 640x400 (938 a tile) 739 -> 407 us, 1M at 1280x720 (260) 531 -> 411,
    // 60k at 480x300 (94) 121 -> 117, 150k at 1280x720 (39) 215 -> 218, 82k
    // (21) 98 -> 101.
    static constexpr uint64_t kCullTris = 64;
    // The engine's launches usually run beside other streams' (the server's
    // batches): a CTA that needs a whole SM would wait there until one is empty
    // (24 requests 1,137 us with k_shade in such CTAs, 1,088 without).
    bool shares_device = false;
    // Pixels per SM (in rounds of 1,024) from which k_shade takes one CTA an SM.
    // Also where the caller has two streams: frames on two streams 4K 662 -> 628
    // us, 2560x1440 448 -> 430, three of 1600x900 275 -> 272, but four of
    // 1920x1080 63 -> 65 where most is sky.
    static constexpr uint64_t kWideShadeRounds = 4;
    // A renderer's first frame waits for each allocation: the three records of a
    // triangle are one (rec_s, rec_r, rec_t by slots), and the buffers sized by
    // tiles and views are one (TileLayout).
    DBuf tables, tri_state, records, fan_base, clip_queue, tile_block;
    DBuf bins, keys, counters, rsqrt_tab;
    DBuf color;                // linear colour of views that need it (padded tile grids)
    bool defer_resolve = false;// the caller resolves (renderer frames with dt > 0)
    static constexpr int kStageRing = 4;
    static constexpr uint64_t kTriCapFromBound = 8u << 20;  // record slots sized from scene bounds, at most
    HBuf h_stage[kStageRing];  // pinned staging of the per-frame tables, one per frame in flight
    std::vector<uint32_t> h_order;  // per-frame node order of every view (capacity kept)
    TableLayout lay;
    cudaEvent_t stage_done[kStageRing] = {};
    bool stage_pending[kStageRing] = {};
    int stage_slot = 0;
    uint32_t retries = 0;
    uint64_t kernel_launches = 0;  // kernels enqueued (graph replays count the graph's kernels)
    DCounters last{};
    DFrameDyn dyn{};
    FrameArgs args{};
    // Graph replay.
    bool use_graph = false;
    // Renderer frames: capture once a frame's arguments (pointers, capacities,
    // kernel variants) have stayed the same for kGraphAfter frames, so that
    // neither a first frame nor alternating scenes pay for a capture.
    bool auto_graph = false;
    static constexpr uint32_t kGraphAfter = 4;
    uint32_t same_frames = 0;
    FrameArgs prev_args{};
    // One graph for each form of the raster and shading kernels: batches of
    // one engine vary in size.
    cudaGraphExec_t graph_exec[4] = {};
    FrameArgs graph_args[4] = {};
    uint32_t graph_kernels[4] = {};  // kernels in the captured graph
    cudaStream_t graph_stream = nullptr;
    cudaStream_t capture_stream = nullptr;  // legacy default streams cannot be captured

    // Staging buffers of frames that a caller captured: the graph's upload reads
    // its buffer at every launch, so the buffer leaves the ring until the graph
    // is gone (its user object tells) or the engine is released.
    struct GraphStage {
        HBuf buf;
        std::shared_ptr<std::atomic<bool>> gone;
    };
    std::vector<GraphStage> graph_stages;
    template <typename F>
    void each_buffer(F f) {
        for (DBuf* b : {&tables, &tri_state, &records, &fan_base, &clip_queue, &tile_block, &bins, &keys, &counters,
                        &rsqrt_tab, &color})
            f(*b);
    }
    void keep_for_graph(cudaStream_t stream, int slot);

    swr_status init(std::string& err);
    // Grows what a frame's counters report as overflowed (bins, clip slots)
    // or, when a tile held too many translucent packets, halves the
    // scheduling tile; SWR_OVERFLOW when nothing is left to grow.
    swr_status grow_for(const DCounters& c, std::string& err);
    void release();
    // captured: the caller captures the stream (stream_captured), so nothing
    // here waits for what is enqueued, nothing is freed, and what the frame
    // reads stays as it is.
    swr_status prepare(const std::vector<const SceneImpl*>& scenes, std::vector<DView>& views,
                       const std::vector<const swr_camera*>& cams, bool captured, std::string& err);
    swr_status launch(cudaStream_t stream, bool captured, cudaEvent_t* ev, std::string& err);
    // prepare + launch (the plain renderer's path).
    swr_status run(const std::vector<const SceneImpl*>& scenes, std::vector<DView>& views,
                   const std::vector<const swr_camera*>& cams, cudaStream_t stream, bool captured, FrameArgs* out_args,
                   std::string& err, cudaEvent_t* ev = nullptr);
};

// Whether the caller is capturing the stream.
bool stream_captured(cudaStream_t stream);

// While a caller's capture is fed: its mode may forbid this thread the queries
// and allocations that a frame makes beside its launches; they touch nothing
// that is captured, so they are made in relaxed mode.
struct CaptureGuard {
    bool on;
    cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
    explicit CaptureGuard(bool captured) : on(captured) {
        if (on) cudaThreadExchangeStreamCaptureMode(&mode);
    }
    ~CaptureGuard() {
        if (on) cudaThreadExchangeStreamCaptureMode(&mode);
    }
    CaptureGuard(const CaptureGuard&) = delete;
    CaptureGuard& operator=(const CaptureGuard&) = delete;
};

// compute_nodes_by_distance (src/renderer.rs:201-210): appends the scene's
// node indices, nearest first, to `out`.
void sort_nodes_by_distance(const SceneImpl& s, const swr_camera& cam, std::vector<uint32_t>& out);

// Fill the view-geometry fields of a DView (tiles, pitches, camera).
void init_view(DView& v, const swr_camera& cam, int32_t width, int32_t height, uint32_t sched_tile);

// Scheduling tile for views of the given sizes when the caller leaves it to
// the library: 64 where that gives the raster kernel at least 8 tiles per SM,
// else 32 where that gives it at least 7, else 16.
uint32_t auto_sched_tile(const int32_t* widths, const int32_t* heights, int32_t n, int num_sms);

// Sets the calling thread's swr_last_error() message.
void set_last_error(const char* msg);

// update_auto_exposure (src/renderer.rs:258-290).
struct ExposureState {
    float exposure = 2.0f;
    float target = 2.0f;
    float ev = 1.0f;  // log2(2.0)
    void update(const float* tile_lum, size_t n, float dt);
};

}  // namespace swr

struct swr_renderer {
    int32_t width = 0, height = 0;
    swr_renderer_opts opts{};
    swr::FrameEngine eng;
    swr::DBuf rgba8, vis, tile_lum;
    // Host memory the shading pass also writes RGBA8 into
    // (swr_renderer_set_blit_target): the caller's pointer, the address the
    // device uses for it, its row pitch in pixels; and the target the last
    // enqueued frame was rendered into.
    uint32_t* blit_target = nullptr;
    uint32_t* blit_target_dev = nullptr;
    size_t blit_stride = 0;
    uint32_t* frame_target = nullptr;
    size_t frame_stride = 0;
    swr::ExposureState expo;
    // Mapped pinned memory for the dt > 0 exposure step.
    float* h_lum = nullptr;
    float* h_expo = nullptr;
    float* d_expo = nullptr;
    cudaEvent_t expo_done = nullptr;
    bool expo_pending = false;
    // What the exposure callback of a frame advances: one step for frames in
    // flight (a frame waits for the step before it), and one for each dt that a
    // caller captured, which its graph's launches read again.
    struct ExposureStep {
        swr_renderer* r;
        float dt;
    };
    ExposureStep step{};
    std::deque<ExposureStep> graph_steps;
    // Last frame, kept for overflow re-runs.
    const swr_scene* last_scene = nullptr;
    swr_camera last_cam{};
    float last_dt = 0.0f;
    cudaStream_t last_stream = nullptr;
    bool have_frame = false;
    bool checked = true;
    // Counters of the last frame, copied back asynchronously so the next
    // frame can adapt capacities without waiting for this one.
    swr::DCounters* h_counters = nullptr;
    cudaEvent_t status_ev = nullptr;
    bool status_pending = false;
    swr::FrameArgs last_args{};
    uint32_t tiles_x = 0, tiles_y = 0;
    // Stage profiling: a ring of event sets, one per in-flight frame.
    static constexpr int kProfRing = 64;
    bool profiling = false;
    cudaEvent_t prof_ev[kProfRing][10] = {};
    bool prof_pending[kProfRing] = {};
    bool prof_resolve[kProfRing] = {};
    int prof_next = 0;
    double prof_ms[SWR_STAGES] = {};
    uint32_t prof_frames = 0;
};
