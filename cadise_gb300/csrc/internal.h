// Library-internal state behind the C ABI (not installed, not part of the ABI).
#pragma once

#include "../../include/cadise_gpu.h"
#include "scene_device.cuh"

#include <cuda_runtime.h>

#include <string>
#include <vector>

namespace cg {

// One render chunk: samples [sample0, sample0 + nsamples) of every pixel of
// one scene; its paths occupy [path_begin, path_begin + npix * nsamples) of
// the batch, sample-major (path = path_begin + s * npix + pixel).
struct Chunk {
    int scene;
    uint32_t path_begin;
    uint32_t npix;
    uint32_t width;
    uint32_t sample0;
    uint32_t nsamples;
    uint32_t pix_begin;  // prefix over chunks of npix (film splat index space)
    uint32_t pixel0;     // first pixel of the scene in this chunk (0 but for the adjoint's frames in parts)
};
constexpr int kMaxChunks = 256;

struct BatchHeader {
    uint32_t num_chunks;
    uint32_t total_paths;
    uint32_t total_pixels;
    int max_depth;
    uint64_t seed;
};

struct FilmD {
    double* sum;    // 3 per pixel
    double* sumsq;  // 3 per pixel
    double* count;  // 1 per pixel
};

// Counters per bounce b at cnt[b * kCntStride + k]:
//   k = 0 continuation rays to extend, 1 unused, 2 shadow rays,
//   3 + kind: hits waiting for the shade kernel of that BSDF kind,
//   8 / 9: rays handed out so far by the persistent extend / shadow kernels,
//   10: unused,
//   11: MIS rays whose direction meets the sampled light's primitive (or that
//       sampled the environment), left for the MIS occlusion pass,
//   12: closest-hit rays of the persistent pass left for k_wf_ties (q_tie).
constexpr int kCntStride = 16;

struct WfBuffers {
    // L.w and Ls.w hold the sample's film position (x, y) for the film filter;
    // the passes update L and Ls in place and leave .w as it is.
    float4 *ray_o, *ray_d, *hit, *thr, *L, *Ls, *mis_a, *mis_b, *mis_d, *sh_d, *sh_c;
    // Sky radiance picked up by an escaped continuation ray.  Kept apart from
    // L: the MIS ray of the same path's last vertex adds to L in the same
    // extend pass.  A path sample is (L + Le) + Ls.
    float4* Le;
    // MIS ray resolved against its light at the vertex: (t, record slot, u, v)
    // of the light's hit, slot -1 for the environment.
    float4* mis_h;
    uint4* meta;      // scene, pixel, sample, rng counter
    int* q_cont[2];
    int* q_mis[2];    // laid out, not used: a MIS ray that meets its light goes to q_mocc
    int* q_shadow[2];
    int* q_mocc[2];   // MIS occlusion queries, ping-pong on the bounce
    int* q_mat[kNumBsdfKinds];
    // closest-hit rays whose persistent traversal met two primitives within
    // the tie reach (persistent_pass), for k_wf_ties: paths
    int* q_tie;
    int* cnt;
    int cnt_depth;    // bounces the counter array covers
};

// Lays the path state of `cap` paths and the counters of `cnt_rows` bounces
// out from `base` (256-byte aligned arrays) and returns the bytes used.  With
// base == nullptr it only measures: the allocation is sized by the same walk
// that carves it.
inline size_t wf_layout(char* base, size_t cap, int cnt_rows, WfBuffers* w) {
    size_t off = 0;
    auto take = [&](size_t bytes) {
        char* r = base ? base + off : nullptr;
        off += (bytes + 255) & ~size_t(255);
        return r;
    };
    float4** f4s[] = {&w->ray_o, &w->ray_d, &w->hit, &w->thr, &w->L, &w->Le, &w->Ls,
                      &w->mis_a, &w->mis_b, &w->mis_d, &w->mis_h, &w->sh_d, &w->sh_c};
    for (float4** f : f4s) *f = reinterpret_cast<float4*>(take(cap * sizeof(float4)));
    w->meta = reinterpret_cast<uint4*>(take(cap * sizeof(uint4)));
    for (int k = 0; k < 2; ++k) {
        w->q_cont[k] = reinterpret_cast<int*>(take(cap * sizeof(int)));
        w->q_mis[k] = reinterpret_cast<int*>(take(cap * sizeof(int)));
        w->q_shadow[k] = reinterpret_cast<int*>(take(cap * sizeof(int)));
        w->q_mocc[k] = reinterpret_cast<int*>(take(cap * sizeof(int)));
    }
    for (int k = 0; k < kNumBsdfKinds; ++k) w->q_mat[k] = reinterpret_cast<int*>(take(cap * sizeof(int)));
    w->q_tie = reinterpret_cast<int*>(take(cap * sizeof(int)));
    w->cnt = reinterpret_cast<int*>(take(size_t(cnt_rows) * kCntStride * sizeof(int)));
    w->cnt_depth = cnt_rows;
    return off;
}

// Static scratch of cgpu_render_noalloc: every device buffer of that call
// lives in one file-scope array of kNoAllocScratchBytes, laid out by
// noalloc_layout.  Limits: a frame of at most kNoAllocMaxPaths pixels (one
// path per pixel per batch), max_depth <= kNoAllocMaxDepth, scene ids below
// kNoAllocMaxScenes (the scene and film tables are indexed by scene id).
constexpr uint32_t kNoAllocMaxPaths = 1u << 18;
constexpr int kNoAllocMaxDepth = 62;
constexpr int kNoAllocMaxScenes = 64;
constexpr size_t kNoAllocScratchBytes = size_t(80) << 20;

struct NoAllocView {
    BatchHeader* header;
    Chunk* chunk;
    SceneD* scenes;               // kNoAllocMaxScenes entries
    FilmD* films;                 // kNoAllocMaxScenes entries
    unsigned long long* counters; // 8
    WfBuffers wf;                 // kNoAllocMaxPaths paths, kNoAllocMaxDepth + 2 counter rows
};

inline size_t noalloc_layout(char* base, NoAllocView* v) {
    size_t off = 0;
    auto take = [&](size_t bytes) {
        char* r = base ? base + off : nullptr;
        off += (bytes + 255) & ~size_t(255);
        return r;
    };
    v->header = reinterpret_cast<BatchHeader*>(take(sizeof(BatchHeader)));
    v->chunk = reinterpret_cast<Chunk*>(take(sizeof(Chunk)));
    v->scenes = reinterpret_cast<SceneD*>(take(sizeof(SceneD) * kNoAllocMaxScenes));
    v->films = reinterpret_cast<FilmD*>(take(sizeof(FilmD) * kNoAllocMaxScenes));
    v->counters = reinterpret_cast<unsigned long long*>(take(8 * sizeof(unsigned long long)));
    return off + wf_layout(base ? base + off : nullptr, kNoAllocMaxPaths, kNoAllocMaxDepth + 2, &v->wf);
}

// Wavefront adjoint (path replay in wavefront form): per path the radiance of
// the whole path from the forward pass (Ltot) and of the vertices replayed so
// far (acc); per path and bounce what the forward pass's rays found, so that
// the replay traces none: the hit, the shade queues, and a byte each for the
// shadow ray and the MIS ray (1: nothing in the way).
struct AdjBufs {
    float4 *Ltot, *acc;
    const float* dLdI;      // d loss / d pixel, 3 per pixel
    double* g_tex;
    const int* tex_offset;  // per texture: first float of its block in g_tex
    double* g_rough;        // per material
    double* g_rad;          // 3 per area light
    int nmat, nlight;
    float inv_spp;
};

// The records of one batch: arrays of `depth` rows, one entry per path in each.
struct AdjRecords {
    size_t stride = 0;  // entries a row
    int depth = 0;
    float4* hit = nullptr;
    int* q_mat[kNumBsdfKinds] = {};
    uint8_t *shadow = nullptr, *mis = nullptr;
};

// Bytes of records a path takes.
inline size_t adj_record_bytes(uint32_t kinds, int depth) {
    size_t row = sizeof(float4) + 2;
    for (int k = 0; k < kNumBsdfKinds; ++k) row += (kinds >> k & 1u) * sizeof(int);
    return row * size_t(depth > 0 ? depth : 1);
}

inline size_t adj_layout(char* base, size_t paths, uint32_t kinds, int depth, AdjBufs* a, AdjRecords* r) {
    size_t off = 0;
    auto take = [&](size_t bytes) {
        char* q = base ? base + off : nullptr;
        off += (bytes + 255) & ~size_t(255);
        return q;
    };
    r->stride = paths;
    r->depth = depth > 0 ? depth : 1;
    const size_t n = paths * size_t(r->depth);
    a->Ltot = reinterpret_cast<float4*>(take(paths * sizeof(float4)));
    a->acc = reinterpret_cast<float4*>(take(paths * sizeof(float4)));
    r->hit = reinterpret_cast<float4*>(take(n * sizeof(float4)));
    for (int k = 0; k < kNumBsdfKinds; ++k) r->q_mat[k] = kinds >> k & 1u ? reinterpret_cast<int*>(take(n * sizeof(int))) : nullptr;
    r->shadow = reinterpret_cast<uint8_t*>(take(n));
    r->mis = reinterpret_cast<uint8_t*>(take(n));
    return off;
}

struct RenderArgs {
    const SceneD* scenes;
    const Chunk* chunks;
    const BatchHeader* header;
    FilmD* films;     // per scene id
    WfBuffers wf;
    unsigned long long* counters;  // closest rays, any rays, nodes, tris, paths
    AdjBufs adj;      // wavefront adjoint only
    // wavefront adjoint: where the passes record (forward) or find (replay) the
    // outcome of one bounce's shadow and MIS rays; null in other renders
    uint8_t *rec_shadow, *rec_mis;
    // reordered closest-hit queue (tuning.reorder): paths
    const uint32_t* sorted;
    // persistent traversal passes: a warp refills its finished lanes once
    // fewer than this many of its lanes still trace (cgpu_tuning)
    int refill_closest, refill_any;
};

// Where the tuning leaves the traversal variant open (traversal 0), the
// persistent passes take batches of kLargeBatch paths through scenes of
// kSmallScene records or more (ms a frame of depth 8, one ray per thread /
// persistent: 2,457,600 paths through 960 triangles 2.83 / 2.99, 3,200 3.78 / 3.73,
// 12,800 4.33 / 4.05, 204,800 6.99 / 5.84; 921,600 through 102,400 2.75 / 2.51).
// Elsewhere one ray per thread, whose three passes of a bounce are one launch, is
// the faster one: 262,144 paths through 960 triangles 0.78 / 0.90, 204,800 1.45 /
// 1.58; 12,288 paths 0.60 / 0.63 and 0.95 / 0.96; an adjoint iteration of 96,520
// paths through 3,842 triangles 1.12 / 1.37; the allocation-free render 0.75 /
// 1.05, always by that one.
constexpr int kSmallScene = 2048;
constexpr uint64_t kLargeBatch = 1u << 19;

// The kernels of a traversal variant (cgpu_tuning::traversal): 0 one ray per
// thread, 1 persistent with ray replacement, 2 / 3 the persistent passes.
// `persistent`: what the library would choose where the tuning leaves it open.
constexpr int kTraversalOpen = 0, kTraversalPerRay = 4;
inline int traversal_kernels(int traversal, bool persistent) {
    return traversal == kTraversalPerRay ? 0 : traversal == kTraversalOpen && persistent ? 3 : traversal;
}

// The refill thresholds of a tuning, 0 replaced by the default.
constexpr int kDefaultRefillLanes = 24;
inline int refill_lanes(int32_t v) { return v > 0 ? v : kDefaultRefillLanes; }

// cgpu_autotune's search: whether it leaves candidate `t` of a pass out, because
// it runs the launches of `best`, which took the kernels `closest` and `any`.
enum { TUNE_TRAVERSAL, TUNE_BLOCK_TRACE, TUNE_BLOCK_SHADE, TUNE_MAX_PATHS, TUNE_REFILL_CLOSEST, TUNE_REFILL_ANY, TUNE_PASSES };
inline bool autotune_skips(int pass, const cgpu_tuning& t, const cgpu_tuning& best, int closest, int any) {
    switch (pass) {
        case TUNE_TRAVERSAL: return traversal_kernels(t.traversal, false) == closest && closest == any;
        case TUNE_BLOCK_TRACE: return t.block_trace == best.block_trace;
        case TUNE_BLOCK_SHADE: return t.block_shade == best.block_shade;
        case TUNE_MAX_PATHS: return t.max_paths == best.max_paths;
        case TUNE_REFILL_CLOSEST: return closest < 2 || refill_lanes(t.refill_closest) == refill_lanes(best.refill_closest);
        default: return any < 3 || refill_lanes(t.refill_any) == refill_lanes(best.refill_any);
    }
}

// Buffers of the ray reordering: keys / values ping-pong for 2 * path_cap
// queue entries, digit counts, scan scratch, the entry count.
struct SortBufs {
    uint32_t* keys[2];
    uint32_t* vals[2];
    uint32_t* hist;
    uint32_t* sums;
    uint32_t* n;
    uint32_t tiles;
};

}  // namespace cg

struct SceneSlot {
    bool live = false;
    cg::SceneD d{};
    // host copies of the differentiable tables (cgpu_params_get / _set)
    std::vector<cg::MaterialD> h_mats;
    std::vector<cg::LightD> h_lights;
    std::vector<cg::TextureD> h_texs;  // device texel pointers
    cg::MaterialD* d_mats = nullptr;
    cg::LightD* d_lights = nullptr;
    int num_area_lights = 0;  // h_lights[0, num_area_lights) are area lights
    std::vector<void*> allocations;
    cgpu_scene_info info{};
    cg::FilmD film{};
    int width = 0, height = 0, spp = 1, max_depth = 1;
    bool has_spheres = false;  // renders of this scene use the kernels with the sphere test
    uint32_t kinds = 0;        // bit k: a material of shade queue k
};

struct cgpu_ctx {
    int device = 0;
    cudaStream_t stream = nullptr;
    cudaStream_t side = nullptr;  // second stream for graph branches
    bool own_stream = false;
    std::string last_error;
    std::vector<SceneSlot> scenes;
    int num_sms = 0;
    bool counting = false;
    cgpu_tuning tuning{128, 128, 0, 0, 0, 0, 0};

    // device tables (rebuilt when the scene set changes)
    cg::SceneD* d_scenes = nullptr;
    cg::FilmD* d_films = nullptr;
    int table_cap = 0;
    bool tables_dirty = true;

    // batch description
    cg::Chunk* d_chunks = nullptr;
    cg::BatchHeader* d_header = nullptr;
    cg::Chunk* h_chunks = nullptr;        // pinned
    cg::BatchHeader* h_header = nullptr;  // pinned

    // per-path buffers
    uint32_t path_cap = 0;
    cg::WfBuffers wf{};
    void* wf_block = nullptr;
    // wavefront adjoint state (Ltot, acc, records), kept between calls up to a size (cg_adjoint_trim)
    // ray reordering buffers (allocated while tuning.reorder is on)
    uint32_t sort_cap = 0;
    cg::SortBufs sort{};
    void* sort_block = nullptr;
    size_t adj_bytes = 0;
    void* adj_block = nullptr;
    // gradient and image buffers of the adjoint calls (adjoint.cu)
    void* grad_block = nullptr;
    size_t grad_cap = 0;
    int adjoint_schedule = CGPU_MODE_WAVEFRONT;
    int bvh_builder = CGPU_BVH_BUILDER_AUTO;
    int tie_order = CGPU_TIE_ORDER_REFERENCE;
    unsigned long long* d_counters = nullptr;
    // device status word: rays whose traversal ran out of its visit budget
    // since the last check (cg_check_status); 0 = automatic budget per scene
    uint32_t* d_status = nullptr;
    uint32_t visit_budget = 0;

    // pinned stage of small host queries and the status word; device buffer of
    // larger ones (trace_host)
    char* h_stage = nullptr;
    void* query_block = nullptr;
    size_t query_cap = 0;

    // captured wavefront graphs: of one ray per thread and of persistent passes
    struct Graph {
        cudaGraphExec_t exec = nullptr;
        int depth = -1;
        uint32_t paths = 0;
        bool spheres = false;
        uint32_t kinds = 0;
        uint32_t launches = 0;  // kernel launches one replay makes
    } graphs[2];
    bool batch_spheres = false;  // a scene of the current render holds spheres
    uint32_t batch_kinds = 0;    // the shade queues of the current render's scenes
    int batch_closest = 0, batch_any = 0;  // its traversal variants (choose_traversal)

    cgpu_render_stats stats{};

    // per-kernel event timing (cgpu_set_profiling)
    bool profiling = false;
    struct ProfEvent { int cls; cudaEvent_t a, b; };
    std::vector<ProfEvent> prof;
    cgpu_kernel_times times{};
};

// implemented in render.cu
cgpu_status cg_render_batches(cgpu_ctx* ctx, const cgpu_render_params* p);
cgpu_status cg_adjoint_wavefront(cgpu_ctx* ctx, int scene, uint32_t spp, uint64_t seed, const cg::AdjBufs& params);
cgpu_status cg_render_paths_raw(cgpu_ctx* ctx, int scene, int mode, uint32_t first, uint32_t count, uint64_t seed,
                                float* host_rgb);
cgpu_status cg_path_radiance(cgpu_ctx* ctx, int scene, int mode, const double* film_xy, const uint64_t* keys,
                             uint32_t n, float* out_rgb);
cgpu_status cg_trace(cgpu_ctx* ctx, int scene, const cgpu_ray* d_rays, uint32_t n, cgpu_hit* d_hits,
                     uint8_t* d_occ, bool any);
cgpu_status cg_camera(cgpu_ctx* ctx, int scene, const double* d_xy, uint32_t n, float* d_out);
cgpu_status cg_film_clear(cgpu_ctx* ctx, int scene);
void cg_free_render_state(cgpu_ctx* ctx);
void cg_drop_graphs(cgpu_ctx* ctx);
// After a backward call: gives a large adjoint state back.
void cg_adjoint_trim(cgpu_ctx* ctx);

// implemented in api.cu
cgpu_status cg_fail(cgpu_ctx* ctx, cgpu_status s, const std::string& msg);
cgpu_status cg_cuda(cgpu_ctx* ctx, cudaError_t e, const char* what);
cgpu_status cg_sync_tables(cgpu_ctx* ctx);
void cg_prefault(void* p, size_t bytes);
// Waits for the context stream (an error is reported as `what`'s); then
// CGPU_ERR_TIMEOUT (and a reset count) if a traversal ran out of its visit
// budget.
cgpu_status cg_check_status(cgpu_ctx* ctx, const char* what);
