// Render kernels: the FP32 megakernel, the wavefront stages, the FP64 film
// splat and the batched ray-query / camera kernels behind the C ABI.
//
// Replaces SamplingRenderer::render + EstimatorTileWork::work
// (source/core/renderer/sampling/samplingRenderer.cpp:33-68,
// source/core/renderer/render-work/estimatorTileWork.cpp:32-61): instead of
// tiles over host threads, a batch holds every path sample of one or more
// scenes for a range of sample indices; each path is independent and owns a
// counter-based random stream keyed by (seed, scene, pixel, sample).
//
// Wavefront schedule of one batch (replayed as one CUDA graph):
//   generate -> for b in [0, max_depth): { extend(b), ties(b) || shadow(b), mis_occl(b) (per ray: all in one launch) ;
//               shade_k(b) for each BSDF kind that the scenes have }
//            -> extend(max_depth) .. mis_occl(max_depth) -> splat
// Queues hold path ids; per-path state lives in SoA arrays indexed by path.
// Queue appends are warp-aggregated (ballot / match + one atomic per group).
#include "film.cuh"
#include "internal.h"
#include "pathtrace.cuh"
#include "persist.cuh"
#include "radix.cuh"

#include <algorithm>
#include <cstring>
#include <mutex>
#include <string>

namespace cg {

// At 128 registers a quarter of an SM holds four warps, so that blocks of up to
// 512 threads launch (uncapped the counting variants take 136: 384 threads).
constexpr int kMegakernelRegs = 128;

template <bool COUNT, bool SPH>
__global__ void __maxnreg__(kMegakernelRegs) k_megakernel(RenderArgs a) {
    const BatchHeader h = *a.header;
    TraceCounters tc{0, 0}, ta{0, 0};
    uint32_t nc = 0, na = 0;
    for (uint32_t p = blockIdx.x * blockDim.x + threadIdx.x; p < h.total_paths; p += gridDim.x * blockDim.x) {
        const PathId id = path_id(a.chunks, int(h.num_chunks), p);
        const SceneD& S = a.scenes[id.scene];
        Rng rng;
        float3 o, d;
        float2 fxy;
        primary_ray(S, id, h.seed, rng, &o, &d, &fxy);
        float3 L, Le, Ls;
        mk_path<COUNT, SPH>(S, o, d, rng, &L, &Le, &Ls, &tc, &ta, &nc, &na);
        a.wf.L[p] = make_float4(L.x, L.y, L.z, fxy.x);
        a.wf.Le[p] = make_float4(Le.x, Le.y, Le.z, 0.0f);
        a.wf.Ls[p] = make_float4(Ls.x, Ls.y, Ls.z, fxy.y);
    }
    count_flush<COUNT>(a.counters, tc, ta, nc, na);
}

// Per-path estimate for explicit film positions and keys (stream from draw 0).
__global__ void k_paths_explicit(const SceneD* scenes, int scene, const double* xy, const uint64_t* keys, uint32_t n,
                                 float* out) {
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const SceneD& S = scenes[scene];
        Rng rng;
        rng.key = keys[i];
        rng.ctr = 0;
        float3 o, d;
        camera_ray(S.cam, float(xy[2 * i]), float(xy[2 * i + 1]), &o, &d);
        float3 L, Le, Ls;
        TraceCounters tc{0, 0}, ta{0, 0};
        uint32_t nc = 0, na = 0;
        mk_path<false>(S, o, d, rng, &L, &Le, &Ls, &tc, &ta, &nc, &na);
        const float3 v = path_sample(L, Le, Ls);
        out[3 * i + 0] = v.x;
        out[3 * i + 1] = v.y;
        out[3 * i + 2] = v.z;
    }
}

// ---------------------------------------------------------------- wavefront --
__global__ void k_wf_generate(RenderArgs a) {
    const BatchHeader h = *a.header;
    const WfBuffers& w = a.wf;
    for (uint32_t p = blockIdx.x * blockDim.x + threadIdx.x; p < h.total_paths; p += gridDim.x * blockDim.x) {
        const PathId id = path_id(a.chunks, int(h.num_chunks), p);
        const SceneD& S = a.scenes[id.scene];
        Rng rng;
        float3 o, d;
        float2 fxy;
        primary_ray(S, id, h.seed, rng, &o, &d, &fxy);
        w.ray_o[p] = make_float4(o.x, o.y, o.z, 0.0f);
        w.ray_d[p] = make_float4(d.x, d.y, d.z, 0.0f);
        w.thr[p] = make_float4(1.0f, 1.0f, 1.0f, __int_as_float(1));
        w.L[p] = make_float4(0.0f, 0.0f, 0.0f, fxy.x);
        w.Le[p] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        w.Ls[p] = make_float4(0.0f, 0.0f, 0.0f, fxy.y);
        w.meta[p] = make_uint4(uint32_t(id.scene), id.pixel, id.sample, rng.ctr);
        w.q_cont[0][p] = int(p);
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) w.cnt[0] = int(h.total_paths);
}

// Append `p` to queue `key` (key < 0: no append); one atomic per group of
// lanes sharing a key.
CG_D void grouped_push(int* const* queues, int* counters, int key, int p) {
    const unsigned active = __activemask();
    const unsigned grp = __match_any_sync(active, key);
    const int lane = threadIdx.x & 31;
    const int leader = __ffs(grp) - 1;
    int base = 0;
    if (lane == leader && key >= 0) base = atomicAdd(counters + key, __popc(grp));
    base = __shfl_sync(grp, base, leader);
    if (key >= 0) queues[key][base + __popc(grp & ((1u << lane) - 1u))] = p;
}

// After the closest-hit trace of path p's continuation ray: a hit is stored
// and its path joins the shade queue of the material; an escaped ray picks up
// the sky.  The queue comes with the record (kind), not by way of the
// material table: two dependent loads less at the few lanes that finish
// together (closest-hit passes of the 1 M-triangle frame 34.5 -> 34.2 ms).
CG_D void extend_finish(const WfBuffers& w, const SceneD& S, int* counters, int p, float t, int slot, int kind) {
    if (slot >= 0) {
        __stcs(&w.hit[p], make_float4(t, __int_as_float(slot), 0.0f, 0.0f));
    } else if (S.env_light >= 0) {
        const float4 tw = w.thr[p];
        if (__float_as_int(tw.w) & 1) {
            const float3 e = f3(tw) * env_radiance(S, f3(w.ray_d[p]));
            w.Le[p] = make_float4(e.x, e.y, e.z, 0.0f);
        }
    }
    grouped_push(w.q_mat, counters, kind, p);
}

// The shade queue of a record's material.
CG_D int kind_of_slot(const SceneD& S, int slot) {
    return slot < 0 ? -1 : int(__float_as_uint(ldg4(reinterpret_cast<const float4*>(S.tris + slot) + 2).w) >> kRecQueueShift);
}

// What an unoccluded MIS ray from o along d adds that meets its light at mh
// (mis_light_hit; mh.y: record, -1 the environment).  X (optional): its
// derivative by the light's radiance.
CG_D float3 mis_add(const SceneD& S, float3 o, float3 d, float4 mh, float3 T, float3 factor, float pdf, float3* X) {
    HitD hit;
    hit.t = mh.x;
    hit.slot = __float_as_int(mh.y);
    hit.u = mh.z;
    hit.v = mh.w;
    if (hit.slot < 0) return mis_resolve_env(S, d, T, factor, pdf);
    return mis_resolve(S, surface_at(S, o, d, hit), o, T, factor, pdf, X);
}

// MIS rays that meet their light (mis_light_hit): unless a primitive comes
// before the light's hit, the BSDF-sampling half of the NEE estimate, added to
// L (and recorded for the adjoint's replay).
template <bool COUNT, bool SPH>
CG_D void mis_rays(const RenderArgs& a, int b, int first, int step) {
    const WfBuffers& w = a.wf;
    const int n = w.cnt[b * kCntStride + 11];
    const int* q = w.q_mocc[b & 1];
    TraceCounters tc{0, 0};
    uint32_t nany = 0;
    for (int i = first; i < n; i += step) {
        const int p = q[i];
        const SceneD& S = a.scenes[w.meta[p].x];
        const RayPre r = ray_prep(f3(w.ray_o[p]), f3(w.mis_d[p]), kRayEps, kFloatMax);
        const float4 mh = w.mis_h[p];
        const int slot = __float_as_int(mh.y);
        const int prim_l = slot >= 0 ? __float_as_int(ldg4(reinterpret_cast<const float4*>(S.tris + slot)).w) : 0x7FFFFFFF;
        if (COUNT) ++nany;
        const bool occluded = occluded_before<COUNT, SPH>(S, r, mh.x, prim_l, slot, &tc);
        if (a.rec_mis) a.rec_mis[p] = occluded ? 0 : 1;
        if (occluded) continue;
        const float4 mb = w.mis_b[p], ma = w.mis_a[p];
        const float3 add = mis_add(S, r.o, r.d, mh, f3(mb), f3(ma), ma.w, nullptr);
        float4 L = w.L[p];
        L.x += add.x;
        L.y += add.y;
        L.z += add.z;
        w.L[p] = L;
    }
    count_flush<COUNT>(a.counters, TraceCounters{0, 0}, tc, 0, nany);
}

template <bool COUNT, bool SPH>
__global__ void k_wf_mis_occl(RenderArgs a, int b) {
    mis_rays<COUNT, SPH>(a, b, blockIdx.x * blockDim.x + threadIdx.x, gridDim.x * blockDim.x);
}

// After the trace of path p's shadow ray (rec: recorded for the adjoint's replay).
CG_D void shadow_finish(const WfBuffers& w, uint8_t* rec, int p, bool occluded) {
    if (rec) rec[p] = occluded ? 0 : 1;
    if (occluded) return;
    const float4 c = w.sh_c[p];
    float4 Ls = w.Ls[p];
    Ls.x += c.x;
    Ls.y += c.y;
    Ls.z += c.z;
    w.Ls[p] = Ls;
}

CG_D uint32_t spread9(uint32_t v) {
    uint32_t x = v & 0x1FFu;
    x = (x | (x << 16)) & 0x030000FFu;
    x = (x | (x << 8)) & 0x0300F00Fu;
    x = (x | (x << 4)) & 0x030C30C3u;
    x = (x | (x << 2)) & 0x09249249u;
    return x;
}

// Sort keys of a closest-hit pass's queue (tuning.reorder): the direction's
// octant above the Morton code of the origin in the scene bounds (`bits` per
// axis, at most 9), so that sorted neighbours leave nearby points in similar
// directions.  Values: paths.  Writes the entry count for the sort.
__global__ void k_ray_keys(RenderArgs a, int b, int bits, uint32_t* keys, uint32_t* vals, uint32_t* n_out) {
    const WfBuffers& w = a.wf;
    const int* cnt = w.cnt + b * kCntStride;
    const int n = cnt[0];
    const int* qc = w.q_cont[b & 1];
    if (blockIdx.x == 0 && threadIdx.x == 0) *n_out = uint32_t(n);
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const int p = qc[i];
        const float3 o = f3(w.ray_o[p]), d = f3(w.ray_d[p]);
        const SceneD& S = a.scenes[w.meta[p].x];
        const float u[3] = {(o.x - S.bounds_lo.x) * S.bounds_inv.x, (o.y - S.bounds_lo.y) * S.bounds_inv.y,
                            (o.z - S.bounds_lo.z) * S.bounds_inv.z};
        const float cells = float((1 << bits) - 1);
        uint32_t q[3];
        for (int k = 0; k < 3; ++k) q[k] = uint32_t(fminf(fmaxf(u[k], 0.0f), 1.0f) * cells);
        const uint32_t oct = (d.x < 0.0f ? 4u : 0u) | (d.y < 0.0f ? 2u : 0u) | (d.z < 0.0f ? 1u : 0u);
        keys[i] = (oct << (3 * bits)) | (spread9(q[0]) << 2) | (spread9(q[1]) << 1) | spread9(q[2]);
        vals[i] = uint32_t(p);
    }
}

template <bool COUNT, bool SPH, bool SORTED = false>
CG_D void extend_rays(const RenderArgs& a, int b, int first, int step) {
    const WfBuffers& w = a.wf;
    int* cnt = w.cnt + b * kCntStride;
    const int n = cnt[0];
    const int* q = SORTED ? reinterpret_cast<const int*>(a.sorted) : w.q_cont[b & 1];
    TraceCounters tc{0, 0};
    uint32_t nclosest = 0;
    for (int i = first; i < n; i += step) {
        const int p = q[i];
        const SceneD& S = a.scenes[w.meta[p].x];
        const RayPre r = ray_prep(f3(w.ray_o[p]), f3(w.ray_d[p]), kRayEps, kFloatMax);
        HitD hit;
        if (COUNT) ++nclosest;
        if (!traverse_warp<COUNT, SPH>(S, r, &hit, &tc)) hit.slot = -1;
        extend_finish(w, S, cnt + 3, p, hit.t, hit.slot, kind_of_slot(S, hit.slot));
    }
    count_flush<COUNT>(a.counters, tc, TraceCounters{0, 0}, nclosest, 0);
}

template <bool COUNT, bool SPH, bool SORTED = false>
__global__ void k_wf_extend(RenderArgs a, int b) {
    extend_rays<COUNT, SPH, SORTED>(a, b, blockIdx.x * blockDim.x + threadIdx.x, gridDim.x * blockDim.x);
}

template <bool COUNT, bool SPH>
CG_D void shadow_rays(const RenderArgs& a, int b, int first, int step) {
    const WfBuffers& w = a.wf;
    const int n = w.cnt[b * kCntStride + 2];
    const int* q = w.q_shadow[b & 1];
    TraceCounters tc{0, 0};
    uint32_t nany = 0;
    for (int i = first; i < n; i += step) {
        const int p = q[i];
        const SceneD& S = a.scenes[w.meta[p].x];
        const float4 sd = w.sh_d[p];
        const RayPre r = ray_prep(f3(w.ray_o[p]), f3(sd), kRayEps, sd.w);
        HitD hit;
        if (COUNT) ++nany;
        shadow_finish(w, a.rec_shadow, p, traverse<true, COUNT, SPH>(S, r, &hit, &tc));
    }
    count_flush<COUNT>(a.counters, TraceCounters{0, 0}, tc, 0, nany);
}

template <bool COUNT, bool SPH>
__global__ void k_wf_shadow(RenderArgs a, int b) {
    shadow_rays<COUNT, SPH>(a, b, blockIdx.x * blockDim.x + threadIdx.x, gridDim.x * blockDim.x);
}

// The three ray passes of a bounce in one launch, for the render on one stream:
// they share no data, and one after the other each waits for the slowest ray of
// the one before.  Every third of the grid takes one pass, the closest hits (the
// longest) first.  (ms: allocation-free render of 320 x 181, 2 samples 1.06 ->
// 0.73.  Against closest hits on one stream beside the other two on a second:
// Cornell box, 256 x 256, 16 samples 1.16 -> 1.09; sphere box, 333 x 251, 9 samples
// 1.98 -> 1.88; adjoint iteration of 127 x 95, 8 samples 1.38 -> 1.10.)
template <bool SPH>
__global__ void k_wf_rays(RenderArgs a, int b) {
    const int third = gridDim.x / 3, pass = blockIdx.x / third;
    const int first = (blockIdx.x - pass * third) * blockDim.x + threadIdx.x, step = third * blockDim.x;
    if (pass == 0) extend_rays<false, SPH>(a, b, first, step);
    else if (pass == 1) shadow_rays<false, SPH>(a, b, first, step);
    else mis_rays<false, SPH>(a, b, first, step);
}

// Persistent variants: each lane takes rays from the queue through a
// warp-aggregated counter and, whenever its ray finishes, the next one, so no
// lane idles while the warp's longest ray is still traversing.
constexpr int kStepsPerFetch = 4;

// Hands the lanes in `need` consecutive entries of [0, n); returns this lane's
// entry or -1 when the queue is drained.
CG_D int warp_take(int* work, bool need, int n) {
    const unsigned mask = __activemask();
    const unsigned nb = __ballot_sync(mask, need);
    if (nb == 0) return -1;
    const int lane = threadIdx.x & 31;
    const int leader = __ffs(nb) - 1;
    int base = 0;
    if (lane == leader) base = atomicAdd(work, __popc(nb));
    base = __shfl_sync(mask, base, leader);
    if (!need) return -1;
    const int k = base + __popc(nb & ((1u << lane) - 1u));
    return k < n ? k : -1;
}

template <bool COUNT, bool SPH>
__global__ void k_wf_extend_dyn(RenderArgs a, int b) {
    const WfBuffers& w = a.wf;
    int* cnt = w.cnt + b * kCntStride;
    const int n = cnt[0];
    const int* q = w.q_cont[b & 1];
    TraceCounters tc{0, 0};
    uint32_t nclosest = 0;
    TravState st;
    RayPre r;
    int i = -1, p = -1;
    bool drained = false;
    for (;;) {
        const bool need = i < 0 && !drained;
        const int k = warp_take(cnt + 8, need, n);
        if (need) {
            if (k < 0) {
                drained = true;
            } else {
                i = k;
                p = q[i];
                r = ray_prep(f3(w.ray_o[p]), f3(w.ray_d[p]), kRayEps, kFloatMax);
                trav_begin(st, r, a.scenes[w.meta[p].x].visit_budget);
                if (COUNT) ++nclosest;
            }
        }
        if (__all_sync(__activemask(), i < 0)) break;
        if (i >= 0) {
            const SceneD& S = a.scenes[w.meta[p].x];
            for (int s = 0; s < kStepsPerFetch && !st.done; ++s) trav_step<false, COUNT, SPH>(S, r, st, &tc);
            if (st.done) {
                extend_finish(w, S, cnt + 3, p, st.tcur, st.hslot, kind_of_slot(S, st.hslot));
                i = -1;
            }
        }
    }
    count_flush<COUNT>(a.counters, tc, TraceCounters{0, 0}, nclosest, 0);
}

// Registers of the persistent passes: 18 blocks of 64 threads an SM.  The
// 1 M-triangle frame's closest-hit / any-hit passes (16 samples) take 34.0 / 17.8
// ms at 56 registers (36 bytes of spills in the ray set-up of the closest-hit
// pass), 34.0 / 18.2 at 64 and 35.6 / 19.0 at 48.
constexpr int kPersistRegs = 56;

// Persistent closest-hit pass (persist.cuh) over the continuation rays.  A ray
// that meets two primitives within the tie reach is left to k_wf_ties.
template <bool COUNT, bool SPH, bool SORTED = false>
__global__ void __maxnreg__(kPersistRegs) k_wf_extend_pww(RenderArgs a, int b) {
    const WfBuffers& w = a.wf;
    int* cnt = w.cnt + b * kCntStride;
    const int n = cnt[0];
    const int* q = SORTED ? reinterpret_cast<const int*>(a.sorted) : w.q_cont[b & 1];
    TraceCounters tc{0, 0};
    uint32_t nclosest = 0;
    persistent_pass<false, COUNT, SPH, false>(
        a.scenes, cnt + 8, n, a.refill_closest,
        [&](int k, float3* o, float3* d, float*, float* tmax, int* scene) {
            const int p = q[k];
            *o = f3(__ldcs(&w.ray_o[p]));
            *d = f3(__ldcs(&w.ray_d[p]));
            *scene = int(__ldcs(&w.meta[p].x));
            *tmax = kFloatMax;
            if (COUNT) ++nclosest;
            return p;
        },
        [&](bool done, int p, float t, int slot, int kind, int other) {
            if (!done) return;
            if (other != -1) {
                w.hit[p] = make_float4(t, __int_as_float(slot), __int_as_float(other), 0.0f);
                w.q_tie[atomicAdd(cnt + 12, 1)] = p;
            } else extend_finish(w, a.scenes[__ldcs(&w.meta[p].x)], cnt + 3, p, t, slot, kind);
        },
        [&](int p) {
            uint32_t* st = a.scenes[w.meta[p].x].status;
            if (st) atomicAdd(st, 1u);
        },
        tc);
    count_flush<COUNT>(a.counters, tc, TraceCounters{0, 0}, nclosest, 0);
}

constexpr int kTieBlock = 64;

// Closest-hit rays the persistent pass left to this kernel (q_tie): two
// primitives within the tie reach of the hit, of which tie_prefers orders those
// within its window by the reference's own test and tie order (tie_hit).  Of two
// the pass has both records and only the comparison is left; of more the ray is
// traced again with the per-ray traversal.  Then it is finished as the persistent
// pass finishes its other rays.  Bound by latency: few rays, and a launch that
// traces some of them from their origins lasts about 100 us whatever their number
// (2 M triangles under a sky, 33 launches: 3.5 ms; 1 M triangles, 26: 0.95).  It
// runs beside the any-hit pass (on the other stream), and its grid strides over
// however few rays it got.
template <bool COUNT, bool SPH>
__global__ void k_wf_ties(RenderArgs a, int b) {
    const WfBuffers& w = a.wf;
    int* cnt = w.cnt + b * kCntStride;
    const int n = cnt[12];
    TraceCounters tc{0, 0};
    uint32_t nties = 0;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        if (COUNT) ++nties;
        const int p = w.q_tie[i];
        const SceneD& S = a.scenes[w.meta[p].x];
        const RayPre r = ray_prep(f3(w.ray_o[p]), f3(w.ray_d[p]), kRayEps, kFloatMax);
        const float4 h4 = w.hit[p];
        HitD hit;
        hit.t = h4.x;
        hit.slot = __float_as_int(h4.y);
        hit = tie_hit<COUNT, SPH>(S, r, hit, __float_as_int(h4.z), &tc);
        extend_finish(w, S, cnt + 3, p, hit.t, hit.slot, kind_of_slot(S, hit.slot));
    }
    count_flush<COUNT>(a.counters, tc, TraceCounters{0, 0}, 0, 0);
    if (COUNT && nties) atomicAdd(a.counters + 6, (unsigned long long)nties);
}

// Persistent any-hit pass over the shadow rays; a ray ends at its first hit.
template <bool COUNT, bool SPH>
__global__ void __maxnreg__(kPersistRegs) k_wf_shadow_pww(RenderArgs a, int b) {
    const WfBuffers& w = a.wf;
    int* cnt = w.cnt + b * kCntStride;
    const int n = cnt[2];
    const int* q = w.q_shadow[b & 1];
    TraceCounters tc{0, 0};
    uint32_t nany = 0;
    persistent_pass<true, COUNT, SPH, false>(
        a.scenes, cnt + 9, n, a.refill_any,
        [&](int k, float3* o, float3* d, float*, float* tmax, int* scene) {
            const int p = q[k];
            const float4 sd = __ldcs(&w.sh_d[p]);
            *o = f3(__ldcs(&w.ray_o[p]));
            *d = f3(sd);
            *tmax = sd.w;
            *scene = int(__ldcs(&w.meta[p].x));
            if (COUNT) ++nany;
            return p;
        },
        [&](bool done, int p, float, int slot, int, int) {
            if (done) shadow_finish(w, a.rec_shadow, p, slot >= 0);
        },
        [&](int p) {
            uint32_t* st = a.scenes[w.meta[p].x].status;
            if (st) atomicAdd(st, 1u);
        },
        tc);
    count_flush<COUNT>(a.counters, TraceCounters{0, 0}, tc, 0, nany);
}

template <bool COUNT, bool SPH>
__global__ void k_wf_shadow_dyn(RenderArgs a, int b) {
    const WfBuffers& w = a.wf;
    int* cnt = w.cnt + b * kCntStride;
    const int n = cnt[2];
    const int* q = w.q_shadow[b & 1];
    TraceCounters tc{0, 0};
    uint32_t nany = 0;
    TravState st;
    RayPre r;
    int i = -1, p = -1;
    bool drained = false;
    for (;;) {
        const bool need = i < 0 && !drained;
        const int k = warp_take(cnt + 9, need, n);
        if (need) {
            if (k < 0) {
                drained = true;
            } else {
                i = k;
                p = q[i];
                const float4 sd = w.sh_d[p];
                r = ray_prep(f3(w.ray_o[p]), f3(sd), kRayEps, sd.w);
                trav_begin(st, r, a.scenes[w.meta[p].x].visit_budget);
                if (COUNT) ++nany;
            }
        }
        if (__all_sync(__activemask(), i < 0)) break;
        if (i >= 0) {
            const SceneD& S = a.scenes[w.meta[p].x];
            for (int s = 0; s < kStepsPerFetch && !st.done; ++s) trav_step<true, COUNT, SPH>(S, r, st, &tc);
            if (st.done) {
                shadow_finish(w, a.rec_shadow, p, st.hslot >= 0);
                i = -1;
            }
        }
    }
    count_flush<COUNT>(a.counters, TraceCounters{0, 0}, tc, 0, nany);
}

// ------------------------------------------------------ wavefront adjoint --
// FP64 block sums of the few roughness / radiance gradients in shared memory
// ([0, nmat) roughness, then 3 per area light), flushed once per block.
CG_D void adj_shared_zero(double* sh, const AdjBufs& A) {
    for (int i = threadIdx.x; i < A.nmat + 3 * A.nlight; i += blockDim.x) sh[i] = 0.0;
    __syncthreads();
}
CG_D void adj_shared_flush(double* sh, const AdjBufs& A) {
    __syncthreads();
    for (int i = threadIdx.x; i < A.nmat; i += blockDim.x)
        if (sh[i] != 0.0) atomicAdd(A.g_rough + i, sh[i]);
    for (int i = threadIdx.x; i < 3 * A.nlight; i += blockDim.x)
        if (sh[A.nmat + i] != 0.0) atomicAdd(A.g_rad + i, sh[A.nmat + i]);
}
CG_D void adj_add(double* sh, int i, double v) {
    if (v != 0.0) atomicAdd(sh + i, v);
}
CG_D void adj_radiance(double* sh, const AdjBufs& A, int light, float3 g) {
    adj_add(sh + A.nmat, 3 * light + 0, g.x);
    adj_add(sh + A.nmat, 3 * light + 1, g.y);
    adj_add(sh + A.nmat, 3 * light + 2, g.z);
}
CG_D float3 adj_delta(const AdjBufs& A, uint32_t pixel) {
    return mk(A.dLdI[3 * pixel] * A.inv_spp, A.dLdI[3 * pixel + 1] * A.inv_spp, A.dLdI[3 * pixel + 2] * A.inv_spp);
}

// Before the replay: every path's total radiance from the forward pass, a zero
// accumulator, and the path's state back at the camera (its shading draws the
// same numbers again).
__global__ void k_adj_begin(RenderArgs a) {
    const BatchHeader h = *a.header;
    const WfBuffers& w = a.wf;
    for (uint32_t p = blockIdx.x * blockDim.x + threadIdx.x; p < h.total_paths; p += gridDim.x * blockDim.x) {
        const float3 v = path_sample(f3(w.L[p]), f3(w.Le[p]), f3(w.Ls[p]));
        a.adj.Ltot[p] = make_float4(v.x, v.y, v.z, 0.0f);
        a.adj.acc[p] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        const PathId id = path_id(a.chunks, int(h.num_chunks), p);
        Rng rng;
        float3 o, d;
        primary_ray(a.scenes[id.scene], id, h.seed, rng, &o, &d);
        w.ray_o[p] = make_float4(o.x, o.y, o.z, 0.0f);
        w.ray_d[p] = make_float4(d.x, d.y, d.z, 0.0f);
        w.thr[p] = make_float4(1.0f, 1.0f, 1.0f, __int_as_float(1));
        w.meta[p] = make_uint4(uint32_t(id.scene), id.pixel, id.sample, rng.ctr);
    }
}

// Bound by latency (long scoreboard, 20 resident warps an SM) and by
// instruction fetch: one kernel over all kinds, grouped in shared memory, took
// 39 to 135 ms where these five take 14.9 (1 M-triangle frame, 16 samples a
// pixel).  96 registers keep five blocks of 128 threads on an SM: 14.9 ms,
// 15.8 uncapped (up to 115 registers), 15.6 at 80, 17.1 at 64.
constexpr int kShadeRegs = 96;

// RECORD: the forward pass of the adjoint.
template <int KIND, bool RECORD = false>
__global__ void __maxnreg__(kShadeRegs) k_wf_shade(RenderArgs a, int b) {
    const WfBuffers& w = a.wf;
    const int n = w.cnt[b * kCntStride + 3 + KIND];
    int* next = w.cnt + (b + 1) * kCntStride;
    const int* q = w.q_mat[KIND];
    const int nb = (b + 1) & 1;
    const uint64_t seed = a.header->seed;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const int p = q[i];
        uint4 meta = w.meta[p];
        const SceneD& S = a.scenes[meta.x];
        const float3 o = f3(w.ray_o[p]), d = f3(w.ray_d[p]);
        const float4 h4 = w.hit[p];
        HitD hit;
        hit.t = h4.x;
        hit.slot = __float_as_int(h4.y);
        hit.u = h4.z;
        hit.v = h4.w;
        const SurfaceD si = surface_at(S, o, d, hit);
        const float4 tw = w.thr[p];
        Rng rng;
        rng.key = path_key(seed, meta.x, meta.y, meta.z);
        rng.ctr = meta.w;
        const VertexPlan pl = plan_vertex<KIND>(S, si, f3(tw), (__float_as_int(tw.w) & 1) != 0, b, rng);
        if (!is_zero(pl.emit)) {
            float4 L = w.L[p];
            L.x += pl.emit.x;
            L.y += pl.emit.y;
            L.z += pl.emit.z;
            w.L[p] = L;
        }
        const bool cont = pl.cont && (b + 1 < S.max_depth);
        if (pl.shadow || pl.mis || cont) w.ray_o[p] = make_float4(si.P.x, si.P.y, si.P.z, 0.0f);
        if (pl.shadow) {
            w.sh_d[p] = make_float4(pl.sdir.x, pl.sdir.y, pl.sdir.z, pl.stmax);
            w.sh_c[p] = make_float4(pl.scontrib.x, pl.scontrib.y, pl.scontrib.z, 0.0f);
        }
        // only MIS rays that meet their light are traced (mis_light_hit)
        bool mocc = false;
        if (pl.mis) {
            float4 mh = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            mocc = mis_light_hit(S, ray_prep(si.P, pl.mdir, kRayEps, kFloatMax), pl.mlight, &mh);
            if (mocc) {
                w.mis_d[p] = make_float4(pl.mdir.x, pl.mdir.y, pl.mdir.z, 0.0f);
                w.mis_a[p] = make_float4(pl.mfactor.x, pl.mfactor.y, pl.mfactor.z, pl.mpdf);
                w.mis_b[p] = make_float4(tw.x, tw.y, tw.z, __int_as_float(pl.mlight));
                w.mis_h[p] = mh;
            }
        }
        if (cont) {
            w.ray_d[p] = make_float4(pl.cdir.x, pl.cdir.y, pl.cdir.z, 0.0f);
            w.thr[p] = make_float4(pl.T.x, pl.T.y, pl.T.z, __int_as_float(pl.count_emission));
        }
        meta.w = rng.ctr;
        w.meta[p] = meta;
        // a shadow ray whose contribution is zero in every channel adds
        // nothing to Ls whatever its outcome (for the adjoint its radiance
        // derivative has to be zero as well)
        const int s_slot = warp_append(next + 2, pl.shadow != 0 && (!is_zero(pl.scontrib) || (RECORD && !is_zero(pl.sx))));
        if (s_slot >= 0) w.q_shadow[nb][s_slot] = p;
        const int o_slot = warp_append(next + 11, mocc);
        if (o_slot >= 0) w.q_mocc[nb][o_slot] = p;
        const int c_slot = warp_append(next + 0, cont);
        if (c_slot >= 0) w.q_cont[nb][c_slot] = p;
    }
}

// The replay of the vertices of bounce b (one shade queue of the forward pass):
// the path's state is shaded again as k_wf_shade does, and what its shadow and
// MIS rays found is taken from the records, so that a vertex's gradients are
// complete at once (A, B and the radiance R = Ltot - acc - A - B of the vertices
// after it give the texel, roughness and radiance terms of adjoint.cuh).  A path
// that carries no gradient (total not finite, zero weight) is left out at every
// vertex.  Bound as k_wf_shade is; 96 registers take as long as 128 and 80 (512 x
// 512, 32 samples, depth 6: 7.21, 7.33 and 7.21 ms the whole backward call).
template <int KIND>
__global__ void __maxnreg__(kShadeRegs) k_adj_replay(RenderArgs a, int b) {
    extern __shared__ double sh[];  // gradient block sums
    const WfBuffers& w = a.wf;
    const AdjBufs& A = a.adj;
    const int n = w.cnt[b * kCntStride + 3 + KIND];
    const int* q = w.q_mat[KIND];
    const uint64_t seed = a.header->seed;
    adj_shared_zero(sh, A);
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const int p = q[i];
        uint4 meta = w.meta[p];
        const float3 delta = adj_delta(A, meta.y);
        const float3 Ltot = f3(A.Ltot[p]);
        if (!finite3(Ltot) || is_zero(delta)) continue;
        const SceneD& S = a.scenes[meta.x];
        const float3 o = f3(w.ray_o[p]), d = f3(w.ray_d[p]);
        const float4 h4 = w.hit[p];
        HitD hit;
        hit.t = h4.x;
        hit.slot = __float_as_int(h4.y);
        hit.u = h4.z;
        hit.v = h4.w;
        const SurfaceD si = surface_at(S, o, d, hit);
        const float4 tw = w.thr[p];
        const bool ce = (__float_as_int(tw.w) & 1) != 0;
        Rng rng;
        rng.key = path_key(seed, meta.x, meta.y, meta.z);
        rng.ctr = meta.w;
        const VertexPlan pl = plan_vertex<KIND>(S, si, f3(tw), ce, b, rng);
        const bool cont = pl.cont && (b + 1 < S.max_depth);
        if (cont) {
            w.ray_o[p] = make_float4(si.P.x, si.P.y, si.P.z, 0.0f);
            w.ray_d[p] = make_float4(pl.cdir.x, pl.cdir.y, pl.cdir.z, 0.0f);
            w.thr[p] = make_float4(pl.T.x, pl.T.y, pl.T.z, __int_as_float(pl.count_emission));
            meta.w = rng.ctr;
            w.meta[p] = meta;
        }
        if (si.light >= 0 && si.light < A.nlight && ce && can_emit(S.lights[si.light], si.wi, si.Ns))
            adj_radiance(sh, A, si.light, delta * f3(tw));
        float3 Av = splat3(0.0f), Bv = splat3(0.0f);
        if (pl.shadow && (!is_zero(pl.scontrib) || !is_zero(pl.sx)) && a.rec_shadow[p]) {
            Av = pl.scontrib;
            if (pl.slight < A.nlight) adj_radiance(sh, A, pl.slight, delta * pl.sx);
        }
        float4 mh = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        if (pl.mis && mis_light_hit(S, ray_prep(si.P, pl.mdir, kRayEps, kFloatMax), pl.mlight, &mh) && a.rec_mis[p]) {
            float3 X = splat3(0.0f);
            Bv = mis_add(S, si.P, pl.mdir, mh, f3(tw), pl.mfactor, pl.mpdf, &X);
            if (__float_as_int(mh.y) >= 0 && pl.mlight >= 0 && pl.mlight < A.nlight) adj_radiance(sh, A, pl.mlight, delta * X);
        }
        const float4 acc4 = A.acc[p];
        const float3 acc = f3(acc4) + pl.emit;
        const float3 after = Ltot - acc - Av - Bv;
        const MaterialD& m = S.materials[si.material];
        if (m.type == BSDF_LAMBERTIAN && m.albedo_tex >= 0) {
            const TextureD& tex = S.textures[m.albedo_tex];
            const float3 alb = texture_rgb(tex, si.uvw);
            const float3 num = delta * (Av + Bv + after);
            double* g = A.g_tex + A.tex_offset[m.albedo_tex] + 3 * texel_index(tex, si.uvw);
            if (alb.x > 0.0f && num.x != 0.0f) atomicAdd(g + 0, double(num.x / alb.x));
            if (alb.y > 0.0f && num.y != 0.0f) atomicAdd(g + 1, double(num.y / alb.y));
            if (alb.z > 0.0f && num.z != 0.0f) atomicAdd(g + 2, double(num.z / alb.z));
        }
        if (m.type == BSDF_CONDUCTOR || m.type == BSDF_DIELECTRIC_GGX) {
            float gr = 0.0f;
            if (!is_zero(Av)) gr += dot(delta, Av) * dlogf_droughness(m, si.wi, pl.sdir, si.Ns);
            if (!is_zero(Bv)) gr += dot(delta, Bv) * dlogf_droughness(m, si.wi, pl.mdir, si.Ns);
            if (pl.cont) gr += dot(delta, after) * dlogf_droughness(m, si.wi, pl.cdir, si.Ns);
            adj_add(sh, si.material, double(gr));
        }
        const float3 nacc = acc + (Av + Bv);
        A.acc[p] = make_float4(nacc.x, nacc.y, nacc.z, 0.0f);
    }
    adj_shared_flush(sh, A);
}

// FP64 accumulation of one batch into the scenes' films.  With the default
// box filter of size 1 a sample at (ix + fx, iy + fy) lands in pixel (ix, iy)
// only; other filters go through splat_filtered.  NaN / Inf samples are
// dropped as FilmTile::addSample does (source/core/film/filmTile.cpp:21-28).
// One warp a block: a filtered frame of 333 x 251 pixels is 327 blocks of 256
// threads, three on some SMs and two on the others (0.68 ms; 0.59 in blocks of
// 128, 0.54 of 64, 0.53 of 32; a 1080p frame 0.66 in any).
constexpr int kSplatBlock = 32;

__global__ void k_splat(RenderArgs a) {
    const BatchHeader h = *a.header;
    for (uint32_t idx = blockIdx.x * blockDim.x + threadIdx.x; idx < h.total_pixels; idx += gridDim.x * blockDim.x) {
        int lo = 0, hi = int(h.num_chunks) - 1;
        while (lo < hi) {
            const int mid = (lo + hi + 1) >> 1;
            if (a.chunks[mid].pix_begin <= idx) lo = mid; else hi = mid - 1;
        }
        const Chunk c = a.chunks[lo];
        const uint32_t pixel = idx - c.pix_begin;
        const FilterD& F = a.scenes[c.scene].filter;
        if (!F.pixel_only) {
            double s[3] = {0, 0, 0}, q[3] = {0, 0, 0}, n = 0;
            const int W = int(c.width);
            auto fetch = [&](uint32_t k, int sx, int sy, float3* v, float2* pos) {
                const uint32_t p = c.path_begin + k * c.npix + uint32_t(sy * W + sx);
                const float4 L = a.wf.L[p], Ls = a.wf.Ls[p];
                *v = path_sample(f3(L), f3(a.wf.Le[p]), f3(Ls));
                *pos = make_float2(L.w, Ls.w);
                return isfinite(v->x) && isfinite(v->y) && isfinite(v->z);
            };
            filter_gather(F, W, int(c.npix / c.width), int(pixel % c.width), int(pixel / c.width), c.nsamples, fetch, s,
                          q, &n);
            const FilmD f = a.films[c.scene];
            for (int k = 0; k < 3; ++k) {
                f.sum[3 * pixel + k] += s[k];
                f.sumsq[3 * pixel + k] += q[k];
            }
            f.count[pixel] += n;
            continue;
        }
        // bound by FP64 (about 1.5 operations a clock and SM): the square of an
        // FP32 value is exact in FP64, so one fused operation adds it with the
        // same rounding as two, and the count is an integer (1 M-triangle frame,
        // 16 samples a pixel: 0.91 -> 0.66 ms)
        double s0 = 0, s1 = 0, s2 = 0, q0 = 0, q1 = 0, q2 = 0;
        uint32_t n = 0;
        for (uint32_t k = 0; k < c.nsamples; ++k) {
            const uint32_t p = c.path_begin + k * c.npix + pixel;
            const float3 v = path_sample(f3(a.wf.L[p]), f3(a.wf.Le[p]), f3(a.wf.Ls[p]));
            const float x = v.x, y = v.y, z = v.z;
            if (!(isfinite(x) && isfinite(y) && isfinite(z))) continue;
            const double dx = x, dy = y, dz = z;
            s0 += dx; s1 += dy; s2 += dz;
            q0 = fma(dx, dx, q0); q1 = fma(dy, dy, q1); q2 = fma(dz, dz, q2);
            ++n;
        }
        const FilmD f = a.films[c.scene];
        f.sum[3 * pixel + 0] += s0;
        f.sum[3 * pixel + 1] += s1;
        f.sum[3 * pixel + 2] += s2;
        f.sumsq[3 * pixel + 0] += q0;
        f.sumsq[3 * pixel + 1] += q1;
        f.sumsq[3 * pixel + 2] += q2;
        f.count[pixel] += double(n);
    }
}

__global__ void k_gather_paths(const float4* L, const float4* Le, const float4* Ls, uint32_t n, float* out) {
    for (uint32_t p = blockIdx.x * blockDim.x + threadIdx.x; p < n; p += gridDim.x * blockDim.x) {
        const float3 v = path_sample(f3(L[p]), f3(Le[p]), f3(Ls[p]));
        out[3 * p + 0] = v.x;
        out[3 * p + 1] = v.y;
        out[3 * p + 2] = v.z;
    }
}

// ------------------------------------------------------------- ray queries --
// The answer of a closest-hit query from its record slot (-1: a miss).
CG_D cgpu_hit query_answer(const SceneD& S, float3 o, float3 d, const HitD& h) {
    cgpu_hit out;
    out.t = 0.0f;
    out.primitive = -1;
    out.u = 0.0f;
    out.v = 0.0f;
    if (h.slot >= 0) {
        const HitPoint hp = hit_point(S, o, d, h);
        out.t = hp.t;
        out.primitive = __float_as_int(ldg4(reinterpret_cast<const float4*>(S.tris + h.slot)).w);
        out.u = hp.rect >= 0 ? hp.p1 : hp.b1;
        out.v = hp.rect >= 0 ? hp.p2 : hp.b2;
    }
    return out;
}

__global__ void k_trace(const SceneD* scenes, int scene, const cgpu_ray* rays, uint32_t n, cgpu_hit* hits,
                        uint8_t* occ) {
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const SceneD& S = scenes[scene];
        const cgpu_ray r = rays[i];
        // the direction is normalised again, as the reference's Ray constructor does (ray.cpp:19-30)
        RayPre pr = ray_prep(mk(r.org[0], r.org[1], r.org[2]), normalize(mk(r.dir[0], r.dir[1], r.dir[2])), r.t_min, r.t_max);
        auto answer = [&](const RayPre& p) {
            HitD h;
            TraceCounters tc{0, 0};
            if (occ) {
                occ[i] = traverse<true, false>(S, p, &h, &tc) ? 1 : 0;
            } else {
                if (!traverse_warp<false>(S, p, &h, &tc)) h.slot = -1;
                hits[i] = query_answer(S, p.o, p.d, h);
            }
        };
        // the mask a constant where it can be (one form for all costs 257 rays 2 %)
        if (r.t_min < 0.0f) {
            answer(pr);
        } else {
            pr.mag = 0xFFFFFFFFu;
            answer(pr);
        }
    }
}

// Large batches of queries: the persistent pass, then (closest hit) one thread
// per ray for the answer.  k_query leaves the traversal's distance in hits[i].t,
// its record slot in hits[i].primitive (-1: a miss) and the record within its
// tie reach in hits[i].u, as the pass reports it; k_query_resolve compares the
// two (tie_hit).
CG_D void load_query(const cgpu_ray& r, float3* o, float3* d, float* tmin, float* tmax) {
    *o = mk(r.org[0], r.org[1], r.org[2]);
    // the direction is normalised again, as the reference's Ray constructor does (ray.cpp:19-30)
    *d = normalize(mk(r.dir[0], r.dir[1], r.dir[2]));
    *tmin = r.t_min;
    *tmax = r.t_max;
}

template <bool ANY, bool SPH>
__global__ void __maxnreg__(kPersistRegs) k_query(const SceneD* scenes, int scene, int* work, const cgpu_ray* rays, uint32_t n,
                                                  int refill, cgpu_hit* hits, uint8_t* occ) {
    TraceCounters tc{0, 0};
    persistent_pass<ANY, false, SPH, true>(
        scenes, work, int(n), refill,
        [&](int k, float3* o, float3* d, float* tmin, float* tmax, int* s) {
            load_query(rays[k], o, d, tmin, tmax);
            *s = scene;
            return k;
        },
        [&](bool done, int k, float t, int slot, int, int other) {
            if (!done) return;
            if (ANY) {
                occ[k] = slot >= 0 ? 1 : 0;
            } else {
                hits[k].t = t;
                hits[k].primitive = slot;
                hits[k].u = __int_as_float(other);
            }
        },
        [&](int) {
            uint32_t* st = scenes[scene].status;
            if (st) atomicAdd(st, 1u);
        },
        tc);
}

__global__ void k_query_resolve(const SceneD* scenes, int scene, const cgpu_ray* rays, uint32_t n, cgpu_hit* hits) {
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const SceneD& S = scenes[scene];
        float3 o, d;
        float tmin, tmax;
        load_query(rays[i], &o, &d, &tmin, &tmax);
        HitD h;
        h.t = hits[i].t;
        h.slot = hits[i].primitive;
        h.u = h.v = 0.0f;
        const int other = __float_as_int(hits[i].u);
        if (h.slot >= 0 && other != -1) {
            TraceCounters tc{0, 0};
            h = tie_hit<false, true>(S, ray_prep(o, d, tmin, tmax), h, other, &tc);
        }
        hits[i] = query_answer(S, o, d, h);
    }
}

__global__ void k_camera(const SceneD* scenes, int scene, const double* xy, uint32_t n, float* out) {
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        float3 o, d;
        camera_ray(scenes[scene].cam, float(xy[2 * i]), float(xy[2 * i + 1]), &o, &d);
        out[6 * i + 0] = o.x; out[6 * i + 1] = o.y; out[6 * i + 2] = o.z;
        out[6 * i + 3] = d.x; out[6 * i + 4] = d.y; out[6 * i + 5] = d.z;
    }
}

}  // namespace cg

// ============================================================== host side ==
using namespace cg;

namespace {

constexpr int kBlock = 128;  // fixed-size utility kernels

template <typename K>
int grid_for(cgpu_ctx* ctx, K kernel, int block, uint64_t work, size_t shared_bytes = 0) {
    int per_sm = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, block, shared_bytes);
    if (per_sm < 1) per_sm = 1;
    const uint64_t full = uint64_t(ctx->num_sms) * uint64_t(per_sm);
    const uint64_t need = (work + block - 1) / block;
    return int(std::max<uint64_t>(1, std::min<uint64_t>(full, need)));
}

// Dynamic shared memory of a traversal launch: the shared-memory part of the
// traversal stacks of the persistent passes (0 for the other variants).  A
// block above the default 48 KB window opts the kernel in first.
template <typename K>
size_t stack_smem(K kernel, bool shared_stack, bool with_t, int block) {
    if (!shared_stack) return 0;
    const size_t bytes = with_t ? persist_bytes(block, true) : persist_bytes(block, false);
    if (bytes > 48 * 1024) cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, int(bytes));
    return bytes;
}

uint32_t paths_capacity(cgpu_ctx* ctx, uint32_t max_npix) {
    uint32_t cap = ctx->tuning.max_paths ? ctx->tuning.max_paths : (1u << 21);
    if (cap < max_npix) cap = max_npix;
    return cap;
}

cgpu_status ensure_path_buffers(cgpu_ctx* ctx, uint32_t cap, int depth) {
    if (ctx->path_cap >= cap && ctx->wf.cnt_depth >= depth + 2) return CGPU_OK;
    cg_free_render_state(ctx);
    const int cdepth = std::max(depth + 2, 34);
    WfBuffers w{};
    const size_t bytes = wf_layout(nullptr, cap, cdepth, &w);
    void* block = nullptr;
    cudaError_t e = cudaMalloc(&block, bytes);
    if (e != cudaSuccess) return cg_fail(ctx, CGPU_ERR_OUT_OF_MEMORY, "path buffers: " + std::string(cudaGetErrorString(e)));
    wf_layout(static_cast<char*>(block), cap, cdepth, &ctx->wf);
    ctx->wf_block = block;
    ctx->path_cap = cap;
    if (!ctx->d_counters) {
        e = cudaMalloc(&ctx->d_counters, 8 * sizeof(unsigned long long));
        if (e != cudaSuccess) return cg_cuda(ctx, e, "counters");
    }
    if (!ctx->d_chunks) {
        if ((e = cudaMalloc(&ctx->d_chunks, sizeof(Chunk) * kMaxChunks)) != cudaSuccess) return cg_cuda(ctx, e, "chunks");
        if ((e = cudaMalloc(&ctx->d_header, sizeof(BatchHeader))) != cudaSuccess) return cg_cuda(ctx, e, "header");
        if ((e = cudaMallocHost(&ctx->h_chunks, sizeof(Chunk) * kMaxChunks)) != cudaSuccess) return cg_cuda(ctx, e, "chunks");
        if ((e = cudaMallocHost(&ctx->h_header, sizeof(BatchHeader))) != cudaSuccess) return cg_cuda(ctx, e, "header");
    }
    return CGPU_OK;
}

uint32_t scan_launches(uint32_t n) {
    const uint32_t nb = radix_tiles(n);
    return 1 + (nb > 1 ? scan_launches(nb) + 1 : 0);
}

// Ray reordering buffers for the path_cap rays a closest-hit pass can have, kept
// while tuning.reorder is on.
cgpu_status ensure_sort_buffers(cgpu_ctx* ctx) {
    if (!ctx->tuning.reorder) return CGPU_OK;
    const uint64_t cap = ctx->path_cap;
    if (ctx->sort_block && ctx->sort_cap >= cap) return CGPU_OK;
    if (ctx->sort_block) cudaFree(ctx->sort_block);
    ctx->sort_block = nullptr;
    ctx->sort_cap = 0;
    const uint32_t tiles = radix_tiles(cap);
    const size_t words[] = {cap, cap, cap, cap, size_t(tiles) * 256, scan_scratch(uint64_t(tiles) * 256), 1};
    size_t total = 0;
    for (size_t w : words) total += (w * sizeof(uint32_t) + 255) & ~size_t(255);
    cudaError_t e = cudaMalloc(&ctx->sort_block, total);
    if (e != cudaSuccess) {
        ctx->sort_block = nullptr;
        return cg_fail(ctx, CGPU_ERR_OUT_OF_MEMORY, "reorder buffers: " + std::string(cudaGetErrorString(e)));
    }
    uint32_t* ptr[7];
    char* base = static_cast<char*>(ctx->sort_block);
    for (int i = 0; i < 7; ++i) {
        ptr[i] = reinterpret_cast<uint32_t*>(base);
        base += (words[i] * sizeof(uint32_t) + 255) & ~size_t(255);
    }
    ctx->sort = SortBufs{{ptr[0], ptr[1]}, {ptr[2], ptr[3]}, ptr[4], ptr[5], ptr[6], tiles};
    ctx->sort_cap = uint32_t(cap);
    return CGPU_OK;
}

RenderArgs make_args(cgpu_ctx* ctx) {
    RenderArgs a{};
    a.scenes = ctx->d_scenes;
    a.chunks = ctx->d_chunks;
    a.header = ctx->d_header;
    a.films = ctx->d_films;
    a.wf = ctx->wf;
    a.counters = ctx->d_counters;
    a.sorted = nullptr;
    a.refill_closest = refill_lanes(ctx->tuning.refill_closest);
    a.refill_any = refill_lanes(ctx->tuning.refill_any);
    return a;
}

// Launch wrapper: with profiling on, bracket the launch with CUDA events on
// the stream it runs on.
template <typename F>
void timed(cgpu_ctx* ctx, int cls, cudaStream_t s, F&& launch) {
    if (!ctx->profiling) {
        launch();
        return;
    }
    cgpu_ctx::ProfEvent ev{cls, nullptr, nullptr};
    cudaEventCreate(&ev.a);
    cudaEventCreate(&ev.b);
    cudaEventRecord(ev.a, s);
    launch();
    cudaEventRecord(ev.b, s);
    ctx->prof.push_back(ev);
}

void collect_profile(cgpu_ctx* ctx) {
    if (ctx->prof.empty()) return;
    cudaDeviceSynchronize();
    for (auto& ev : ctx->prof) {
        float ms = 0.0f;
        cudaEventElapsedTime(&ms, ev.a, ev.b);
        ctx->times.ms[ev.cls] += ms;
        ctx->times.launches[ev.cls] += 1;
        cudaEventDestroy(ev.a);
        cudaEventDestroy(ev.b);
    }
    ctx->prof.clear();
}

// The traversal variants of the current render's passes: the tuning's, or where
// it leaves them open the persistent ones as the caller asks.  Counting renders
// then keep one ray per thread, whose node visits do not depend on which rays
// happen to share a warp.
void choose_traversal(cgpu_ctx* ctx, bool closest, bool any) {
    ctx->batch_closest = traversal_kernels(ctx->tuning.traversal, closest && !ctx->counting);
    ctx->batch_any = traversal_kernels(ctx->tuning.traversal, any && !ctx->counting);
}
bool large_batch(const cgpu_ctx* ctx, uint64_t paths) { return std::min<uint64_t>(paths, ctx->path_cap) >= kLargeBatch; }

// The shade kernels of the queues that the render's scenes have materials for.
// An empty launch still costs 2 to 4 us between two passes (Cornell box, 256 x
// 256, 16 samples, depth 6: 1.28 -> 1.20 ms without four of them a bounce).
uint32_t launch_shade(cgpu_ctx* ctx, const RenderArgs& a, int b, const int (&grid)[kNumBsdfKinds]) {
    static void (*const plain[kNumBsdfKinds])(RenderArgs, int) = {k_wf_shade<0>, k_wf_shade<1>, k_wf_shade<2>, k_wf_shade<3>,
                                                                  k_wf_shade<4>};
    static void (*const record[kNumBsdfKinds])(RenderArgs, int) = {k_wf_shade<0, true>, k_wf_shade<1, true>, k_wf_shade<2, true>,
                                                                   k_wf_shade<3, true>, k_wf_shade<4, true>};
    auto& kernel = a.rec_shadow ? record : plain;
    uint32_t launches = 0;
    for (int k = 0; k < kNumBsdfKinds; ++k) {
        if (!(ctx->batch_kinds >> k & 1u)) continue;
        kernel[k]<<<grid[k], ctx->tuning.block_shade, 0, ctx->stream>>>(a, b);
        ++launches;
    }
    return launches;
}

// Enqueue the wavefront schedule for one batch on ctx->stream.
void set_records(RenderArgs& a, const AdjRecords& r, int b, int outcomes);

// The film splat of the batch in h_header.
void launch_splat(cgpu_ctx* ctx, const RenderArgs& a) {
    const int grid = grid_for(ctx, k_splat, kSplatBlock, ctx->h_header->total_pixels);
    timed(ctx, CGPU_KERNEL_SPLAT, ctx->stream, [&] { k_splat<<<grid, kSplatBlock, 0, ctx->stream>>>(a); });
    ctx->stats.kernel_launches += 1;
}

// rec (optional): the batch's rays are recorded there, for the adjoint.
cgpu_status enqueue_wavefront(cgpu_ctx* ctx, int depth, uint32_t paths, bool counting, const AdjRecords* rec = nullptr) {
    RenderArgs a = make_args(ctx);
    // With per-kernel timing on, the shadow pass runs after the extend pass on
    // the same stream, so that each event pair brackets one kernel alone.
    cudaStream_t s = ctx->stream, side = ctx->profiling ? ctx->stream : ctx->side;
    cudaEvent_t fork = nullptr, join = nullptr;
    cudaEventCreateWithFlags(&fork, cudaEventDisableTiming);
    cudaEventCreateWithFlags(&join, cudaEventDisableTiming);
    cudaMemsetAsync(ctx->wf.cnt, 0, size_t(depth + 2) * kCntStride * sizeof(int), s);
    uint32_t launches = 1;
    const int bt = ctx->tuning.block_trace, bs = ctx->tuning.block_shade;
    const int ggen = grid_for(ctx, k_wf_generate, kBlock, paths);
    timed(ctx, CGPU_KERNEL_GENERATE, s, [&] { k_wf_generate<<<ggen, kBlock, 0, s>>>(a); });
    const int trav = ctx->batch_closest, trav_any = ctx->batch_any;
    const bool sph = ctx->batch_spheres;
#define CG_PICK(K) (sph ? (counting ? K<true, true> : K<false, true>) : (counting ? K<true, false> : K<false, false>))
    auto ext_kernel = trav == 1 ? CG_PICK(k_wf_extend_dyn)
                      : (trav == 2 || trav == 3) ? CG_PICK(k_wf_extend_pww) : CG_PICK(k_wf_extend);
    auto sh_kernel = trav_any == 1 ? CG_PICK(k_wf_shadow_dyn) : trav_any == 3 ? CG_PICK(k_wf_shadow_pww) : CG_PICK(k_wf_shadow);
    auto mocc_kernel = CG_PICK(k_wf_mis_occl);
    auto ties_kernel = CG_PICK(k_wf_ties);
#undef CG_PICK
    // reordered closest-hit passes after the first (the primary rays are in pixel order already)
    const bool reorder = ctx->tuning.reorder != 0 && trav != 1 && ctx->sort_block != nullptr;
#define CG_PICK_SORTED(C, S) (trav >= 2 ? k_wf_extend_pww<C, S, true> : k_wf_extend<C, S, true>)
    auto ext_sorted = sph ? (counting ? CG_PICK_SORTED(true, true) : CG_PICK_SORTED(false, true))
                          : (counting ? CG_PICK_SORTED(true, false) : CG_PICK_SORTED(false, false));
#undef CG_PICK_SORTED
    // reorder 1 / 2 / 3 / 4: 9 / 7 / 4 / 0 Morton bits per axis, 4 / 3 / 2 / 1 sort passes of 8 bits
    // (4: the direction octant alone); an odd pass count leaves the sorted values in the second buffer
    const int sort_bits = ctx->tuning.reorder == 1 ? 9 : ctx->tuning.reorder == 2 ? 7 : ctx->tuning.reorder == 3 ? 4 : 0;
    const int sort_passes = (3 + 3 * sort_bits + 7) / 8;
    if (reorder) a.sorted = ctx->sort.vals[sort_passes & 1];
    const int gkeys = grid_for(ctx, k_ray_keys, 256, paths);
    // the persistent passes keep the bottom of their traversal stacks in shared memory
    const size_t ext_sm = stack_smem(ext_kernel, trav >= 2, true, bt);
    const size_t ext_sorted_sm = stack_smem(ext_sorted, trav >= 2, true, bt);
    const size_t sh_sm = stack_smem(sh_kernel, trav_any == 3, false, bt);
    const int gext = grid_for(ctx, ext_kernel, bt, paths, ext_sm);
    const int gsh = grid_for(ctx, sh_kernel, bt, paths, sh_sm);
    const int gmo = grid_for(ctx, mocc_kernel, bt, paths);
    const int gties = grid_for(ctx, ties_kernel, kTieBlock, paths);
    const int gsd[kNumBsdfKinds] = {grid_for(ctx, k_wf_shade<0>, bs, paths), grid_for(ctx, k_wf_shade<1>, bs, paths),
                                    grid_for(ctx, k_wf_shade<2>, bs, paths), grid_for(ctx, k_wf_shade<3>, bs, paths),
                                    grid_for(ctx, k_wf_shade<4>, bs, paths)};
    auto rays = sph ? k_wf_rays<true> : k_wf_rays<false>;
    const int grays = 3 * grid_for(ctx, rays, bt, paths);
    const bool one = trav == 0 && trav_any == 0 && !counting && !reorder && !ctx->profiling;
    for (int b = 0; b <= depth; ++b) {
        if (rec) set_records(a, *rec, b, b - 1);
        if (one && b > 0) {
            rays<<<grays, bt, 0, s>>>(a, b);
            launches += 1;
            if (b == depth) break;
            launches += launch_shade(ctx, a, b, gsd);
            continue;
        }
        cudaEventRecord(fork, s);
        cudaStreamWaitEvent(side, fork, 0);
        if (reorder && b > 0) {
            const SortBufs& q = ctx->sort;
            timed(ctx, CGPU_KERNEL_REORDER, s, [&] {
                k_ray_keys<<<gkeys, 256, 0, s>>>(a, b, sort_bits, q.keys[0], q.vals[0], q.n);
                radix_sort_pairs<uint32_t>(q.keys, q.vals, 0, q.n, q.tiles, sort_passes, q.hist, q.sums, s);
            });
            launches += 1 + sort_passes * (2 + scan_launches(q.tiles * 256));
            timed(ctx, CGPU_KERNEL_EXTEND, s, [&] { ext_sorted<<<gext, bt, ext_sorted_sm, s>>>(a, b); });
        } else {
            timed(ctx, CGPU_KERNEL_EXTEND, s, [&] { ext_kernel<<<gext, bt, ext_sm, s>>>(a, b); });
        }
        if (trav >= 2) {
            // the persistent pass's rays within the tie reach
            timed(ctx, CGPU_KERNEL_TIES, s, [&] { ties_kernel<<<gties, kTieBlock, 0, s>>>(a, b); });
            launches += 1;
        }
        timed(ctx, CGPU_KERNEL_SHADOW, side, [&] { sh_kernel<<<gsh, bt, sh_sm, side>>>(a, b); });
        // the MIS rays of the vertices of bounce b - 1 that meet their light
        if (b > 0) {
            timed(ctx, CGPU_KERNEL_MIS_OCCL, side, [&] { mocc_kernel<<<gmo, bt, 0, side>>>(a, b); });
            launches += 1;
        }
        cudaEventRecord(join, side);
        cudaStreamWaitEvent(s, join, 0);
        launches += 2;
        if (b == depth) break;
        timed(ctx, CGPU_KERNEL_SHADE, s, [&] { launches += launch_shade(ctx, a, b, gsd); });
    }
    cudaEventDestroy(fork);
    cudaEventDestroy(join);
    ctx->stats.kernel_launches += launches;
    return cg_cuda(ctx, cudaGetLastError(), "wavefront launch");
}

cgpu_status run_batch(cgpu_ctx* ctx, int mode, int depth, uint32_t paths, bool splat, bool use_graph) {
    const bool counting = ctx->counting;
    if (mode == CGPU_MODE_MEGAKERNEL) {
        RenderArgs a = make_args(ctx);
        const int bt = ctx->tuning.block_trace;
        const bool sph = ctx->batch_spheres;
        if (counting) {
            auto k = sph ? k_megakernel<true, true> : k_megakernel<true, false>;
            k<<<grid_for(ctx, k, bt, paths), bt, 0, ctx->stream>>>(a);
        } else {
            auto k = sph ? k_megakernel<false, true> : k_megakernel<false, false>;
            const int g = grid_for(ctx, k, bt, paths);
            timed(ctx, CGPU_KERNEL_MEGAKERNEL, ctx->stream, [&] { k<<<g, bt, 0, ctx->stream>>>(a); });
        }
        ctx->stats.kernel_launches += 1;
        if (splat) launch_splat(ctx, a);
        return cg_cuda(ctx, cudaGetLastError(), "megakernel launch");
    }
    if (!use_graph || counting || !splat || ctx->profiling) {
        const cgpu_status st = enqueue_wavefront(ctx, depth, paths, counting);
        if (st != CGPU_OK || !splat) return st;
        launch_splat(ctx, make_args(ctx));
        return cg_cuda(ctx, cudaGetLastError(), "splat launch");
    }
    // one graph per traversal variant, captured anew when the depth, the path capacity or the other
    // kernels change; the batch itself lives in device memory.  The splat follows it: its grid goes by
    // the batch's own pixels (with the grid of the batch that was captured first, a 24 x 20 frame, a
    // 1280 x 720 frame of 16 samples took 59.4 ms instead of 13.5; with the grid of the path capacity, a
    // 333 x 251 frame 1.91 instead of 1.88).
    cgpu_ctx::Graph& G = ctx->graphs[ctx->batch_closest >= 2 ? 1 : 0];
    if (!G.exec || G.depth != depth || G.paths != ctx->path_cap || G.spheres != ctx->batch_spheres ||
        G.kinds != ctx->batch_kinds) {
        if (G.exec) {
            cudaGraphExecDestroy(G.exec);
            G.exec = nullptr;
        }
        cudaGraph_t g = nullptr;
        cudaError_t e = cudaStreamBeginCapture(ctx->stream, cudaStreamCaptureModeThreadLocal);
        if (e != cudaSuccess) return cg_cuda(ctx, e, "begin capture");
        const uint32_t before = ctx->stats.kernel_launches;
        // capture for the full capacity: kernels read the live path count from the header
        cgpu_status st = enqueue_wavefront(ctx, depth, ctx->path_cap, false);
        e = cudaStreamEndCapture(ctx->stream, &g);
        if (st != CGPU_OK) return st;
        if (e != cudaSuccess) return cg_cuda(ctx, e, "end capture");
        e = cudaGraphInstantiate(&G.exec, g, 0);
        cudaGraphDestroy(g);
        if (e != cudaSuccess) return cg_cuda(ctx, e, "graph instantiate");
        G.depth = depth;
        G.paths = ctx->path_cap;
        G.spheres = ctx->batch_spheres;
        G.kinds = ctx->batch_kinds;
        G.launches = ctx->stats.kernel_launches - before;
        ctx->stats.kernel_launches = before;
    }
    ctx->stats.kernel_launches += G.launches;
    const cudaError_t e = cudaGraphLaunch(G.exec, ctx->stream);
    if (e != cudaSuccess) return cg_cuda(ctx, e, "graph launch");
    launch_splat(ctx, make_args(ctx));
    return cg_cuda(ctx, cudaGetLastError(), "splat launch");
}

}  // namespace

void cg_drop_graphs(cgpu_ctx* ctx) {
    for (cgpu_ctx::Graph& G : ctx->graphs) {
        if (G.exec) cudaGraphExecDestroy(G.exec);
        G = cgpu_ctx::Graph{};
    }
}

void cg_free_render_state(cgpu_ctx* ctx) {
    cg_drop_graphs(ctx);
    if (ctx->wf_block) {
        cudaFree(ctx->wf_block);
        ctx->wf_block = nullptr;
    }
    ctx->wf = WfBuffers{};
    ctx->path_cap = 0;
    if (ctx->adj_block) {
        cudaFree(ctx->adj_block);
        ctx->adj_block = nullptr;
    }
    ctx->adj_bytes = 0;
    if (ctx->sort_block) {
        cudaFree(ctx->sort_block);
        ctx->sort_block = nullptr;
    }
    ctx->sort = SortBufs{};
    ctx->sort_cap = 0;
}

// Split the requested samples of every scene into batches of at most
// path_cap paths and run them.
cgpu_status cg_render_batches(cgpu_ctx* ctx, const cgpu_render_params* p) {
    if (!p || !p->scenes || p->num_scenes == 0 || p->num_scenes > uint32_t(kMaxChunks))
        return cg_fail(ctx, CGPU_ERR_INVALID_ARGUMENT, "render: bad scene list");
    if (p->mode != CGPU_MODE_MEGAKERNEL && p->mode != CGPU_MODE_WAVEFRONT)
        return cg_fail(ctx, CGPU_ERR_INVALID_ARGUMENT, "render: unknown mode");
    uint32_t max_npix = 0;
    int depth = 1;
    for (uint32_t i = 0; i < p->num_scenes; ++i) {
        const int s = p->scenes[i];
        if (s < 0 || s >= int(ctx->scenes.size()) || !ctx->scenes[s].live)
            return cg_fail(ctx, CGPU_ERR_NOT_FOUND, "render: unknown scene id");
        const SceneSlot& sl = ctx->scenes[s];
        max_npix = std::max<uint32_t>(max_npix, uint32_t(sl.width) * uint32_t(sl.height));
        depth = std::max(depth, sl.max_depth);
    }
    ctx->batch_spheres = false;
    ctx->batch_kinds = 0;
    int records = 0;  // of the largest scene
    for (uint32_t i = 0; i < p->num_scenes; ++i) {
        records = std::max(records, ctx->scenes[p->scenes[i]].d.num_tris);
        ctx->batch_spheres |= ctx->scenes[p->scenes[i]].has_spheres;
        ctx->batch_kinds |= ctx->scenes[p->scenes[i]].kinds;
    }
    cgpu_status st = cg_sync_tables(ctx);
    if (st != CGPU_OK) return st;
    st = ensure_path_buffers(ctx, paths_capacity(ctx, max_npix), depth);
    if (st != CGPU_OK) return st;
    st = ensure_sort_buffers(ctx);
    if (st != CGPU_OK) return st;
    ctx->stats = cgpu_render_stats{};
    ctx->times = cgpu_kernel_times{};
    if (ctx->counting) cudaMemsetAsync(ctx->d_counters, 0, 8 * sizeof(unsigned long long), ctx->stream);
    // remaining samples per scene
    std::vector<uint32_t> next(p->num_scenes, p->first_sample), end(p->num_scenes);
    for (uint32_t i = 0; i < p->num_scenes; ++i) {
        const uint64_t n = p->scene_samples ? p->scene_samples[i] : p->num_samples;
        if (uint64_t(p->first_sample) + n > 0xFFFFFFFFull)
            return cg_fail(ctx, CGPU_ERR_INVALID_ARGUMENT, "render: sample range overflows 32 bits");
        end[i] = p->first_sample + uint32_t(n);
    }
    uint64_t asked = 0;
    for (uint32_t i = 0; i < p->num_scenes; ++i) {
        const SceneSlot& sl = ctx->scenes[p->scenes[i]];
        asked += uint64_t(sl.width) * uint64_t(sl.height) * (end[i] - next[i]);
    }
    const bool persistent = records >= kSmallScene && large_batch(ctx, asked);
    choose_traversal(ctx, persistent, persistent);
    uint64_t total_paths = 0;
    for (;;) {
        uint32_t used = 0, pix = 0, nch = 0;
        for (uint32_t i = 0; i < p->num_scenes && nch < uint32_t(kMaxChunks); ++i) {
            if (next[i] >= end[i]) continue;
            const SceneSlot& sl = ctx->scenes[p->scenes[i]];
            const uint32_t npix = uint32_t(sl.width) * uint32_t(sl.height);
            const uint32_t room = (ctx->path_cap - used) / npix;
            if (room == 0) continue;
            const uint32_t k = std::min(room, end[i] - next[i]);
            Chunk& c = ctx->h_chunks[nch++];
            c.scene = p->scenes[i];
            c.path_begin = used;
            c.npix = npix;
            c.width = uint32_t(sl.width);
            c.sample0 = next[i];
            c.nsamples = k;
            c.pix_begin = pix;
            c.pixel0 = 0;
            used += k * npix;
            pix += npix;
            next[i] += k;
        }
        if (nch == 0) break;
        BatchHeader& h = *ctx->h_header;
        // the previous batch may still read the pinned staging copies
        cudaStreamSynchronize(ctx->stream);
        h.num_chunks = nch;
        h.total_paths = used;
        h.total_pixels = pix;
        h.max_depth = depth;
        h.seed = p->seed;
        cudaMemcpyAsync(ctx->d_chunks, ctx->h_chunks, sizeof(Chunk) * nch, cudaMemcpyHostToDevice, ctx->stream);
        cudaMemcpyAsync(ctx->d_header, ctx->h_header, sizeof(BatchHeader), cudaMemcpyHostToDevice, ctx->stream);
        st = run_batch(ctx, p->mode, depth, used, true, p->use_graph != 0);
        if (st != CGPU_OK) return st;
        total_paths += used;
        ctx->stats.batches += 1;
        ctx->stats.h2d_bytes += sizeof(Chunk) * nch + sizeof(BatchHeader);
        collect_profile(ctx);
    }
    ctx->stats.paths = total_paths;
    if (ctx->counting) {
        unsigned long long c[8];
        cudaMemcpyAsync(c, ctx->d_counters, sizeof(c), cudaMemcpyDeviceToHost, ctx->stream);
        cudaStreamSynchronize(ctx->stream);
        ctx->stats.closest_rays = c[0];
        ctx->stats.any_rays = c[1];
        ctx->stats.node_visits = c[2];
        ctx->stats.triangle_tests = c[3];
        ctx->stats.any_node_visits = c[4];
        ctx->stats.any_triangle_tests = c[5];
        ctx->stats.tie_rays = c[6];
    }
    return cg_cuda(ctx, cudaGetLastError(), "render");
}

cgpu_status cg_render_paths_raw(cgpu_ctx* ctx, int scene, int mode, uint32_t first, uint32_t count, uint64_t seed,
                                float* host_rgb) {
    if (scene < 0 || scene >= int(ctx->scenes.size()) || !ctx->scenes[scene].live)
        return cg_fail(ctx, CGPU_ERR_NOT_FOUND, "render_paths: unknown scene id");
    const SceneSlot& sl = ctx->scenes[scene];
    const uint32_t npix = uint32_t(sl.width) * uint32_t(sl.height);
    ctx->batch_spheres = sl.has_spheres;
    ctx->batch_kinds = sl.kinds;
    cgpu_status st = cg_sync_tables(ctx);
    if (st != CGPU_OK) return st;
    st = ensure_path_buffers(ctx, paths_capacity(ctx, npix), sl.max_depth);
    if (st != CGPU_OK) return st;
    st = ensure_sort_buffers(ctx);
    if (st != CGPU_OK) return st;
    const bool persistent = sl.d.num_tris >= kSmallScene && large_batch(ctx, uint64_t(count) * npix);
    choose_traversal(ctx, persistent, persistent);
    float* d_out = nullptr;
    const uint32_t per = std::max<uint32_t>(1, ctx->path_cap / npix);
    cudaError_t e = cudaMalloc(&d_out, size_t(per) * npix * 3 * sizeof(float));
    if (e != cudaSuccess) return cg_cuda(ctx, e, "render_paths buffer");
    for (uint32_t done = 0; done < count;) {
        const uint32_t k = std::min(per, count - done);
        cudaStreamSynchronize(ctx->stream);
        Chunk& c = ctx->h_chunks[0];
        c = Chunk{scene, 0, npix, uint32_t(sl.width), first + done, k, 0, 0};
        BatchHeader& h = *ctx->h_header;
        h.num_chunks = 1;
        h.total_paths = k * npix;
        h.total_pixels = npix;
        h.max_depth = sl.max_depth;
        h.seed = seed;
        cudaMemcpyAsync(ctx->d_chunks, ctx->h_chunks, sizeof(Chunk), cudaMemcpyHostToDevice, ctx->stream);
        cudaMemcpyAsync(ctx->d_header, ctx->h_header, sizeof(BatchHeader), cudaMemcpyHostToDevice, ctx->stream);
        st = run_batch(ctx, mode, sl.max_depth, k * npix, false, false);
        if (st != CGPU_OK) break;
        k_gather_paths<<<grid_for(ctx, k_gather_paths, 256, k * npix), 256, 0, ctx->stream>>>(ctx->wf.L, ctx->wf.Le, ctx->wf.Ls, k * npix, d_out);
        cg_prefault(host_rgb + size_t(done) * npix * 3, size_t(k) * npix * 3 * sizeof(float));
        cudaMemcpyAsync(host_rgb + size_t(done) * npix * 3, d_out, size_t(k) * npix * 3 * sizeof(float),
                        cudaMemcpyDeviceToHost, ctx->stream);
        done += k;
    }
    cudaStreamSynchronize(ctx->stream);
    cudaFree(d_out);
    if (st != CGPU_OK) return st;
    return cg_cuda(ctx, cudaGetLastError(), "render_paths");
}

cgpu_status cg_path_radiance(cgpu_ctx* ctx, int scene, int mode, const double* film_xy, const uint64_t* keys,
                             uint32_t n, float* out_rgb) {
    (void)mode;  // one path per thread either way: both modes share plan_vertex / resolve
    cgpu_status st = cg_sync_tables(ctx);
    if (st != CGPU_OK) return st;
    double* d_xy = nullptr;
    uint64_t* d_keys = nullptr;
    float* d_out = nullptr;
    cudaError_t e = cudaMalloc(&d_xy, size_t(n) * 16);
    if (e == cudaSuccess) e = cudaMalloc(&d_keys, size_t(n) * 8);
    if (e == cudaSuccess) e = cudaMalloc(&d_out, size_t(n) * 12);
    if (e == cudaSuccess) e = cudaMemcpyAsync(d_xy, film_xy, size_t(n) * 16, cudaMemcpyHostToDevice, ctx->stream);
    if (e == cudaSuccess) e = cudaMemcpyAsync(d_keys, keys, size_t(n) * 8, cudaMemcpyHostToDevice, ctx->stream);
    if (e == cudaSuccess) {
        k_paths_explicit<<<grid_for(ctx, k_paths_explicit, kBlock, n), kBlock, 0, ctx->stream>>>(ctx->d_scenes, scene, d_xy,
                                                                                                d_keys, n, d_out);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) cg_prefault(out_rgb, size_t(n) * 12);
    if (e == cudaSuccess) e = cudaMemcpyAsync(out_rgb, d_out, size_t(n) * 12, cudaMemcpyDeviceToHost, ctx->stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(ctx->stream);
    cudaFree(d_xy);
    cudaFree(d_keys);
    cudaFree(d_out);
    return cg_cuda(ctx, e, "path_radiance");
}

// From this many rays the persistent pass answers ray queries, below it one
// thread per ray (us, one thread per ray against the pass, incoherent rays
// through the 1 M-triangle field: closest hit 65,536 rays 120 / 126, 131,072
// 196 / 201 (40,960 triangles: 82 / 78), 524,288 515 / 320, 2,000,003
// 1794 / 757; any hit 1,024 72 / 62, 32,768 85 / 77, 2,000,003 1265 / 600).
constexpr uint32_t kPersistentClosestRays = 1u << 17, kPersistentAnyRays = 1u << 10;
constexpr int kQueryRefill = 28;  // 2,000,003 closest-hit rays: 757 us, 768 at 24, 798 at 20

cgpu_status cg_trace(cgpu_ctx* ctx, int scene, const cgpu_ray* d_rays, uint32_t n, cgpu_hit* d_hits, uint8_t* d_occ,
                     bool any) {
    cgpu_status st = cg_sync_tables(ctx);
    if (st != CGPU_OK) return st;
    if (n == 0) return CGPU_OK;
    if (n >= (any ? kPersistentAnyRays : kPersistentClosestRays)) {
        int* work = reinterpret_cast<int*>(ctx->d_status + 1);
        const bool sph = ctx->scenes[size_t(scene)].has_spheres;
        auto k = any ? (sph ? k_query<true, true> : k_query<true, false>) : (sph ? k_query<false, true> : k_query<false, false>);
        constexpr int block = 64;
        const size_t sm = stack_smem(k, true, !any, block);
        for (uint32_t i = 0; i < n;) {  // the pass counts its rays in an int
            const uint32_t m = std::min<uint32_t>(n - i, 1u << 30);
            cudaMemsetAsync(work, 0, sizeof(int), ctx->stream);
            k<<<grid_for(ctx, k, block, m, sm), block, sm, ctx->stream>>>(ctx->d_scenes, scene, work, d_rays + i, m, kQueryRefill,
                                                                         any ? nullptr : d_hits + i, any ? d_occ + i : nullptr);
            i += m;
        }
        if (!any)
            k_query_resolve<<<grid_for(ctx, k_query_resolve, kBlock, n), kBlock, 0, ctx->stream>>>(ctx->d_scenes, scene, d_rays, n,
                                                                                                 d_hits);
    } else {
        // few rays: a warp per block, so that each has an SM's pipes and L1 to itself
        const int block = n < uint32_t(ctx->num_sms) * kBlock ? 32 : kBlock;
        k_trace<<<grid_for(ctx, k_trace, block, n), block, 0, ctx->stream>>>(ctx->d_scenes, scene, d_rays, n,
                                                                            any ? nullptr : d_hits, any ? d_occ : nullptr);
    }
    return cg_cuda(ctx, cudaGetLastError(), "trace launch");
}

cgpu_status cg_camera(cgpu_ctx* ctx, int scene, const double* d_xy, uint32_t n, float* d_out) {
    cgpu_status st = cg_sync_tables(ctx);
    if (st != CGPU_OK) return st;
    if (n == 0) return CGPU_OK;
    k_camera<<<grid_for(ctx, k_camera, kBlock, n), kBlock, 0, ctx->stream>>>(ctx->d_scenes, scene, d_xy, n, d_out);
    return cg_cuda(ctx, cudaGetLastError(), "camera launch");
}

cgpu_status cg_film_clear(cgpu_ctx* ctx, int scene) {
    SceneSlot& sl = ctx->scenes[scene];
    const size_t npix = size_t(sl.width) * sl.height;
    cudaMemsetAsync(sl.film.sum, 0, npix * 3 * sizeof(double), ctx->stream);
    cudaMemsetAsync(sl.film.sumsq, 0, npix * 3 * sizeof(double), ctx->stream);
    cudaMemsetAsync(sl.film.count, 0, npix * sizeof(double), ctx->stream);
    return cg_cuda(ctx, cudaGetLastError(), "film clear");
}

// ======================================================= wavefront adjoint ==
// cgpu_adjoint_backward on the wavefront schedule.  Per batch: (A) the forward
// wavefront render without the film splat, whose per-path radiance is the Ltot
// of each path and whose passes record what every ray found; (B) the same paths
// shaded again bounce by bounce from the records (k_adj_replay), without a ray:
// 26 bytes a path and bounce with two kinds of material.  With the rays of (B)
// traced again, each vertex's terms kept for a kernel behind them (120 bytes a
// path), the backward call of 512 x 512 pixels, 32 samples, depth 6 took 12.3 ms,
// now 7.2; of 127 x 95, 8 samples, depth 4 1.20 and 0.75.
namespace {

// Most bytes of records a batch takes: 13 million paths of depth 12 through three
// kinds of material.  Beyond that the frame is done in parts.
constexpr uint64_t kAdjRecordBytes = uint64_t(4) << 30;
// Most bytes of state and records the context keeps between calls (all of a batch
// of 11 million paths of depth 6 through two kinds of material); what is larger is
// given back when the call ends.
constexpr size_t kAdjKeep = size_t(2) << 30;

// The launches of bounce b of a batch with records: hits and shade queues are
// the row's own, and so are the outcomes of the rays that the shadow and MIS
// passes of row `outcomes` trace.
void set_records(RenderArgs& a, const AdjRecords& r, int b, int outcomes) {
    const size_t row = size_t(std::min(std::max(b, 0), r.depth - 1)) * r.stride;
    const size_t out = size_t(std::min(std::max(outcomes, 0), r.depth - 1)) * r.stride;
    a.wf.hit = r.hit + row;
    for (int k = 0; k < kNumBsdfKinds; ++k)
        if (r.q_mat[k]) a.wf.q_mat[k] = r.q_mat[k] + row;
    a.rec_shadow = r.shadow + out;
    a.rec_mis = r.mis + out;
}

void enqueue_adjoint_replay(cgpu_ctx* ctx, RenderArgs a, const AdjRecords& rec, int depth, uint32_t paths, size_t shared_bytes) {
    cudaStream_t s = ctx->stream;
    static void (*const replay[kNumBsdfKinds])(RenderArgs, int) = {k_adj_replay<0>, k_adj_replay<1>, k_adj_replay<2>,
                                                                   k_adj_replay<3>, k_adj_replay<4>};
    const int bs = ctx->tuning.block_shade;
    k_adj_begin<<<grid_for(ctx, k_adj_begin, kBlock, paths), kBlock, 0, s>>>(a);
    int grid[kNumBsdfKinds];
    for (int k = 0; k < kNumBsdfKinds; ++k) grid[k] = grid_for(ctx, replay[k], bs, paths, shared_bytes);
    ctx->stats.kernel_launches += 1;
    for (int b = 0; b < depth; ++b) {
        set_records(a, rec, b, b);
        for (int k = 0; k < kNumBsdfKinds; ++k)
            if (ctx->batch_kinds >> k & 1u) {
                replay[k]<<<grid[k], bs, shared_bytes, s>>>(a, b);
                ctx->stats.kernel_launches += 1;
            }
    }
}

// Room for the adjoint state of *paths paths (cg_adjoint_trim).  Where the
// device has not that much left, *paths is halved until it has.
cgpu_status ensure_adj_buffers(cgpu_ctx* ctx, int depth, uint32_t* paths, AdjBufs* a, AdjRecords* r) {
    cudaError_t e = cudaSuccess;
    for (uint32_t n = *paths;; n = (n + 1) / 2) {
        const size_t bytes = adj_layout(nullptr, n, ctx->batch_kinds, depth, a, r);
        e = cudaSuccess;
        if (bytes > ctx->adj_bytes) {
            if (ctx->adj_block) cudaFree(ctx->adj_block);
            ctx->adj_block = nullptr;
            ctx->adj_bytes = 0;
            e = cudaMalloc(&ctx->adj_block, bytes);
            if (e == cudaSuccess) ctx->adj_bytes = bytes;
            else ctx->adj_block = nullptr;
        }
        if (e == cudaSuccess) {
            *paths = n;
            adj_layout(static_cast<char*>(ctx->adj_block), n, ctx->batch_kinds, depth, a, r);
            return CGPU_OK;
        }
        cudaGetLastError();
        if (e != cudaErrorMemoryAllocation || n <= 4096) break;
    }
    return cg_fail(ctx, CGPU_ERR_OUT_OF_MEMORY, "adjoint buffers: " + std::string(cudaGetErrorString(e)));
}

}  // namespace

void cg_adjoint_trim(cgpu_ctx* ctx) {
    if (ctx->adj_bytes <= kAdjKeep) return;
    cudaFree(ctx->adj_block);
    ctx->adj_block = nullptr;
    ctx->adj_bytes = 0;
}

cgpu_status cg_adjoint_wavefront(cgpu_ctx* ctx, int scene, uint32_t spp, uint64_t seed, const AdjBufs& params) {
    const SceneSlot& sl = ctx->scenes[scene];
    const uint32_t npix = uint32_t(sl.width) * uint32_t(sl.height);
    ctx->batch_spheres = sl.has_spheres;
    ctx->batch_kinds = sl.kinds;
    cgpu_status st = cg_sync_tables(ctx);
    if (st != CGPU_OK) return st;
    st = ensure_path_buffers(ctx, paths_capacity(ctx, npix), sl.max_depth);
    if (st != CGPU_OK) return st;
    const int depth = sl.max_depth;
    const size_t shared_bytes = size_t(params.nmat + 3 * params.nlight) * sizeof(double);
    RenderArgs a = make_args(ctx);
    a.adj = params;
    // a batch: whole samples of the frame or, where the records of one sample
    // take more than kAdjRecordBytes, parts of one
    const uint64_t want = std::min<uint64_t>({ctx->path_cap, uint64_t(spp) * npix,
                                              std::max<uint64_t>(1, kAdjRecordBytes / adj_record_bytes(sl.kinds, depth))});
    uint32_t room = uint32_t(want);
    AdjRecords rec;
    st = ensure_adj_buffers(ctx, depth, &room, &a.adj, &rec);
    if (st != CGPU_OK) return st;
    if (shared_bytes > 48 * 1024) {
        const int sb = int(shared_bytes);
        cudaFuncSetAttribute(k_adj_replay<0>, cudaFuncAttributeMaxDynamicSharedMemorySize, sb);
        cudaFuncSetAttribute(k_adj_replay<1>, cudaFuncAttributeMaxDynamicSharedMemorySize, sb);
        cudaFuncSetAttribute(k_adj_replay<2>, cudaFuncAttributeMaxDynamicSharedMemorySize, sb);
        cudaFuncSetAttribute(k_adj_replay<3>, cudaFuncAttributeMaxDynamicSharedMemorySize, sb);
        cudaFuncSetAttribute(k_adj_replay<4>, cudaFuncAttributeMaxDynamicSharedMemorySize, sb);
    }
    ctx->stats = cgpu_render_stats{};
    const bool persistent = sl.d.num_tris >= kSmallScene && large_batch(ctx, uint64_t(spp) * npix);
    choose_traversal(ctx, persistent, persistent);
    const uint32_t per = std::max<uint32_t>(1, room / npix), part = std::min(room, npix);
    for (uint32_t done = 0, pixel0 = 0; done < spp;) {
        const uint32_t pixels = std::min(part, npix - pixel0);
        const uint32_t k = std::min(per, spp - done);
        const uint32_t paths = k * pixels;
        cudaStreamSynchronize(ctx->stream);
        ctx->h_chunks[0] = Chunk{scene, 0, pixels, uint32_t(sl.width), done, k, 0, pixel0};
        BatchHeader& h = *ctx->h_header;
        h.num_chunks = 1;
        h.total_paths = paths;
        h.total_pixels = pixels;
        h.max_depth = depth;
        h.seed = seed;
        cudaMemcpyAsync(ctx->d_chunks, ctx->h_chunks, sizeof(Chunk), cudaMemcpyHostToDevice, ctx->stream);
        cudaMemcpyAsync(ctx->d_header, ctx->h_header, sizeof(BatchHeader), cudaMemcpyHostToDevice, ctx->stream);
        st = enqueue_wavefront(ctx, depth, paths, false, &rec);
        if (st != CGPU_OK) return st;
        enqueue_adjoint_replay(ctx, a, rec, depth, paths, shared_bytes);
        st = cg_cuda(ctx, cudaGetLastError(), "adjoint wavefront launch");
        if (st != CGPU_OK) return st;
        ctx->stats.batches += 1;
        pixel0 += pixels;
        if (pixel0 == npix) {
            pixel0 = 0;
            done += k;
        }
    }
    ctx->stats.paths = uint64_t(spp) * npix;
    collect_profile(ctx);  // the forward passes' events, with profiling on
    return CGPU_OK;
}

// =========================================================== no-alloc render ==
// cgpu_render_noalloc: the wavefront render of one scene with every device
// buffer the call needs in a static array of this library, so that the call
// itself allocates nothing.  Same kernels as cgpu_render; the batch tables are
// written by a one-block setup kernel (arguments by value, no copies), and the
// ray passes of a bounce are one launch on the context stream (with traversal 0
// and 4; else one after the other: no side stream, no events, no graph).

static __device__ __align__(256) unsigned char g_noalloc_scratch[kNoAllocScratchBytes];

namespace cg {

// Writes the batch tables and zeroes the queue counters of one batch.
__global__ void k_noalloc_setup(NoAllocView v, BatchHeader h, Chunk c, SceneD sd, FilmD fd, int scene, int cnt_ints) {
    for (int i = threadIdx.x; i < cnt_ints; i += blockDim.x) v.wf.cnt[i] = 0;
    if (threadIdx.x == 0) {
        *v.header = h;
        *v.chunk = c;
        v.scenes[scene] = sd;
        v.films[scene] = fd;
    }
}

}  // namespace cg

namespace {

constexpr int kNoAllocMaxDevices = 64;
std::mutex g_noalloc_mu;
char* g_noalloc_base[kNoAllocMaxDevices] = {};

// Device address of the scratch, looked up once per device (the caller has
// made ctx->device current).
cgpu_status noalloc_base(cgpu_ctx* ctx, char** out) {
    if (ctx->device < 0 || ctx->device >= kNoAllocMaxDevices)
        return cg_fail(ctx, CGPU_ERR_INVALID_ARGUMENT, "render_noalloc: device index out of range");
    std::lock_guard<std::mutex> lock(g_noalloc_mu);
    char*& p = g_noalloc_base[ctx->device];
    if (!p) {
        void* a = nullptr;
        const cudaError_t e = cudaGetSymbolAddress(&a, g_noalloc_scratch);
        if (e != cudaSuccess) return cg_cuda(ctx, e, "render_noalloc: scratch address");
        p = static_cast<char*>(a);
    }
    *out = p;
    return CGPU_OK;
}

void enqueue_wavefront_serial(cgpu_ctx* ctx, const RenderArgs& a, int depth, uint32_t paths, uint32_t npix) {
    cudaStream_t s = ctx->stream;
    const int bt = ctx->tuning.block_trace, bs = ctx->tuning.block_shade;
    const int trav = ctx->batch_closest, trav_any = ctx->batch_any;
    const bool sph = ctx->batch_spheres;
    auto ext = trav == 1   ? (sph ? k_wf_extend_dyn<false, true> : k_wf_extend_dyn<false, false>)
               : trav >= 2 ? (sph ? k_wf_extend_pww<false, true> : k_wf_extend_pww<false, false>)
                           : (sph ? k_wf_extend<false, true> : k_wf_extend<false, false>);
    auto sh = trav_any == 1   ? (sph ? k_wf_shadow_dyn<false, true> : k_wf_shadow_dyn<false, false>)
              : trav_any == 3 ? (sph ? k_wf_shadow_pww<false, true> : k_wf_shadow_pww<false, false>)
                          : (sph ? k_wf_shadow<false, true> : k_wf_shadow<false, false>);
    k_wf_generate<<<grid_for(ctx, k_wf_generate, kBlock, paths), kBlock, 0, s>>>(a);
    const size_t ext_sm = stack_smem(ext, trav >= 2, true, bt), sh_sm = stack_smem(sh, trav_any == 3, false, bt);
    const int gext = grid_for(ctx, ext, bt, paths, ext_sm), gsh = grid_for(ctx, sh, bt, paths, sh_sm);
    const int gsd[kNumBsdfKinds] = {grid_for(ctx, k_wf_shade<0>, bs, paths), grid_for(ctx, k_wf_shade<1>, bs, paths),
                                    grid_for(ctx, k_wf_shade<2>, bs, paths), grid_for(ctx, k_wf_shade<3>, bs, paths),
                                    grid_for(ctx, k_wf_shade<4>, bs, paths)};
    auto mocc = sph ? k_wf_mis_occl<false, true> : k_wf_mis_occl<false, false>;
    auto ties = sph ? k_wf_ties<false, true> : k_wf_ties<false, false>;
    const int gmo = grid_for(ctx, mocc, bt, paths);
    const int gties = grid_for(ctx, ties, kTieBlock, paths);
    auto rays = sph ? k_wf_rays<true> : k_wf_rays<false>;
    const int grays = 3 * grid_for(ctx, rays, bt, paths);
    const bool one = trav == 0 && trav_any == 0;
    for (int b = 0; b <= depth; ++b) {
        if (one && b > 0) {
            rays<<<grays, bt, 0, s>>>(a, b);
        } else {
            ext<<<gext, bt, ext_sm, s>>>(a, b);
            if (trav >= 2) ties<<<gties, kTieBlock, 0, s>>>(a, b);
            if (b > 0) sh<<<gsh, bt, sh_sm, s>>>(a, b);
            if (b > 0) mocc<<<gmo, bt, 0, s>>>(a, b);
        }
        if (b == depth) break;
        ctx->stats.kernel_launches += launch_shade(ctx, a, b, gsd);
    }
    k_splat<<<grid_for(ctx, k_splat, kSplatBlock, npix), kSplatBlock, 0, s>>>(a);
    ctx->stats.kernel_launches += uint32_t(4 + (one ? depth : 3 * depth) + (trav >= 2 ? depth + 1 : 0));
}

}  // namespace

extern "C" cgpu_status cgpu_render_noalloc(cgpu_ctx* ctx, int32_t scene, uint32_t first_sample, uint32_t num_samples,
                                           uint64_t seed) {
    if (!ctx) return CGPU_ERR_INVALID_ARGUMENT;
    if (scene < 0 || scene >= int32_t(ctx->scenes.size()) || !ctx->scenes[size_t(scene)].live)
        return cg_fail(ctx, CGPU_ERR_NOT_FOUND, "render_noalloc: unknown scene id");
    const SceneSlot& sl = ctx->scenes[size_t(scene)];
    const uint64_t npix = uint64_t(sl.width) * uint64_t(sl.height);
    if (scene >= kNoAllocMaxScenes)
        return cg_fail(ctx, CGPU_ERR_INVALID_ARGUMENT, "render_noalloc: scene id " + std::to_string(scene) +
                                                           " is not below the static scratch's " +
                                                           std::to_string(kNoAllocMaxScenes) + " scene slots");
    if (npix > kNoAllocMaxPaths)
        return cg_fail(ctx, CGPU_ERR_INVALID_ARGUMENT, "render_noalloc: " + std::to_string(sl.width) + " x " +
                                                           std::to_string(sl.height) + " pixels exceed the " +
                                                           std::to_string(kNoAllocMaxPaths) +
                                                           " paths of the static scratch");
    if (sl.max_depth > kNoAllocMaxDepth)
        return cg_fail(ctx, CGPU_ERR_INVALID_ARGUMENT, "render_noalloc: max depth " + std::to_string(sl.max_depth) +
                                                           " exceeds " + std::to_string(kNoAllocMaxDepth));
    if (uint64_t(first_sample) + num_samples > 0xFFFFFFFFull)
        return cg_fail(ctx, CGPU_ERR_INVALID_ARGUMENT, "render_noalloc: sample range overflows 32 bits");
    if (num_samples == 0) return CGPU_OK;
    cudaError_t e = cudaSetDevice(ctx->device);
    if (e != cudaSuccess) return cg_cuda(ctx, e, "render_noalloc: set device");
    char* base = nullptr;
    cgpu_status st = noalloc_base(ctx, &base);
    if (st != CGPU_OK) return st;
    NoAllocView v;
    if (noalloc_layout(base, &v) > kNoAllocScratchBytes)
        return cg_fail(ctx, CGPU_ERR_UNSUPPORTED, "render_noalloc: scratch layout exceeds the static array");
    RenderArgs a{};
    a.scenes = v.scenes;
    a.chunks = v.chunk;
    a.header = v.header;
    a.films = v.films;
    a.wf = v.wf;
    a.counters = v.counters;
    a.refill_closest = refill_lanes(ctx->tuning.refill_closest);
    a.refill_any = refill_lanes(ctx->tuning.refill_any);
    const uint32_t n = uint32_t(npix);
    choose_traversal(ctx, false, false);
    const uint32_t per = kNoAllocMaxPaths / n;  // samples per batch
    const int depth = sl.max_depth;
    ctx->batch_spheres = sl.has_spheres;
    ctx->batch_kinds = sl.kinds;
    ctx->stats = cgpu_render_stats{};
    for (uint32_t done = 0; done < num_samples;) {
        const uint32_t k = std::min(per, num_samples - done);
        BatchHeader h;
        h.num_chunks = 1;
        h.total_paths = k * n;
        h.total_pixels = n;
        h.max_depth = depth;
        h.seed = seed;
        const Chunk c{scene, 0, n, uint32_t(sl.width), first_sample + done, k, 0, 0};
        k_noalloc_setup<<<1, 256, 0, ctx->stream>>>(v, h, c, sl.d, sl.film, scene, (depth + 2) * kCntStride);
        enqueue_wavefront_serial(ctx, a, depth, k * n, n);
        ctx->stats.batches += 1;
        ctx->stats.paths += uint64_t(k) * n;
        done += k;
    }
    return cg_cuda(ctx, cudaGetLastError(), "render_noalloc launch");
}
