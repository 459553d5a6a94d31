// CPU execution of what follows the persistent passes' closest hits (tie_hit)
// and of queries against every record of a scene (test infrastructure, never
// part of the library).
#include "../../cadise_gb300/csrc/scene_build.h"
#include "../../cadise_gb300/csrc/traverse.cuh"

#include <cmath>
#include <cstdint>
#include <cstdio>
#include <memory>
#include <string>

namespace {
struct Scene {
    cg::HostScene hs;
    cg::SceneD S;
};

cg::RayPre prep(const float* r) {
    return cg::ray_prep(cg::mk(r[0], r[1], r[2]), cg::normalize(cg::mk(r[4], r[5], r[6])), r[3], r[7]);
}

bool record_hit(const cg::SceneD& S, const cg::RayPre& r, size_t i, float bound, float* t) {
    const float4 a = S.tris[i].v0, b = S.tris[i].v1, c = S.tris[i].v2;
    float u, v;
    if ((__float_as_uint(c.w) & 3u) == cg::kRecSphere) return cg::sphere_test(r, cg::f3(a), b.x, bound, t);
    return cg::tri_test(r, cg::f3(a), cg::f3(b), cg::f3(c), bound, t, &u, &v);
}
}  // namespace

extern "C" {

void* tc_create(const cgpu_scene_desc* d, char* err, int errlen) {
    auto s = std::make_unique<Scene>();
    std::string e;
    if (cg::build_host_scene(d, &s->hs, &e) != CGPU_OK) {
        std::snprintf(err, size_t(errlen), "%s", e.c_str());
        return nullptr;
    }
    s->S = cg::host_view(s->hs, d);
    return s.release();
}

void tc_destroy(void* p) { delete static_cast<Scene*>(p); }

// Per ray (8 floats): the record with the smallest distance of all (held[0], -1
// a miss; held[1] how many records lie within the tie window of it, itself
// included), the record that tie_hit returns for it with several others within
// the window, and the record of the traversal from the origin.
void tc_several(void* p, const float* rays, uint32_t n, int32_t* held, int32_t* resolved, int32_t* general) {
    const Scene& sc = *static_cast<Scene*>(p);
    const cg::SceneD& S = sc.S;
    for (uint32_t i = 0; i < n; ++i) {
        const cg::RayPre r = prep(rays + 8 * size_t(i));
        cg::HitD h{r.tmax, -1, 0.0f, 0.0f};
        for (size_t k = 0; k < sc.hs.tris.size(); ++k) {
            float t;
            if (record_hit(S, r, k, h.t, &t) && (h.slot < 0 || t < h.t)) {
                h.t = t;
                h.slot = int(k);
            }
        }
        held[2 * i] = h.slot;
        held[2 * i + 1] = 0;
        resolved[i] = -1;
        cg::TraceCounters tc{0, 0};
        cg::HitD g;
        general[i] = cg::traverse<false, false>(S, r, &g, &tc) ? g.slot : -1;
        if (h.slot < 0) continue;
        for (size_t k = 0; k < sc.hs.tris.size(); ++k) {
            float t;
            held[2 * i + 1] += record_hit(S, r, k, cg::tie_hi(S, r, h.t), &t);
        }
        resolved[i] = cg::tie_hit<false, true>(S, r, h, -2, &tc).slot;
    }
}

// Per ray (8 floats): t[3 i] the smallest distance of all records, t[3 i + 1] that
// of the traversal, t[3 i + 2] that of the warp traversal (3.4e38: a miss);
// any[i] the any-hit traversal's answer; window[i] how far two distances may lie
// apart and still be ordered by the reference's rule.
void tc_closest(void* p, const float* rays, uint32_t n, float* t, int32_t* any, float* window) {
    const Scene& sc = *static_cast<Scene*>(p);
    const cg::SceneD& S = sc.S;
    for (uint32_t i = 0; i < n; ++i) {
        const cg::RayPre r = prep(rays + 8 * size_t(i));
        float best = r.tmax, tk;
        bool found = false;
        for (size_t k = 0; k < sc.hs.tris.size(); ++k)
            if (record_hit(S, r, k, best, &tk) && tk <= best) {
                best = tk;
                found = true;
            }
        cg::TraceCounters tc{0, 0};
        cg::HitD a, b, c;
        t[3 * i] = found ? best : 3.4e38f;
        t[3 * i + 1] = cg::traverse<false, false>(S, r, &a, &tc) ? a.t : 3.4e38f;
        t[3 * i + 2] = cg::traverse_warp<false>(S, r, &b, &tc) ? b.t : 3.4e38f;
        any[i] = cg::traverse<true, false>(S, r, &c, &tc);
        window[i] = std::fabs(cg::tie_hi(S, r, best) - best);
    }
}

}  // extern "C"
