// CPU execution of the persistent passes' own triangle test (test
// infrastructure, never part of the library).
#include "../../cadise_gb300/csrc/traverse.cuh"

#include <cstdint>

extern "C" {

// tri_test and tri_test_rot of n (ray, triangle) pairs: rays 8 floats (org,
// t_min, dir, t_max), triangles 9.  hit[2 i] / t[2 i] from tri_test, the odd
// entries from tri_test_rot.
void pc_tri(const float* rays, const float* tris, uint32_t n, int32_t* hit, float* t) {
    for (uint32_t i = 0; i < n; ++i) {
        const float* r = rays + 8 * size_t(i);
        const float* v = tris + 9 * size_t(i);
        const float3 A = cg::mk(v[0], v[1], v[2]), B = cg::mk(v[3], v[4], v[5]), C = cg::mk(v[6], v[7], v[8]);
        const float3 o = cg::mk(r[0], r[1], r[2]), d = cg::mk(r[4], r[5], r[6]);
        const cg::RayPre p = cg::ray_prep(o, d, r[3], r[7]);
        float u, w;
        t[2 * i] = t[2 * i + 1] = 0.0f;
        hit[2 * i] = cg::tri_test(p, A, B, C, r[7], t + 2 * i, &u, &w);
        // the shear as the persistent passes compute it: kz, then the next two axes in turn
        const int kz = p.kz, kx = (kz + 1) % 3, ky = (kz + 2) % 3;
        const float dz = cg::comp(d, kz);
        hit[2 * i + 1] = cg::tri_test_rot(o, kz, cg::comp(d, kx) / dz, cg::comp(d, ky) / dz, 1.0f / dz, r[3], A, B, C,
                                          r[7], t + 2 * i + 1);
    }
}

}  // extern "C"
