// The persistent traversal pass: warps that stay on the chip, hand every
// finished lane the next ray of the queue, and vote at each step whether the
// whole warp visits inner nodes or tests triangles.
//
// What bounds it: the ALU pipe (73 % busy), issue slots and L1 / L2 latency of
// divergent node fetches; the scene sits in L2 and DRAM is idle.  So the pass
// is built for few instructions and full steps:
//  * One step visits one node, or tests one triangle, in every lane that has
//    one pending (a while-while loop with postponed leaves, Aila & Laine, HPG
//    2009, cut into uniform steps): 21 of 32 lanes active per instruction,
//    against 11.6 when every lane ran its own inner loop.
//  * The bookkeeping of a step is straight-line predicated code: the loops of
//    branches that popped, culled and promoted entries cost more than the box
//    tests (BRA / BSSY / BSYNC 17 % of all instructions, now 8 %).
//  * Children: the nearest next, the others onto the stack in slot order; a
//    full sort visits 3 % fewer nodes but costs more.
//  * A node comes in two 32-byte loads instead of four of 16 (L1 tag look-ups
//    halved).
// Closest-hit passes of the 1 M-triangle 1080p frame, 16 samples a pixel:
// 52.5 ms with the inner loops, 34.1 here; any-hit passes 25.0 and 17.8 ms.
#pragma once

#include "traverse.cuh"

#ifdef __CUDACC__
namespace cg {

constexpr unsigned kFullWarp = 0xFFFFFFFFu;
// Rays a warp reserves from the queue with one atomic.
constexpr int kFetchChunk = 32;
// The warp takes triangles once kLeafLanes lanes hold a leaf, or when fewer
// than kNodeLanes still have a node (ms of the frame above: 8 / 12 71.2,
// 12 / 12 72.0, 8 / 16 73.9).
constexpr int kNodeLanes = 8, kLeafLanes = 12;
// Steps between two looks at the refill threshold: finished lanes wait a few
// steps, so that a refill serves several (ms at thresholds 24 / 26 and 28 / 32:
// every step 71.2 and 74.7, every 4th 70.2 and 71.4, every 6th 70.1 and 70.3).
constexpr int kRoundSteps = 6;

// This lane's traversal stack: kSmemStack entries in shared memory, entry k of
// lane l at row k of its warp (neighbouring lanes in neighbouring banks).  `sp`
// is the shared address of the next free entry.  A ray that runs out of them
// (2 in 100,000 on the million-triangle field) moves its oldest kSpill entries
// to local memory and takes them back when it has emptied the rest.
// Closest hit: an entry is (child entry, distance); any hit: the child entry.
// More rows cost L1 capacity, fewer cost spills: 16 rows 34.1 ms of closest-hit
// passes, 12 rows 36.3, 11 rows 37.5.
constexpr int kSmemStack = 16, kSpill = 8;
// the dynamic shared memory of a persistent traversal launch
extern __shared__ __align__(16) uint32_t trav_stack_smem[];

constexpr int kSlotMask = int(kMaxTriSlots);

// Shared memory of a block of `threads` threads.
constexpr CG_HD uint32_t persist_warp_bytes(bool with_t) { return uint32_t(kSmemStack) * 32u * (with_t ? 8u : 4u); }
constexpr size_t persist_bytes(int threads, bool with_t) { return size_t(threads / 32) * persist_warp_bytes(with_t); }

template <bool WITH_T>
struct PStack {
    static constexpr uint32_t kEntry = WITH_T ? 8u : 4u;
    static constexpr uint32_t kRow = 32u * kEntry;
    uint32_t base, sp;
    int spilled;
    static constexpr int kOver = kStackSize - kSmemStack + kSpill;

    CG_D void bind() {
        base = uint32_t(__cvta_generic_to_shared(trav_stack_smem)) + (threadIdx.x >> 5) * persist_warp_bytes(WITH_T) +
               (threadIdx.x & 31u) * kEntry;
        clear();
    }
    CG_D void clear() {
        sp = base;
        spilled = 0;
    }
    static CG_D uint2 load(uint32_t at) {
        uint2 e{0u, 0u};
        if (WITH_T) asm volatile("ld.shared.v2.b32 {%0, %1}, [%2];" : "=r"(e.x), "=r"(e.y) : "r"(at));
        else asm volatile("ld.shared.b32 %0, [%1];" : "=r"(e.x) : "r"(at));
        return e;
    }
    static CG_D void store(uint32_t at, uint2 e) {
        if (WITH_T) asm volatile("st.shared.v2.b32 [%0], {%1, %2};" ::"r"(at), "r"(e.x), "r"(e.y));
        else asm volatile("st.shared.b32 [%0], %1;" ::"r"(at), "r"(e.x));
    }
};

// The rare moves between the shared rows and local memory, out of line so that
// they cost the passes no registers.  Both return (sp, spilled).
template <bool WITH_T>
__device__ __noinline__ uint2 stack_spill_out(uint32_t base, uint32_t sp, uint32_t* over, int spilled) {
    using St = PStack<WITH_T>;
    constexpr int W = WITH_T ? 2 : 1;
    // (a tree within the upload's depth limit never needs more than kOver)
    if (spilled <= St::kOver - kSpill) {
        for (int i = 0; i < kSpill; ++i) {
            const uint2 e = St::load(base + uint32_t(i) * St::kRow);
            over[(spilled + i) * W] = e.x;
            if (WITH_T) over[(spilled + i) * W + 1] = e.y;
        }
        spilled += kSpill;
    }
    for (uint32_t at = base; at + kSpill * St::kRow < sp; at += St::kRow) St::store(at, St::load(at + kSpill * St::kRow));
    return make_uint2(sp - kSpill * St::kRow, uint32_t(spilled));
}
template <bool WITH_T>
__device__ __noinline__ uint2 stack_spill_in(uint32_t base, const uint32_t* over, int spilled) {
    using St = PStack<WITH_T>;
    constexpr int W = WITH_T ? 2 : 1;
    spilled -= kSpill;
    for (int i = 0; i < kSpill; ++i)
        St::store(base + uint32_t(i) * St::kRow, make_uint2(over[(spilled + i) * W], WITH_T ? over[(spilled + i) * W + 1] : 0u));
    return make_uint2(base + kSpill * St::kRow, uint32_t(spilled));
}

// What the pass keeps of a ray.
template <bool SPH>
struct PRay {
    float3 o, inv;
    float Sx, Sy, Sz;
    int kz;
};
template <>
struct PRay<true> : PRay<false> {
    float3 d;
};

// The ray's part of tri_test and child_hits (ray_prep), with 1 / d from the
// reciprocal unit (kBoxSlack covers its rounding) but the shear exact.
template <bool SPH>
CG_D void pray_prep(PRay<SPH>& r, float3 d) {
    const float e = 1e-30f;
    auto rcp = [e](float x) {
        const float y = fabsf(x) < e ? copysignf(e, x) : x;
        float i;
        asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(i) : "f"(y));
        return i;
    };
    r.inv = mk(rcp(d.x), rcp(d.y), rcp(d.z));
    const float ax = fabsf(d.x), ay = fabsf(d.y), az = fabsf(d.z);
    int kz = 0;
    if (ay > ax) kz = 1;
    if (az > fmaxf(ax, ay)) kz = 2;
    r.kz = kz;
    const float dz = kz == 0 ? d.x : kz == 1 ? d.y : d.z;
    r.Sx = (kz == 0 ? d.y : kz == 1 ? d.z : d.x) / dz;
    r.Sy = (kz == 0 ? d.z : kz == 1 ? d.x : d.y) / dz;
    r.Sz = 1.0f / dz;
    if constexpr (SPH) r.d = d;
}

// One pass over the `n` rays of a queue.  fetch(k, &o, &d, &tmin, &tmax, &scene)
// loads entry k and returns the caller's id of the ray; finish(done, id, t,
// slot, kind, other) is called by the whole warp with the lanes whose ray is done
// (slot < 0: a miss; kind: the record's shade queue; other: the record that met
// the ray within the tie reach of slot, -1 none, -2 more than one);
// exhausted(id): the ray ran out of its visit budget.
// The tie reach of a hit is three tie windows wide, and closest-hit rays cull by
// its far end, so that every record within it is met, whatever the order of the
// visits.  Two windows hold all records that tie with the hit or with one that
// ties with it: of a hit and a single other in its reach the two alone decide
// (tie_hit).  The third stands in for box_widen.
// GENERAL (ray queries): every ray has its own tmin, which may be negative; the
// render's rays all start at kRayEps.
template <bool ANY, bool COUNT, bool SPH, bool GENERAL, class Fetch, class Finish, class Exhausted>
CG_D void persistent_pass(const SceneD* scenes, int* work, int n, int refill, Fetch&& fetch, Finish&& finish,
                          Exhausted&& exhausted, TraceCounters& tc) {
    PStack<!ANY> stack;
    uint32_t over[PStack<!ANY>::kOver * (ANY ? 1 : 2)];  // the entries beyond the shared rows
    stack.bind();
    PRay<SPH> r{};
    const Bvh4Node* nodes = nullptr;
    const TriRecord* tris = nullptr;
    float tie_abs = 0.0f;  // the absolute part of the tie reach
    float tcur = 0.0f, ray_tmin = 0.0f;
    int hslot = -1;
    int other = -1;      // the record within the tie reach of hslot: -1 none, -2 more than one
    int left = 0;        // node and leaf visits left, negative once the budget is exceeded
    int cur = -1;        // next entry: an inner node (>= 0), a leaf (< -1), -1 none
    int leaf = -1;       // postponed leaf, -1 none
    int p = -1;          // this lane's ray (< 0: none)
    int pool = 0, pool_end = 0;
    bool drained = false;
    const int lane = threadIdx.x & 31;
    float box_abs = 0.0f;
    // the far end of the tie reach, and box_widen: at a negative t the relative part
    // shrinks the bound, and the absolute parts make up for it
    auto reach = [&](float t) { return fmaf(t, 1.0f + 3.0f * kTieSlack, tie_abs); };
    auto widen = [&](float t) { return GENERAL ? fmaf(t, 1.0f + kBoxSlack, box_abs) : t * (1.0f + kBoxSlack); };

    for (;;) {
        // ---- finished lanes take the next rays of the warp's share of the queue
        unsigned need = __ballot_sync(kFullWarp, p < 0);
        while (need != 0 && !drained) {
            if (pool == pool_end) {
                int base = 0;
                if (lane == 0) base = atomicAdd(work, kFetchChunk);
                pool = __shfl_sync(kFullWarp, base, 0);
                pool_end = min(pool + kFetchChunk, n);
                if (pool >= pool_end) {
                    pool = pool_end = 0;
                    drained = true;
                    break;
                }
            }
            const int rank = __popc(need & ((1u << lane) - 1u));
            if (p < 0 && rank < pool_end - pool) {
                float3 d;
                int scene = 0;
                tcur = kFloatMax;
                p = fetch(pool + rank, &r.o, &d, &ray_tmin, &tcur, &scene);
                const SceneD* S = scenes + scene;
                nodes = S->nodes;
                tris = S->tris;
                if (!ANY) tie_abs = 3.0f * S->tie_abs;
                if (GENERAL) {
                    // no distance in the scene is below -far
                    const float far = fminf(fmaxf(-ray_tmin, 0.0f),
                                            fabsf(r.o.x) + fabsf(r.o.y) + fabsf(r.o.z) + 0x1p17f * S->tie_abs);
                    box_abs = 2.0f * kBoxSlack * far;
                    if (!ANY) tie_abs += 6.0f * kTieSlack * far;
                }
                left = int(min(S->visit_budget, 0x7FFFFFFFu));
                pray_prep(r, d);
                hslot = -1;
                other = -1;
                cur = 0;
                leaf = -1;
                stack.clear();
            }
            pool += min(__popc(need), pool_end - pool);
            need = __ballot_sync(kFullWarp, p < 0);
        }
        if (need == kFullWarp) break;
        // ---- steps
        for (int round = kRoundSteps - 1;;) {
            const float tmin = GENERAL ? ray_tmin : kRayEps;
            const float tlim = ANY ? widen(tcur) : reach(tcur);
            // a leaf is postponed (once); a lane without a node takes its next
            // stack entry (one a step: a culled one costs it the step)
            if (cur < -1 && leaf == -1) {
                leaf = cur;
                cur = -1;
                --left;
            }
            if (ANY) {
                asm volatile(
                    "{\n\t.reg .pred p;\n\t"
                    "setp.ne.u32 p, %1, %2;\n\t"
                    "setp.eq.and.s32 p, %0, -1, p;\n\t"
                    "@p sub.u32 %1, %1, 128;\n\t"
                    "@p ld.shared.b32 %0, [%1];\n\t}"
                    : "+r"(cur), "+r"(stack.sp)
                    : "r"(stack.base));
            } else {
                asm volatile(
                    "{\n\t.reg .pred p, q;\n\t.reg .b32 e;\n\t.reg .f32 t;\n\t"
                    "mov.f32 t, 0f00000000;\n\t"
                    "mov.b32 e, 0;\n\t"
                    "setp.ne.u32 p, %1, %2;\n\t"
                    "setp.eq.and.s32 p, %0, -1, p;\n\t"
                    "@p sub.u32 %1, %1, 256;\n\t"
                    "@p ld.shared.v2.b32 {e, t}, [%1];\n\t"
                    "setp.le.and.f32 q, t, %3, p;\n\t"
                    "@q mov.b32 %0, e;\n\t}"
                    : "+r"(cur), "+r"(stack.sp)
                    : "r"(stack.base), "f"(tlim));
            }
            if (cur < -1 && leaf == -1) {
                leaf = cur;
                cur = -1;
                --left;
            }
            const bool inner = cur >= 0 && left > 0, tri = leaf != -1 && left >= 0;
            const unsigned bi = __ballot_sync(kFullWarp, inner);
            const unsigned bl = __ballot_sync(kFullWarp, tri);
            if ((bi | bl) == 0 || --round < 0) {
                round = kRoundSteps - 1;
                // lanes whose stack entry was culled go on as well
                const unsigned pend = __ballot_sync(kFullWarp, cur == -1 && stack.sp != stack.base && left >= 0);
                const int live = __popc(bi | bl | pend);
                if (live < refill && (live == 0 || !drained)) break;
                if ((bi | bl) == 0) continue;
            }
            const int ni = __popc(bi), nl = __popc(bl);
            if (ni != 0 && nl < kLeafLanes && (ni >= kNodeLanes || nl == 0)) {
                if (inner) {
                    --left;
                    float4 nd[4];
                    load_node(nodes, uint32_t(cur), nd);
                    if (COUNT) tc.nodes++;
                    float tn[4];
                    child_hits(r.o, r.inv, tmin, nd, tlim, widen, tn);
                    const uint32_t ce[4] = {__float_as_uint(nd[1].x), __float_as_uint(nd[1].y),
                                            __float_as_uint(nd[1].z), __float_as_uint(nd[1].w)};
                    // room for the three children a visit may push
                    if (stack.sp > stack.base + uint32_t(kSmemStack - 3) * PStack<!ANY>::kRow) {
                        const uint2 m = stack_spill_out<!ANY>(stack.base, stack.sp, over, stack.spilled);
                        stack.sp = m.x;
                        stack.spilled = int(m.y);
                    }
                    if (ANY) {
                        cur = -1;
#pragma unroll
                        for (int i = 3; i >= 0; --i) {
                            // a hit child takes the place of the one before it, which goes onto the stack
                            asm volatile(
                                "{\n\t.reg .pred p, q;\n\t"
                                "setp.lt.f32 p, %2, 0f7F800000;\n\t"
                                "setp.ne.and.s32 q, %1, -1, p;\n\t"
                                "@q st.shared.b32 [%0], %1;\n\t"
                                "@q add.u32 %0, %0, 128;\n\t"
                                "@p mov.b32 %1, %3;\n\t}"
                                : "+r"(stack.sp), "+r"(cur)
                                : "f"(tn[i]), "r"(ce[i]));
                        }
                    } else {
                        // the nearest child next, the others onto the stack in slot order
                        const float m = fminf(fminf(tn[0], tn[1]), fminf(tn[2], tn[3]));
                        asm volatile(
                            "{\n\t.reg .pred c0, c1, c2, c01, c012, p;\n\t"
                            "setp.eq.f32 c0, %2, %6;\n\t"
                            "setp.eq.and.f32 c1, %3, %6, !c0;\n\t"
                            "or.pred c01, c0, c1;\n\t"
                            "setp.eq.and.f32 c2, %4, %6, !c01;\n\t"
                            "or.pred c012, c01, c2;\n\t"
                            "setp.lt.and.f32 p, %5, 0f7F800000, c012;\n\t"
                            "@p st.shared.v2.b32 [%0], {%10, %5};\n\t"
                            "@p add.u32 %0, %0, 256;\n\t"
                            "setp.lt.and.f32 p, %4, 0f7F800000, !c2;\n\t"
                            "@p st.shared.v2.b32 [%0], {%9, %4};\n\t"
                            "@p add.u32 %0, %0, 256;\n\t"
                            "setp.lt.and.f32 p, %3, 0f7F800000, !c1;\n\t"
                            "@p st.shared.v2.b32 [%0], {%8, %3};\n\t"
                            "@p add.u32 %0, %0, 256;\n\t"
                            "setp.lt.and.f32 p, %2, 0f7F800000, !c0;\n\t"
                            "@p st.shared.v2.b32 [%0], {%7, %2};\n\t"
                            "@p add.u32 %0, %0, 256;\n\t"
                            "selp.b32 %1, %9, %10, c2;\n\t"
                            "selp.b32 %1, %8, %1, c1;\n\t"
                            "selp.b32 %1, %7, %1, c0;\n\t"
                            "setp.lt.f32 p, %6, 0f7F800000;\n\t"
                            "selp.b32 %1, %1, -1, p;\n\t}"
                            : "+r"(stack.sp), "+r"(cur)
                            : "f"(tn[0]), "f"(tn[1]), "f"(tn[2]), "f"(tn[3]), "f"(m), "r"(ce[0]), "r"(ce[1]), "r"(ce[2]),
                              "r"(ce[3]));
                    }
                }
            } else if (tri) {
                const uint32_t slot = leaf_first(uint32_t(leaf));
                const float4* tp = reinterpret_cast<const float4*>(tris + slot);
                const float4 a = ldg4(tp), b = ldg4(tp + 1), c = ldg4(tp + 2);
                if (COUNT) tc.tris++;
                leaf = (leaf & 0x70000000) ? leaf - 0x10000000 + 1 : -1;
                const float bound = ANY ? tcur : tlim;
                float t;
                bool hit;
                bool sphere = false;
                if constexpr (SPH) {
                    sphere = (__float_as_uint(c.w) & 3u) == kRecSphere;
                    if (sphere) {
                        RayPre q;
                        q.o = r.o;
                        q.d = r.d;
                        q.tmin = tmin;
                        hit = sphere_test(q, f3(a), b.x, bound, &t);
                    }
                }
                if (!sphere) hit = tri_test_rot(r.o, r.kz, r.Sx, r.Sy, r.Sz, tmin, f3(a), f3(b), f3(c), bound, &t);
                if (hit) {
                    if (ANY) {
                        hslot = int(slot);
                        cur = leaf = -1;
                        stack.clear();
                    } else {
                        const bool first = hslot < 0;
                        const int held = hslot & kSlotMask;
                        const bool nearer = first ? t <= tcur : (t < tcur || (t == tcur && int(slot) < held));
                        // a hit nearer by more than the reach clears what the held one was tied with
                        const bool tied = !first && reach(t) >= tcur;
                        if (tied) other = other == -1 ? (nearer ? held : int(slot)) : -2;
                        else if (nearer) other = -1;
                        if (nearer) {
                            // the record's shade queue rides above its 28 slot bits
                            hslot = int(slot | (__float_as_uint(c.w) >> kRecQueueShift << 28));
                            tcur = t;
                        }
                    }
                }
            }
        }
        // ---- finished rays
        if (cur == -1 && stack.sp == stack.base && stack.spilled != 0) {
            const uint2 m = stack_spill_in<!ANY>(stack.base, over, stack.spilled);
            stack.sp = m.x;
            stack.spilled = int(m.y);
        }
        const bool over = left < 0 || (left == 0 && cur >= 0);
        const bool done = p >= 0 && (over || (cur == -1 && leaf == -1 && stack.sp == stack.base));
        if (done && over) exhausted(p);
        finish(done, p, tcur, hslot < 0 ? -1 : hslot & kSlotMask, hslot >> 28, other);
        if (done) {
            p = -1;
            cur = leaf = -1;
            stack.clear();
        }
    }
}

}  // namespace cg
#endif
