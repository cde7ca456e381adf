// traverse.cuh -- two-level walk of the 8-wide quantised BVH (TLAS over instances, one BLAS per mesh).
//
// Semantics follow SceneRenderProxy::Intersect<AnyHit> (SceneRenderProxy.cpp:82-126) over
// MeshRenderProxy's BLAS (MeshRenderProxy.cpp:94-194) and SphereRenderProxy (SphereRenderProxy.cpp:5-38):
//  * closest hit: a triangle is accepted when Möller–Trumbore passes in local space and its world t,
//    computed the reference's way from the x component only (Ray::InverseAt, Ray.h:43-47), satisfies
//    0 < world_t < best (strict, so the first of equal t is kept);
//  * any hit (reference semantics): the first Möller–Trumbore pass (local t > Eps) or sphere with a
//    non-negative discriminant ends the walk (the reference does not test the sphere's t sign);
//  * occlusion (for next-event estimation): a hit with Eps < t < tmax ends the walk.
// Differences from the reference walk that cannot change a closest hit: the reference never lowers the
// ray's tmax (every box along the ray is visited); this walk prunes boxes that start beyond the current
// best t plus a bound on the x-only world-t rounding error, and visits children in an octant order.
// Two hits with bit-identical t go to the smaller (instance, face) rather than to the first visited, so
// the result never depends on the visit order (the reference's winner among exact ties does).
// One deliberate difference: for a direction component with |d| <= FLT_EPSILON, bvh v2's fast slab test
// uses 1/d = +-FLT_MAX and its -inv*org term overflows to +-inf once |org| > 1 on that axis, which culls
// every box of the level; here that axis is tested as an exact containment test instead.
//
// The walk is a resumable state machine (Walker::step) so persistent warps can replace finished rays
// with new ones while the others are still walking (dynamic ray fetch). A persistent warp collects the triangles its
// rays reach and tests 32 at a time, one per lane (TriangleQueue).
#pragma once

#include "device_scene.cuh"

namespace spk {

enum : int { kTraceClosest = 0, kTraceAnyRef = 1, kTraceOcclusion = 2 };
enum : uint32_t { kErrStackOverflow = 1u, kErrIterationBudget = 2u, kErrQueueOverflow = 4u };

// Tunables (compile-time; the autotuner builds variants by defining them).
#ifndef SPK_REFILL_LANES
#define SPK_REFILL_LANES 22  // persistent warps refill idle lanes once fewer than this are walking
#endif
#ifndef SPK_WIDE_RAYS_PER_BLOCK
#define SPK_WIDE_RAYS_PER_BLOCK 12  // launches of at most this many rays per block walk one ray per warp (walk_rays)
#endif
#ifndef SPK_TAIL_STEPS
#define SPK_TAIL_STEPS 4  // steps between the rounds of a persistent warp that has no more rays to fetch
#endif
#ifndef SPK_WALK_MIN_BLOCKS
#define SPK_WALK_MIN_BLOCKS 7  // resident 128-thread blocks per SM of the closest-hit walks (72 registers)
#endif
#ifndef SPK_SHADOW_MIN_BLOCKS
#define SPK_SHADOW_MIN_BLOCKS 7  // the same for the occlusion walk of the shadow stage
#endif
#ifndef SPK_PACKET_MIN_BLOCKS
#define SPK_PACKET_MIN_BLOCKS 8  // resident 128-thread blocks per SM the packet walk is compiled for
#endif
#ifndef SPK_PACKET2_MIN_BLOCKS
#define SPK_PACKET2_MIN_BLOCKS 6  // resident 128-thread blocks per SM the two-rays-per-lane packet walk is compiled for
#endif
#ifndef SPK_FRUSTUM_SPREAD
#define SPK_FRUSTUM_SPREAD 0.25f  // largest relative spread of a packet's slab reciprocals tested as one
#endif
#ifndef SPK_PACKET_FRUSTUM
#define SPK_PACKET_FRUSTUM 1  // 1: packets of one octant test each node once for all rays (0: every lane its own ray)
#endif
#ifndef SPK_PACKET_WORLD_SMEM
#define SPK_PACKET_WORLD_SMEM 1  // 1: packet walks keep each lane's world rays in shared memory, not registers
#endif
#ifndef SPK_PACKET_SIBLINGS
#define SPK_PACKET_SIBLINGS 4  // sibling nodes a packet tests at once (one per 8-lane group), 1..4
#endif
constexpr int kStackSize = 48;
constexpr uint32_t kFewNodes = 16;  // scenes of at most this many nodes (TLAS and BLASes) have short walks (launch_trace)
constexpr int kWalkThreads = 128;  // threads per block of every persistent walking kernel
constexpr uint32_t kMaxIterations = 1u << 20;
constexpr uint32_t kPacketSiblings = SPK_PACKET_SIBLINGS;
constexpr uint32_t kPacketStack = 64;  // packet walks push up to 2 * kPacketSiblings - 1 groups per node step
static_assert(kPacketSiblings >= 1 && kPacketSiblings <= 4, "one to four 8-lane groups");

// 65536 + byte `c` of `word`: the byte, times 128, added to the bits of 65536.f (whose last place is 1/128). The byte dot
// product does it in one instruction of the FMA pipe, where a byte permute, or an extraction and a conversion, would
// go to the ALU pipe, the walk's busiest (it also takes the slab minima and maxima).
__device__ __forceinline__ float raised_plane(uint32_t word, int c) {
    return __uint_as_float(__dp4a(word, 128u << (8 * c), 0x47800000u));
}
// Packed single-precision fused multiply-add (the halves rounded as fmaf rounds them).
__device__ __forceinline__ unsigned long long pack_f2(float lo, float hi) {
    unsigned long long d;
    asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "f"(lo), "f"(hi));
    return d;
}
__device__ __forceinline__ void fma_f2(unsigned long long a, unsigned long long b, unsigned long long c, float &lo,
                                       float &hi) {
    unsigned long long d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(d));
}

// Bytes `c` and `c` + 1 of `word` as floats: 65536 is taken off again two at a time, without rounding.
__device__ __forceinline__ unsigned long long planes_f2(uint32_t word, int c) {
    const unsigned long long raised = pack_f2(raised_plane(word, c), raised_plane(word, c + 1));
    unsigned long long d;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(raised), "l"(pack_f2(-65536.f, -65536.f)));
    return d;
}

struct TraceResult {
    float t, u, v;
    uint32_t inst;  // caller instance index, kInvalid on a miss
    uint32_t face;  // original face index, kInvalid for spheres and misses
};

// Per-thread traffic counters of the instrumented walk (wide nodes visited, triangles tested).
struct TraceCounts {
    uint32_t nodes = 0, tris = 0;
};

struct LevelRay {
    f3 o, d, inv;
    uint32_t oct;  // bit k set when direction component k is negative
};

// Reciprocal for the slab test, correctly rounded; a component with |d| <= FLT_EPSILON gets +-2^100 so that
// (bound - o) * inv keeps its exact sign without overflowing (an exact containment test on that axis).
__device__ __forceinline__ float slab_inverse(float x) {
    return fabsf(x) <= 1.1920928955078125e-07f ? copysignf(0x1p100f, x) : 1.f / x;
}

__device__ __forceinline__ void setup_level(LevelRay &r, f3 o, f3 d) {
    r.o = o;
    r.d = d;
    r.inv = mk3(slab_inverse(d.x), slab_inverse(d.y), slab_inverse(d.z));
    r.oct = (signbit(d.x) ? 1u : 0u) | (signbit(d.y) ? 2u : 0u) | (signbit(d.z) ? 4u : 0u);
}

// Upper bound on the t a box may start at and still hold a hit closer than `best` (in world-t terms).
__device__ __forceinline__ float prune_limit(float best, float wox, float wdx, float scene_abs_x) {
    if (!(best < kFltMax)) return kFltMax;
    float r;  // 1 / |wdx| within 2^-23; infinite below 2^-126, which leaves the limit open
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(fabsf(wdx)));
    const float slack = (fabsf(wox) + scene_abs_x) * 0x1.00001p-18f * r;
    const float lim = best * (1.f + 0x1p-14f) + slack;
    return isfinite(lim) ? lim : kFltMax;
}

// Slots of a node in a ray's visiting order: first[oct][mask] is the slot s of `mask` (a non-zero set of the 8
// slots) with the smallest s ^ oct, the child nearest along a ray of octant `oct`.
struct SlotOrder {
    uint8_t first[8][256];
    constexpr SlotOrder() : first() {
        for (int oct = 0; oct < 8; ++oct)
            for (int mask = 1; mask < 256; ++mask)
                for (int k = 7; k >= 0; --k)
                    if ((mask >> (k ^ oct)) & 1) first[oct][mask] = static_cast<uint8_t>(k ^ oct);
    }
};
static __device__ const SlotOrder kSlotOrder{};

// Slot mask with slot s moved to bit s ^ oct (the packet walk's groups: lowest bit first is the visiting order).
__device__ __forceinline__ uint32_t order_slots(uint32_t mask, uint32_t oct) {
    if (oct & 1u) mask = ((mask & 0x55u) << 1) | ((mask >> 1) & 0x55u);
    if (oct & 2u) mask = ((mask & 0x33u) << 2) | ((mask >> 2) & 0x33u);
    if (oct & 4u) mask = ((mask & 0x0Fu) << 4) | (mask >> 4);
    return mask;
}

// What a ray's slab tests found in a node.
struct NodeHits {
    uint32_t child_base, item_base;
    uint32_t imask;       // slots that hold inner nodes
    uint32_t hit;         // slots whose box the ray enters
    uint32_t meta[2];     // per slot: leaf items (unary count << 5 | first item) or an inner child's marker
};

// Slab test of the 8 children of node `idx` against one ray, in pairs of children (packed multiply-adds).
//
// Bound: instruction issue and the ALU pipe, which runs at half the issue rate. With the byte planes converted one by
// one and every hit child's item bits assembled here a visit took 277 warp instructions, 159 of them on the ALU pipe. The
// planes come from byte dot products and packed adds (FMA pipe), the packed operands are two children's (which needs no
// register moves), and only the slot mask is built here (leaf items are decoded by the few rays that reach a leaf).
//
// The test is fma(q, a, o) on the plane bytes q, with a = scale * inv and o = (p - r.o) * inv, bit for bit the one of
// walk_wide and of a packet's single rays. That matters: Moeller-Trumbore accepts rays that pass an edge by a rounding
// error outside, so a triangle can be hit through a box that the exact ray misses, and a walk whose boxes are wider by a
// slack, which would save the adds and the division (6% of a walk), finds hits that the others do not.
__device__ __forceinline__ NodeHits visit_slots(const uint4 *__restrict__ nodes, uint32_t idx, const LevelRay &r,
                                                float tmax) {
    const uint4 *np = nodes + static_cast<size_t>(idx) * 5;
    const uint4 n0 = __ldg(np), n1 = __ldg(np + 1), n2 = __ldg(np + 2), n3 = __ldg(np + 3), n4 = __ldg(np + 4);
    float a[3], o[3];
    const float p[3] = {__uint_as_float(n0.x), __uint_as_float(n0.y), __uint_as_float(n0.z)};
    const float ro[3] = {r.o.x, r.o.y, r.o.z}, ri[3] = {r.inv.x, r.inv.y, r.inv.z};
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        a[k] = __uint_as_float(((n0.w >> (8 * k)) & 0xFFu) << 23) * ri[k];
        o[k] = (p[k] - ro[k]) * ri[k];
    }
    NodeHits h{n1.x, n1.y, n0.w >> 24, 0u, {n1.z, n1.w}};
    const uint32_t lo[3][2] = {{n2.x, n2.y}, {n2.z, n2.w}, {n3.x, n3.y}};
    const uint32_t hi[3][2] = {{n3.z, n3.w}, {n4.x, n4.y}, {n4.z, n4.w}};
#pragma unroll
    for (int half = 0; half < 2; ++half) {
        uint32_t nw[3], fw[3];
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            const bool neg = (r.oct >> k) & 1u;
            nw[k] = neg ? hi[k][half] : lo[k][half];
            fw[k] = neg ? lo[k][half] : hi[k][half];
        }
#pragma unroll
        for (int c = 0; c < 4; c += 2) {
            float tn[3][2], tf[3][2];
#pragma unroll
            for (int k = 0; k < 3; ++k) {
                const unsigned long long a2 = pack_f2(a[k], a[k]), o2 = pack_f2(o[k], o[k]);
                fma_f2(planes_f2(nw[k], c), a2, o2, tn[k][0], tn[k][1]);
                fma_f2(planes_f2(fw[k], c), a2, o2, tf[k][0], tf[k][1]);
            }
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                const float t0 = fmaxf(fmaxf(tn[0][e], tn[1][e]), fmaxf(tn[2][e], 0.f));
                const float t1 = fminf(fminf(tf[0][e], tf[1][e]), fminf(tf[2][e], tmax));
                if (t0 <= t1) h.hit |= 1u << (4 * half + c + e);
            }
        }
    }
    return h;
}

// The triangle (or TLAS item) bits of the leaf slots `leaf` of a node.
__device__ __forceinline__ uint32_t leaf_items(uint32_t leaf, const uint32_t (&meta)[2]) {
    uint32_t bits = 0u;
    for (; leaf != 0u; leaf &= leaf - 1u) {
        const uint32_t m = __byte_perm(meta[0], meta[1], __ffs(leaf) - 1);
        bits |= ((m >> 5) & 7u) << (m & 31u);
    }
    return bits;
}

// Möller–Trumbore (MeshRenderProxy.cpp:128-194) of triangle record `idx` in the level ray's (the instance's
// local) space: true when the ray passes with local t > Eps, with (t, u, v) and the record's face index.
__device__ __forceinline__ bool triangle_hit(const float4 *__restrict__ tris, uint32_t idx, const LevelRay &ray,
                                             float &t, float &u, float &v, uint32_t &face) {
    const float4 *tp = tris + static_cast<size_t>(idx) * 3;
    const float4 a4 = __ldg(tp), b4 = __ldg(tp + 1), c4 = __ldg(tp + 2);
    const f3 p0 = mk3(a4.x, a4.y, a4.z), e1 = mk3(a4.w, b4.x, b4.y), e2 = mk3(b4.z, b4.w, c4.x);
    const f3 h = cross(ray.d, e2);
    const float det = dot3(e1, h);
    if (fabsf(det) < kEps) return false;
    const f3 s = ray.o - p0;
    const float f = __frcp_rn(det);  // the bits of 1.f / det
    u = f * dot3(s, h);
    if (u < 0.f || u > 1.f) return false;
    const f3 q = cross(s, e1);
    v = f * dot3(ray.d, q);
    if (v < 0.f || u + v > 1.f) return false;
    t = f * dot3(e2, q);
    face = __float_as_uint(c4.y);
    return t > kEps;
}

// World t of a local hit at `t`, the reference's way: from the x component only (Ray::InverseAt, Ray.h:43-47).
__device__ __forceinline__ float world_t(const DevInstance &I, const LevelRay &ray, float t, f3 wo, f3 wd) {
    const f3 wp = xform_point(I.m, ray.o + ray.d * t);
    return (wp.x - wo.x) / wd.x;
}

// SphereRenderProxy::IntersectInternal (SphereRenderProxy.cpp:5-38) in world space: false when the
// discriminant is negative, else true with the root the reference takes (the near one from outside).
__device__ __forceinline__ bool sphere_hit(const DevInstance &I, f3 wo, f3 wd, float &t) {
    const f3 center = mk3(I.m[3], I.m[7], I.m[11]);
    const f3 co = wo - center;
    const float half_b = dot3(wd, co);
    const float c = sqnorm(co) - I.radius * I.radius;
    const float disc = half_b * half_b - 1.f * c;
    if (disc < 0.f) return false;
    const float sq = sqrtf(disc);
    t = (-half_b + (c >= 0.f ? -sq : sq)) / 1.f;
    return true;
}

// The traversal stack of one ray in local memory (it hits in L1; the stack is about 1% of a walk's instructions).
struct LocalStack {
    uint2 e[kStackSize];
    __device__ __forceinline__ void put(int i, uint2 v) { e[i] = v; }
    __device__ __forceinline__ uint2 take(int i) { return e[i]; }
};

// True when a hit at world t `t` on (inst, face) replaces `best`: a smaller t, or an exact tie on a smaller
// (instance, face). The reference keeps the first of equal t (IntersectionCandidate::IsCloserHit is a strict <),
// which depends on the visit order; this rule makes every hit independent of scheduling.
__device__ __forceinline__ bool closer_hit(const TraceResult &best, float t, uint32_t inst, uint32_t face) {
    if (t < best.t) return true;
    return t == best.t && (inst < best.inst || (inst == best.inst && face < best.face));
}

// What a walk keeps but rarely touches: its world ray and where in its best triangle the hit is. A one-thread walk:
// registers. A persistent walk: a column of the block's shared memory (word k of thread t at [k][t]: lanes that read
// their own or distinct lanes' columns meet no bank conflict), so that other lanes of the warp can test its triangles
// (TriangleQueue), and because the registers would spill in the node visit (two spilled words cost the walk 2-4%). 11
// words a thread keep 7 blocks within a 64 KB shared-memory share of the SM; 14 words take the next share from the L1.
struct RegState {
    f3 ro, rd;
    float hit_u, hit_v;
    uint32_t hit_face;
    __device__ __forceinline__ void set_ray(f3 a, f3 b) {
        ro = a;
        rd = b;
    }
    __device__ __forceinline__ f3 o() const { return ro; }
    __device__ __forceinline__ f3 d() const { return rd; }
    __device__ __forceinline__ void set_hit(float u, float v, uint32_t face) {
        hit_u = u;
        hit_v = v;
        hit_face = face;
    }
    __device__ __forceinline__ float u() const { return hit_u; }
    __device__ __forceinline__ float v() const { return hit_v; }
    __device__ __forceinline__ uint32_t face() const { return hit_face; }
};
struct SharedState {
    static constexpr int kWords = 11;
    float *w;  // word 0 of this thread
    __device__ __forceinline__ float &at(int k) const { return w[k * kWalkThreads]; }
    __device__ __forceinline__ void set_ray(f3 a, f3 b) const {
        const float v[6] = {a.x, a.y, a.z, b.x, b.y, b.z};
#pragma unroll
        for (int k = 0; k < 6; ++k) at(k) = v[k];
    }
    __device__ __forceinline__ f3 o() const { return mk3(at(0), at(1), at(2)); }
    __device__ __forceinline__ f3 d() const { return mk3(at(3), at(4), at(5)); }
    __device__ __forceinline__ void set_hit(float u, float v, uint32_t face) const {
        at(6) = u;
        at(7) = v;
        at(8) = __uint_as_float(face);
    }
    __device__ __forceinline__ float u() const { return at(6); }
    __device__ __forceinline__ float v() const { return at(7); }
    __device__ __forceinline__ uint32_t face() const { return __float_as_uint(at(8)); }
    __device__ __forceinline__ void set_item(unsigned long long q) const {
        at(9) = __uint_as_float(static_cast<uint32_t>(q));
        at(10) = __uint_as_float(static_cast<uint32_t>(q >> 32));
    }
    __device__ __forceinline__ unsigned long long item() const {
        return __float_as_uint(at(9)) | (static_cast<unsigned long long>(__float_as_uint(at(10))) << 32);
    }
};

// Resumable two-level walk of one ray. init() starts it; step() advances by one node visit and returns true when
// the walk is over (result in best()).
template <int kMode, bool kCount, class State>
struct Walker {
    State st;
    LevelRay ray;
    uint2 ngroup;
    int sp;
    int blas_sp;  // stack height the BLAS was entered at; -1 at the TLAS level, -2 there before `ray` is the world ray again
    uint32_t cur_inst;
    uint32_t steps_left;
    float tmax_box;
    float best_t;
    uint32_t best_inst;

    // `root` is the TLAS root node of the ray's scene (S.tlas_root for a single-scene context).
    __device__ __forceinline__ void init(const DevScene &S, uint32_t root, f3 o, f3 d, float tmax) {
        st.set_ray(o, d);
        setup_level(ray, o, d);
        ngroup = make_uint2(root, root == kInvalid ? 0u : (1u << 24));
        sp = 0;
        blas_sp = -1;
        cur_inst = 0;
        steps_left = S.walk_budget ? S.walk_budget : kMaxIterations;
        tmax_box = (kMode == kTraceOcclusion) ? tmax : kFltMax;
        best_t = kFltMax;
        best_inst = kInvalid;
        st.set_hit(0.f, 0.f, kInvalid);
    }

    __device__ __forceinline__ TraceResult best() const { return TraceResult{best_t, st.u(), st.v(), best_inst, st.face()}; }

    // Takes the hit when it is closer than the best one (ties as closer_hit has them).
    __device__ __forceinline__ bool take(float t, float u, float v, uint32_t inst, uint32_t face) {
        if (!(t < best_t) && !(t == best_t && closer_hit(best(), t, inst, face))) return false;
        best_t = t;
        best_inst = inst;
        st.set_hit(u, v, face);
        return true;
    }

    template <class Stack>
    __device__ __forceinline__ void push(Stack &stack, uint2 v, uint32_t &err) {
        if (sp < kStackSize) {
            stack.put(sp++, v);
        } else {
            err |= kErrStackOverflow;
        }
    }

    // Instances and spheres of a TLAS leaf group, until one opens a BLAS. True: an any-hit walk is over.
    template <class Stack>
    __device__ __forceinline__ bool items(const DevScene &S, Stack &stack, uint2 tgroup, uint32_t &err) {
        while (tgroup.y != 0u) {
            const uint32_t k = __ffs(tgroup.y) - 1;
            tgroup.y &= tgroup.y - 1u;
            const uint32_t inst = __ldg(S.tlas_items + tgroup.x + k);
            const DevInstance &I = S.instances[inst];
            if (I.type == 1u) {
                // SphereRenderProxy::IntersectInternal (SphereRenderProxy.cpp:5-38), world space: sphere_hit's
                // test, written out so the any-hit modes stop before the square root.
                const f3 wo = st.o(), wd = st.d();
                const f3 center = mk3(I.m[3], I.m[7], I.m[11]);
                const f3 co = wo - center;
                const float half_b = dot3(wd, co);
                const float c = sqnorm(co) - I.radius * I.radius;
                const float disc = half_b * half_b - 1.f * c;
                if (disc < 0.f) continue;
                if (kMode == kTraceAnyRef) {
                    best_inst = inst;
                    return true;
                }
                const float sq = sqrtf(disc);
                const float t = (-half_b + (c >= 0.f ? -sq : sq)) / 1.f;
                if (kMode == kTraceOcclusion) {
                    if (t > kEps && t < tmax_box) {
                        best_inst = inst;
                        return true;
                    }
                    continue;
                }
                if (t > 0.f && take(t, 0.f, 0.f, inst, kInvalid)) tmax_box = prune_limit(t, wo.x, wd.x, S.scene_abs_x);
            } else if (I.blas_root != kInvalid) {
                // Enter the BLAS: park the rest of this TLAS level on the stack.
                if (tgroup.y != 0u) push(stack, tgroup, err);
                if (ngroup.y > 0x00FFFFFFu) push(stack, ngroup, err);
                blas_sp = sp;
                cur_inst = inst;
                setup_level(ray, xform_point(I.minv, st.o()), xform_dir(I.minv, st.d()));
                ngroup = make_uint2(I.blas_root, 1u << 24);
                tgroup.y = 0u;
            }
        }
        return false;
    }

    // Tests the triangles of a group at once. True: a hit ends the walk.
    __device__ __forceinline__ bool test(const DevScene &S, uint2 tg) {
        for (; tg.y != 0u; tg.y &= tg.y - 1u) {
            float t, u, v;
            uint32_t face;
            if (!triangle_hit(S.tris, tg.x + __ffs(tg.y) - 1, ray, t, u, v, face)) continue;
            if (kMode == kTraceAnyRef || (kMode == kTraceOcclusion && t < tmax_box)) {
                best_inst = cur_inst;
                return true;
            }
            if (kMode == kTraceOcclusion) continue;
            const f3 wo = st.o(), wd = st.d();
            const float wt = world_t(S.instances[cur_inst], ray, t, wo, wd);
            if (wt > 0.f && take(wt, u, v, cur_inst, face)) tmax_box = prune_limit(wt, wo.x, wd.x, S.scene_abs_x);
        }
        return false;
    }

    // `leaves(item_base, slots, meta)` and `group(tgroup)` take the triangles of the leaf slots reached in a node, and
    // of a group that came back from the stack; either returns true when a hit ends the walk.
    template <class Stack, class Leaves, class Group>
    __device__ __forceinline__ bool step(const DevScene &S, Stack &stack, uint32_t &err, TraceCounts *counts,
                                         Leaves &&leaves, Group &&group) {
        if (steps_left-- == 0u) {
            err |= kErrIterationBudget;
            return true;
        }
        uint2 tgroup = make_uint2(0u, 0u);  // TLAS items
        if (ngroup.y > 0x00FFFFFFu) {
            const uint32_t slot = __ldg(&kSlotOrder.first[ray.oct][ngroup.y >> 24]);
            ngroup.y &= ~(1u << (slot + 24));
            const uint32_t node_idx = ngroup.x + __popc(ngroup.y & 0xFFu & ((1u << slot) - 1u));
            if (ngroup.y > 0x00FFFFFFu) push(stack, ngroup, err);
            const NodeHits h = visit_slots(S.nodes, node_idx, ray, tmax_box);
            ngroup = make_uint2(h.child_base, ((h.hit & h.imask) << 24) | h.imask);
            const uint32_t leaf = h.hit & ~h.imask;
            if (kCount) ++counts->nodes;
            if (leaf != 0u) {
                if (blas_sp >= 0) {
                    if (kCount) counts->tris += __popc(leaf_items(leaf, h.meta));
                    if (leaves(h.item_base, leaf, h.meta)) return true;
                } else {
                    tgroup = make_uint2(h.item_base, leaf_items(leaf, h.meta));
                }
            }
        } else {
            tgroup = ngroup;
            ngroup = make_uint2(0u, 0u);
            if (blas_sp >= 0) {
                if (group(tgroup)) return true;
                tgroup.y = 0u;
            }
        }
        if (tgroup.y != 0u && items(S, stack, tgroup, err)) return true;
        if (ngroup.y <= 0x00FFFFFFu) {
            if (sp == 0) return true;
            if (sp == blas_sp) blas_sp = -2;
            ngroup = stack.take(--sp);
            if (blas_sp == -2 && ngroup.y > 0x00FFFFFFu) {
                setup_level(ray, st.o(), st.d());
                blas_sp = -1;
            }
        }
        return false;
    }
};

// Whole walk of one ray by one thread, its triangles tested as they are reached.
template <int kMode, bool kCount = false>
__device__ __forceinline__ TraceResult trace_ray(const DevScene &S, f3 wo, f3 wd, float tmax_occl, uint32_t &err,
                                                 TraceCounts *counts = nullptr) {
    LocalStack stack;
    Walker<kMode, kCount, RegState> w;
    w.init(S, S.tlas_root, wo, wd, tmax_occl);
    auto group = [&](uint2 tg) { return w.test(S, tg); };
    auto leaves = [&](uint32_t base, uint32_t slots, const uint32_t (&meta)[2]) {
        return group(make_uint2(base, leaf_items(slots, meta)));
    };
    while (!w.step(S, stack, err, counts, leaves, group)) {
    }
    return w.best();
}

// The triangles a warp's rays have reached and not tested yet: (triangle, instance) pairs with the lane that owns
// the ray. Tested in the lane that reached them, triangles ran at 3.2 of 32 lanes (secondary rays of the 1024^2
// terrain: 2 warp executions per ray, 30% of the walk's instructions); queued, a round tests 32 pairs with 26 lanes on
// average. With this and the packed slab tests bounces 1 to 7 of a 64-sample 1080p frame went from 523 to 444 warp
// instructions per ray. Queueing groups instead of triangles saves the writes but costs a scan per round (+4%
// instructions).
constexpr uint32_t kQueueCap = 64;  // a round leaves fewer than 32, a step adds about 8 (the rest goes to the stack)
struct TriangleQueue {
    uint2 pair[kQueueCap];      // triangle record, instance
    uint8_t owner[kQueueCap];
    uint32_t count;             // pairs handed a place; those past kQueueCap were not stored
    uint32_t pad;
};

// Persistent walk over a work list: each warp pulls batches of items from `cursor` and refills lanes whose
// ray has finished once fewer than `kRefillLanes` lanes are still walking. `fetch(i, o, d, tmax)` loads item
// i's ray (tmax starts at the call's `tmax`; an occlusion walk may lower it per ray) and returns the TLAS
// root of its scene; `finish(i, result)` stores its result. Every lane of every warp of the block must call
// this, and the block must have kWalkThreads threads (the shared memory is laid out for that many).
//
// A step visits one node per walking lane and queues the triangles of the leaves it reaches; once 32 pairs are
// queued the whole warp tests them, lane i pair i, with the owner's world ray from shared memory taken into the
// pair's instance space (the same operations as at the BLAS entry, so the same bits). A hit goes back to its
// owner, whose best t then prunes as before: a few steps later than if tested at once, which adds node visits (+1.6%)
// but cannot change a result. When fewer than kRefillLanes lanes walk, every pair is tested, the walks that are over
// store their results, and idle lanes are refilled (22: 16 and 26 are 0.6 and 1.6% slower on a 64-sample 1080p frame). 72 registers (7 blocks per SM) hold a
// walk without touching local memory in the node visits; more state in shared memory instead (8 blocks) takes L1 from
// the nodes: measured even.
// `kDirect`: nothing is queued, a lane tests the triangles of a leaf when it reaches it (launch_trace says when).
constexpr int kRefillLanes = SPK_REFILL_LANES;
constexpr uint32_t kTailSteps = SPK_TAIL_STEPS;

template <int kMode, bool kCount, bool kDirect, class Fetch, class Finish>
__device__ __forceinline__ void walk_persistent(const DevScene &S, unsigned long long *cursor, unsigned long long n,
                                                float tmax, uint32_t &err, TraceCounts *counts, Fetch &&fetch,
                                                Finish &&finish) {
    constexpr uint32_t kAll = 0xFFFFFFFFu;
    __shared__ float state[SharedState::kWords * kWalkThreads];
    __shared__ TriangleQueue queues[kWalkThreads / 32];
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t lt_mask = (1u << lane) - 1u;
    TriangleQueue &Q = queues[threadIdx.x >> 5];
    LocalStack stack;
    Walker<kMode, kCount, SharedState> w;
    w.st.w = state + threadIdx.x;
    bool walking = false, over = false;  // over: the walk has ended, its pairs may still be queued
    bool exhausted = false;
    uint32_t tail_steps = 0;
    if (lane == 0) Q.count = 0u;
    __syncwarp();

    // Queues `cnt` consecutive triangles (at most 3) of this lane's ray from record `first` on; returns how many found
    // no room.
    auto enqueue = [&](uint32_t first, uint32_t cnt) {
        const uint32_t pos = atomicAdd(&Q.count, cnt);
#pragma unroll
        for (uint32_t k = 0; k < 3; ++k) {
            if (k < cnt && pos + k < kQueueCap) {
                Q.pair[pos + k] = make_uint2(first + k, w.cur_inst);
                Q.owner[pos + k] = static_cast<uint8_t>(lane);
            }
        }
        return pos + cnt > kQueueCap ? min(pos + cnt - kQueueCap, cnt) : 0u;
    };
    // What does not fit goes back to the stack.
    auto leaves = [&](uint32_t base, uint32_t slots, const uint32_t (&meta)[2]) {
        uint32_t left = 0u;
        for (; slots != 0u; slots &= slots - 1u) {
            const uint32_t m = __byte_perm(meta[0], meta[1], __ffs(slots) - 1);
            const uint32_t at = m & 31u, cnt = __popc(m & 0xE0u);
            const uint32_t rest = enqueue(base + at, cnt);
            if (rest != 0u) left |= ((1u << rest) - 1u) << (at + cnt - rest);
        }
        if (left != 0u) w.push(stack, make_uint2(base, left), err);
        return false;
    };
    auto group = [&](uint2 tg) {
        while (tg.y != 0u) {
            const uint32_t k = __ffs(tg.y) - 1;
            if (enqueue(tg.x + k, 1u) != 0u) {
                w.push(stack, tg, err);
                break;
            }
            tg.y &= tg.y - 1u;
        }
        return false;
    };
    auto test_group = [&](uint2 tg) { return w.test(S, tg); };
    auto test_leaves = [&](uint32_t base, uint32_t slots, const uint32_t (&meta)[2]) {
        return w.test(S, make_uint2(base, leaf_items(slots, meta)));
    };
    auto step = [&] {
        if constexpr (kDirect) {
            return w.step(S, stack, err, counts, test_leaves, test_group);
        } else {
            return w.step(S, stack, err, counts, leaves, group);
        }
    };
    // One round: lane i tests pair i (of `cnt`); hits go to their owners; the pairs past 32 move to the front.
    auto round = [&](uint32_t cnt) {
        bool hit = false;
        float t = 0.f, u = 0.f, v = 0.f;
        uint32_t face = kInvalid, own = lane, inst = kInvalid;
        if (lane < cnt) {
            const uint2 e = Q.pair[lane];
            own = Q.owner[lane];
            inst = e.y;
            const SharedState ow{state + (threadIdx.x & ~31u) + own};
            const DevInstance &I = S.instances[inst];
            const f3 wo = ow.o(), wd = ow.d();
            LevelRay r;
            r.o = xform_point(I.minv, wo);
            r.d = xform_dir(I.minv, wd);
            hit = triangle_hit(S.tris, e.x, r, t, u, v, face);
            if (kMode == kTraceClosest && hit) {
                t = world_t(I, r, t, wo, wd);
                hit = t > 0.f;
            }
        }
        if (kMode == kTraceClosest) {
            bool closer = false;
            for (uint32_t m = __ballot_sync(kAll, hit); m != 0u; m &= m - 1u) {
                const int src = __ffs(m) - 1;
                const uint32_t o = __shfl_sync(kAll, own, src);
                const TraceResult c{__shfl_sync(kAll, t, src), __shfl_sync(kAll, u, src), __shfl_sync(kAll, v, src),
                                    __shfl_sync(kAll, inst, src), __shfl_sync(kAll, face, src)};
                if (o == lane && w.take(c.t, c.u, c.v, c.inst, c.face)) closer = true;
            }
            if (closer) w.tmax_box = prune_limit(w.best_t, w.st.at(0), w.st.at(3), S.scene_abs_x);
        } else if (kMode == kTraceOcclusion) {
            const float limit = __shfl_sync(kAll, w.tmax_box, static_cast<int>(own));
            const uint32_t blocked = __reduce_or_sync(kAll, hit && t < limit ? 1u << own : 0u);
            if ((blocked >> lane) & 1u) {
                w.best_inst = 0u;  // (which instance it was is not asked for)
                over = over || walking;
                walking = false;
            }
        } else {
            for (uint32_t m = __ballot_sync(kAll, hit); m != 0u; m &= m - 1u) {
                const int src = __ffs(m) - 1;
                const uint32_t o = __shfl_sync(kAll, own, src), ci = __shfl_sync(kAll, inst, src);
                if (o == lane) {
                    w.best_inst = ci;
                    over = over || walking;
                    walking = false;
                }
            }
        }
        const uint32_t rem = cnt > 32u ? cnt - 32u : 0u;
        uint2 e = make_uint2(0u, 0u);
        uint32_t o = 0;
        if (lane < rem) {
            e = Q.pair[32u + lane];
            o = Q.owner[32u + lane];
        }
        __syncwarp();
        if (lane < rem) {
            Q.pair[lane] = e;
            Q.owner[lane] = static_cast<uint8_t>(o);
        }
        if (lane == 0) Q.count = rem;
        __syncwarp();
    };

    for (;;) {
        const uint32_t idle = __ballot_sync(kAll, !walking && !over);
        if (!exhausted && idle != 0u) {
            // A list of fewer than 32 rays per block is spread over as many warps as there are blocks, one fetch
            // each: lanes of different warps do not wait for each other (335x202 pixels of the large scene: 1026 ->
            // 947 us a frame; over all warps, four times as many, they crowd each other: 65536 rays of the box 28 ->
            // 33 us).
            const uint32_t quota = n < 32ull * gridDim.x ? static_cast<uint32_t>((n + gridDim.x - 1) / gridDim.x) : 32u;
            const uint32_t cnt = min(static_cast<uint32_t>(__popc(idle)), quota);
            unsigned long long base = 0;
            if (lane == 0) base = atomicAdd(cursor, static_cast<unsigned long long>(cnt));
            base = __shfl_sync(kAll, base, 0);
            exhausted = base + cnt >= n || quota < 32u;
            if (!walking && !over) {
                const uint32_t rank = __popc(idle & lt_mask);
                const unsigned long long q = base + rank;
                if (rank < cnt && q < n) {
                    w.st.set_item(q);
                    f3 o, d;
                    float tm = tmax;
                    const uint32_t root = fetch(q, o, d, tm);
                    w.init(S, root, o, d, tm);
                    walking = true;
                }
            }
        }
        if (__ballot_sync(kAll, walking) == 0u) {  // (no walk is over with pairs left: the loop below drained them)
            if (exhausted) break;
            continue;
        }
        for (;;) {
            if (walking && step()) {
                walking = false;
                over = true;
            }
            __syncwarp();
            const uint32_t walkers = __popc(__ballot_sync(kAll, walking));
            // Once the list is exhausted there is nothing to refill: every few steps, which keeps a round's latency
            // out of most steps of the last, longest walks (a round every 1 / 4 / 8 / 16 steps, us: 65536 rays of the
            // 3.4M-triangle scene 140 / 129 / 129 / 135, 12769 of 11392 triangles 72 / 68 / 69 / 68, a 1080p frame of one
            // sample 3076 / 3044 / 3034 / 3054).
            const bool drain = !exhausted ? walkers < kRefillLanes : walkers == 0u || (++tail_steps % kTailSteps) == 0u;
            while (!kDirect) {  // (direct: nothing is queued)
                const uint32_t cnt = min(__shfl_sync(kAll, Q.count, 0), kQueueCap);
                if (cnt < 32u && !(drain && cnt != 0u)) break;
                round(cnt);
            }
            if (drain) {  // the queue is empty: every walk that is over has its result
                if (over) finish(w.st.item(), w.best());
                over = false;
                if (!exhausted || walkers == 0u) break;
            }
        }
    }
}

// Walk of few rays, one ray per warp: the warp visits up to four of the ray's nearest pending nodes at once, lane 8 g + k
// testing child slot k ^ octant of node g (so that the ballot is in visiting order), and tests the triangles of the
// leaves reached in the lanes that reached them. A launch of few rays lasts as long as its longest walk, whatever the
// rest of the chip does: the last bounces of a 1080p frame (a few thousand rays) take hundreds of dependent steps. Here a
// step is a few loads and some 60 instructions before the next ones are known, where walk_persistent's lane runs 250 and
// visits one node. Same boxes (the plain slab test with a correctly rounded reciprocal), triangles and tie rule, so the
// same results. `fetch` and `finish` as for walk_persistent; `finish` runs in one lane.
// 4097 rays: 49 -> 22 us (11392 triangles). It takes 6 times the instructions per ray, so more rays soon do better with
// a ray per lane: beyond 12 rays per block (12768 on 152 SMs), or, in scenes of few nodes, whose walks are over in a
// few steps, 5/8 of the nodes, at least 4. One per warp / per lane, us a closest-hit query: 12768 rays of 1188, 33423 and 312823
// nodes 58 / 69, 62 / 78, 71 / 100; of 13 nodes 5320 rays 32 / 34, 8512 rays 36 / 36, 12768 rays 40 / 36; of 8 nodes 4097
// rays 35 / 35, 6385 rays 40 / 36, 12768 rays 52 / 38.
constexpr int kWideStack = 96;  // a step pushes at most 8 groups
// Not inlined, so that its registers do not count against walk_persistent's in the same kernel. Returns error bits.
template <int kMode, bool kCount, class Fetch, class Finish>
__device__ __noinline__ uint32_t walk_wide(const DevScene &S, unsigned long long *cursor, unsigned long long n,
                                           float tmax, TraceCounts *counts, Fetch fetch, Finish finish) {
    uint32_t err = 0;
    constexpr uint32_t kAll = 0xFFFFFFFFu;
    const uint32_t lane = threadIdx.x & 31u, grp = lane >> 3;
    uint2 stack[kWideStack];
    for (;;) {
        unsigned long long q = 0;
        if (lane == 0) q = atomicAdd(cursor, 1ull);
        q = __shfl_sync(kAll, q, 0);
        if (q >= n) break;
        f3 wo, wd;
        float limit = tmax;  // boxes that start beyond it hold nothing closer; an occlusion walk's own limit
        const uint32_t root = fetch(q, wo, wd, limit);
        if (kMode != kTraceOcclusion) limit = kFltMax;
        LevelRay ray;
        setup_level(ray, wo, wd);
        TraceResult best{kFltMax, 0.f, 0.f, kInvalid, kInvalid};
        uint2 ng = make_uint2(root, root == kInvalid ? 0u : (1u << 24));  // inner children in visiting order, or TLAS items
        uint32_t left = S.walk_budget ? S.walk_budget : kMaxIterations;
        uint32_t cur_inst = kInvalid;
        int sp = 0, blas_sp = -1;  // blas_sp as in Walker
        auto push = [&](uint2 g) {
            if (sp < kWideStack) {
                stack[sp++] = g;
            } else {
                err |= kErrStackOverflow;
            }
        };
        for (bool done = ng.y == 0u; !done;) {
            if (ng.y > 0x00FFFFFFu) {
                const uint32_t inner = ng.y >> 24, imask = ng.y & 0xFFu;
                const uint32_t cnt = sp + 8 <= kWideStack ? min(__popc(inner), 4) : 1;
                if (left < cnt) {
                    err |= kErrIterationBudget;
                    break;
                }
                left -= cnt;
                if (kCount && lane == 0) counts->nodes += cnt;
                uint32_t rest = inner, mine = inner;
#pragma unroll
                for (uint32_t k = 0; k < 4; ++k) {
                    if (k < grp && k + 1 < cnt) mine &= mine - 1u;  // (groups past `cnt` repeat its last node)
                    if (k < cnt) rest &= rest - 1u;
                }
                const uint32_t parent_slot = (__ffs(mine) - 1) ^ ray.oct;
                const uint32_t node = ng.x + __popc(imask & ((1u << parent_slot) - 1u));
                if (rest != 0u) push(make_uint2(ng.x, (rest << 24) | imask));
                const uint4 *np = S.nodes + static_cast<size_t>(node) * 5;
                const uint4 n0 = __ldg(np), n1 = __ldg(np + 1);
                const uint32_t slot = (lane & 7u) ^ ray.oct;
                const uint8_t *lo = reinterpret_cast<const uint8_t *>(np + 2) + slot, *hi = lo + 24;
                float tn[3], tf[3];
                const float p[3] = {__uint_as_float(n0.x), __uint_as_float(n0.y), __uint_as_float(n0.z)};
                const float ro[3] = {ray.o.x, ray.o.y, ray.o.z}, ri[3] = {ray.inv.x, ray.inv.y, ray.inv.z};
#pragma unroll
                for (int k = 0; k < 3; ++k) {
                    const bool neg = (ray.oct >> k) & 1u;
                    const float a = __uint_as_float(((n0.w >> (8 * k)) & 0xFFu) << 23) * ri[k];
                    const float o = (p[k] - ro[k]) * ri[k];
                    tn[k] = fmaf(static_cast<float>(__ldg((neg ? hi : lo) + 8 * k)), a, o);
                    tf[k] = fmaf(static_cast<float>(__ldg((neg ? lo : hi) + 8 * k)), a, o);
                }
                const float t0 = fmaxf(fmaxf(tn[0], tn[1]), fmaxf(tn[2], 0.f));
                const float t1 = fminf(fminf(tf[0], tf[1]), fminf(tf[2], limit));
                const uint32_t meta = __byte_perm(n1.z, n1.w, slot) & 0xFFu;
                const bool reached = grp < cnt && meta != 0u && t0 <= t1;
                const bool leaf = (meta & 0x18u) != 0x18u;
                const uint32_t inner_hits = __ballot_sync(kAll, reached && !leaf);
                uint32_t items = reached && leaf ? (meta >> 5) << (meta & 31u) : 0u;
                const bool in_blas = blas_sp >= 0;
                if (in_blas) {
                    // The lane's triangles (at most 3), then the closest over the warp.
                    bool hit = false;
                    float bt = kFltMax, bu = 0.f, bv = 0.f;
                    uint32_t bface = kInvalid;
                    if (kCount) counts->tris += __popc(items);
                    while (__any_sync(kAll, items != 0u)) {
                        if (items != 0u) {
                            const uint32_t idx = n1.y + __ffs(items) - 1;
                            items &= items - 1u;
                            float t, u, v;
                            uint32_t face;
                            if (triangle_hit(S.tris, idx, ray, t, u, v, face)) {
                                if (kMode == kTraceClosest) {
                                    t = world_t(S.instances[cur_inst], ray, t, wo, wd);
                                    if (t > 0.f && (t < bt || (t == bt && face < bface))) {
                                        hit = true;
                                        bt = t;
                                        bu = u;
                                        bv = v;
                                        bface = face;
                                    }
                                } else {
                                    hit = hit || kMode == kTraceAnyRef || t < limit;
                                }
                            }
                        }
                    }
                    if (__any_sync(kAll, hit)) {
                        if (kMode != kTraceClosest) {
                            best.inst = cur_inst;
                            break;
                        }
                        const uint32_t key = hit ? __float_as_uint(bt) : 0xFFFFFFFFu;  // t > 0: ordered as an integer
                        const uint32_t first = __reduce_min_sync(kAll, key);
                        const uint32_t face = __reduce_min_sync(kAll, key == first ? bface : kInvalid);
                        const int src = __ffs(__ballot_sync(kAll, key == first && bface == face)) - 1;
                        const TraceResult c{__uint_as_float(first), __shfl_sync(kAll, bu, src), __shfl_sync(kAll, bv, src),
                                            cur_inst, face};
                        if (closer_hit(best, c.t, c.inst, c.face)) {
                            best = c;
                            limit = prune_limit(best.t, wo.x, wd.x, S.scene_abs_x);
                        }
                    }
                } else {  // the items of each TLAS node as one group
#pragma unroll
                    for (int d = 1; d < 8; d <<= 1) items |= __shfl_xor_sync(kAll, items, d);
                }
                // Farthest node's groups first onto the stack, the nearest node's last: it is taken next.
                ng.y = 0u;
                for (int g = static_cast<int>(cnt) - 1; g >= 0; --g) {
                    const uint32_t hits = (inner_hits >> (8 * g)) & 0xFFu;
                    const uint32_t base = __shfl_sync(kAll, n1.x, 8 * g), im = __shfl_sync(kAll, n0.w, 8 * g) >> 24;
                    if (hits != 0u) {
                        if (ng.y != 0u) push(ng);
                        ng = make_uint2(base, (hits << 24) | im);
                    }
                    if (!in_blas) {
                        const uint32_t ib = __shfl_sync(kAll, n1.y, 8 * g), bits = __shfl_sync(kAll, items, 8 * g);
                        if (bits != 0u) {
                            if (ng.y != 0u) push(ng);
                            ng = make_uint2(ib, bits);
                        }
                    }
                }
            } else {  // TLAS items
                const uint32_t inst = __ldg(S.tlas_items + ng.x + __ffs(ng.y) - 1);
                ng.y &= ng.y - 1u;
                const DevInstance &I = S.instances[inst];
                if (I.type == 1u) {
                    float t;
                    if (kMode == kTraceClosest) {
                        if (sphere_hit(I, wo, wd, t) && t > 0.f && closer_hit(best, t, inst, kInvalid)) {
                            best = TraceResult{t, 0.f, 0.f, inst, kInvalid};
                            limit = prune_limit(t, wo.x, wd.x, S.scene_abs_x);
                        }
                    } else if (sphere_hit(I, wo, wd, t) && (kMode == kTraceAnyRef || (t > kEps && t < limit))) {
                        best.inst = inst;
                        break;
                    }
                } else if (I.blas_root != kInvalid) {
                    if (ng.y != 0u) push(ng);
                    blas_sp = sp;
                    cur_inst = inst;
                    setup_level(ray, xform_point(I.minv, wo), xform_dir(I.minv, wd));
                    ng = make_uint2(I.blas_root, 1u << 24);
                }
            }
            if (ng.y == 0u) {
                if (sp == 0) break;
                if (sp == blas_sp) blas_sp = -2;
                ng = stack[--sp];
                if (blas_sp == -2 && ng.y > 0x00FFFFFFu) {
                    setup_level(ray, wo, wd);
                    blas_sp = -1;
                }
            }
        }
        if (lane == 0) finish(q, best);
    }
    return err;
}

// The walk of a launch's rays: one per warp while there are few, else persistent warps with a ray per lane.
template <int kMode, bool kCount, bool kDirect = false, class Fetch, class Finish>
__device__ __forceinline__ void walk_rays(const DevScene &S, unsigned long long *cursor, unsigned long long n,
                                          float tmax, uint32_t &err, TraceCounts *counts, Fetch &&fetch,
                                          Finish &&finish) {
    const uint32_t per_block = max(4u, min(static_cast<uint32_t>(SPK_WIDE_RAYS_PER_BLOCK), min(S.num_nodes, 64u) * 5u / 8u));
    if (n <= static_cast<unsigned long long>(gridDim.x) * per_block) {
        TraceCounts c;
        err |= walk_wide<kMode, kCount>(S, cursor, n, tmax, kCount ? &c : nullptr, fetch, finish);
        if (kCount) *counts = c;
    } else {
        walk_persistent<kMode, kCount, kDirect>(S, cursor, n, tmax, err, counts, fetch, finish);
    }
}

// Order-preserving map of a float to an int (and back) for warp min / max reductions.
__device__ __forceinline__ int float_key(float x) {
    const int b = __float_as_int(x);
    return b ^ ((b >> 31) & 0x7FFFFFFF);
}
__device__ __forceinline__ float key_float(int k) { return __int_as_float(k ^ ((k >> 31) & 0x7FFFFFFF)); }
__device__ __forceinline__ float warp_min(float x) { return key_float(__reduce_min_sync(0xFFFFFFFFu, float_key(x))); }
__device__ __forceinline__ float warp_max(float x) { return key_float(__reduce_max_sync(0xFFFFFFFFu, float_key(x))); }

// Bounds of a packet's level rays: origins and slab reciprocals per axis over the warp's 32 lanes.
struct PacketFrustum {
    f3 omin, omax, imin, imax;
};

// Fills `f` from the level rays of every lane (kRays per lane) and returns true when the packet can be tested
// as one: every ray's direction lies in octant `order` and no component is small enough for slab_inverse's
// 2^100 stand-in (so every bound below stays finite). Every lane of the warp must call this.
template <int kRays>
__device__ __forceinline__ bool make_frustum(const LevelRay (&r)[kRays], uint32_t order, PacketFrustum &f) {
    bool ok = true;
    f3 omin = r[0].o, omax = r[0].o, imin = r[0].inv, imax = r[0].inv;
#pragma unroll
    for (int k = 0; k < kRays; ++k) {
        ok = ok && r[k].oct == order && fabsf(r[k].inv.x) < 0x1p24f && fabsf(r[k].inv.y) < 0x1p24f &&
             fabsf(r[k].inv.z) < 0x1p24f;
        if (k > 0) {
            omin = mk3(fminf(omin.x, r[k].o.x), fminf(omin.y, r[k].o.y), fminf(omin.z, r[k].o.z));
            omax = mk3(fmaxf(omax.x, r[k].o.x), fmaxf(omax.y, r[k].o.y), fmaxf(omax.z, r[k].o.z));
            imin = mk3(fminf(imin.x, r[k].inv.x), fminf(imin.y, r[k].inv.y), fminf(imin.z, r[k].inv.z));
            imax = mk3(fmaxf(imax.x, r[k].inv.x), fmaxf(imax.y, r[k].inv.y), fmaxf(imax.z, r[k].inv.z));
        }
    }
    if (!__all_sync(0xFFFFFFFFu, ok)) return false;
    f.omin = mk3(warp_min(omin.x), warp_min(omin.y), warp_min(omin.z));
    f.omax = mk3(warp_max(omax.x), warp_max(omax.y), warp_max(omax.z));
    f.imin = mk3(warp_min(imin.x), warp_min(imin.y), warp_min(imin.z));
    f.imax = mk3(warp_max(imax.x), warp_max(imax.y), warp_max(imax.z));
    // The bounds of (p - org) * inv widen with the spread of inv relative to its size: past a few tens of
    // percent (a component near zero in some rays) the packet test stops culling and walks far more nodes
    // than its rays need, so such a packet tests with its own rays instead.
    const float k = SPK_FRUSTUM_SPREAD;
    return f.imax.x - f.imin.x <= k * fminf(fabsf(f.imin.x), fabsf(f.imax.x)) &&
           f.imax.y - f.imin.y <= k * fminf(fabsf(f.imin.y), fabsf(f.imax.y)) &&
           f.imax.z - f.imin.z <= k * fminf(fabsf(f.imin.z), fabsf(f.imax.z));
}

// Bounds over the packet of one axis's slab terms: a = s * inv and o = (p - org) * inv, the two values
// a ray's slab test is made of (t = fma(q, a, o) for a plane byte q). Each is a product or difference of the
// lanes' values, so rounding to nearest keeps them within the products and differences of the extremes.
__device__ __forceinline__ void axis_bounds(float p, float s, float omin, float omax, float imin, float imax,
                                            float &alo, float &ahi, float &olo, float &ohi) {
    alo = s * imin;
    ahi = s * imax;
    const float nlo = p - omax, nhi = p - omin;
    const float c0 = nlo * imin, c1 = nlo * imax, c2 = nhi * imin, c3 = nhi * imax;
    olo = fminf(fminf(c0, c1), fminf(c2, c3));
    ohi = fmaxf(fmaxf(c0, c1), fmaxf(c2, c3));
}

// The slab test for a whole packet at once: each 8-lane group of the warp visits node `idx` (its own: the groups
// may visit different nodes), lane k testing child slot k mod 8 against the packet's bounds, and the group
// ORs the results. fma(q, a, o) grows with a (q >= 0) and with o, so the lower bound of each near-plane t and
// the upper bound of each far-plane t take the extremes of a and o: a child passes whenever it passes for at
// least one lane's own ray with that lane's tmax (<= `tmax`), in that form, and may pass for
// none (the packet then visits a node that none of its rays needs, which only costs time). Every lane of the
// warp must call this; the result is the same in every lane of a group.
__device__ __forceinline__ void visit_node_frustum(const uint4 *__restrict__ nodes, uint32_t idx,
                                                   const PacketFrustum &f, uint32_t order, float tmax,
                                                   uint2 &ngroup, uint2 &tgroup) {
    const uint4 *np = nodes + static_cast<size_t>(idx) * 5;
    const uint4 n0 = __ldg(np), n1 = __ldg(np + 1), n2 = __ldg(np + 2), n3 = __ldg(np + 3), n4 = __ldg(np + 4);
    float axlo, axhi, oxlo, oxhi, aylo, ayhi, oylo, oyhi, azlo, azhi, ozlo, ozhi;
    axis_bounds(__uint_as_float(n0.x), __uint_as_float((n0.w & 0xFFu) << 23), f.omin.x, f.omax.x, f.imin.x,
                f.imax.x, axlo, axhi, oxlo, oxhi);
    axis_bounds(__uint_as_float(n0.y), __uint_as_float(((n0.w >> 8) & 0xFFu) << 23), f.omin.y, f.omax.y, f.imin.y,
                f.imax.y, aylo, ayhi, oylo, oyhi);
    axis_bounds(__uint_as_float(n0.z), __uint_as_float(((n0.w >> 16) & 0xFFu) << 23), f.omin.z, f.omax.z,
                f.imin.z, f.imax.z, azlo, azhi, ozlo, ozhi);
    const uint32_t slot = threadIdx.x & 7u, h = slot >> 2, c = slot & 3u;
    const uint32_t meta4 = h ? n1.w : n1.z;
    const uint32_t lox = h ? n2.y : n2.x, loy = h ? n2.w : n2.z, loz = h ? n3.y : n3.x;
    const uint32_t hix = h ? n3.w : n3.z, hiy = h ? n4.y : n4.x, hiz = h ? n4.w : n4.z;
    const uint32_t nx = (order & 1u) ? hix : lox, fx = (order & 1u) ? lox : hix;
    const uint32_t ny = (order & 2u) ? hiy : loy, fy = (order & 2u) ? loy : hiy;
    const uint32_t nz = (order & 4u) ? hiz : loz, fz = (order & 4u) ? loz : hiz;
    const uint32_t sel = 0x4440u | c;
    const float t0 = fmaxf(fmaxf(fmaf(static_cast<float>(__byte_perm(nx, 0u, sel)), axlo, oxlo),
                                 fmaf(static_cast<float>(__byte_perm(ny, 0u, sel)), aylo, oylo)),
                           fmaxf(fmaf(static_cast<float>(__byte_perm(nz, 0u, sel)), azlo, ozlo), 0.f));
    const float t1 = fminf(fminf(fmaf(static_cast<float>(__byte_perm(fx, 0u, sel)), axhi, oxhi),
                                 fmaf(static_cast<float>(__byte_perm(fy, 0u, sel)), ayhi, oyhi)),
                           fminf(fmaf(static_cast<float>(__byte_perm(fz, 0u, sel)), azhi, ozhi), tmax));
    const uint32_t m = __byte_perm(meta4, 0u, sel);
    uint32_t bits = 0u;
    if (m != 0u && t0 <= t1) {
        uint32_t bit = m & 0x1Fu;
        if ((m & 0x18u) == 0x18u) bit ^= order;
        bits = ((m >> 5) & 7u) << bit;
    }
    uint32_t any = bits | __shfl_xor_sync(0xFFFFFFFFu, bits, 1);
    any |= __shfl_xor_sync(0xFFFFFFFFu, any, 2);
    any |= __shfl_xor_sync(0xFFFFFFFFu, any, 4);
    ngroup = make_uint2(n1.x, (any & 0xFF000000u) | (n0.w >> 24));
    tgroup = make_uint2(n1.y, any & 0x00FFFFFFu);
}

// Closest-hit walk of coherent rays in packets (primary rays: the samples of one pixel, or neighbouring
// pixels). Each warp takes 32 * kRays consecutive items of the work list (lane l the items l, l + 32, ...)
// and walks them together: one node or triangle group at a time for the whole warp, in the order of the
// leader's octant, every lane testing its own rays against each triangle. When all the packet's rays share
// that octant (checked per level, TLAS and each BLAS), a node's 8 children are tested once for the whole
// packet (visit_node_frustum: one child per lane against the bounds of all its rays); otherwise every lane
// tests them with its own rays (visit_slots) and takes only the children they hit. Either way a ray is tested
// against every box and triangle its own walk would reach, and pruned only beyond its own best t; it may be
// tested against more. Its result is still the smallest world t over every triangle and sphere it hits
// (exact ties to the smaller (instance, face)), which no visiting order or extra test changes: the results
// are walk_persistent's. `fetch(i, o, d, tmax)` and `finish(i, result)` as for walk_persistent (`fetch` may
// be called more than once for an item, `finish` must find the item from i alone); every lane of the warp
// must call this. `counts` (kCount) takes each node and triangle once per packet: one fetch serves its rays.
template <bool kCount, int kRays, class Fetch, class Finish>
__device__ __forceinline__ void walk_packets(const DevScene &S, unsigned long long *cursor, unsigned long long n,
                                             uint32_t &err, TraceCounts *counts, Fetch &&fetch, Finish &&finish) {
    static_assert(kRays == 1 || kRays == 2, "one or two rays per lane");
    constexpr uint32_t kAll = 0xFFFFFFFFu;
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t budget = S.walk_budget ? S.walk_budget : kMaxIterations;
    uint2 groups[kPacketStack];  // the shared groups (the same in every lane)
    uint32_t own[kPacketStack];  // this lane's hit bits of each
#if SPK_PACKET_WORLD_SMEM
    // Each lane's world rays (origin, direction per ray) wait in shared memory, read only at a BLAS exit and
    // for a candidate hit's world t: entry k of thread t at [k][t], consecutive lanes in consecutive words.
    __shared__ float4 world[2 * kRays][kWalkThreads];
    auto world_o = [&](int r) { const float4 v = world[2 * r][threadIdx.x]; return mk3(v.x, v.y, v.z); };
    auto world_d = [&](int r) { const float4 v = world[2 * r + 1][threadIdx.x]; return mk3(v.x, v.y, v.z); };
#endif
    unsigned long long base = 0;
    bool todo[kRays];  // this lane's items not walked yet
#pragma unroll
    for (int r = 0; r < kRays; ++r) todo[r] = false;
    for (;;) {
        bool any_todo = false;
#pragma unroll
        for (int r = 0; r < kRays; ++r) any_todo = any_todo || todo[r];
        if (!__any_sync(kAll, any_todo)) {
            unsigned long long b = 0;
            if (lane == 0) b = atomicAdd(cursor, 32ull * kRays);
            base = __shfl_sync(kAll, b, 0);
            if (base >= n) break;
#pragma unroll
            for (int r = 0; r < kRays; ++r) todo[r] = base + lane + 32u * r < n;  // lane 0's first always
            any_todo = todo[0];
        }
        // One packet per TLAS root among the items (a batch of requests holds several scenes; almost every
        // warp has one). The packet is the rays with the leader's root (its lowest pending item's); the
        // others, and items past the end of the list, walk a copy of that ray and drop their results, which
        // keeps the packet's bounds and octant those of its real rays.
        const int leader = __ffs(__ballot_sync(kAll, any_todo)) - 1;
        f3 wo[kRays], wd[kRays];
        uint32_t root[kRays];
        bool valid[kRays];
#pragma unroll
        for (int r = 0; r < kRays; ++r) {
            wo[r] = mk3(0.f, 0.f, 0.f);
            wd[r] = mk3(1.f, 1.f, 1.f);
            root[r] = kInvalid;
            if (todo[r]) {
                float tm = kFltMax;
                root[r] = fetch(base + lane + 32u * r, wo[r], wd[r], tm);
            }
        }
        uint32_t first_root = root[0];
        f3 first_o = wo[0], first_d = wd[0];
        if (kRays > 1 && !todo[0]) {
            first_root = root[kRays - 1];
            first_o = wo[kRays - 1];
            first_d = wd[kRays - 1];
        }
        const uint32_t lroot = __shfl_sync(kAll, first_root, leader);
        const f3 o0 = mk3(__shfl_sync(kAll, first_o.x, leader), __shfl_sync(kAll, first_o.y, leader),
                          __shfl_sync(kAll, first_o.z, leader));
        const f3 d0 = mk3(__shfl_sync(kAll, first_d.x, leader), __shfl_sync(kAll, first_d.y, leader),
                          __shfl_sync(kAll, first_d.z, leader));
        LevelRay ray[kRays];
        TraceResult best[kRays];
        float tmax_box[kRays];
#pragma unroll
        for (int r = 0; r < kRays; ++r) {
            valid[r] = todo[r] && root[r] == lroot;
            todo[r] = todo[r] && !valid[r];
            if (!valid[r]) {
                wo[r] = o0;
                wd[r] = d0;
            }
            setup_level(ray[r], wo[r], wd[r]);
            best[r] = TraceResult{kFltMax, 0.f, 0.f, kInvalid, kInvalid};
            tmax_box[r] = kFltMax;
#if SPK_PACKET_WORLD_SMEM
            world[2 * r][threadIdx.x] = make_float4(wo[r].x, wo[r].y, wo[r].z, 0.f);
            world[2 * r + 1][threadIdx.x] = make_float4(wd[r].x, wd[r].y, wd[r].z, 0.f);
#endif
        }
        const uint32_t top_order = __shfl_sync(kAll, ray[0].oct, leader);  // the leader's ray: o0, d0
        uint32_t order = top_order;
        PacketFrustum frustum;
        bool packed = make_frustum(ray, order, frustum);  // the level's nodes are tested once for the packet
        uint2 ngroup = make_uint2(lroot, lroot == kInvalid ? 0u : (1u << 24)), tgroup = make_uint2(0u, 0u);
        uint32_t nown = 1u << 24, town = 0u;
        int sp = 0, blas_sp = 0;
        bool in_blas = false;
        uint32_t cur_inst = 0, iter = 0;
        auto push = [&](uint2 g, uint32_t mine) {
            if (sp < kPacketStack) {
                groups[sp] = g;
                own[sp] = mine;
                ++sp;
            } else {
                err |= kErrStackOverflow;
            }
        };
        auto lane_tmax = [&]() {
            float t = tmax_box[0];
#pragma unroll
            for (int r = 1; r < kRays; ++r) t = fmaxf(t, tmax_box[r]);
            return t;
        };
        for (;;) {
            if (++iter > budget) {
                err |= kErrIterationBudget;
                break;
            }
            if (ngroup.y > 0x00FFFFFFu && packed && SPK_PACKET_FRUSTUM) {
                // The nearest inner children of the group (up to kPacketSiblings, while the stack has room for
                // their groups), one per 8-lane group, each tested once for the packet against the largest
                // tmax of the rays of the lanes that reached any of them (tmax_box is never negative). A lane
                // takes every child that passes in the nodes it reached.
                const uint32_t imask = ngroup.y & 0xFFu, inner = ngroup.y >> 24;
                const uint32_t room = sp + 2 * kPacketSiblings <= kPacketStack ? kPacketSiblings : 1u;
                const uint32_t cnt = min(static_cast<uint32_t>(__popc(inner)), room);
                const uint32_t grp = (threadIdx.x >> 3) & 3u;
                uint32_t rest = inner, from = inner;
                for (uint32_t k = 0; k < cnt; ++k) {
                    if (k == grp) from = rest;
                    rest &= rest - 1u;
                }
                const uint32_t slot = (__ffs(from) - 1) ^ order;  // groups past `cnt` repeat the first child
                const uint32_t node_idx = ngroup.x + __popc(imask & ((1u << slot) - 1u));
                const uint32_t taken = inner & ~rest;
                const uint32_t mine_taken = (nown >> 24) & taken;
                ngroup.y = (rest << 24) | imask;
                nown &= ~(taken << 24);
                if (rest) push(ngroup, nown);
                if (kCount && lane == 0) counts->nodes += cnt;
                const float tmax =
                    __uint_as_float(__reduce_max_sync(kAll, mine_taken ? __float_as_uint(lane_tmax()) : 0u));
                uint2 ng, tg;
                visit_node_frustum(S.nodes, node_idx, frustum, order, tmax, ng, tg);
                // Hand each child's groups out, farthest first onto the stack so the nearest comes back first.
                uint32_t left = taken;
                for (int g = static_cast<int>(cnt) - 1; g >= 0; --g) {
                    const uint32_t b = 31 - __clz(left);
                    left &= ~(1u << b);
                    const bool mine = (mine_taken >> b) & 1u;
                    const uint2 n_g = make_uint2(__shfl_sync(kAll, ng.x, 8 * g), __shfl_sync(kAll, ng.y, 8 * g));
                    const uint2 t_g = make_uint2(__shfl_sync(kAll, tg.x, 8 * g), __shfl_sync(kAll, tg.y, 8 * g));
                    if (g == 0) {
                        ngroup = n_g;
                        tgroup = t_g;
                        nown = mine ? (n_g.y & 0xFF000000u) : 0u;
                        town = mine ? t_g.y : 0u;
                    } else {
                        if (n_g.y > 0x00FFFFFFu) push(n_g, mine ? (n_g.y & 0xFF000000u) : 0u);
                        if (t_g.y != 0u) push(t_g, mine ? t_g.y : 0u);
                    }
                }
            } else if (ngroup.y > 0x00FFFFFFu) {
                const uint32_t bit = __ffs(ngroup.y >> 24) - 1;
                const uint32_t keep = ~(1u << (bit + 24));
                const bool mine = (nown >> (bit + 24)) & 1u;
                ngroup.y &= keep;
                nown &= keep;
                const uint32_t slot = bit ^ order;
                const uint32_t node_idx = ngroup.x + __popc(ngroup.y & 0xFFu & ((1u << slot) - 1u));
                if (ngroup.y > 0x00FFFFFFu) push(ngroup, nown);
                if (kCount && lane == 0) ++counts->nodes;
                // Rays of several octants: every lane tests the node with its own rays; a lane that did not
                // reach it tests against t <= -1 (no hits).
                uint32_t hits = 0u;
#pragma unroll
                for (int r = 0; r < kRays; ++r) {
                    const NodeHits h = visit_slots(S.nodes, node_idx, ray[r], mine ? tmax_box[r] : -1.f);
                    hits |= (order_slots(h.hit & h.imask, order) << 24) | leaf_items(h.hit & ~h.imask, h.meta);
                    ngroup.x = h.child_base;
                    tgroup.x = h.item_base;
                    ngroup.y = (ngroup.y & ~0xFFu) | h.imask;  // the child's imask
                }
                nown = hits & 0xFF000000u;
                town = hits & 0x00FFFFFFu;
                const uint32_t any = __reduce_or_sync(kAll, hits);
                ngroup.y = (any & 0xFF000000u) | (ngroup.y & 0xFFu);
                tgroup.y = any & 0x00FFFFFFu;
            } else {
                tgroup = ngroup;
                town = nown;
                ngroup = make_uint2(0u, 0u);
                nown = 0u;
            }
            while (tgroup.y != 0u) {
                const uint32_t k = __ffs(tgroup.y) - 1;
                tgroup.y &= tgroup.y - 1u;
                const bool mine = (town >> k) & 1u;
                const uint32_t idx = tgroup.x + k;
                if (in_blas) {
                    if (kCount && lane == 0) ++counts->tris;
                    if (!mine) continue;
#pragma unroll
                    for (int r = 0; r < kRays; ++r) {
                        float t, u, v;
                        uint32_t face;
                        if (!triangle_hit(S.tris, idx, ray[r], t, u, v, face)) continue;
#if SPK_PACKET_WORLD_SMEM
                        const f3 ro = world_o(r), rd = world_d(r);
#else
                        const f3 ro = wo[r], rd = wd[r];
#endif
                        const float wt = world_t(S.instances[cur_inst], ray[r], t, ro, rd);
                        if (wt > 0.f && closer_hit(best[r], wt, cur_inst, face)) {
                            best[r] = TraceResult{wt, u, v, cur_inst, face};
                            tmax_box[r] = prune_limit(wt, ro.x, rd.x, S.scene_abs_x);
                        }
                    }
                } else {
                    const uint32_t inst = __ldg(S.tlas_items + idx);
                    const DevInstance &I = S.instances[inst];
                    if (I.type == 1u) {
                        if (!mine) continue;
#pragma unroll
                        for (int r = 0; r < kRays; ++r) {
                            float t;
                            // (at the TLAS level the level ray is the world ray)
                            if (sphere_hit(I, ray[r].o, ray[r].d, t) && t > 0.f &&
                                closer_hit(best[r], t, inst, kInvalid)) {
                                best[r] = TraceResult{t, 0.f, 0.f, inst, kInvalid};
                                tmax_box[r] = prune_limit(t, ray[r].o.x, ray[r].d.x, S.scene_abs_x);
                            }
                        }
                    } else if (I.blas_root != kInvalid) {
                        // Enter the BLAS with every lane (those that did not reach it take no part); the
                        // rest of this TLAS level waits on the stack.
                        if (tgroup.y != 0u) push(tgroup, town);
                        if (ngroup.y > 0x00FFFFFFu) push(ngroup, nown);
                        blas_sp = sp;
                        in_blas = true;
                        cur_inst = inst;
#pragma unroll
                        for (int r = 0; r < kRays; ++r)
                            setup_level(ray[r], xform_point(I.minv, ray[r].o), xform_dir(I.minv, ray[r].d));
                        const uint32_t entering = __ballot_sync(kAll, mine);  // not empty: the group had bit k
                        order = __shfl_sync(kAll, ray[0].oct, __ffs(entering) - 1);
                        packed = make_frustum(ray, order, frustum);
                        ngroup = make_uint2(I.blas_root, 1u << 24);
                        nown = mine ? (1u << 24) : 0u;
                        tgroup.y = 0u;
                        break;
                    }
                }
            }
            if (ngroup.y <= 0x00FFFFFFu) {
                if (in_blas && sp == blas_sp) {
                    in_blas = false;
#pragma unroll
                    for (int r = 0; r < kRays; ++r) {
#if SPK_PACKET_WORLD_SMEM
                        setup_level(ray[r], world_o(r), world_d(r));
#else
                        setup_level(ray[r], wo[r], wd[r]);
#endif
                    }
                    order = top_order;
                    if (sp != 0) packed = make_frustum(ray, order, frustum);
                }
                if (sp == 0) break;
                --sp;
                ngroup = groups[sp];
                nown = own[sp];
            }
        }
#pragma unroll
        for (int r = 0; r < kRays; ++r)
            if (valid[r]) finish(base + lane + 32u * r, best[r]);
    }
}

}  // namespace spk
