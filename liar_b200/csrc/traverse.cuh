// traverse.cuh -- sm_100a closest-hit / any-hit traversal of the 4-wide tree (qbvh.h).
//
// Replaces the per-ray Lass traversal behind TriangleMesh::doIntersect / doIsIntersecting
// (src/liar/scenery/triangle_mesh.cpp:291-330) and ObjectTree::doIntersect / doIsIntersecting
// (src/liar/scenery/object_trees.h:110-143).
//
// Organisation (one lane per ray, persistent warps with per-lane refill):
//   * a grid of (SM count x resident blocks) blocks; each warp takes batches of BATCH ray indices
//     (up to 256, sized so that the n rays cover every resident warp), its first one by its own
//     number and further ones from one atomic work counter, and hands them to its lanes one by one:
//     whenever at least REFILL lanes have finished their ray, those lanes store their hits and load
//     the next rays of the batch, so short rays (most random rays miss the mesh after a node or two)
//     do not leave lanes idle while a long ray of the same warp is still traversing (dynamic
//     fetch, Aila & Laine 2009);
//   * one loop turn (trace_turn) = a node phase, a leaf phase and a pop: every lane still descending
//     visits one node, lanes that have reached a leaf wait until LEAF_AT of them have (or none
//     descends any more) and then test their leaves together, lanes left without a node pop one.
//     Compared with running each lane down to its next leaf per turn, lanes idle far less (random
//     rays of very different lengths);
//   * a node is 64 bytes, its child boxes quantised to a byte a plane (qbvh.h), read with four 16-byte
//     loads that carry an L2 evict-last policy; rays and hits stream with evict-first, so the 512 MiB
//     ray stream does not push the tree out of L2. With every lane at its own node a 16-byte load
//     costs an L1 wavefront per lane, and with unquantised planes (seven such loads a visit) those
//     wavefronts bound the kernel (86% of their peak, issue 60%); with four they are at 62% and the
//     issue slots (72%) are the limit. 16.7M random rays on the 1.31M-triangle icosphere, closest hit:
//     2.74 ms unquantised, 2.44 ms with centre and half-extent rows in 32-byte loads (each still two
//     wavefronts), 1.94 ms quantised, decoded by a byte permutation a plane and packed FMAs;
//   * hit children are ordered by entry distance (5-comparator network on distance-bit keys; any hit
//     takes them as they come); the farther ones are pushed with their key onto a per-lane stack
//     whose top S entries live in shared memory (column per lane: conflict-free) and whose deeper
//     entries spill to local memory; popped entries farther than the current closest hit are dropped;
//   * the last rays of a warp, and all rays of launches with a few rays per warp, are traced one at a
//     time by the whole warp (trace_coop), which takes a fraction of the time of a lone lane;
//   * triangles are tested with the exact Moller-Trumbore of tri_exact.h, so t is bit-identical
//     to the CPU restatement, and equal t resolves to the lower original triangle index.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "../../include/liar_gpu.h"
#include "qbvh.h"
#include "tri_exact.h"

namespace liar_gpu {

// device-side status bits (ORed into the status word of a launch)
enum : uint32_t { STATUS_STACK_OVERFLOW = 1u, STATUS_BAD_NODE = 2u };

// total stack entries per lane (shared top + local spill); the host refuses deeper trees
constexpr int kTraceStackTotal = 64;

// Where trace_coop takes over: at once in a launch that gives every warp at most kCoopBatch rays and
// no more, else when a warp without further rays to fetch has held at most kCoopRays unfinished ones
// for kCoopTurns turns (the short rays of small scenes end before that: one by one they would take
// longer). Measured on 1.31M triangles, random rays: 70,000 rays 179 -> 72 us, 300,000 193 -> 100 us;
// 1000 rays on 5,120 triangles 26 -> 14 us; 2 or 8 rays instead of 4: the same there, guided rendering
// 2% slower at 8.
constexpr uint32_t kCoopRays = 4, kCoopBatch = 8, kCoopTurns = 12;

struct TraceCounters {
    unsigned long long nodes;
    unsigned long long tris;
};

// ---- loads and stores with L2 eviction policies (PTX createpolicy / cache_hint)
__device__ __forceinline__ uint64_t policy_evict_last() {
    uint64_t p;
    asm("createpolicy.fractional.L2::evict_last.b64 %0, 1.0;" : "=l"(p));
    return p;
}
__device__ __forceinline__ uint64_t policy_evict_first() {
    uint64_t p;
    asm("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(p));
    return p;
}
__device__ __forceinline__ float4 ld_hint(const void* ptr, uint64_t pol) {
    float4 v;
    asm("ld.global.nc.L2::cache_hint.v4.f32 {%0, %1, %2, %3}, [%4], %5;"
        : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
        : "l"(ptr), "l"(pol));
    return v;
}
__device__ __forceinline__ int4 ld_hint_i(const void* ptr, uint64_t pol) {
    int4 v;
    asm("ld.global.nc.L2::cache_hint.v4.s32 {%0, %1, %2, %3}, [%4], %5;"
        : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
        : "l"(ptr), "l"(pol));
    return v;
}
__device__ __forceinline__ void st_hint(void* ptr, int a, int b, uint64_t pol) {
    asm volatile("st.global.L2::cache_hint.v2.s32 [%0], {%1, %2}, %3;" ::"l"(ptr), "r"(a), "r"(b), "l"(pol) : "memory");
}

__device__ __forceinline__ float safe_rcp(float d) {
    // keeps 1/d finite, so that inverted (empty) boxes can never produce NaN slab distances; the
    // approximate reciprocal (within 1 ulp) only enters the box tests, whose padding covers it
    const float ad = fabsf(d);
    float r;
    asm("rcp.approx.f32 %0, %1;" : "=f"(r) : "f"(ad > 1e-20f ? d : copysignf(1e-20f, d)));
    return r;
}

__device__ __forceinline__ uint64_t f2_splat2(float a) {
    uint64_t r;
    asm("mov.b64 %0, {%1, %1};" : "=l"(r) : "f"(a));
    return r;
}
__device__ __forceinline__ uint64_t f2_pair(float a, float b) {
    uint64_t r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ uint64_t f2_fma2(uint64_t a, uint64_t b, uint64_t c) {
    uint64_t d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}
__device__ __forceinline__ void f2_split2(uint64_t v, float& lo, float& hi) {
    asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
}
// three-input minimum and maximum
__device__ __forceinline__ float max3f(float a, float b, float c) {
    float d;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
    return d;
}
__device__ __forceinline__ float min3f(float a, float b, float c) {
    float d;
    asm("min.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
    return d;
}
__device__ __forceinline__ int sel4i(const int4& v, uint32_t s) {
    const int a = (s & 1u) ? v.y : v.x, b = (s & 1u) ? v.w : v.z;
    return (s & 2u) ? b : a;
}
__device__ __forceinline__ void cswap(int& a, int& b) {
    const int lo = min(a, b), hi = max(a, b);
    a = lo;
    b = hi;
}

// Rays that are retired untraced, as misses: non-finite origins or directions, NaN limits, and
// directions with a component of minus zero (whose reciprocal is negative although the component
// is not below zero: the boxes of such a ray have always been entered from the wrong side)
__device__ __forceinline__ bool traceable(const float4& r0, const float4& r1) {
    const uint32_t nz = 0x80000000u;
    return isfinite(r0.x) && isfinite(r0.y) && isfinite(r0.z) && isfinite(r1.x) && isfinite(r1.y) && isfinite(r1.z) &&
           !isnan(r0.w) && !isnan(r1.w) && __float_as_uint(r1.x) != nz && __float_as_uint(r1.y) != nz &&
           __float_as_uint(r1.z) != nz;
}

// no node left here (pop the next), and no node left at all; real leaves lie below both (their
// counts are <= 8, so that the packed word is at most 0xc7ffffff)
constexpr int kNodeNone = -1, kNodeDone = -2;

// Per-lane traversal state.
struct RayState {
    float ox, oy, oz, tmin, dx, dy, dz, tmax;
    float idx, idy, idz, oix, oiy, oiz;
    float tbest;
    int best;
    int node;
    int sp;
};

// The stack of a lane: (node or leaf, sort key of visit_node).
template <int S, int BLOCK>
struct LaneStack {
    static constexpr int L = kTraceStackTotal - S > 0 ? kTraceStackTotal - S : 1;
    uint2* s_ent;  // this lane's column: entry sp at s_ent[sp * BLOCK]
    uint2 l_ent[L];

    __device__ __forceinline__ void push(int sp, int node, uint32_t key) {
        const uint2 e = make_uint2((uint32_t)node, key);
        if (sp < S) s_ent[sp * BLOCK] = e;
        else l_ent[sp - S] = e;
    }
    __device__ __forceinline__ void get(int sp, int& node, float& t) const {
        const uint2 e = sp < S ? s_ent[sp * BLOCK] : l_ent[sp - S];
        node = (int)e.x;
        t = __uint_as_float(e.y & ~3u);
    }
};

// byte i of w as its plane value (qbvh.h): the float with bits 0x40qq0000
template <int I>
__device__ __forceinline__ float plane_float(uint32_t w) {
    return __uint_as_float(__byte_perm(w, 0x40000000u, 0x7044 | (I << 8)));
}

// One inner node: st.node >= 0 on entry. Its hit children are ordered by entry distance, the
// farther ones pushed; on exit st.node is the nearest hit child (inner node or leaf), or kNodeNone
// when no child is hit.
template <bool ANY, int S, int BLOCK, bool COUNT>
__device__ __forceinline__ void visit_node(const QNode* __restrict__ nodes, RayState& st, LaneStack<S, BLOCK>& stack,
                                           uint64_t pol_tree, uint32_t& status, uint32_t& n_nodes) {
    if (COUNT) ++n_nodes;
    const char* qb = reinterpret_cast<const char*>(nodes + st.node);
    const float4 r0 = ld_hint(qb, pol_tree);
    const int4 r1 = ld_hint_i(qb + 16, pol_tree), r2 = ld_hint_i(qb + 32, pol_tree), ch = ld_hint_i(qb + 48, pol_tree);
    // t of a plane with value v on axis a: v * A + B
    const float Ax = r0.w * st.idx, Ay = __int_as_float(r1.x) * st.idy, Az = __int_as_float(r1.y) * st.idz;
    const float Bx = fmaf(r0.x, st.idx, -st.oix), By = fmaf(r0.y, st.idy, -st.oiy), Bz = fmaf(r0.z, st.idz, -st.oiz);
    // the codes of the planes a ray meets first along each axis, all four children at once
    const bool nx = st.idx < 0.0f, ny = st.idy < 0.0f, nz = st.idz < 0.0f;
    const uint32_t lx = r1.z, ly = r1.w, lz = r2.x, hx = r2.y, hy = r2.z, hz = r2.w;
    const uint32_t nwx = nx ? hx : lx, fwx = nx ? lx : hx, nwy = ny ? hy : ly, fwy = ny ? ly : hy, nwz = nz ? hz : lz,
                   fwz = nz ? lz : hz;
    float tn[4], tf[4];
    const uint64_t Ax2 = f2_splat2(Ax), Ay2 = f2_splat2(Ay), Az2 = f2_splat2(Az), Bx2 = f2_splat2(Bx), By2 = f2_splat2(By), Bz2 = f2_splat2(Bz);
#define LIAR_CHILD2(k)                                                                                             \
    {                                                                                                              \
        float n[3][2], f[3][2];                                                                                    \
        f2_split2(f2_fma2(f2_pair(plane_float<k>(nwx), plane_float<k + 1>(nwx)), Ax2, Bx2), n[0][0], n[0][1]);     \
        f2_split2(f2_fma2(f2_pair(plane_float<k>(nwy), plane_float<k + 1>(nwy)), Ay2, By2), n[1][0], n[1][1]);     \
        f2_split2(f2_fma2(f2_pair(plane_float<k>(nwz), plane_float<k + 1>(nwz)), Az2, Bz2), n[2][0], n[2][1]);     \
        f2_split2(f2_fma2(f2_pair(plane_float<k>(fwx), plane_float<k + 1>(fwx)), Ax2, Bx2), f[0][0], f[0][1]);     \
        f2_split2(f2_fma2(f2_pair(plane_float<k>(fwy), plane_float<k + 1>(fwy)), Ay2, By2), f[1][0], f[1][1]);     \
        f2_split2(f2_fma2(f2_pair(plane_float<k>(fwz), plane_float<k + 1>(fwz)), Az2, Bz2), f[2][0], f[2][1]);     \
        tn[k] = max3f(n[0][0], n[1][0], fmaxf(n[2][0], st.tmin));                                                  \
        tn[k + 1] = max3f(n[0][1], n[1][1], fmaxf(n[2][1], st.tmin));                                              \
        tf[k] = min3f(f[0][0], f[1][0], fminf(f[2][0], st.tbest));                                                 \
        tf[k + 1] = min3f(f[0][1], f[1][1], fminf(f[2][1], st.tbest));                                             \
    }
    LIAR_CHILD2(0)
    LIAR_CHILD2(2)
#undef LIAR_CHILD2
    if (ANY) {
        // in any order, without distances
        const bool room = st.sp <= S - 3;
        int next = kNodeNone;
#pragma unroll
        for (int k = 3; k >= 0; --k) {
            if (!(tn[k] <= tf[k])) continue;
            if (next != kNodeNone) {
                if (room) stack.s_ent[st.sp * BLOCK] = make_uint2((uint32_t)next, 0u);
                else if (st.sp < kTraceStackTotal) stack.push(st.sp, next, 0u);
                else status |= STATUS_STACK_OVERFLOW, --st.sp;
                ++st.sp;
            }
            next = k == 0 ? ch.x : k == 1 ? ch.y : k == 2 ? ch.z : ch.w;
        }
        st.node = next;
        return;
    }
    // sortable keys: entry distance bits as a signed number with the slot in the two low bits
    // (negative distances, possible when tmin < 0, come first, in no order); misses become kMiss
    constexpr int kMiss = 0x7fffffff;
    int key[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) key[k] = tn[k] <= tf[k] ? ((__float_as_int(tn[k]) & ~3) | k) : kMiss;
    cswap(key[0], key[1]);
    cswap(key[2], key[3]);
    cswap(key[0], key[2]);
    cswap(key[1], key[3]);
    cswap(key[1], key[2]);
    if (key[0] == kMiss) {
        st.node = kNodeNone;  // nothing hit below this node
        return;
    }
    // push the other hit children, farthest first
    if (st.sp <= S - 3) {
        uint2* top = stack.s_ent + st.sp * BLOCK;
#pragma unroll
        for (int k = 3; k >= 1; --k) {
            if (key[k] != kMiss) {
                *top = make_uint2((uint32_t)sel4i(ch, (uint32_t)key[k]), (uint32_t)key[k]);
                top += BLOCK;
                ++st.sp;
            }
        }
    } else {
#pragma unroll
        for (int k = 3; k >= 1; --k) {
            if (key[k] == kMiss) continue;
            if (st.sp >= kTraceStackTotal) {
                status |= STATUS_STACK_OVERFLOW;
                continue;
            }
            stack.push(st.sp, sel4i(ch, (uint32_t)key[k]), (uint32_t)key[k]);
            ++st.sp;
        }
    }
    st.node = sel4i(ch, (uint32_t)key[0]);
}

// The primitive at tp against the ray: true with its distance t (range not checked) and index.
__device__ __forceinline__ bool test_prim(const QTri* tp, const RayState& st, uint64_t pol_tree, float& t, int& prim) {
    const float4 a = ld_hint(&tp->v0, pol_tree), e1 = ld_hint(&tp->e1, pol_tree), e2 = ld_hint(&tp->e2, pol_tree);
    float u, v;
    prim = __float_as_int(a.w);
    if (e1.w != 0.0f) {
        // a sphere: its nearer root beyond tmin, else the farther one
        float t1;
        const bool hit = sphere_intersect_exact(st.ox, st.oy, st.oz, st.dx, st.dy, st.dz, a.x, a.y, a.z, e1.x, t, t1);
        if (hit && !(t > st.tmin)) t = t1;
        return hit;
    }
    return tri_intersect_exact(st.ox, st.oy, st.oz, st.dx, st.dy, st.dz, a.x, a.y, a.z, e1.x, e1.y, e1.z, e2.x, e2.y, e2.z,
                               t, u, v);
}

// Tests the leaf st.node (packed 0x80000000 | count << 27 | first). True when an any-hit ray is
// finished by it.
template <bool ANY, bool COUNT>
__device__ __forceinline__ bool test_leaf(const QTri* __restrict__ tris, RayState& st, uint64_t pol_tree,
                                          uint32_t& n_tris) {
    const uint32_t packed = (uint32_t)st.node;
    const uint32_t count = (packed >> 27) & 15u;
    const uint32_t first = packed & 0x07ffffffu;
    for (uint32_t k = 0; k < count; ++k) {
        if (COUNT) ++n_tris;
        float t;
        int prim;
        if (test_prim(tris + first + k, st, pol_tree, t, prim)) {
            if (ANY) {
                if (t > st.tmin && t < st.tmax) {
                    st.best = prim;
                    st.tbest = t;
                    return true;
                }
            } else if (t > st.tmin && (t < st.tbest || (t == st.tbest && prim < st.best))) {
                st.tbest = t;
                st.best = prim;
            }
        }
    }
    return false;
}

// Takes the next entry that can still hold a closer hit into st.node, or kNodeDone.
template <bool ANY, int S, int BLOCK>
__device__ __forceinline__ void pop_next(RayState& st, const LaneStack<S, BLOCK>& stack) {
    // entry distances below zero never cull (their low bits raise them); the low bits of the others
    // hold the slot and are cleared, which lowers them
    const float far = fmaxf(st.tbest, 0.0f);
    while (st.sp > 0) {
        --st.sp;
        int nd;
        float te;
        stack.get(st.sp, nd, te);
        if (ANY || te <= far) {
            st.node = nd;
            return;
        }
    }
    st.node = kNodeDone;
}

// A new ray (r0: origin, tmin; r1: direction, tmax) at the root of its tree.
template <bool ANY>
__device__ __forceinline__ void start_ray(const float4& r0, const float4& r1, RayState& st) {
    st.ox = r0.x;
    st.oy = r0.y;
    st.oz = r0.z;
    st.tmin = r0.w;
    st.dx = r1.x;
    st.dy = r1.y;
    st.dz = r1.z;
    st.tmax = r1.w;
    st.idx = safe_rcp(st.dx);
    st.idy = safe_rcp(st.dy);
    st.idz = safe_rcp(st.dz);
    st.oix = st.ox * st.idx;
    st.oiy = st.oy * st.idy;
    st.oiz = st.oz * st.idz;
    // closest hit keeps candidates strictly below range_far(tmax); any hit below tmax
    st.tbest = ANY ? st.tmax : range_far(st.tmax);
    st.best = -1;
    st.sp = 0;
    st.node = traceable(r0, r1) ? 0 : kNodeDone;
}

// The finished ray's hit to memory.
template <bool ANY>
__device__ __forceinline__ void store_hit(const RayState& st, liar_hit* hit, uint64_t pol) {
    int prim = st.best;
    float t = st.tbest;
    if (!ANY && prim >= 0 && !(t > range_near(st.tmin))) prim = -1;  // BoundedRay::inRange near side
    if (prim < 0) t = INFINITY;
    st_hint(hit, prim, __float_as_int(t), pol);
}

// One turn of a warp's rays (see the head of this file): every descending lane visits a node, the
// lanes at a leaf test it once LEAF_AT of them wait (or none descends), and lanes left without a
// node pop one. A lane is done with its ray when st.node is kNodeDone.
template <bool ANY, int S, int BLOCK, bool COUNT, int LEAF_AT>
__device__ __forceinline__ void trace_turn(const QNode* __restrict__ nodes, const QTri* __restrict__ tris, RayState& st,
                                           LaneStack<S, BLOCK>& stack, uint64_t pol_tree, uint32_t& status,
                                           uint32_t& n_nodes, uint32_t& n_tris) {
    if (st.node >= 0) visit_node<ANY, S, BLOCK, COUNT>(nodes, st, stack, pol_tree, status, n_nodes);
    const bool at_leaf = st.node < kNodeDone;
    const uint32_t leafw = __ballot_sync(0xffffffffu, at_leaf);
    if (leafw) {
        if ((uint32_t)__popc(leafw) >= (uint32_t)LEAF_AT || !__any_sync(0xffffffffu, st.node >= 0)) {
            if (at_leaf) st.node = test_leaf<ANY, COUNT>(tris, st, pol_tree, n_tris) ? kNodeDone : kNodeNone;
        }
    }
    if (st.node == kNodeNone) pop_next<ANY, S, BLOCK>(st, stack);
}

// One ray traced by a whole warp, for launches (and the ends of launches) with few rays, which last
// as long as their longest ray: a ray along the surface visits hundreds of nodes, one after the other
// in trace_turn. Here eight entries come off the stack at once, four lanes to an entry: a lane tests
// one child box of a node or one primitive of a leaf. The rays the lanes hold are taken one by one,
// from the root (with the hits they have), their stacks' shared memory as one stack. Every lane of
// the warp calls this; on return every ray is finished.
// Not inlined, and given the rays by their index: its registers are not those of the main loop.
struct CoopResult {
    int best;
    float tbest;
    uint32_t n_nodes, n_tris;
};
template <bool ANY, int S, int BLOCK, bool COUNT>
__device__ __forceinline__ CoopResult trace_coop(const QNode* lane_nodes, const QTri* lane_tris, const liar_ray* rays, int rid,
                                              int best, float tbest, uint2* s_warp, uint32_t* status_word) {
    constexpr int kCap = S * 32;  // entry e at s_warp[(e / 32) * BLOCK + e % 32]
    const uint32_t lane = threadIdx.x & 31u, c = lane & 3u, group = lane >> 2;
    const uint64_t pol_tree = policy_evict_last();
    const auto slot = [&](int e) { return s_warp + (e >> 5) * BLOCK + (e & 31); };
    CoopResult out{best, tbest, 0u, 0u};
    uint32_t& n_nodes = out.n_nodes;
    uint32_t& n_tris = out.n_tris;
    uint32_t todo = __ballot_sync(0xffffffffu, rid >= 0);
    while (todo) {
        const int src = __ffs(todo) - 1;
        todo &= todo - 1;
        const float4* rp = reinterpret_cast<const float4*>(rays + __shfl_sync(0xffffffffu, rid, src));
        RayState st;
        start_ray<ANY>(__ldg(rp), __ldg(rp + 1), st);
        st.tbest = __shfl_sync(0xffffffffu, tbest, src);
        st.best = __shfl_sync(0xffffffffu, best, src);
        const QNode* nodes = reinterpret_cast<const QNode*>(__shfl_sync(0xffffffffu, (unsigned long long)lane_nodes, src));
        const QTri* tris = reinterpret_cast<const QTri*>(__shfl_sync(0xffffffffu, (unsigned long long)lane_tris, src));
        const bool nx = st.idx < 0.0f, ny = st.idy < 0.0f, nz = st.idz < 0.0f;
        int node = group == 0 ? 0 : kNodeNone;  // this lane's entry; the first step takes the root
        int sp = 0;
        while (true) {
            // inner nodes: child c of the node
            bool hit = false;
            int child = 0, key = 0x7fffffff;
            if (node >= 0) {
                if (COUNT && c == 0) ++n_nodes;
                const char* qb = reinterpret_cast<const char*>(nodes + node);
                const float4 r0 = ld_hint(qb, pol_tree);
                const int4 r1 = ld_hint_i(qb + 16, pol_tree), r2 = ld_hint_i(qb + 32, pol_tree);
                child = __ldg(reinterpret_cast<const int*>(qb + 48) + c);
                const float Ax = r0.w * st.idx, Ay = __int_as_float(r1.x) * st.idy, Az = __int_as_float(r1.y) * st.idz;
                const float Bx = fmaf(r0.x, st.idx, -st.oix), By = fmaf(r0.y, st.idy, -st.oiy), Bz = fmaf(r0.z, st.idz, -st.oiz);
                const uint32_t sel = 0x7044u | (c << 8);
                const auto plane = [&](int w) { return __uint_as_float(__byte_perm((uint32_t)w, 0x40000000u, sel)); };
                const float lx = fmaf(plane(r1.z), Ax, Bx), ly = fmaf(plane(r1.w), Ay, By), lz = fmaf(plane(r2.x), Az, Bz);
                const float hx = fmaf(plane(r2.y), Ax, Bx), hy = fmaf(plane(r2.z), Ay, By), hz = fmaf(plane(r2.w), Az, Bz);
                const float tn = max3f(nx ? hx : lx, ny ? hy : ly, fmaxf(nz ? hz : lz, st.tmin));
                const float tf = min3f(nx ? lx : hx, ny ? ly : hy, fminf(nz ? lz : hz, st.tbest));
                hit = tn <= tf;
                if (hit) key = (__float_as_int(tn) & ~3) | (int)c;
            }
            // leaves: primitives c, c + 4 of the leaf
            float t_hit = INFINITY;
            int prim_hit = -1;
            if (node < kNodeDone) {
                const uint32_t count = ((uint32_t)node >> 27) & 15u, first = (uint32_t)node & 0x07ffffffu;
                for (uint32_t k = c; k < count; k += 4) {
                    if (COUNT) ++n_tris;
                    float t;
                    int prim;
                    if (test_prim(tris + first + k, st, pol_tree, t, prim) && t > st.tmin) {
                        if (ANY ? t < st.tmax : (t < st.tbest || (t == st.tbest && prim < st.best))) {
                            if (prim_hit < 0 || t < t_hit || (t == t_hit && prim < prim_hit)) {
                                t_hit = t;
                                prim_hit = prim;
                            }
                        }
                    }
                }
            }
            if (__any_sync(0xffffffffu, prim_hit >= 0)) {
                // the nearest (the lower index among equals) of the lanes' hits
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) {
                    const float t = __shfl_xor_sync(0xffffffffu, t_hit, o);
                    const int prim = __shfl_xor_sync(0xffffffffu, prim_hit, o);
                    if (prim >= 0 && (prim_hit < 0 || t < t_hit || (t == t_hit && prim < prim_hit))) {
                        t_hit = t;
                        prim_hit = prim;
                    }
                }
                st.tbest = t_hit;
                st.best = prim_hit;
                if (ANY) break;
            }
            // push the children hit, the nearest node's on top, within a node by distance
            const uint32_t hits = __ballot_sync(0xffffffffu, hit);
            if (hits) {
                const int k1 = __shfl_xor_sync(0xffffffffu, key, 1), k2 = __shfl_xor_sync(0xffffffffu, key, 2),
                          k3 = __shfl_xor_sync(0xffffffffu, key, 3);
                const uint32_t quad = (hits >> (lane & 28u)) & 15u;
                const uint32_t above = lane >= 28u ? 0u : hits >> ((lane & 28u) + 4u);
                const int rank = (k1 < key) + (k2 < key) + (k3 < key);
                const int at = sp + __popc(above) + __popc(quad) - 1 - rank;
                if (sp + __popc(hits) > kCap) {  // cannot happen: the steps below leave room
                    atomicOr(status_word, STATUS_STACK_OVERFLOW);
                    break;
                }
                if (hit) *slot(at) = make_uint2((uint32_t)child, (uint32_t)key);
                sp += __popc(hits);
            }
            if (sp == 0) break;
            __syncwarp();
            // the next entries: eight while that leaves room to finish them one at a time
            const int room = (kCap - kTraceStackTotal - sp) / 3;
            const int m = min(sp, max(1, min(8, room)));
            node = kNodeNone;
            if ((int)group < m) {
                const uint2 e = *slot(sp - 1 - (int)group);
                if (ANY || __uint_as_float(e.y & ~3u) <= fmaxf(st.tbest, 0.0f)) node = (int)e.x;
            }
            sp -= m;
            __syncwarp();
        }
        __syncwarp();
        if ((int)lane == src) {
            out.tbest = st.tbest;
            out.best = st.best;
        }
    }
    return out;
}

// Rays a warp takes at once, of n spread over `warps` warps: whole 32s up to 256 where there are
// enough rays to fill the lanes, else an even share.
__host__ __device__ __forceinline__ uint32_t trace_batch(uint32_t n, uint32_t warps) {
    const uint32_t per = warps ? (n + warps - 1) / warps : n;
    if (per <= 32u) return per ? per : 1u;
    const uint32_t b = (per + 31u) & ~31u;
    return b > 256u ? 256u : b;
}

// Warps that share n rays, of `resident` that fit the GPU: too few rays to fill them all go to
// kSpreadWarps warps per SM, however few lanes that fills: such a launch takes as long as its slowest
// warp, and a warp with fewer rays has fewer turns (5,000 rays on 328k triangles: 80 us with full
// warps, 29 us at 16 warps per SM, 23 us at 32; 20,000: 90, 46, 39 us).
constexpr uint32_t kSpreadWarps = 32;
inline uint32_t trace_warps(uint32_t n, uint32_t resident, uint32_t sms) {
    const uint32_t full = (n + 31u) / 32u, spread = n < sms * kSpreadWarps ? n : sms * kSpreadWarps;
    const uint32_t w = full > spread ? full : spread;
    return w < 1u ? 1u : w > resident ? resident : w;
}

// REFILL: idle lanes that trigger a refill; LEAF_AT: lanes waiting at a leaf that start the leaf
// phase (see below); MINB: resident blocks the register allocation must allow
template <bool ANY, int S, int BLOCK, bool COUNT, int REFILL = 8, int LEAF_AT = 8, int MINB = 1024 / BLOCK>
__global__ void __launch_bounds__(BLOCK, MINB) trace_kernel(const QNode* __restrict__ nodes, const QTri* __restrict__ tris,
                                                      const liar_ray* __restrict__ rays, liar_hit* __restrict__ hits,
                                                      uint32_t n_rays, uint32_t* __restrict__ work_counter,
                                                      uint32_t* __restrict__ status_word,
                                                      TraceCounters* __restrict__ counters, uint32_t BATCH,
                                                      const uint32_t* __restrict__ n_dev, uint32_t* __restrict__ zero_word) {
    // BATCH: ray indices a warp takes at once (trace_batch: n spread over all resident warps, at most
    // 256, so that a small wave still keeps every warp busy).
    // zero_word: a word that this launch clears (the size of the queue that the next kernel fills), null
    // for none
    if (zero_word && blockIdx.x == 0 && threadIdx.x == 0) *zero_word = 0u;
    // n_dev: the ray count in device memory, at most n_rays (a queue whose size the host does not
    // wait for); the launch was sized for n_rays
    if (n_dev) {
        n_rays = min(*n_dev, n_rays);
        BATCH = trace_batch(n_rays, gridDim.x * (BLOCK / 32));
    }
    extern __shared__ uint2 trace_smem[];  // S * BLOCK stack entries
    LaneStack<S, BLOCK> stack;
    stack.s_ent = trace_smem + threadIdx.x;
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t lt_mask = (1u << lane) - 1u;
    const uint64_t pol_tree = policy_evict_last();
    const uint64_t pol_stream = policy_evict_first();
    uint32_t status = 0, n_nodes = 0, n_tris = 0;

    // the warp's current batch [w_next, w_end), uniform; the first is its own, the counter hands out
    // those after
    const uint32_t n_warps = gridDim.x * (BLOCK / 32), first = (blockIdx.x * (BLOCK / 32) + (threadIdx.x >> 5)) * BATCH;
    uint32_t w_next = min(first, n_rays), w_end = min(first + BATCH, n_rays);
    const bool more = (uint64_t)n_warps * BATCH < n_rays;  // rays are left for the counter to hand out
    const bool all_coop = !more && BATCH <= kCoopBatch;
    uint32_t waited = 0;
    bool exhausted = false;          // uniform: the warp has its last rays
    int rid = -1;                    // this lane's ray, -1 for none
    RayState st;
    st.node = kNodeDone;

    while (true) {
        const uint32_t idle = __ballot_sync(0xffffffffu, st.node == kNodeDone);
        if (exhausted) {
            const uint32_t left = __popc(~idle);
            if (left == 0u || all_coop || (left <= kCoopRays && ++waited > kCoopTurns)) break;
        } else if ((uint32_t)__popc(idle) >= (uint32_t)REFILL) {
            if (w_next >= w_end) {
                uint32_t b = n_rays;
                if (more) {
                    if (lane == 0) b = atomicAdd(work_counter, BATCH);
                    b = __shfl_sync(0xffffffffu, b, 0) + n_warps * BATCH;
                }
                if (b >= n_rays) {
                    exhausted = true;
                } else {
                    w_next = b;
                    w_end = min(b + BATCH, n_rays);
                }
            }
            if (!exhausted) {
                const uint32_t avail = w_end - w_next;
                const uint32_t rank = __popc(idle & lt_mask);
                if (st.node == kNodeDone && rank < avail) {
                    // hits are stored here, by all idle lanes at once, rather than as each ray ends
                    if (rid >= 0) store_hit<ANY>(st, hits + rid, pol_stream);
                    rid = (int)(w_next + rank);
                    const float4* rp = reinterpret_cast<const float4*>(rays + rid);
                    const float4 r0 = ld_hint(rp, pol_stream), r1 = ld_hint(rp + 1, pol_stream);
                    start_ray<ANY>(r0, r1, st);
                }
                w_next += min(avail, (uint32_t)__popc(idle));
                if (!more && w_next >= w_end) {
                    exhausted = true;
                    continue;
                }
            }
        }
        trace_turn<ANY, S, BLOCK, COUNT, LEAF_AT>(nodes, tris, st, stack, pol_tree, status, n_nodes, n_tris);
    }
    if (__any_sync(0xffffffffu, st.node != kNodeDone)) {
        const CoopResult r = trace_coop<ANY, S, BLOCK, COUNT>(nodes, tris, rays, st.node != kNodeDone ? rid : -1, st.best, st.tbest,
                                                          trace_smem + (threadIdx.x & ~31u), status_word);
        st.best = r.best;
        st.tbest = r.tbest;
        n_nodes += r.n_nodes;
        n_tris += r.n_tris;
    }
    if (rid >= 0) store_hit<ANY>(st, hits + rid, pol_stream);
    if (status) atomicOr(status_word, status);
    if (COUNT) {
        unsigned long long a = n_nodes, b = n_tris;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            a += __shfl_down_sync(0xffffffffu, a, o);
            b += __shfl_down_sync(0xffffffffu, b, o);
        }
        if (lane == 0) {
            atomicAdd(&counters->nodes, a);
            atomicAdd(&counters->tris, b);
        }
    }
}

// ---- many trees in one launch (batched rendering): each ray names its scene, whose tree comes
// from a table; the ray count is read from device memory, so the launch can sit in a CUDA graph
// whose queue sizes are only known on the device
struct TreeRoot {
    const QNode* nodes;
    const QTri* tris;
};

template <int S, int BLOCK>
__global__ void __launch_bounds__(BLOCK, 1024 / BLOCK) trace_multi_kernel(const TreeRoot* __restrict__ roots,
                                                            const liar_ray* __restrict__ rays,
                                                            const uint32_t* __restrict__ ray_scene,
                                                            liar_hit* __restrict__ hits, const uint32_t* __restrict__ n_dev,
                                                            uint32_t* __restrict__ work_counter,
                                                            uint32_t* __restrict__ status_word) {
    constexpr int REFILL = 8, LEAF_AT = 8;  // as trace_kernel
    extern __shared__ uint2 trace_smem[];
    LaneStack<S, BLOCK> stack;
    stack.s_ent = trace_smem + threadIdx.x;
    const uint32_t n_rays = *n_dev;
    const uint32_t BATCH = trace_batch(n_rays, gridDim.x * (BLOCK / 32));
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t lt_mask = (1u << lane) - 1u;
    const uint64_t pol_tree = policy_evict_last();
    const uint64_t pol_stream = policy_evict_first();
    uint32_t status = 0, n_nodes = 0, n_tris = 0;
    const uint32_t n_warps = gridDim.x * (BLOCK / 32), first = (blockIdx.x * (BLOCK / 32) + (threadIdx.x >> 5)) * BATCH;
    uint32_t w_next = min(first, n_rays), w_end = min(first + BATCH, n_rays);
    const bool more = (uint64_t)n_warps * BATCH < n_rays;
    const bool all_coop = !more && BATCH <= kCoopBatch;
    uint32_t waited = 0;
    bool exhausted = false;
    int rid = -1;
    RayState st;
    st.node = kNodeDone;
    const QNode* nodes = nullptr;
    const QTri* tris = nullptr;
    while (true) {
        const uint32_t idle = __ballot_sync(0xffffffffu, st.node == kNodeDone);
        if (exhausted) {
            const uint32_t left = __popc(~idle);
            if (left == 0u || all_coop || (left <= kCoopRays && ++waited > kCoopTurns)) break;
        } else if ((uint32_t)__popc(idle) >= (uint32_t)REFILL) {
            if (w_next >= w_end) {
                uint32_t b = n_rays;
                if (more) {
                    if (lane == 0) b = atomicAdd(work_counter, BATCH);
                    b = __shfl_sync(0xffffffffu, b, 0) + n_warps * BATCH;
                }
                if (b >= n_rays) {
                    exhausted = true;
                } else {
                    w_next = b;
                    w_end = min(b + BATCH, n_rays);
                }
            }
            if (!exhausted) {
                const uint32_t avail = w_end - w_next;
                const uint32_t rank = __popc(idle & lt_mask);
                if (st.node == kNodeDone && rank < avail) {
                    if (rid >= 0) store_hit<false>(st, hits + rid, pol_stream);
                    rid = (int)(w_next + rank);
                    const TreeRoot root = roots[ray_scene[rid]];
                    nodes = root.nodes;
                    tris = root.tris;
                    const float4* rp = reinterpret_cast<const float4*>(rays + rid);
                    const float4 r0 = ld_hint(rp, pol_stream), r1 = ld_hint(rp + 1, pol_stream);
                    start_ray<false>(r0, r1, st);
                }
                w_next += min(avail, (uint32_t)__popc(idle));
                if (!more && w_next >= w_end) {
                    exhausted = true;
                    continue;
                }
            }
        }
        trace_turn<false, S, BLOCK, false, LEAF_AT>(nodes, tris, st, stack, pol_tree, status, n_nodes, n_tris);
    }
    if (__any_sync(0xffffffffu, st.node != kNodeDone)) {
        const CoopResult r = trace_coop<false, S, BLOCK, false>(nodes, tris, rays, st.node != kNodeDone ? rid : -1, st.best, st.tbest,
                                                          trace_smem + (threadIdx.x & ~31u), status_word);
        st.best = r.best;
        st.tbest = r.tbest;
        n_nodes += r.n_nodes;
        n_tris += r.n_tris;
    }
    if (rid >= 0) store_hit<false>(st, hits + rid, pol_stream);
    if (status) atomicOr(status_word, status);
}

}  // namespace liar_gpu
