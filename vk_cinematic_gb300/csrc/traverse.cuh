// Closest-hit traversal of the two-level scene (device code).
//
// Semantics follow sp_RayIntersectScene / sp_RayIntersectMesh
// (src/sp_scene.cpp:127-339):
//   * an object is a candidate iff its world AABB passes the reference's
//     slab test (src/simd.h:198-271) for the world ray;
//   * the ray enters object space through the inverse model matrix and its
//     direction is re-normalised there (src/sp_scene.cpp:274-276);
//   * a triangle is a candidate iff its own AABB passes the slab test in
//     object space (the reference collects exactly those BVH leaves,
//     src/bvh.cpp:203-311) and the Moller-Trumbore test hits with t > 0;
//   * per object the smallest object-space t wins, its hit point goes back
//     to world space and t = dot(worldHit - o, d) (src/sp_scene.cpp:302-308);
//     the smallest world t over objects wins.
// Node boxes here are exact unions of the reference's leaf boxes, and the
// slab test is monotone in the box, so interior tests never drop a leaf the
// reference would test.  Unlike the reference, the walk is ordered and
// prunes boxes that start beyond the best hit so far; pruning keeps a
// relative margin of 2^-10 so that a triangle whose rounded t lands just
// under its box's rounded entry distance is still tested.  Exact t ties go
// to the lower triangle (or object) index instead of the reference's
// BVH-order-dependent first find.
#pragma once

#include "gbsp_common.cuh"

namespace gbsp {

constexpr int kStackSize = 96;

// One traversal stack entry: a node or leaf reference and its entry
// distance, kept together so that a push or a pop is one 8-byte access.
struct __align__(8) StackEntry {
    uint32_t ref;
    float t;
};
constexpr float kInf = __builtin_huge_valf();

struct RayHit {
    float t;       // world t, +inf = miss
    float u, v;    // barycentrics of the winning triangle
    int32_t prim;  // leaf-order triangle index in the pool, -1 = miss
    int32_t inst;  // instance index (object-BVH leaf order), -1 = miss
};

struct TraceCounters {
    uint32_t topNodes, meshNodes, boxTests, triTests, meshTests;
};

// The rows of an instance's transform: three 128-bit loads (an instance is
// 16-byte aligned) instead of twelve scalar ones, each its own L1 lookup per
// lane.  1080p benchmark frame 77.1 -> 76.3 ms.
__device__ __forceinline__ Affine load_affine(const Affine *a)
{
    const float4 *p = reinterpret_cast<const float4 *>(a);
    const float4 x = __ldg(p), y = __ldg(p + 1), z = __ldg(p + 2);
    return Affine{{x.x, x.y, x.z, x.w, y.x, y.y, y.z, y.w, z.x, z.y, z.z, z.w}};
}

__device__ __forceinline__ float prune_bound(float t) { return t + t * 0.0009765625f; }

// Tests the children of a node (4 per quad, `quads` = 1 or 2) against the
// ray, pushing hits nearest-last.  kWT: the watertight mode's robust slab
// test.  With kKeepNearest the nearest hit child is not pushed but returned
// (ref kEmptyChild when no child is hit), for the caller to visit straight
// away: one stack store and load fewer per node visit.  Without it the
// return value is an empty entry.
// kFastSlab: slab_entry_node instead of the reference's slab_entry (see
// visit_node for when that is allowed).
template <bool kCount, bool kWT, bool kKeepNearest, bool kFastSlab>
__device__ __forceinline__ StackEntry visit_node_impl(const float4 *__restrict__ pool,
    uint32_t quads, uint32_t ref, V3 o, V3 invd, float bound, StackEntry *stack, int &sp,
    uint32_t *status, TraceCounters &cnt)
{
    const float4 *p = pool + node_offset(ref, quads);
    // a node pushes at most 4 * quads entries: one room check per visit instead
    // of one per push (a walk out of room reports the overflow and skips the node)
    if (sp > kStackSize - 4 * (int)kMaxNodeQuads) {
        atomicOr(status, kStatusStackOverflow);
        return StackEntry{kEmptyChild, 0.0f};
    }
    uint32_t nearRef = kEmptyChild;
    float nearT = kInf;
#pragma unroll
    for (int half = 0; half < (int)kMaxNodeQuads; half++) {
        if (half >= (int)quads) break;
        float4 lx = __ldg(p + 0 * quads + half), hx = __ldg(p + 1 * quads + half);
        float4 ly = __ldg(p + 2 * quads + half), hy = __ldg(p + 3 * quads + half);
        float4 lz = __ldg(p + 4 * quads + half), hz = __ldg(p + 5 * quads + half);
        uint4 ch = __ldg(reinterpret_cast<const uint4 *>(p + 6 * quads + half));
        float lxs[4] = {lx.x, lx.y, lx.z, lx.w}, hxs[4] = {hx.x, hx.y, hx.z, hx.w};
        float lys[4] = {ly.x, ly.y, ly.z, ly.w}, hys[4] = {hy.x, hy.y, hy.z, hy.w};
        float lzs[4] = {lz.x, lz.y, lz.z, lz.w}, hzs[4] = {hz.x, hz.y, hz.z, hz.w};
        uint32_t chs[4] = {ch.x, ch.y, ch.z, ch.w};
#pragma unroll
        for (int k = 0; k < 4; k++) {
            uint32_t c = chs[k];
            if (c == kEmptyChild) continue;
            if (kCount) cnt.boxTests++;
            V3 bl = v3(lxs[k], lys[k], lzs[k]), bh = v3(hxs[k], hys[k], hzs[k]);
            float te = kWT ? slab_entry_robust(bl, bh, o, invd)
                           : (kFastSlab ? slab_entry_node(bl, bh, o, invd)
                                        : slab_entry(bl, bh, o, invd));
            if (te < 0.0f || te > bound) continue;
            if (te < nearT) {
                if (nearRef != kEmptyChild) {
                    stack[sp] = StackEntry{nearRef, nearT};
                    sp++;
                }
                nearRef = c;
                nearT = te;
            } else {
                stack[sp] = StackEntry{c, te};
                sp++;
            }
        }
    }
    if constexpr (kKeepNearest) {
        return StackEntry{nearRef, nearT};
    } else {
        if (nearRef != kEmptyChild) {
            stack[sp] = StackEntry{nearRef, nearT};
            sp++;
        }
        return StackEntry{kEmptyChild, 0.0f};
    }
}

// ---- 8-wide nodes: one 256-bit load per box component -----------------------------
struct Floats8 {
    unsigned long long p[4];  // packed pairs of floats
};

__device__ __forceinline__ Floats8 load8(const void *a)
{
    Floats8 r;
    asm("ld.global.nc.v4.b64 {%0, %1, %2, %3}, [%4];"
        : "=l"(r.p[0]), "=l"(r.p[1]), "=l"(r.p[2]), "=l"(r.p[3])
        : "l"(a));
    return r;
}

__device__ __forceinline__ unsigned long long pack2(float a, float b)
{
    unsigned long long r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}

__device__ __forceinline__ void unpack2(unsigned long long v, float &a, float &b)
{
    asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v));
}

// (a + b) * c on two floats, each operation rounded once as in the scalar form
__device__ __forceinline__ unsigned long long add_mul2(unsigned long long a, unsigned long long b,
    unsigned long long c)
{
    unsigned long long r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(r), "l"(c));
    return r;
}

__device__ __forceinline__ float max3(float a, float b, float c)
{
    float r;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
    return r;
}

__device__ __forceinline__ float min3(float a, float b, float c)
{
    float r;
    asm("min.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
    return r;
}

// Tests the children of an 8-wide node against a ray whose inverse direction
// is finite, pushes the hit ones but the nearest and returns that one
// (kEmptyChild when none is hit); boxes += the children tested.
//
// Bound: issue slots and the L1's one-line-per-cycle lookups (each lane reads
// its own node).  A component of all eight children is one aligned 32-byte
// sector, read with one 256-bit load: 7 loads instead of 14.  The sign of the
// direction picks each axis' near and far plane, so no per-axis min / max is
// left: with lo <= hi, (lo - o) * invd <= (hi - o) * invd for invd > 0 also
// after rounding (subtraction and multiplication round monotonically), and
// the other way round for invd < 0.  Two children share one f32x2 operation,
// each half rounded like the scalar one: entry distances and decisions are
// those of slab_entry_node, also for an origin that is NaN in some or all
// components, and those of slab_entry_robust unless o.z is NaN.  1080p benchmark frame: 85.3 -> 79.1 ms, 2^20
// rays against 2^18 triangles 2,366 -> 1,905 us (both at 6 blocks per SM).
template <bool kWT>
__device__ __forceinline__ uint32_t visit_node8(const float4 *__restrict__ pool, uint32_t ref,
    V3 o, V3 invd, float bound, StackEntry *stack, int &sp, uint32_t *status, uint32_t &boxes)
{
    if (sp > kStackSize - 4 * (int)kMaxNodeQuads) {
        atomicOr(status, kStatusStackOverflow);
        return kEmptyChild;
    }
    const char *n = reinterpret_cast<const char *>(pool) + (size_t)ref * sizeof(Node8);
    const uint32_t sx = invd.x < 0.0f ? 32u : 0u, sy = invd.y < 0.0f ? 32u : 0u,
                   sz = invd.z < 0.0f ? 32u : 0u;
    const Floats8 nx = load8(n + sx), fx = load8(n + (32u - sx));
    const Floats8 ny = load8(n + 64 + sy), fy = load8(n + 64 + (32u - sy));
    const Floats8 nz = load8(n + 128 + sz), fz = load8(n + 128 + (32u - sz));
    const Floats8 ch = load8(n + 192);
    const unsigned long long ox = pack2(-o.x, -o.x), oy = pack2(-o.y, -o.y), oz = pack2(-o.z, -o.z);
    const unsigned long long ix = pack2(invd.x, invd.x), iy = pack2(invd.y, invd.y),
                             iz = pack2(invd.z, invd.z);
    uint32_t nearRef = kEmptyChild;
    float nearT = kInf;
#pragma unroll
    for (int k = 0; k < 4; k++) {
        float a[2], b[2], c[2], d[2], e[2], f[2];
        unpack2(add_mul2(nx.p[k], ox, ix), a[0], a[1]);
        unpack2(add_mul2(fx.p[k], ox, ix), b[0], b[1]);
        unpack2(add_mul2(ny.p[k], oy, iy), c[0], c[1]);
        unpack2(add_mul2(fy.p[k], oy, iy), d[0], d[1]);
        unpack2(add_mul2(nz.p[k], oz, iz), e[0], e[1]);
        unpack2(add_mul2(fz.p[k], oz, iz), f[0], f[1]);
        const uint32_t cc[2] = {(uint32_t)ch.p[k], (uint32_t)(ch.p[k] >> 32)};
#pragma unroll
        for (int j = 0; j < 2; j++) {
            const float tn = fmaxf(max3(a[j], c[j], e[j]), 0.0f);
            float tf = min3(b[j], d[j], f[j]);
            if (kWT) tf = tf * 1.0000004f;
            const bool present = cc[j] != kEmptyChild;
            boxes += present ? 1u : 0u;
            // tf is NaN (a miss) when the origin is NaN in every component; fminf(tf,
            // bound) would drop it and take every box.  In time the same as fminf was;
            // min.NaN cost frames and rays 2% and a batch 4%, `&& tn <= bound` rays 3%
            const bool hit = present && tn <= tf && !(tn > bound);
            const bool closer = tn < nearT;
            const StackEntry push{closer ? nearRef : cc[j], closer ? nearT : tn};
            if (hit && push.ref != kEmptyChild) {
                stack[sp] = push;
                sp++;
            }
            if (hit && closer) {
                nearRef = cc[j];
                nearT = tn;
            }
        }
    }
    return nearRef;
}

// The same for any ray (a zero direction component makes an infinite inverse,
// for which the reference's slab form has its own NaN rules), one child after
// another: the rare path of the 8-wide walks, kept small.
template <bool kWT>
__device__ __forceinline__ uint32_t visit_node8_any(const float4 *__restrict__ pool, uint32_t ref,
    V3 o, V3 invd, float bound, StackEntry *stack, int &sp, uint32_t *status, uint32_t &boxes)
{
    if (sp > kStackSize - 4 * (int)kMaxNodeQuads) {
        atomicOr(status, kStatusStackOverflow);
        return kEmptyChild;
    }
    const float *n = reinterpret_cast<const float *>(pool + node_offset(ref, 2));
    uint32_t nearRef = kEmptyChild;
    float nearT = kInf;
#pragma unroll 1
    for (int k = 0; k < 8; k++) {
        const uint32_t c = __float_as_uint(__ldg(n + 48 + k));
        if (c == kEmptyChild) continue;
        boxes++;
        const V3 bl = v3(__ldg(n + k), __ldg(n + 16 + k), __ldg(n + 32 + k));
        const V3 bh = v3(__ldg(n + 8 + k), __ldg(n + 24 + k), __ldg(n + 40 + k));
        const float te = kWT ? slab_entry_robust(bl, bh, o, invd) : slab_entry(bl, bh, o, invd);
        if (te < 0.0f || te > bound) continue;
        const bool closer = te < nearT;
        const StackEntry push{closer ? nearRef : c, closer ? nearT : te};
        if (push.ref != kEmptyChild) {
            stack[sp] = push;
            sp++;
        }
        if (closer) {
            nearRef = c;
            nearT = te;
        }
    }
    return nearRef;
}

// Interior nodes take the min/max-instruction slab test when every component
// of the inverse direction is finite: then no NaN can arise and it decides
// exactly as the reference's form.  A ray with a zero direction component (an
// infinite inverse, where (lo - o) * invd can be NaN and the reference's form
// has its own NaN rules) keeps the reference's form, whose decisions below a
// node are a superset of its leaves'.
template <bool kCount, bool kWT = false, bool kKeepNearest = false>
__device__ __forceinline__ StackEntry visit_node(const float4 *__restrict__ pool, uint32_t quads,
    uint32_t ref, V3 o, V3 invd, float bound, StackEntry *stack, int &sp, uint32_t *status,
    TraceCounters &cnt)
{
    if (kWT || !(isfinite(invd.x) && isfinite(invd.y) && isfinite(invd.z)))
        return visit_node_impl<kCount, kWT, kKeepNearest, false>(pool, quads, ref, o, invd, bound,
            stack, sp, status, cnt);
    return visit_node_impl<kCount, kWT, kKeepNearest, true>(pool, quads, ref, o, invd, bound,
        stack, sp, status, cnt);
}

// The walks' node visit: pushes the hit children but the nearest and returns
// that one.  kQ = 2: every node is 8-wide; 0: `quads` says.
template <bool kWT, int kQ>
__device__ __forceinline__ uint32_t visit_nearest(const float4 *__restrict__ pool, uint32_t quads,
    uint32_t ref, V3 o, V3 invd, float bound, StackEntry *stack, int &sp, uint32_t *status,
    uint32_t &boxes)
{
    if constexpr (kQ == 2) {
        // slab_entry_robust misses every box from an origin with a NaN in z and has no
        // constraint from one in x or y, as the instructions of visit_node8 have for all three
        if (isfinite(invd.x) && isfinite(invd.y) && isfinite(invd.z) && (!kWT || o.z == o.z))
            return visit_node8<kWT>(pool, ref, o, invd, bound, stack, sp, status, boxes);
        return visit_node8_any<kWT>(pool, ref, o, invd, bound, stack, sp, status, boxes);
    } else {
        TraceCounters cnt = {0, 0, 0, 0, 0};
        const uint32_t r = visit_node<true, kWT, true>(pool, quads, ref, o, invd, bound, stack, sp,
            status, cnt).ref;
        boxes += cnt.boxTests;
        return r;
    }
}

// Triangle candidates of one mesh leaf, in object space.  kWT: the
// watertight test on every candidate (no box gate: a rounded box test could
// reject an edge ray); otherwise the reference's gate and MT test.  A closer
// hit updates bestT and bestPrim and hands its barycentrics to keepUV(u, v).
template <bool kCount, bool kWT, class KeepUV>
__device__ __forceinline__ void visit_leaf_uv(const SceneView &sv, uint32_t ref, V3 lo, V3 ld,
    V3 linvd, float &bestT, int32_t &bestPrim, KeepUV keepUV, TraceCounters &cnt)
{
    uint32_t first = leaf_first(ref), count = leaf_count(ref);
    for (uint32_t k = 0; k < count; k++) {
        uint32_t j = first + k;
        const float4 *tp = reinterpret_cast<const float4 *>(sv.tris + j);
        float4 A = __ldg(tp + 0), B = __ldg(tp + 1), C = __ldg(tp + 2);
        V3 a = v3(A.x, A.y, A.z), b = v3(B.x, B.y, B.z), c = v3(C.x, C.y, C.z);
        if (kCount) cnt.triTests++;
        TriHit h;
        if constexpr (kWT) {
            h = ray_triangle_watertight(lo, ld, a, b, c, v3(A.w, B.w, C.w));
        } else {
            // the three conditions of a hit, cheapest first (each is a pure
            // predicate, so the order changes no result): the face culling of
            // RayIntersectTriangleMT (src/ray_intersection.cpp:181-182), the
            // triangle's own box (the reference only reaches triangles whose
            // box passes), then the test itself
            if (!(dot(ld, v3(A.w, B.w, C.w)) < 0.0f)) continue;
            V3 bl = vmin(a, vmin(b, c)), bh = vmax(a, vmax(b, c));
            if (slab_entry(bl, bh, lo, linvd) < 0.0f) continue;
            h = ray_triangle_mt(lo, ld, a, b, c, v3(A.w, B.w, C.w));
        }
        if (!h.hit || !(h.t > 0.0f)) continue;
        bool take = h.t < bestT;
        if (!take && h.t == bestT && bestPrim >= 0)
            take = __ldg(sv.triIds + j) < __ldg(sv.triIds + bestPrim);
        if (take) {
            bestT = h.t;
            keepUV(h.u, h.v);
            bestPrim = (int32_t)j;
        }
    }
}

template <bool kCount, bool kWT = false>
__device__ __forceinline__ void visit_leaf(const SceneView &sv, uint32_t ref, V3 lo, V3 ld,
    V3 linvd, float &bestT, float &bestU, float &bestV, int32_t &bestPrim, TraceCounters &cnt)
{
    visit_leaf_uv<kCount, kWT>(sv, ref, lo, ld, linvd, bestT, bestPrim,
        [&](float u, float v) {
            bestU = u;
            bestV = v;
        },
        cnt);
}

template <bool kCount, bool kWT = false, int kQ = 0>
__device__ RayHit trace_closest(const SceneView &sv, V3 o, V3 d, uint32_t *status,
    TraceCounters &cnt)
{
    RayHit best;
    best.t = kInf;
    best.u = best.v = 0.0f;
    best.prim = -1;
    best.inst = -1;
    if (sv.tlasRoot == kEmptyChild) return best;
    StackEntry stack[kStackSize];
    // State used only when entering or leaving an object, kept in memory
    // (local, L1-resident) on purpose so that the walks hold just the current
    // level's ray, bounds and stack in registers.  Words: world origin 0-2,
    // direction 3-5, inverse direction 6-8; best hit over objects u 9, v 10,
    // triangle 11, object 12; the object's best triangle's u 13, v 14.
    volatile uint32_t cold[15];
    const auto put3 = [&](int w, V3 v) {
        cold[w] = __float_as_uint(v.x);
        cold[w + 1] = __float_as_uint(v.y);
        cold[w + 2] = __float_as_uint(v.z);
    };
    const auto get3 = [&](int w) {
        return v3(__uint_as_float(cold[w]), __uint_as_float(cold[w + 1]),
            __uint_as_float(cold[w + 2]));
    };
    int sp = 0;
    V3 invd = inverse(d);
    put3(0, o);
    put3(3, d);
    put3(6, invd);
    cold[9] = 0u;
    cold[10] = 0u;
    cold[11] = 0xFFFFFFFFu;
    cold[12] = 0xFFFFFFFFu;
    // the node or leaf to visit next (the nearest child of the last node
    // visit), kept out of the stack; no hit is recorded between its test and
    // its visit, so its entry distance is still within the bound
    uint32_t next = sv.tlasRoot;
    const float4 *__restrict__ nodes = sv.nodes;
    const uint32_t quads = sv.nodeQuads;
    // trees are validated at build time (children after parents), so the
    // walk is finite; the guard only bounds it against corrupted memory
    for (int guard = 0; next != kEmptyChild || sp > 0; guard++) {
        if (guard >= (1 << 20)) {
            atomicOr(status, kStatusStackOverflow);
            break;
        }
        uint32_t ref = next;
        next = kEmptyChild;
        if (ref == kEmptyChild) {
            sp--;
            const StackEntry top = stack[sp];
            if (top.t > prune_bound(best.t)) continue;
            ref = top.ref;
        }
        if (!child_is_leaf(ref)) {
            if (kCount) cnt.topNodes++;
            next = visit_nearest<kWT, kQ>(nodes, quads, ref, o, invd, prune_bound(best.t), stack,
                sp, status, cnt.boxTests);
            continue;
        }
        // an object whose world box passed: descend into its mesh
        uint32_t inst = leaf_first(ref);
        const Instance &in = sv.instances[inst];
        const Affine inv = load_affine(&in.inv);
        const V3 lo = transform_point(inv, o);
        float len;
        const V3 ld = normalize(transform_vector(inv, get3(3)), &len);
        const V3 linvd = inverse(ld);
        if (kCount) cnt.meshTests++;
        float lBestT = kInf;
        int32_t lPrim = -1;
        float bound = prune_bound(best.t * len);
        const int base = sp;
        uint32_t lnext = __ldg(&in.blasRoot);
        for (int guard = 0; (lnext != kEmptyChild || sp > base) && guard < (1 << 22); guard++) {
            uint32_t r2 = lnext;
            lnext = kEmptyChild;
            if (r2 == kEmptyChild) {
                sp--;
                const StackEntry top = stack[sp];
                if (top.t > bound) continue;
                r2 = top.ref;
            }
            if (!child_is_leaf(r2)) {
                if (kCount) cnt.meshNodes++;
                lnext = visit_nearest<kWT, kQ>(nodes, quads, r2, lo, linvd, bound, stack, sp,
                    status, cnt.boxTests);
            } else {
                visit_leaf_uv<kCount, kWT>(sv, r2, lo, ld, linvd, lBestT, lPrim,
                    [&](float u, float v) {
                        cold[13] = __float_as_uint(u);
                        cold[14] = __float_as_uint(v);
                    },
                    cnt);
                bound = rmin(prune_bound(lBestT), bound);
            }
        }
        sp = base;
        // the world ray comes back from memory: it was not held through the mesh walk
        o = get3(0);
        invd = get3(6);
        if (lPrim < 0) continue;
        const Affine model = load_affine(&in.model);
        V3 localHit = add(lo, mul(ld, lBestT));
        V3 worldHit = transform_point(model, localHit);
        float tw = dot(sub(worldHit, o), get3(3));
        if (tw < best.t || (tw == best.t && (int32_t)inst < (int32_t)cold[12])) {
            best.t = tw;
            cold[9] = cold[13];
            cold[10] = cold[14];
            cold[11] = (uint32_t)lPrim;
            cold[12] = inst;
        }
    }
    best.u = __uint_as_float(cold[9]);
    best.v = __uint_as_float(cold[10]);
    best.prim = (int32_t)cold[11];
    best.inst = (int32_t)cold[12];
    return best;
}

// Texture coordinates of a hit (src/sp_scene.cpp:189-215).
__device__ __forceinline__ void hit_uv(const SceneView &sv, const RayHit &h, float &uvx, float &uvy)
{
    const float4 *ap = reinterpret_cast<const float4 *>(sv.attrs + h.prim);
    float4 a2 = __ldg(ap + 2), a3 = __ldg(ap + 3);
    float w = 1.0f - h.u - h.v;
    // uv0 = (a2.y, a2.z), uv1 = (a2.w, a3.x), uv2 = (a3.y, a3.z)
    uvx = a2.y * w + a2.w * h.u + a3.y * h.v;
    uvy = a2.z * w + a3.x * h.u + a3.z * h.v;
}

// World-space normal of a hit (src/sp_scene.cpp:189-215, 302-312): the face
// normal in the w lanes of the triangle record, or the interpolated vertex
// normals of a smooth mesh (only those read the attributes).
__device__ __forceinline__ V3 hit_normal(const SceneView &sv, const RayHit &h)
{
    const Instance &in = sv.instances[h.inst];
    V3 ln;
    if (__ldg(&in.smooth)) {
        const float4 *ap = reinterpret_cast<const float4 *>(sv.attrs + h.prim);
        float4 a0 = __ldg(ap + 0), a1 = __ldg(ap + 1);
        float a2x = __ldg(&ap[2].x);
        float w = 1.0f - h.u - h.v;
        V3 n0 = v3(a0.x, a0.y, a0.z), n1 = v3(a0.w, a1.x, a1.y), n2 = v3(a1.z, a1.w, a2x);
        ln = normalize(add(add(mul(n0, w), mul(n1, h.u)), mul(n2, h.v)));
    } else {
        const TriRecord *t = sv.tris + h.prim;
        ln = v3(__ldg(&t->a_nx.w), __ldg(&t->b_ny.w), __ldg(&t->c_nz.w));
    }
    return normalize(transform_vector(load_affine(&in.model), ln));
}

// World-space normal and uv of a hit.
__device__ __forceinline__ void hit_surface(const SceneView &sv, const RayHit &h, V3 &normal,
    float &uvx, float &uvy)
{
    normal = hit_normal(sv, h);
    hit_uv(sv, h, uvx, uvy);
}

}  // namespace gbsp
