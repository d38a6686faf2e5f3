// The reference's compute-shader path tracer (src/shaders/test_compute.comp.glsl)
// as a CUDA kernel.
//
// Semantics kept from the shader: one 16x16 (configurable) tile per work item,
// the tile's RNG seeded (tileIndex + 1) * 0xF51C0E49 and drawn in scanline
// order through the tile (2 jitter draws per pixel, 3 per hit), a brute-force
// closest hit over every entity's triangles in entity order (no BVH, no
// back-face culling, strict < so the first triangle wins ties), three bounces,
// hard-coded materials (0 red albedo, 2 checkerboard texture, 5 white light)
// and the normalize(N + rand3) bounce.
//
// GB300 layout: the tile's RNG chain makes its pixels sequential, so a whole
// block works on one tile and on one ray at a time.  Each mesh's triangles are
// grouped into clusters of 16 (cpt_clusters.h); per ray
//   1. warp 0 moves the ray into up to 32 entities' spaces, one lane each;
//   2. all warps test 32 clusters of one entity per step and list (each warp
//      for itself) the clusters whose triangles the float test could accept -
//      the rejected ones provably contain no accepted triangle, so the set of
//      hits is the brute-force loop's, rounding included;
//   3. half-warps run the shader's test on the listed clusters; an entity's
//      answer is the smallest t, lowest triangle index among equal t, kept by
//      an atomic minimum on (t, index) in shared memory;
//   4. warp 0 takes each entity's winner to world space, one lane each, and
//      reduces in entity order (strict <), then shades and makes the next ray.
// Texture coordinates are read only for the winner.
//
// Bound: the serial chain of a tile (two barriers, one pass over the clusters
// and warp 0's shading per ray, 5.5 us a ray with one tile on an SM; the
// longest tile has 768 rays).  A ray among 18 spheres of 1,280 triangles costs
// 1,440 cluster tests and the tests of about 55 listed clusters instead of
// 23,042 triangle tests.  512 x 384 pixels of that scene: 107.5 ms with a warp
// per tile and every triangle staged through shared memory, 5.6 to 5.8 ms now
// (three machines; 0.4 more before the cluster test's sums were fused multiply-adds
// and the winner a minimum reduction).  Before those two: 4 blocks of 8 warps per SM (64
// registers) 5.88 ms, unbounded (2 blocks) 7.4, 4 warps 6.6 and 2 warps per
// tile 9.8 ms.  Worse since: clusters of 8 or 32 triangles 6.4 and 7.7 ms, one
// list for all warps of a tile (a barrier more) 6.1, the next clusters loaded
// ahead (registers) 7.0, 5 blocks per SM 5.7.
//
// Built-ins are fixed to one IEEE definition shared with the oracle (dot in
// x, y, z order; normalize = v * (1 / sqrt(dot)); mat4 * vec4 summed over
// columns 0..3; GLSL max(x, y) = x < y ? y : x) and compiled without
// contraction.

#include <vector>

#include "cpt_clusters.h"
#include "gbsp_internal.h"

namespace gbsp {
namespace cpt {

constexpr float kF32Max = 3.402823466e+38f;
constexpr uint32_t kMaterialRed = 0, kMaterialCheckerBoard = 2, kMaterialWhiteLight = 5,
                   kMaterialBlack = 6;
constexpr int kMaxBounces = 3;
struct EntityDev {
    float model[16];
    float inv[16];
    uint32_t triBegin, triCount, material;
    uint32_t clusterBegin, clusterCount, pad[3];
};

struct Triangles {
    // cluster c: 9 components (a, e1, e2) of 16 triangles each, from 144 c;
    // NaN in the places no triangle fills
    const float *clustered;
    const uint32_t *index;    // the clusters' triangles, as indices in their mesh
    const Cluster *clusters;
    const float *plain;       // 9 floats per triangle, in mesh order
    const float2 *uv;         // 3 per triangle, in mesh order
};

struct View {
    V3 right, up, position, center;
    float halfWidth, halfHeight, halfPixelWidth, halfPixelHeight, invW, invH;
    uint32_t width, height, tileW, tileH, tileCountX;
};

struct Counters {
    unsigned long long *rays, *hits, *tests, *paths;
};

__device__ __forceinline__ V3 cnormalize(V3 v)
{
    float inv = 1.0f / sqrtf(cdot(v, v));
    return v3(v.x * inv, v.y * inv, v.z * inv);
}
__device__ __forceinline__ float glsl_max(float x, float y) { return x < y ? y : x; }

__device__ __forceinline__ V3 mat_mul(const float *m, V3 v, float w)
{
    V3 r;
    r.x = ((__ldg(m + 0) * v.x + __ldg(m + 4) * v.y) + __ldg(m + 8) * v.z) + __ldg(m + 12) * w;
    r.y = ((__ldg(m + 1) * v.x + __ldg(m + 5) * v.y) + __ldg(m + 9) * v.z) + __ldg(m + 13) * w;
    r.z = ((__ldg(m + 2) * v.x + __ldg(m + 6) * v.y) + __ldg(m + 10) * v.z) + __ldg(m + 14) * w;
    return r;
}

struct Rng {
    uint32_t s;
    __device__ __forceinline__ float bilateral()
    {
        uint32_t x = s;
        x ^= x << 13;
        x ^= x >> 17;
        x ^= x << 5;
        s = x;
        float u = __uint2float_rn(x) / 4294967296.0f;  // float(x) / float(U32_MAX)
        return -1.0f + 2.0f * u;
    }
};

__device__ __forceinline__ float wrap_coord(float u, uint32_t n, int32_t &i0, int32_t &i1)
{
    float x = u * (float)n - 0.5f;
    if (!(fabsf(x) < 1.0e9f)) {
        i0 = 0;
        i1 = n > 1 ? 1 : 0;
        return 0.0f;
    }
    float f = floorf(x);
    float a = x - f;
    // |f| < 1e9: 32-bit remainders (64-bit ones cost hundreds of instructions)
    int32_t m;
    if (n <= 0x7FFFFFFFu) {
        m = (int32_t)f % (int32_t)n;
        if (m < 0) m += (int32_t)n;
    } else {
        m = (int32_t)f;  // n is larger than any |f|
        if (m < 0) m = (int32_t)(uint32_t)((long long)m + (long long)n);
    }
    i0 = m;
    i1 = (uint32_t)m + 1u == n ? 0 : m + 1;
    return a;
}

// Vulkan linear filter at the base level with REPEAT addressing (the
// reference's defaultSampler, src/vulkan_renderer.cpp:986-1001).
__device__ V3 sample_bilinear(const float4 *tex, uint32_t w, uint32_t h, float u, float v)
{
    if (!tex || !w || !h) return v3(0.0f, 0.0f, 0.0f);
    int32_t x0, x1, y0, y1;
    float a = wrap_coord(u, w, x0, x1);
    float b = wrap_coord(v, h, y0, y1);
    float w00 = (1.0f - a) * (1.0f - b), w10 = a * (1.0f - b), w01 = (1.0f - a) * b, w11 = a * b;
    float4 t00 = __ldg(&tex[(size_t)y0 * w + x0]), t10 = __ldg(&tex[(size_t)y0 * w + x1]);
    float4 t01 = __ldg(&tex[(size_t)y1 * w + x0]), t11 = __ldg(&tex[(size_t)y1 * w + x1]);
    V3 r = v3(t00.x * w00, t00.y * w00, t00.z * w00);
    r = v3(r.x + t10.x * w10, r.y + t10.y * w10, r.z + t10.z * w10);
    r = v3(r.x + t01.x * w01, r.y + t01.y * w01, r.z + t01.z * w01);
    r = v3(r.x + t11.x * w11, r.y + t11.y * w11, r.z + t11.z * w11);
    return r;
}

struct SceneHit {
    float t;
    uint32_t material;
    V3 normal;
    float u, v;
};

struct PathVertex {
    uint32_t material;
    V3 incoming, normal;
    float u, v;
};

// Radiance of a finished path (test_compute.comp.glsl:441-481): lane i of the
// warp holds vertex i and evaluates its material, the reverse pass then takes
// them from the last to the first.
__device__ __forceinline__ V3 path_radiance_cpt(const PathVertex &vertex, int len, int lane,
    const float4 *__restrict__ tex, uint32_t texW, uint32_t texH)
{
    V3 emission = v3(0.0f, 0.0f, 0.0f), albedo = v3(0.0f, 0.0f, 0.0f);
    float cosine = 0.0f;
    if (lane < len) {
        const uint32_t m = vertex.material;
        if (m == kMaterialRed)
            albedo = v3(0.18f, 0.1f, 0.1f);
        else if (m == kMaterialCheckerBoard)
            albedo = sample_bilinear(tex, texW, texH, vertex.u, vertex.v);
        else if (m == kMaterialWhiteLight)
            emission = v3(1.0f, 1.0f, 1.0f);
        cosine = glsl_max(0.0f, cdot(vertex.normal, vertex.incoming));
    }
    V3 radiance = v3(0.0f, 0.0f, 0.0f);
#pragma unroll
    for (int i = kMaxBounces - 1; i >= 0; i--) {
        const V3 e = v3(__shfl_sync(0xFFFFFFFFu, emission.x, i), __shfl_sync(0xFFFFFFFFu, emission.y, i),
            __shfl_sync(0xFFFFFFFFu, emission.z, i));
        const V3 a = v3(__shfl_sync(0xFFFFFFFFu, albedo.x, i), __shfl_sync(0xFFFFFFFFu, albedo.y, i),
            __shfl_sync(0xFFFFFFFFu, albedo.z, i));
        const float c = __shfl_sync(0xFFFFFFFFu, cosine, i);
        if (i < len)
            radiance = v3(e.x + (a.x * radiance.x) * c, e.y + (a.y * radiance.y) * c,
                e.z + (a.z * radiance.z) * c);
    }
    return radiance;
}

constexpr int kEntChunk = 32;     // entities whose clusters a ray tests together: one lane of warp 0 each
constexpr int kListCap = 128;     // clusters a warp lists before it runs their triangles

template <int kWarps>
__global__ void __launch_bounds__(32 * kWarps, kWarps == 8 ? 4 : 1) k_compute_pt(const EntityDev *__restrict__ ents,
    uint32_t entityCount, uint64_t triangleTests, Triangles tri, const float4 *__restrict__ tex,
    uint32_t texW, uint32_t texH, View view, const uint32_t *__restrict__ tiles,
    float4 *__restrict__ image, Counters counters)
{
    __shared__ float sRay[kEntChunk][6];                // the ray in each entity's space
    __shared__ unsigned long long sBest[kEntChunk];     // (t bits, triangle) of its closest hit
    __shared__ uint32_t sUnits[kEntChunk + 1];          // units of 32 clusters before each entity
    __shared__ uint32_t sBegin[kEntChunk], sClusters[kEntChunk];
    __shared__ uint32_t sLists[kWarps][kListCap];       // each warp's listed clusters
    __shared__ uint8_t sEntities[kWarps][kListCap];     // and their entities
    __shared__ uint32_t sActive, sNone;                 // sNone: entities the ray cannot hit
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const uint32_t laneMaskLt = (1u << lane) - 1u;
    uint32_t *sList = sLists[warp];
    uint8_t *sEntity = sEntities[warp];
    const uint32_t tileIndex = __ldg(&tiles[blockIdx.x]);
    const uint32_t tx = tileIndex % view.tileCountX, ty = tileIndex / view.tileCountX;
    const uint32_t minX = tx * view.tileW, minY = ty * view.tileH;
    const uint32_t maxX = min(view.width, (tx + 1) * view.tileW);
    const uint32_t maxY = min(view.height, (ty + 1) * view.tileH);
    bool active = minX < maxX && minY < maxY;
    Rng rng{(tileIndex + 1u) * 0xF51C0E49u};
    uint64_t rays = 0, hits = 0, paths = 0;
    uint32_t x = minX, y = minY;
    int len = 0, bounce = 0;
    PathVertex vertex = {kMaterialBlack, v3(0.0f, 0.0f, 0.0f), v3(0.0f, 0.0f, 0.0f), 0.0f, 0.0f};  // lane i: vertex i
    V3 o = v3(0.0f, 0.0f, 0.0f), d = v3(0.0f, 0.0f, 0.0f);
    // camera ray of pixel (x, y): test_compute.comp.glsl:510-540
    auto start_pixel = [&]() {
        float px = (float)x + 0.5f, py = (float)y + 0.5f;
        float jx = view.halfPixelWidth * rng.bilateral();
        float jy = view.halfPixelHeight * rng.bilateral();
        px = px + jx;
        py = py + jy;
        float fx = px * view.invW, fy = py * view.invH;
        fy = 1.0f - fy;
        fx = fx * 2.0f - 1.0f;
        fy = fy * 2.0f - 1.0f;
        V3 filmP = view.center;
        float sx = view.halfWidth * fx, sy = view.halfHeight * fy;
        filmP = v3(filmP.x + view.right.x * sx, filmP.y + view.right.y * sx,
            filmP.z + view.right.z * sx);
        filmP = v3(filmP.x + view.up.x * sy, filmP.y + view.up.y * sy, filmP.z + view.up.z * sy);
        o = view.position;
        d = cnormalize(v3(filmP.x - o.x, filmP.y - o.y, filmP.z - o.z));
        len = 0;
        bounce = 0;
    };
    // the ray's state lives in warp 0 (every lane holds it)
    if (warp == 0 && active) start_pixel();
    const uint32_t chunks = (entityCount + kEntChunk - 1) / kEntChunk;
    for (uint32_t guard = 0; guard < (1u << 30); guard++) {
        // ---- trace: test_compute.comp.glsl:320-430
        SceneHit res;
        res.t = kF32Max;
        res.material = kMaterialBlack;
        res.normal = v3(0.0f, 0.0f, 0.0f);
        res.u = res.v = 0.0f;
        uint32_t chunk = 0;
        bool done = false;
        do {
            const uint32_t e = chunk * kEntChunk + lane;  // warp 0: the lane's entity
            const bool mine = warp == 0 && e < entityCount;
            V3 lo = v3(0.0f, 0.0f, 0.0f), ld = lo;
            if (warp == 0) {
                if (mine) {
                    lo = mat_mul(ents[e].inv, o, 1.0f);
                    ld = cnormalize(mat_mul(ents[e].inv, d, 0.0f));
                    sRay[lane][0] = lo.x;
                    sRay[lane][1] = lo.y;
                    sRay[lane][2] = lo.z;
                    sRay[lane][3] = ld.x;
                    sRay[lane][4] = ld.y;
                    sRay[lane][5] = ld.z;
                }
                if (guard == 0 || chunks > 1) {  // a single chunk's tables stay
                    const uint32_t clusters = mine ? __ldg(&ents[e].clusterCount) : 0u;
                    sBegin[lane] = mine ? __ldg(&ents[e].clusterBegin) : 0u;
                    sClusters[lane] = clusters;
                    uint32_t units = (clusters + 31) / 32;
                    for (int off = 1; off < 32; off <<= 1) {
                        uint32_t v = __shfl_up_sync(0xFFFFFFFFu, units, off);
                        if (lane >= off) units += v;
                    }
                    sUnits[lane + 1] = units;
                    if (lane == 0) sUnits[0] = 0;
                }
                sBest[lane] = ~0ull;
                // a ray with a NaN is never accepted: every numerator of the test
                // has it.  (A path that leaves the scene can go on as one: an
                // entity's miss at t = FLT_MAX may pass the world-space test and
                // has no normal.)
                const bool nan = !(lo.x + lo.y + lo.z == lo.x + lo.y + lo.z) ||
                    !(ld.x + ld.y + ld.z == ld.x + ld.y + ld.z);
                const uint32_t none = __ballot_sync(0xFFFFFFFFu, !mine || nan);
                if (lane == 0) {
                    sActive = active ? 1u : 0u;
                    sNone = none;
                }
            }
            __syncthreads();
            if (!sActive) {
                done = true;
                break;
            }
            const uint32_t none = sNone;
            const uint32_t before = sUnits[lane], total = none == 0xFFFFFFFFu ? 0u : sUnits[kEntChunk];
            uint32_t listed = 0;
            for (uint32_t u = warp; u < total; u += kWarps) {
                // the entity of unit u: the last one that starts at or before it
                const int el = __popc(__ballot_sync(0xFFFFFFFFu, before <= u)) - 1;
                const uint32_t c = 32u * (u - sUnits[el]) + lane;
                bool may = false;
                uint32_t cluster = 0;
                if (c < sClusters[el] && !(none >> el & 1u)) {
                    cluster = sBegin[el] + c;
                    const float4 *p = reinterpret_cast<const float4 *>(tri.clusters + cluster);
                    may = cluster_may_hit(__ldg(p), __ldg(p + 1), __ldg(p + 2),
                        v3(sRay[el][0], sRay[el][1], sRay[el][2]),
                        v3(sRay[el][3], sRay[el][4], sRay[el][5]));
                }
                const uint32_t m = __ballot_sync(0xFFFFFFFFu, may);
                if (may) {
                    const uint32_t at = listed + __popc(m & laneMaskLt);
                    sList[at] = cluster;
                    sEntity[at] = (uint8_t)el;
                }
                listed += __popc(m);
                if (u + kWarps < total && listed <= kListCap - 32) continue;
                // run the listed clusters' triangles, a half-warp each
                __syncwarp();
                for (uint32_t k = lane / kClusterTris; k < listed; k += 32 / kClusterTris) {
                    const uint32_t lc = sList[k], le = sEntity[k], j = lane % kClusterTris;
                    const float *p = tri.clustered + (size_t)lc * (9 * kClusterTris) + j;
                    const V3 a = v3(__ldg(p), __ldg(p + kClusterTris), __ldg(p + 2 * kClusterTris));
                    const V3 e1 = v3(__ldg(p + 3 * kClusterTris), __ldg(p + 4 * kClusterTris),
                        __ldg(p + 5 * kClusterTris));
                    const V3 e2 = v3(__ldg(p + 6 * kClusterTris), __ldg(p + 7 * kClusterTris),
                        __ldg(p + 8 * kClusterTris));
                    const MtHit h = mt_test(v3(sRay[le][0], sRay[le][1], sRay[le][2]),
                        v3(sRay[le][3], sRay[le][4], sRay[le][5]), a, e1, e2, kF32Max);
                    // t >= 0 orders as its bits (+ 0 makes a zero positive)
                    if (h.ok)
                        atomicMin(&sBest[le],
                            (unsigned long long)__float_as_uint(h.t + 0.0f) << 32 |
                                __ldg(tri.index + (size_t)lc * kClusterTris + j));
                }
                listed = 0;
                __syncwarp();
            }
            __syncthreads();
            if (warp == 0) {
                // each lane's entity in world space, then the sequential loop's
                // answer over entities: the smallest t, the first one of equals
                float t = kF32Max, hu = 0.0f, hv = 0.0f;
                V3 normal = v3(0.0f, 0.0f, 0.0f);
                bool cand = false;
                if (mine) {
                    const EntityDev &ent = ents[e];
                    float meshT = kF32Max;
                    V3 localNormal = v3(0.0f, 0.0f, 0.0f);
                    if (sBest[lane] != ~0ull) {
                        const uint32_t g = __ldg(&ent.triBegin) + (uint32_t)sBest[lane];
                        const float *p = tri.plain + (size_t)g * 9;
                        const V3 e1 = v3(__ldg(p + 3), __ldg(p + 4), __ldg(p + 5));
                        const V3 e2 = v3(__ldg(p + 6), __ldg(p + 7), __ldg(p + 8));
                        const MtHit h = mt_test(lo, ld, v3(__ldg(p), __ldg(p + 1), __ldg(p + 2)), e1, e2,
                            kF32Max);
                        localNormal = cnormalize(ccross(e1, e2));
                        const float w = 1.0f - h.u - h.v;
                        const float2 t0 = __ldg(&tri.uv[(size_t)g * 3 + 0]);
                        const float2 t1 = __ldg(&tri.uv[(size_t)g * 3 + 1]);
                        const float2 t2 = __ldg(&tri.uv[(size_t)g * 3 + 2]);
                        meshT = h.t;
                        hu = (t0.x * w + t1.x * h.u) + t2.x * h.v;
                        hv = (t0.y * w + t1.y * h.u) + t2.y * h.v;
                    }
                    const V3 localHit = v3(lo.x + ld.x * meshT, lo.y + ld.y * meshT, lo.z + ld.z * meshT);
                    const V3 worldHit = mat_mul(ent.model, localHit, 1.0f);
                    t = cdot(v3(worldHit.x - o.x, worldHit.y - o.y, worldHit.z - o.z), d);
                    normal = cnormalize(mat_mul(ent.model, localNormal, 0.0f));
                    cand = t >= 0.0f && t < res.t;
                }
                // t >= 0 orders as its bits (+ 0 makes a zero positive)
                const uint32_t key = cand ? __float_as_uint(t + 0.0f) : 0xFFFFFFFFu;
                const uint32_t best = __reduce_min_sync(0xFFFFFFFFu, key);
                const int who = best == 0xFFFFFFFFu ? 32 : __ffs(__ballot_sync(0xFFFFFFFFu, key == best)) - 1;
                if (who < 32) {
                    res.t = __shfl_sync(0xFFFFFFFFu, t, who);
                    res.normal.x = __shfl_sync(0xFFFFFFFFu, normal.x, who);
                    res.normal.y = __shfl_sync(0xFFFFFFFFu, normal.y, who);
                    res.normal.z = __shfl_sync(0xFFFFFFFFu, normal.z, who);
                    res.u = __shfl_sync(0xFFFFFFFFu, hu, who);
                    res.v = __shfl_sync(0xFFFFFFFFu, hv, who);
                    res.material = __ldg(&ents[chunk * kEntChunk + who].material);
                }
            }
            chunk++;
        } while (chunk < chunks);
        if (done) break;  // the same in every thread
        if (warp != 0) continue;
        // ---- shade: test_compute.comp.glsl:558-600 (the same in every lane)
        rays++;
        bool more = false;
        if (res.t > 0.0f && res.t < kF32Max) {
            hits++;
            float r0 = rng.bilateral();
            float r1 = rng.bilateral();
            float r2 = rng.bilateral();
            V3 dir = cnormalize(v3(res.normal.x + r0, res.normal.y + r1, res.normal.z + r2));
            if (cdot(dir, res.normal) < 0.0f) dir = v3(-dir.x, -dir.y, -dir.z);
            if (lane == len) vertex = PathVertex{res.material, dir, res.normal, res.u, res.v};
            len++;
            V3 wp = v3(o.x + d.x * res.t, o.y + d.y * res.t, o.z + d.z * res.t);
            o = v3(wp.x + res.normal.x * 0.001f, wp.y + res.normal.y * 0.001f,
                wp.z + res.normal.z * 0.001f);
            d = dir;
            bounce++;
            more = bounce < kMaxBounces;
        } else {
            if (lane == len)
                vertex = PathVertex{kMaterialBlack, v3(0.0f, 0.0f, 0.0f), v3(0.0f, 0.0f, 0.0f), 0.0f, 0.0f};
            len++;
        }
        if (!more) {
            V3 radiance = path_radiance_cpt(vertex, len, lane, tex, texW, texH);
            paths++;
            if (lane == 0)
                image[(size_t)y * view.width + x] = make_float4(0.0f + radiance.x * 1.0f,
                    0.0f + radiance.y * 1.0f, 0.0f + radiance.z * 1.0f, 1.0f);
            // next pixel of the tile in scanline order
            if (++x >= maxX) {
                x = minX;
                y++;
            }
            if (y >= maxY)
                active = false;
            else
                start_pixel();
        }
    }
    if (tid == 0) {
        atomicAdd(counters.rays, (unsigned long long)rays);
        atomicAdd(counters.hits, (unsigned long long)hits);
        atomicAdd(counters.tests, (unsigned long long)(rays * triangleTests));
        atomicAdd(counters.paths, (unsigned long long)paths);
    }
}

}  // namespace cpt
}  // namespace gbsp

using namespace gbsp;

struct gbsp_cpt_scene {
    gbsp_runtime *rt = nullptr;
    uint32_t entityCount = 0, texW = 0, texH = 0;
    DeviceBuffer<cpt::EntityDev> entities;
    uint64_t triangleTests = 0, units = 0;  // per ray: triangles, and steps of 32 clusters
    DeviceBuffer<float> plain, clustered;  // cpt::Triangles
    DeviceBuffer<uint32_t> index;
    DeviceBuffer<cpt::Cluster> clusters;
    DeviceBuffer<float2> uv;
    DeviceBuffer<float4> tex;
    DeviceBuffer<uint32_t> tiles;
};

extern "C" {

int gbsp_cpt_scene_create(gbsp_runtime *rt, const gbsp_vertex *vertices, uint32_t vertexCount,
    const uint32_t *indices, uint32_t indexCount, const gbsp_cpt_mesh *meshes, uint32_t meshCount,
    const float *modelMatrices, const float *invModelMatrices, uint32_t matrixCount,
    const gbsp_cpt_entity *entities, uint32_t entityCount, const float *checkerBoard,
    uint32_t texWidth, uint32_t texHeight, gbsp_cpt_scene **out)
{
    if (!rt || !out) return set_error(GBSP_ERR_INVALID_ARGUMENT, "NULL argument");
    *out = nullptr;
    if ((entityCount && (!entities || !meshes || !modelMatrices || !invModelMatrices)) ||
        (indexCount && !indices) || (vertexCount && !vertices))
        return set_error(GBSP_ERR_INVALID_ARGUMENT, "NULL array with a non-zero count");
    if ((texWidth || texHeight) && (!checkerBoard || !texWidth || !texHeight))
        return set_error(GBSP_ERR_INVALID_ARGUMENT, "texture needs pixels, width and height");
    // triangles per mesh, expanded once (entities share meshes)
    std::vector<uint64_t> meshBegin(meshCount), meshTris(meshCount);
    uint64_t total = 0;
    for (uint32_t m = 0; m < meshCount; m++) {
        const gbsp_cpt_mesh &mesh = meshes[m];
        uint64_t tris = mesh.indexCount / 3;
        if ((uint64_t)mesh.indicesOffset + tris * 3 > indexCount)
            return set_error(GBSP_ERR_INVALID_ARGUMENT, "mesh %u: indices out of range", m);
        for (uint64_t k = 0; k < tris * 3; k++) {
            uint64_t vi = (uint64_t)indices[mesh.indicesOffset + k] + mesh.vertexDataOffset;
            if (vi >= vertexCount)
                return set_error(GBSP_ERR_INVALID_ARGUMENT, "mesh %u: vertex index out of range", m);
        }
        meshBegin[m] = total;
        meshTris[m] = tris;
        total += tris;
    }
    if (total > 0xFFFFFFF0ull) return set_error(GBSP_ERR_CAPACITY, "too many triangles");
    std::vector<cpt::EntityDev> ents(entityCount);
    for (uint32_t e = 0; e < entityCount; e++) {
        const gbsp_cpt_entity &en = entities[e];
        if (en.meshIndex >= meshCount || en.modelMatrixIndex >= matrixCount)
            return set_error(GBSP_ERR_INVALID_ARGUMENT, "entity %u: mesh or matrix out of range", e);
        cpt::EntityDev &d = ents[e];
        memset(&d, 0, sizeof(d));
        for (int k = 0; k < 16; k++) {
            d.model[k] = modelMatrices[(size_t)en.modelMatrixIndex * 16 + k];
            d.inv[k] = invModelMatrices[(size_t)en.modelMatrixIndex * 16 + k];
        }
        d.triBegin = (uint32_t)meshBegin[en.meshIndex];
        d.triCount = (uint32_t)meshTris[en.meshIndex];
        d.material = en.materialId;
    }
    std::vector<float> plain((size_t)total * 9), clustered;
    std::vector<float2> uv((size_t)total * 3);
    std::vector<cpt::Cluster> clusters;
    std::vector<uint32_t> index;
    std::vector<uint32_t> clusterBegin(meshCount), clusterCount(meshCount);
    std::vector<V3> ma, me1, me2;
    for (uint32_t m = 0; m < meshCount; m++) {
        const gbsp_cpt_mesh &mesh = meshes[m];
        ma.resize(meshTris[m]);
        me1.resize(meshTris[m]);
        me2.resize(meshTris[m]);
        for (uint64_t k = 0; k < meshTris[m]; k++) {
            uint64_t g = meshBegin[m] + k;
            const gbsp_vertex *v[3];
            for (int j = 0; j < 3; j++)
                v[j] = &vertices[indices[mesh.indicesOffset + k * 3 + j] + mesh.vertexDataOffset];
            const float *a = v[0]->position, *b = v[1]->position, *c = v[2]->position;
            ma[k] = v3(a[0], a[1], a[2]);
            me1[k] = v3(b[0] - a[0], b[1] - a[1], b[2] - a[2]);
            me2[k] = v3(c[0] - a[0], c[1] - a[1], c[2] - a[2]);
            const float comp[9] = {ma[k].x, ma[k].y, ma[k].z, me1[k].x, me1[k].y, me1[k].z, me2[k].x,
                me2[k].y, me2[k].z};
            memcpy(plain.data() + 9 * g, comp, sizeof(comp));
            for (int j = 0; j < 3; j++) uv[g * 3 + j] = make_float2(v[j]->uv[0], v[j]->uv[1]);
        }
        const size_t c0 = clusters.size();
        cpt::build_clusters({ma.data(), me1.data(), me2.data(), (uint32_t)meshTris[m]}, clusters, index);
        clusterBegin[m] = (uint32_t)c0;
        clusterCount[m] = (uint32_t)(clusters.size() - c0);
        clustered.resize(clusters.size() * 9 * cpt::kClusterTris, nanf(""));
        for (size_t i = c0 * cpt::kClusterTris; i < index.size(); i++) {
            if (index[i] == 0xFFFFFFFFu) continue;
            const size_t c = i / cpt::kClusterTris, j = i % cpt::kClusterTris;
            for (int q = 0; q < 9; q++)
                clustered[(c * 9 + q) * cpt::kClusterTris + j] = plain[9 * (meshBegin[m] + index[i]) + q];
        }
    }
    uint64_t triangleTests = 0, units = 0;
    std::vector<uint32_t> openBegin(meshCount, 0xFFFFFFFFu);  // a mesh's clusters without a bound
    for (uint32_t e = 0; e < entityCount; e++) {
        const uint32_t m = entities[e].meshIndex;
        ents[e].clusterBegin = clusterBegin[m];
        if (!cpt::unit_directions(ents[e].inv)) {
            if (openBegin[m] == 0xFFFFFFFFu) {
                openBegin[m] = (uint32_t)clusters.size();
                const size_t b = clusterBegin[m], n = clusterCount[m];
                cpt::Cluster open = {};
                open.sphere.w = INFINITY;
                clusters.resize(clusters.size() + n, open);
                index.resize(index.size() + n * cpt::kClusterTris);
                std::copy_n(index.begin() + b * cpt::kClusterTris, n * cpt::kClusterTris,
                    index.end() - n * cpt::kClusterTris);
                clustered.resize(clustered.size() + n * 9 * cpt::kClusterTris);
                std::copy_n(clustered.begin() + b * 9 * cpt::kClusterTris, n * 9 * cpt::kClusterTris,
                    clustered.end() - n * 9 * cpt::kClusterTris);
            }
            ents[e].clusterBegin = openBegin[m];
        }
        ents[e].clusterCount = clusterCount[m];
        triangleTests += meshTris[m];
        units += (clusterCount[m] + 31) / 32;
    }
    int rrc = runtime_retain(rt);
    if (rrc) return rrc;
    gbsp_cpt_scene *s = new gbsp_cpt_scene();
    s->rt = rt;
    s->entityCount = entityCount;
    s->triangleTests = triangleTests;
    s->units = units;
    s->texW = texWidth;
    s->texH = texHeight;
    cudaStream_t st = rt->stream;
    int rc = GBSP_OK;
    if (entityCount) rc = s->entities.upload(ents.data(), ents.size(), st);
    if (!rc && total) rc = s->plain.upload(plain.data(), plain.size(), st);
    if (!rc && total) rc = s->clustered.upload(clustered.data(), clustered.size(), st);
    if (!rc && total) rc = s->index.upload(index.data(), index.size(), st);
    if (!rc && total) rc = s->clusters.upload(clusters.data(), clusters.size(), st);
    if (!rc && total) rc = s->uv.upload(uv.data(), uv.size(), st);
    if (!rc && texWidth)
        rc = s->tex.upload(reinterpret_cast<const float4 *>(checkerBoard),
            (size_t)texWidth * texHeight, st);
    if (!rc && cudaStreamSynchronize(st) != cudaSuccess)
        rc = set_error(GBSP_ERR_CUDA, "compute path tracer scene upload failed");
    if (rc) {
        delete s;
        runtime_release(rt);
        return rc;
    }
    *out = s;
    return GBSP_OK;
}

int gbsp_cpt_scene_destroy(gbsp_cpt_scene *scene)
{
    if (!scene) return GBSP_OK;
    gbsp_runtime *rt = scene->rt;
    cudaStreamSynchronize(rt->stream);
    delete scene;
    runtime_release(rt);
    return GBSP_OK;
}

int gbsp_cpt_render_tiles(gbsp_cpt_scene *scene, const gbsp_cpt_view *view,
    const uint32_t *tileIndices, uint32_t tileCount, float *deviceImage, gbsp_metrics *metrics)
{
    if (!scene || !view || (tileCount && (!tileIndices || !deviceImage)))
        return set_error(GBSP_ERR_INVALID_ARGUMENT, "NULL argument");
    if (!view->width || !view->height || !view->tileWidth || !view->tileHeight ||
        view->width < view->tileWidth)
        return set_error(GBSP_ERR_INVALID_ARGUMENT, "bad image or tile size");
    gbsp_runtime *rt = scene->rt;
    cudaStream_t s = rt->stream;
    if (!tileCount) return GBSP_OK;
    int rc = scene->tiles.upload(tileIndices, tileCount, s);
    if (rc) return rc;
    // main() of the shader: film and camera (test_compute.comp.glsl:615-668)
    cpt::View v;
    float planeW = (float)view->width, planeH = (float)view->height;
    float filmWidth = 1.0f, filmHeight = 1.0f;
    if (planeW > planeH)
        filmHeight = planeH / planeW;
    else if (planeW < planeH)
        filmWidth = planeW / planeH;
    const float *ct = view->cameraTransform;
    v.right = v3(ct[0], ct[1], ct[2]);
    v.up = v3(ct[4], ct[5], ct[6]);
    V3 forward = v3(ct[8], ct[9], ct[10]);
    v.position = v3(ct[12], ct[13], ct[14]);
    v.halfWidth = filmWidth * 0.5f;
    v.halfHeight = filmHeight * 0.5f;
    v.halfPixelWidth = 0.5f / planeW;
    v.halfPixelHeight = 0.5f / planeH;
    float fd = view->filmDistance;
    v.center = v3(v.position.x + forward.x * fd, v.position.y + forward.y * fd,
        v.position.z + forward.z * fd);
    v.invW = 1.0f / planeW;
    v.invH = 1.0f / planeH;
    v.width = view->width;
    v.height = view->height;
    v.tileW = view->tileWidth;
    v.tileH = view->tileHeight;
    v.tileCountX = view->width / view->tileWidth;
    cpt::Triangles tri;
    tri.clustered = scene->clustered.ptr;
    tri.index = scene->index.ptr;
    tri.clusters = scene->clusters.ptr;
    tri.plain = scene->plain.ptr;
    tri.uv = scene->uv.ptr;
    cpt::Counters c;
    c.rays = rt->dCounters + GBSP_METRIC_RAYS_TRACED;
    c.hits = rt->dCounters + GBSP_METRIC_RAY_HIT_COUNT;
    c.tests = rt->dCounters + GBSP_METRIC_TRIANGLE_TESTS;
    c.paths = rt->dCounters + GBSP_METRIC_PATHS_TRACED;
    GBSP_CUDA_TRY(cudaMemsetAsync(rt->dCounters, 0, sizeof(unsigned long long) * GBSP_METRIC_COUNT, s));
    if (metrics) GBSP_CUDA_TRY(cudaEventRecord(rt->ev[0], s));
    // warps per tile: as many as there are steps of 32 clusters to share (57
    // steps: 8 warps 5.9, 4 warps 6.6, 2 warps 9.8 ms; 10 steps: 4 warps 2.7,
    // 8 warps 2.9 ms, both at 512 x 384)
    auto kern = scene->units <= 4 ? cpt::k_compute_pt<2>
        : scene->units <= 16      ? cpt::k_compute_pt<4>
                                  : cpt::k_compute_pt<8>;
    const unsigned threads = scene->units <= 4 ? 64 : scene->units <= 16 ? 128 : 256;
    kern<<<tileCount, threads, 0, s>>>(scene->entities.ptr, scene->entityCount, scene->triangleTests, tri,
        scene->tex.ptr, scene->texW, scene->texH, v, scene->tiles.ptr,
        reinterpret_cast<float4 *>(deviceImage), c);
    GBSP_CUDA_TRY(cudaGetLastError());
    if (!metrics) return GBSP_OK;
    GBSP_CUDA_TRY(cudaEventRecord(rt->ev[1], s));
    unsigned long long cnt[GBSP_METRIC_COUNT];
    GBSP_CUDA_TRY(cudaMemcpyAsync(cnt, rt->dCounters, sizeof(cnt), cudaMemcpyDeviceToHost, s));
    GBSP_CUDA_TRY(cudaStreamSynchronize(s));
    float ms = 0.0f;
    cudaEventElapsedTime(&ms, rt->ev[0], rt->ev[1]);
    for (int i = 0; i < GBSP_METRIC_COUNT; i++) metrics->values[i] += cnt[i];
    metrics->values[GBSP_METRIC_RAY_MISS_COUNT] +=
        cnt[GBSP_METRIC_RAYS_TRACED] - cnt[GBSP_METRIC_RAY_HIT_COUNT];
    metrics->values[GBSP_METRIC_ELAPSED_NS] += (uint64_t)((double)ms * 1.0e6);
    metrics->values[GBSP_METRIC_KERNEL_LAUNCHES] += 1;
    return GBSP_OK;
}

}  // extern "C"
