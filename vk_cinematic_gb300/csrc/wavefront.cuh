// Wave kernels shared by the frame renderer (pathtrace.cu) and the batched
// wavefront (batch.cu).  See pathtrace.cu for the stage structure.  The
// trace and shade kernels are templates over a scene source: OneScene for a
// frame, a per-path item table for a batch of scenes.
#pragma once

#include "gbsp_internal.h"
#include "launch.cuh"
#include "traverse.cuh"
#include "shading.cuh"

namespace gbsp {

// Work/queue control words (u32) behind the metric counters.  The queue of
// bounce b has its length in word kCtlQueues + b % 3: while bounce b is shaded
// (reads word b, fills word b + 1), nothing reads word b + 2, so the shade
// kernel zeroes it and the trace kernel's work counter for the next bounce.
// A reset kernel of its own before every bounce and wave had cost a small
// frame 7 of 180 us on the device and four launches.
enum Ctl : int {
    kCtlTraceWork = 0,
    kCtlQueues = 2,
    kCtlCount = 8
};
__host__ __device__ __forceinline__ int queue_word(uint32_t bounce) { return kCtlQueues + (int)(bounce % 3u); }

// A new wave's control words, by the kernel that fills its first queue.
__device__ __forceinline__ void reset_wave_ctl(unsigned int *ctl, uint32_t paths)
{
    ctl[kCtlTraceWork] = 0;
    ctl[queue_word(0)] = paths;
    ctl[queue_word(1)] = ctl[queue_word(2)] = 0;
}

struct WaveBuffers {
    // a queued ray carries its path's state: the path id and the RNG state ride
    // in the w lanes, and its path length is the bounce number of the queue
    float4 *rayO;      // 2 * cap: (origin, path id bits)
    float4 *rayD;      // 2 * cap: (direction, RNG state bits)
    int4 *hitA;        // cap: (t, u, v, prim) bits
    int *hitInst;      // cap
    float4 *vert;      // 2 per vertex, (maxBounces - 1) * cap vertices of paths that go on:
                       // (emission xyz, cosine), (A xyz, 0)
    float4 *pathRad;   // cap
    float4 *pathAov;   // 2 * cap first-hit G-buffer per path, or null
    uint32_t cap;
};

struct WaveParams {
    CameraParams cam;
    uint32_t x0, y0, regionW;
    // optional list of rectangles rendered instead of the region: tile i is
    // (x0, y0, width, height) = tiles[i], its pixels numbered row-major from
    // tileStart[i] (an exclusive prefix sum over the tiles' pixel counts)
    const uint4 *tiles;
    const uint64_t *tileStart;
    uint32_t tileCount;
    // optional per-tile sample counts of a tile list: tile i renders
    // tileSpp[i] samples per pixel, its paths numbered pixel-major from
    // tilePath[i] (an exclusive prefix sum over pixels x spp); null: `spp`
    // samples for every pixel
    const uint32_t *tileSpp;
    const uint64_t *tilePath;
    uint64_t pixelBase;   // first pixel (row-major in the region) of this wave
    uint32_t pixels;      // pixels in this wave
    uint64_t pathBase;    // first path of this wave (with tileSpp)
    uint32_t paths;       // paths in this wave
    uint32_t spp;
    uint32_t maxBounces;
    uint32_t seed;
    float clampValue;
    uint32_t nanPolicy;
    float invSpp;
    float4 *aovImage;     // 2 float4 per image pixel, or null
    // split accumulation (0: off): samples [0, splitSpp) of a pixel go to the
    // image (and the G-buffers), samples [splitSpp, spp) to image2
    uint32_t splitSpp;
    float4 *image2;
};

// Scene source of the wave kernels: everything a path needs from its scene.
// OneScene: one scene for the whole launch (a frame or a tile).
struct OneScene {
    static constexpr bool kManyScenes = false;
    SceneView sv;
    MaterialView mv;
    uint32_t maxBounces;
    float clampValue;
    __device__ __forceinline__ const SceneView &scene(uint32_t) const { return sv; }
    __device__ __forceinline__ const MaterialView &materials(uint32_t) const { return mv; }
    __device__ __forceinline__ uint32_t bounces(uint32_t) const { return maxBounces; }
    __device__ __forceinline__ float clamp(uint32_t) const { return clampValue; }
};

// ---------------------------------------------------------------------------
// Stage kernels
// ---------------------------------------------------------------------------
// Stable counting sort of a ray queue by direction octant (sign bits of d),
// so that the lanes of a warp walk the tree with the same near-to-far child
// order.  Queue order otherwise follows path order (neighbouring pixels'
// samples), which the sort keeps within each octant.  Three launches over a
// fixed grid of kSortBlocks blocks (the count lives on the device):
// per-block octant histograms, one exclusive scan over (octant, block), and
// the scatter, which ranks rays inside each 256-ray tile with warp ballots.
constexpr int kSortBlocks = 512;

__device__ __forceinline__ uint32_t dir_octant(float4 d)
{
    return (d.x < 0.0f ? 1u : 0u) | (d.y < 0.0f ? 2u : 0u) | (d.z < 0.0f ? 4u : 0u);
}

__device__ __forceinline__ void sort_chunk(uint32_t n, uint32_t &begin, uint32_t &end)
{
    uint32_t chunk = (n + kSortBlocks - 1) / kSortBlocks;
    chunk = (chunk + 255u) & ~255u;
    begin = min(n, blockIdx.x * chunk);
    end = min(n, begin + chunk);
}

static __global__ void __launch_bounds__(256) k_octant_count(const float4 *__restrict__ rayD,
    const unsigned int *ctl, int queue, uint32_t *hist)
{
    __shared__ uint32_t sh[8];
    if (threadIdx.x < 8) sh[threadIdx.x] = 0;
    __syncthreads();
    uint32_t begin, end;
    sort_chunk(ctl[queue], begin, end);
    for (uint32_t i = begin + threadIdx.x; i < end; i += 256) atomicAdd(&sh[dir_octant(rayD[i])], 1u);
    __syncthreads();
    if (threadIdx.x < 8) hist[threadIdx.x * kSortBlocks + blockIdx.x] = sh[threadIdx.x];
}

// Exclusive scan of hist[8][kSortBlocks] in (octant, block) order.
static __global__ void __launch_bounds__(1024) k_octant_scan(uint32_t *hist)
{
    constexpr int kPer = 8 * kSortBlocks / 1024;
    __shared__ uint32_t warpSum[32];
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    uint32_t v[kPer], sum = 0;
#pragma unroll
    for (int k = 0; k < kPer; k++) {
        v[k] = hist[t * kPer + k];
        sum += v[k];
    }
    uint32_t incl = sum;
    for (int off = 1; off < 32; off <<= 1) {
        uint32_t o = __shfl_up_sync(0xFFFFFFFFu, incl, off);
        if (lane >= off) incl += o;
    }
    if (lane == 31) warpSum[warp] = incl;
    __syncthreads();
    if (warp == 0) {
        uint32_t w = warpSum[lane], wi = w;
        for (int off = 1; off < 32; off <<= 1) {
            uint32_t o = __shfl_up_sync(0xFFFFFFFFu, wi, off);
            if (lane >= off) wi += o;
        }
        warpSum[lane] = wi - w;
    }
    __syncthreads();
    uint32_t run = warpSum[warp] + incl - sum;
#pragma unroll
    for (int k = 0; k < kPer; k++) {
        hist[t * kPer + k] = run;
        run += v[k];
    }
}

static __global__ void __launch_bounds__(256) k_octant_scatter(const float4 *__restrict__ srcO,
    const float4 *__restrict__ srcD, const unsigned int *ctl, int queue,
    const uint32_t *__restrict__ offsets, float4 *__restrict__ dstO, float4 *__restrict__ dstD)
{
    __shared__ uint32_t base[8], warpCount[8][8];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (threadIdx.x < 8) base[threadIdx.x] = offsets[threadIdx.x * kSortBlocks + blockIdx.x];
    uint32_t begin, end;
    sort_chunk(ctl[queue], begin, end);
    __syncthreads();
    for (uint32_t t0 = begin; t0 < end; t0 += 256) {
        const uint32_t i = t0 + threadIdx.x;
        const bool valid = i < end;
        float4 o = make_float4(0, 0, 0, 0), d = o;
        uint32_t oct = 8u;
        if (valid) {
            o = srcO[i];
            d = srcD[i];
            oct = dir_octant(d);
        }
        uint32_t rank = 0;
#pragma unroll
        for (uint32_t k = 0; k < 8; k++) {
            uint32_t m = __ballot_sync(0xFFFFFFFFu, oct == k);
            if (lane == 0) warpCount[k][warp] = __popc(m);
            if (oct == k) rank = __popc(m & ((1u << lane) - 1u));
        }
        __syncthreads();
        if (valid) {
            uint32_t before = 0;
            for (int w = 0; w < warp; w++) before += warpCount[oct][w];
            const uint32_t dst = base[oct] + before + rank;
            dstO[dst] = o;
            dstD[dst] = d;
        }
        __syncthreads();
        if (threadIdx.x < 8) {
            uint32_t tot = 0;
            for (int w = 0; w < 8; w++) tot += warpCount[threadIdx.x][w];
            base[threadIdx.x] += tot;
        }
        __syncthreads();
    }
}

// Image position of pixel `pix` of a wave's pixel numbering: row-major in
// the region, or in the tile list (binary search over the tiles' first
// pixels).
// The tile holding item `key` of a list numbered by the exclusive prefix sum
// `start` (binary search: the last tile whose start is <= key).
__device__ __forceinline__ uint32_t tile_of(const uint64_t *start, uint32_t count, uint64_t key)
{
    uint32_t lo = 0, hi = count - 1;
    while (lo < hi) {
        uint32_t mid = (lo + hi + 1) >> 1;
        if (__ldg(start + mid) <= key)
            lo = mid;
        else
            hi = mid - 1;
    }
    return lo;
}

__device__ __forceinline__ void tile_pixel(const WaveParams &wp, uint32_t t, uint64_t local,
    uint32_t &x, uint32_t &y)
{
    const uint4 r = __ldg(wp.tiles + t);
    x = r.x + (uint32_t)(local % r.z);
    y = r.y + (uint32_t)(local / r.z);
}

__device__ __forceinline__ void wave_pixel(const WaveParams &wp, uint64_t pix, uint32_t &x,
    uint32_t &y)
{
    if (!wp.tiles) {
        x = wp.x0 + (uint32_t)(pix % wp.regionW);
        y = wp.y0 + (uint32_t)(pix / wp.regionW);
        return;
    }
    const uint32_t t = tile_of(wp.tileStart, wp.tileCount, pix);
    tile_pixel(wp, t, pix - __ldg(wp.tileStart + t), x, y);
}

static __global__ void __launch_bounds__(256) k_generate(WaveParams wp, WaveBuffers wb, unsigned int *ctl)
{
    uint32_t p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p == 0) reset_wave_ctl(ctl, wp.paths);
    if (p >= wp.paths) return;
    uint32_t x, y, s;
    if (wp.tileSpp) {
        const uint64_t gp = wp.pathBase + p;
        const uint32_t t = tile_of(wp.tilePath, wp.tileCount, gp);
        const uint32_t n = __ldg(wp.tileSpp + t);
        const uint64_t local = gp - __ldg(wp.tilePath + t), lp = local / n;
        s = (uint32_t)(local - lp * n);
        tile_pixel(wp, t, lp, x, y);
    } else {
        s = p % wp.spp;
        wave_pixel(wp, wp.pixelBase + p / wp.spp, x, y);
    }
    uint32_t rng = sample_seed(wp.seed, x, y, s);
    V3 o, d;
    camera_ray(wp.cam, x, y, rng, o, d);
    wb.rayO[p] = make_float4(o.x, o.y, o.z, __int_as_float((int)p));
    wb.rayD[p] = make_float4(d.x, d.y, d.z, __uint_as_float(rng));
}

// Closest hit, 32 queued rays per warp (primary rays by default: they are
// coherent, 27.7 lanes active per instruction, and the per-lane kernel's vote
// then only costs: a 1080p frame took 72.4 ms with it for the primary rays too,
// 69.5 ms with this one).  7 blocks of 128 per SM (72 registers); 6 measured
// the same.
template <class Src, bool kWT, int kQ>
__global__ void __launch_bounds__(128, 7) k_trace(Src src, const float4 *rayO,
    const float4 *rayD, const unsigned int *queueCount, int4 *hitA, int *hitInst,
    unsigned int *ctl, unsigned long long *counters, uint32_t *status)
{
    stage_begin();
    int lane = threadIdx.x & 31;
    uint32_t count = *queueCount;
    TraceCounters cnt = {0, 0, 0, 0, 0};
    uint32_t done = 0, hits = 0;
    for (uint32_t guard = 0; guard <= count / 32 + 1; guard++) {
        uint32_t base = 0;
        if (lane == 0) base = atomicAdd(&ctl[kCtlTraceWork], 32u);
        base = __shfl_sync(0xFFFFFFFFu, base, 0);
        if (base >= count) break;
        uint32_t i = base + lane;
        if (i < count) {
            float4 o4 = rayO[i], d4 = rayD[i];
            const SceneView &sv = src.scene((uint32_t)__float_as_int(o4.w));
            RayHit h = trace_closest<true, kWT, kQ>(sv, v3(o4.x, o4.y, o4.z), v3(d4.x, d4.y, d4.z),
                status, cnt);
            hitA[i] = make_int4(__float_as_int(h.t), __float_as_int(h.u), __float_as_int(h.v),
                h.prim);
            hitInst[i] = h.inst;
            done++;
            hits += (h.prim >= 0 && h.t > 0.0f) ? 1u : 0u;
        }
    }
    uint32_t v[7] = {done, hits, cnt.topNodes, cnt.meshNodes, cnt.triTests, cnt.boxTests,
        cnt.meshTests};
#pragma unroll
    for (int k = 0; k < 7; k++)
        for (int off = 16; off; off >>= 1) v[k] += __shfl_xor_sync(0xFFFFFFFFu, v[k], off);
    if (lane == 0) {
        atomicAdd(&counters[GBSP_METRIC_RAYS_TRACED], (unsigned long long)v[0]);
        atomicAdd(&counters[GBSP_METRIC_RAY_HIT_COUNT], (unsigned long long)v[1]);
        atomicAdd(&counters[GBSP_METRIC_RAY_MISS_COUNT], (unsigned long long)(v[0] - v[1]));
        atomicAdd(&counters[GBSP_METRIC_BROADPHASE_NODE_VISITS], (unsigned long long)v[2]);
        atomicAdd(&counters[GBSP_METRIC_MIDPHASE_NODE_VISITS], (unsigned long long)v[3]);
        atomicAdd(&counters[GBSP_METRIC_TRIANGLE_TESTS], (unsigned long long)v[4]);
        atomicAdd(&counters[GBSP_METRIC_MIDPHASE_BOX_TESTS], (unsigned long long)v[5]);
        atomicAdd(&counters[GBSP_METRIC_MESH_TESTS_PERFORMED], (unsigned long long)v[6]);
    }
}

// Per-lane variant of k_trace (bounce rays by default).  Every lane keeps
// its own ray and stack; a lane whose ray is done takes the next queue index,
// so short rays do not wait for the warp's longest one.
//
// Bound: issue slots and load latency on diverged lanes, not memory (DRAM
// under 2%, L1 55-60% busy).  A walk is a sequence of steps of five kinds (a
// node visit, a triangle leaf, entering an object, leaving it, storing a
// finished ray and fetching the next); when every iteration runs each lane's
// next step, the warp issues all five kinds for a few lanes each (9.6 of 32
// lanes active per instruction).  Here an iteration runs ONE kind, the one
// most lanes want, and the other lanes wait for theirs to win: 17.3 lanes
// active, and one load latency per iteration instead of up to five.  The
// vote is one __reduce_add_sync over 6-bit counters (32 lanes fit in 6 bits).
// Some lane always advances, and a waiting kind gains lanes until it wins.
// 1080p benchmark frame (64 spp, 5 bounces): 85.3 ms before; 76.3 ms with the
// 256-bit node visits (visit_node8) and 128-bit transform loads; 68.4 ms with
// the vote; 67.8 ms with the weights below (steps that cost less than a node
// visit win with fewer lanes).  2^20 incoherent rays against 2^18 triangles:
// 2,366, 1,865, 1,737 and 1,768 us.
// Queues shorter than the grid's lanes use as few lanes per warp as spread them
// over all warps: a 128 x 128 x 4 crop of a dense part of that scene 692 -> 543
// us, 641 x 359 x 7 watertight 1,183 -> 1,045 us (at least 4, 8 or 16 lanes
// instead of 1: 560, 595 and 630 us for the crop).
//
// Every full-mask intrinsic stands at the loop head or in a branch taken on
// the vote's (warp-uniform) result; the only exit is the vote's zero.  Same
// candidate sets, arithmetic and tie rules as trace_closest, hence the same
// hit records.
//
// Blocks per SM: 7 of 128 threads (72 registers): 69.5 ms against 71.0 at 8
// (64 registers, spills) and 71.4 at 6 on the frame above.  The watertight
// test and the per-path scenes of a batch need more registers: 6 (a
// 641 x 359 x 7 watertight frame 1.20 against 1.22 ms at 7; an uneven batch
// 3.27 against 3.28).
constexpr uint32_t kMaxLaneRaySteps = 1u << 22;
constexpr int kLaneThreads = 128;  // block size of k_trace_lane
constexpr uint32_t kMaxLaneIterations = 1u << 28;
enum LaneStep : int { kStepNode = 0, kStepLeaf, kStepEnter, kStepLeave, kStepRay };
constexpr int kWeightNode = 3, kWeightLeaf = 3, kWeightEnter = 4, kWeightLeave = 5, kWeightRay = 3;

template <class Src, bool kWT, int kQ>
__global__ void __launch_bounds__(kLaneThreads, kWT || Src::kManyScenes ? 6 : 7) k_trace_lane(Src src, const float4 *rayO,
    const float4 *rayD, const unsigned int *queueCount, int4 *hitA, int *hitInst,
    unsigned int *ctl, unsigned long long *counters, uint32_t *status)
{
    stage_begin();
    const int lane = threadIdx.x & 31;
    const uint32_t count = *queueCount;
    unsigned int *work = &ctl[kCtlTraceWork];
    TraceCounters cnt = {0, 0, 0, 0, 0};
    uint32_t done = 0, hits = 0;
    StackEntry stack[kStackSize];
    // State a lane touches only when it fetches a ray, enters or leaves an
    // object, tests a leaf or stores a hit, kept in shared memory on purpose:
    // the walk itself then holds just the current level's ray, bound and
    // stack pointer in registers.  (In a local array its stores were written
    // through to L2; shared memory keeps them on the SM: 1,556 against
    // 1,552 Msamples/s on the 1080p benchmark frame.)  Word w of the lane
    // is column threadIdx.x of row w, so a warp's accesses to one word are
    // contiguous.  Words: world origin 0-2, direction 3-5, inverse direction
    // 6-8; best hit over objects u 9, v 10, triangle 11, object 12; queue
    // slot 13; object being walked 14; its best triangle's u 15, v 16; the
    // object-space direction 17-19.
    __shared__ uint32_t coldWords[20 * kLaneThreads];
    struct ColdWords {
        volatile uint32_t *p;
        __device__ __forceinline__ volatile uint32_t &operator[](int w) const
        {
            return p[w * kLaneThreads];
        }
    };
    const ColdWords cold{coldWords + threadIdx.x};
    // the node or leaf to visit next; kEmptyChild when none
    uint32_t ref = kEmptyChild;
    // Short queues are spread over every warp: only this many lanes of a warp
    // take rays.  Each lane's steps then wait for fewer others (the longest
    // ray's chain of steps is what a short launch takes).
    const uint32_t warps = gridDim.x * (kLaneThreads / 32);
    const uint32_t quota = (count + warps - 1) / warps;
    // base: stack height at which the object being walked is done, -1 at
    // object level, -2 without a ray, -3 when the queue is drained
    int sp = 0, base = (uint32_t)lane < quota ? -2 : -3;
    uint32_t steps = 0;
    // the ray of the level being walked (world or object space); `bound` is the
    // largest entry distance still worth a visit at that level
    V3 ro = v3(0, 0, 0), rinvd = v3(0, 0, 0);
    float bestT = kInf, bound = kInf, lBestT = kInf;
    int32_t lPrim = -1;
    uint32_t pathId = 0;
    bool drained = false;
    const auto put3 = [&](int w, V3 v) {
        cold[w] = __float_as_uint(v.x);
        cold[w + 1] = __float_as_uint(v.y);
        cold[w + 2] = __float_as_uint(v.z);
    };
    const auto get3 = [&](int w) {
        return v3(__uint_as_float(cold[w]), __uint_as_float(cold[w + 1]),
            __uint_as_float(cold[w + 2]));
    };
    for (uint32_t it = 0; it < kMaxLaneIterations; it++) {
        // ---- what each lane needs next
        if (ref == kEmptyChild) {
            const int floor = max(base, 0);
            while (sp > floor) {
                sp--;
                steps++;
                const StackEntry top = stack[sp];
                if (!(top.t > bound)) {
                    ref = top.ref;
                    break;
                }
            }
        }
        // children that are nodes have bit 31 clear; leaves and "none" have it set
        int cls = base >= 0 ? kStepLeave : kStepRay;
        if (!child_is_leaf(ref))
            cls = kStepNode;
        else if (ref != kEmptyChild)
            cls = base >= 0 ? kStepLeaf : kStepEnter;
        const uint32_t sums = __reduce_add_sync(0xFFFFFFFFu, base == -3 ? 0u : 1u << (6 * cls));
        if (sums == 0) {
            drained = true;
            break;
        }
        // the kind with the most lanes, weighted; its number rides in the low bits
        const int k0 = (int)(sums & 63u) * (8 * kWeightNode) + kStepNode,
                  k1 = (int)(sums >> 6 & 63u) * (8 * kWeightLeaf) + kStepLeaf,
                  k2 = (int)(sums >> 12 & 63u) * (8 * kWeightEnter) + kStepEnter,
                  k3 = (int)(sums >> 18 & 63u) * (8 * kWeightLeave) + kStepLeave,
                  k4 = (int)(sums >> 24) * (8 * kWeightRay) + kStepRay;
        const int best = __vimax3_s32(__vimax3_s32(k0, k1, k2), k3, k4) & 7;
        const bool mine = cls == best && base != -3;
        if (best == kStepNode) {
            if (mine) {
                if (base < 0)
                    cnt.topNodes++;
                else
                    cnt.meshNodes++;
                ref = visit_nearest<kWT, kQ>(src.scene(pathId).nodes, src.scene(pathId).nodeQuads,
                    ref, ro, rinvd, bound, stack, sp, status, cnt.boxTests);
            }
        } else if (best == kStepLeaf) {
            if (mine) {
                visit_leaf_uv<true, kWT>(src.scene(pathId), ref, ro, get3(17), rinvd, lBestT, lPrim,
                    [&](float u, float v) {
                        cold[15] = __float_as_uint(u);
                        cold[16] = __float_as_uint(v);
                    },
                    cnt);
                bound = rmin(prune_bound(lBestT), bound);
                ref = kEmptyChild;
            }
        } else if (best == kStepEnter) {
            if (mine) {
                // an object whose world box passed: enter its mesh
                const uint32_t inst = leaf_first(ref);
                cold[14] = inst;
                const Instance &in = src.scene(pathId).instances[inst];
                const Affine inv = load_affine(&in.inv);
                const V3 d = get3(3);
                ro = transform_point(inv, ro);
                float len;
                const V3 ld = normalize(transform_vector(inv, d), &len);
                put3(17, ld);
                rinvd = inverse(ld);
                cnt.meshTests++;
                lBestT = kInf;
                lPrim = -1;
                bound = prune_bound(bestT * len);
                base = sp;
                ref = __ldg(&in.blasRoot);
            }
        } else if (best == kStepLeave) {
            if (mine) {
                // leaving an object: its closest triangle goes back to world space
                const V3 o = get3(0);
                if (lPrim >= 0) {
                    const uint32_t inst = cold[14];
                    const Instance &in = src.scene(pathId).instances[inst];
                    const Affine model = load_affine(&in.model);
                    V3 worldHit = transform_point(model, add(ro, mul(get3(17), lBestT)));
                    float tw = dot(sub(worldHit, o), get3(3));
                    if (tw < bestT || (tw == bestT && (int32_t)inst < (int32_t)cold[12])) {
                        bestT = tw;
                        cold[9] = cold[15];
                        cold[10] = cold[16];
                        cold[11] = (uint32_t)lPrim;
                        cold[12] = inst;
                    }
                }
                ro = o;
                rinvd = get3(6);
                bound = prune_bound(bestT);
                base = -1;
            }
        } else {
            // a finished ray is stored and the next one fetched: one atomic for
            // the lanes that need a ray
            const uint32_t m = __ballot_sync(0xFFFFFFFFu, mine);
            uint32_t first = 0;
            if (lane == 0) first = atomicAdd(work, (unsigned int)__popc(m));
            first = __shfl_sync(0xFFFFFFFFu, first, 0);
            if (mine) {
                if (base == -1) {
                    const int32_t bestPrim = (int32_t)cold[11];
                    const uint32_t slot = cold[13];
                    hitA[slot] = make_int4(__float_as_int(bestT), (int)cold[9], (int)cold[10],
                        bestPrim);
                    hitInst[slot] = (int)cold[12];
                    done++;
                    hits += (bestPrim >= 0 && bestT > 0.0f) ? 1u : 0u;
                }
                const uint32_t idx = first + __popc(m & ((1u << lane) - 1u));
                if (idx < count) {
                    float4 o4 = rayO[idx], d4 = rayD[idx];
                    ro = v3(o4.x, o4.y, o4.z);
                    const V3 d = v3(d4.x, d4.y, d4.z);
                    pathId = (uint32_t)__float_as_int(o4.w);
                    rinvd = inverse(d);
                    put3(0, ro);
                    put3(3, d);
                    put3(6, rinvd);
                    cold[9] = 0u;
                    cold[10] = 0u;
                    cold[11] = 0xFFFFFFFFu;
                    cold[12] = 0xFFFFFFFFu;
                    cold[13] = idx;
                    bestT = kInf;
                    bound = kInf;
                    sp = 0;
                    steps = 0;
                    ref = src.scene(pathId).tlasRoot;
                    base = -1;
                } else {
                    base = -3;
                }
            }
        }
        if (steps > kMaxLaneRaySteps) {
            // store the best hit found so far
            atomicOr(status, kStatusRayStepLimit);
            steps = 0;
            base = -1;
            sp = 0;
            ref = kEmptyChild;
        }
    }
    if (!drained) atomicOr(status, kStatusQueueOverflow);
    __syncwarp();
    uint32_t v[7] = {done, hits, cnt.topNodes, cnt.meshNodes, cnt.triTests, cnt.boxTests,
        cnt.meshTests};
#pragma unroll
    for (int k = 0; k < 7; k++)
        for (int off = 16; off; off >>= 1) v[k] += __shfl_xor_sync(0xFFFFFFFFu, v[k], off);
    if (lane == 0) {
        atomicAdd(&counters[GBSP_METRIC_RAYS_TRACED], (unsigned long long)v[0]);
        atomicAdd(&counters[GBSP_METRIC_RAY_HIT_COUNT], (unsigned long long)v[1]);
        atomicAdd(&counters[GBSP_METRIC_RAY_MISS_COUNT], (unsigned long long)(v[0] - v[1]));
        atomicAdd(&counters[GBSP_METRIC_BROADPHASE_NODE_VISITS], (unsigned long long)v[2]);
        atomicAdd(&counters[GBSP_METRIC_MIDPHASE_NODE_VISITS], (unsigned long long)v[3]);
        atomicAdd(&counters[GBSP_METRIC_TRIANGLE_TESTS], (unsigned long long)v[4]);
        atomicAdd(&counters[GBSP_METRIC_MIDPHASE_BOX_TESTS], (unsigned long long)v[5]);
        atomicAdd(&counters[GBSP_METRIC_MESH_TESTS_PERFORMED], (unsigned long long)v[6]);
    }
}

// Shading of one bounce.  A warp walks batches of up to kShadeRows x 32 queue
// entries, sorts their indices into hits and misses (order kept, by ballot)
// and shades each kind with full warps.
//
// Bound, before: the one counter every warp took 32 entries from and the one
// every warp reserved its outputs at.  Atomics on one address complete at
// about 0.8 ns each, two per 32 rays: 1.2 to 2 ms of the 4.9 ms a wave of 2^25
// paths spent here.  Batches are now dealt out by index (their cost is even),
// and a batch reserves its outputs at once (a batch launch, whose items end at
// different bounces, still does per 32).  Now: the chain of dependent loads of
// a vertex (ray and hit, instance, triangle, material), so that there are few
// of them: a flat hit reads 12 bytes of its triangle instead of 112
// (attributes only for smooth meshes or textured albedo), a stored vertex is
// one 32-byte sector, and a path's last vertex, which adds only its emission
// (last_vertex_is_emission), skips the BRDF.  1080p benchmark frame (64 spp, 5
// bounces) 67.8 -> 54.6 ms with this kernel, uneven batch 3.24 -> 2.45 ms;
// 1, 2, 4 and 8 rows with an atomic per batch: 67.7, 63.7, 61.1 and 59.3 ms;
// by index 8 rows 55.3 and 4 rows 55.1 ms, and 4 are the better ones on short
// queues (641 x 359 x 7: 1.106 and 1.091 ms).  8, 10 and 12 blocks per SM
// measured the same; unbounded (72 registers, 7 blocks) the batch took 2.78 ms.
constexpr uint32_t kShadeRows = 4;
constexpr int kShadeThreads = 128;

template <class Src>
__global__ void __launch_bounds__(kShadeThreads, 8) k_shade(Src src, WaveBuffers wb, uint32_t bounce,
    uint32_t side, unsigned int *ctl, unsigned long long *counters)
{
    stage_begin();
    const int lane = threadIdx.x & 31;
    const uint32_t laneMaskLt = (1u << lane) - 1u;
    __shared__ uint8_t lists[kShadeThreads / 32][32 * kShadeRows];
    uint8_t *list = lists[threadIdx.x >> 5];  // hits from the front, misses from the back
    const uint32_t count = ctl[queue_word(bounce)];
    const int outQueue = queue_word(bounce + 1);
    if (blockIdx.x == 0 && threadIdx.x == 0) ctl[queue_word(bounce + 2)] = ctl[kCtlTraceWork] = 0;
    const float4 *inO = wb.rayO + (side ? wb.cap : 0);
    const float4 *inD = wb.rayD + (side ? wb.cap : 0);
    float4 *outO = wb.rayO + (side ? 0 : wb.cap);
    float4 *outD = wb.rayD + (side ? 0 : wb.cap);
    // short queues: fewer rows, so that every warp gets some entries
    const uint32_t warps = gridDim.x * (kShadeThreads / 32);
    const uint32_t rows = min(kShadeRows, max(1u, count / (32u * warps)));
    uint32_t finished = 0;
    // counts stay below 2^31, so the index does not wrap
    for (uint32_t base = (blockIdx.x * (kShadeThreads / 32) + (threadIdx.x >> 5)) * 32u * rows;
         base < count; base += warps * 32u * rows) {
        uint32_t hits = 0, misses = 0;
        for (uint32_t r = 0; r < rows; r++) {
            const uint32_t i = base + 32u * r + lane;
            bool hit = false;
            if (i < count) {
                const int4 h = wb.hitA[i];
                hit = h.w >= 0 && __int_as_float(h.x) > 0.0f;
            }
            const uint32_t mh = __ballot_sync(0xFFFFFFFFu, hit);
            const uint32_t mm = __ballot_sync(0xFFFFFFFFu, i < count && !hit);
            if (hit)
                list[hits + __popc(mh & laneMaskLt)] = (uint8_t)(32u * r + lane);
            else if (i < count)
                list[32u * kShadeRows - 1u - misses - __popc(mm & laneMaskLt)] = (uint8_t)(32u * r + lane);
            hits += __popc(mh);
            misses += __popc(mm);
        }
        __syncwarp();
        finished += lane == 0 ? misses : 0u;
        // a frame's hits all go on or all end: one queue reservation per batch
        uint32_t outBase = 0;
        if (!Src::kManyScenes && bounce + 1 < src.bounces(0)) {
            if (lane == 0 && hits) outBase = atomicAdd(&ctl[outQueue], hits);
            outBase = __shfl_sync(0xFFFFFFFFu, outBase, 0);
        }
        for (uint32_t k0 = 0; k0 < hits; k0 += 32) {
            // hit vertex (src/simd_path_tracer.cpp:268-288)
            bool cont = false;
            float4 newO = make_float4(0, 0, 0, 0), newD = make_float4(0, 0, 0, 0);
            if (k0 + lane < hits) {
                const uint32_t i = base + list[k0 + lane];
                const float4 o4 = inO[i], d4 = inD[i];
                const int4 hA = wb.hitA[i];
                RayHit h;
                h.t = __int_as_float(hA.x);
                h.u = __int_as_float(hA.y);
                h.v = __int_as_float(hA.z);
                h.prim = hA.w;
                h.inst = wb.hitInst[i];
                const uint32_t p = (uint32_t)__float_as_int(o4.w);
                const SceneView &sv = src.scene(p);
                const MaterialView &mv = src.materials(p);
                const V3 o = v3(o4.x, o4.y, o4.z), d = v3(d4.x, d4.y, d4.z);
                const V3 n = hit_normal(sv, h);
                const SurfaceMaterial sm = surface_material(mv, mv.instanceSlot[h.inst], neg(d),
                    [&](float &u, float &v) { hit_uv(sv, h, u, v); });
                if (wb.pathAov && bounce == 0) {
                    wb.pathAov[2 * (size_t)p] = make_float4(sm.albedo.x, sm.albedo.y, sm.albedo.z, h.t);
                    wb.pathAov[2 * (size_t)p + 1] = make_float4(n.x, n.y, n.z, 1.0f);
                }
                uint32_t rng = __float_as_uint(d4.w);
                const V3 dir = random_hemisphere(n, rng);
                // every path in this queue has `bounce` vertices so far
                cont = bounce + 1 < src.bounces(p);
                V3 r = add(sm.emission, v3(0.0f, 0.0f, 0.0f));
                if (cont || !last_vertex_is_emission(sm, n, dir, neg(d), src.clamp(p))) {
                    V3 A;
                    float cosine;
                    brdf_terms(sm, n, dir, neg(d), A, cosine);
                    const float4 ec = make_float4(sm.emission.x, sm.emission.y, sm.emission.z, cosine);
                    const float4 aa = make_float4(A.x, A.y, A.z, 0.0f);
                    if (cont) {
                        store_vertex(wb.vert, (size_t)bounce * wb.cap + p, ec, aa);
                        const V3 pos = add(o, mul(d, h.t));
                        const V3 no = add(pos, mul(n, 0.0001f));
                        newO = make_float4(no.x, no.y, no.z, o4.w);
                        newD = make_float4(dir.x, dir.y, dir.z, __uint_as_float(rng));
                    } else {
                        r = radiance_step(v3(0.0f, 0.0f, 0.0f), ec, aa, src.clamp(p));
                    }
                }
                if (!cont) {
                    r = path_radiance_from(r, wb.vert, wb.cap, p, bounce, src.clamp(p));
                    wb.pathRad[p] = make_float4(r.x, r.y, r.z, 0.0f);
                    finished++;
                }
            }
            // compaction: one atomic per warp for the continuing rays
            const uint32_t mask = __ballot_sync(0xFFFFFFFFu, cont);
            if (Src::kManyScenes) {
                if (lane == 0 && mask) outBase = atomicAdd(&ctl[outQueue], (unsigned)__popc(mask));
                outBase = __shfl_sync(0xFFFFFFFFu, outBase, 0);
            }
            if (cont) {
                const uint32_t slot = outBase + (Src::kManyScenes ? 0u : k0) + __popc(mask & laneMaskLt);
                outO[slot] = newO;
                outD[slot] = newD;
            }
        }
        for (uint32_t k0 = 0; k0 < misses; k0 += 32) {
            // miss: background vertex, path ends (:302-314)
            if (k0 + lane < misses) {
                const uint32_t i = base + list[32u * kShadeRows - 1u - k0 - lane];
                const float4 d4 = inD[i];
                const uint32_t p = (uint32_t)__float_as_int(inO[i].w);
                const MaterialView &mv = src.materials(p);
                const V3 z = v3(0.0f, 0.0f, 0.0f), V = neg(v3(d4.x, d4.y, d4.z));
                const SurfaceMaterial sm = surface_material(mv, mv.backgroundSlot, V,
                    [&](float &u, float &v) { u = v = 0.0f; });
                V3 r = add(sm.emission, z);
                if (!last_vertex_is_emission(sm, z, z, V, src.clamp(p))) {
                    V3 A;
                    float cosine;
                    brdf_terms(sm, z, z, V, A, cosine);
                    r = radiance_step(z, make_float4(sm.emission.x, sm.emission.y, sm.emission.z, cosine),
                        make_float4(A.x, A.y, A.z, 0.0f), src.clamp(p));
                }
                if (wb.pathAov && bounce == 0) {
                    wb.pathAov[2 * (size_t)p] = make_float4(0, 0, 0, 0);
                    wb.pathAov[2 * (size_t)p + 1] = make_float4(0, 0, 0, 0);
                }
                r = path_radiance_from(r, wb.vert, wb.cap, p, bounce, src.clamp(p));
                wb.pathRad[p] = make_float4(r.x, r.y, r.z, 0.0f);
            }
        }
        __syncwarp();
    }
    for (int off = 16; off; off >>= 1) finished += __shfl_xor_sync(0xFFFFFFFFu, finished, off);
    if (lane == 0 && finished)
        atomicAdd(&counters[GBSP_METRIC_PATHS_TRACED], (unsigned long long)finished);
}

static __global__ void __launch_bounds__(256) k_accumulate(WaveParams wp, WaveBuffers wb, float4 *image,
    uint32_t imageWidth, unsigned long long *counters)
{
    stage_begin();
    uint32_t k = blockIdx.x * blockDim.x + threadIdx.x;
    uint32_t nans = 0;
    if (k < wp.pixels) {
        uint64_t pix = wp.pixelBase + k;
        uint32_t x, y, n = wp.spp;
        size_t first = (size_t)k * wp.spp;  // this pixel's first path in the wave
        float inv = wp.invSpp;
        if (wp.tileSpp) {
            const uint32_t t = tile_of(wp.tileStart, wp.tileCount, pix);
            const uint64_t lp = pix - __ldg(wp.tileStart + t);
            n = __ldg(wp.tileSpp + t);
            first = (size_t)(__ldg(wp.tilePath + t) + lp * n - wp.pathBase);
            inv = 1.0f / (float)n;
            tile_pixel(wp, t, lp, x, y);
        } else {
            wave_pixel(wp, pix, x, y);
        }
        // with a split, the image holds the first splitSpp samples, image2 the rest
        const uint32_t nFirst = wp.splitSpp ? wp.splitSpp : n;
        if (wp.splitSpp) inv = 1.0f / (float)nFirst;
        CSum acc[3] = {{0, 0}, {0, 0}, {0, 0}};
        for (uint32_t s = 0; s < nFirst; s++) {
            float4 r = wb.pathRad[first + s];
            if (isnan(r.x) || isnan(r.y) || isnan(r.z)) {
                nans++;
                if (wp.nanPolicy == GBSP_NAN_ZERO) continue;
            }
            csum_add(acc[0], r.x * inv);
            csum_add(acc[1], r.y * inv);
            csum_add(acc[2], r.z * inv);
        }
        image[(size_t)y * imageWidth + x] =
            make_float4(csum_value(acc[0]), csum_value(acc[1]), csum_value(acc[2]), 1.0f);
        if (wp.splitSpp) {
            const float inv2 = 1.0f / (float)(n - nFirst);
            CSum acc2[3] = {{0, 0}, {0, 0}, {0, 0}};
            for (uint32_t s = nFirst; s < n; s++) {
                float4 r = wb.pathRad[first + s];
                if (isnan(r.x) || isnan(r.y) || isnan(r.z)) {
                    nans++;
                    if (wp.nanPolicy == GBSP_NAN_ZERO) continue;
                }
                csum_add(acc2[0], r.x * inv2);
                csum_add(acc2[1], r.y * inv2);
                csum_add(acc2[2], r.z * inv2);
            }
            wp.image2[(size_t)y * imageWidth + x] =
                make_float4(csum_value(acc2[0]), csum_value(acc2[1]), csum_value(acc2[2]), 1.0f);
        }
        if (wp.aovImage) {
            float4 a = make_float4(0, 0, 0, 0), b = make_float4(0, 0, 0, 0);
            for (uint32_t s = 0; s < nFirst; s++) {
                float4 u = wb.pathAov[2 * (first + s)];
                float4 v = wb.pathAov[2 * (first + s) + 1];
                a = make_float4(a.x + u.x, a.y + u.y, a.z + u.z, a.w + u.w);
                b = make_float4(b.x + v.x, b.y + v.y, b.z + v.z, b.w + v.w);
            }
            float is = inv;
            size_t o = 2 * ((size_t)y * imageWidth + x);
            wp.aovImage[o] = make_float4(a.x * is, a.y * is, a.z * is, a.w * is);
            wp.aovImage[o + 1] = make_float4(b.x * is, b.y * is, b.z * is, b.w * is);
        }
    }
    for (int off = 16; off; off >>= 1) nans += __shfl_xor_sync(0xFFFFFFFFu, nans, off);
    if ((threadIdx.x & 31) == 0 && nans)
        atomicAdd(&counters[GBSP_METRIC_NAN_SAMPLES], (unsigned long long)nans);
}

// Persistent grid of k_shade: every block an SM can hold (the kernel waits on
// scattered loads, so more resident warps hide more of that latency).
template <class Src>
int shade_grid(int smCount)
{
    static int perSm = 0;
    if (perSm == 0) {
        int n = 0;
        if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, k_shade<Src>, kShadeThreads, 0) !=
                cudaSuccess || n < 1)
            n = 8;
        perSm = n;
    }
    return smCount * perSm;
}

// Persistent grid of the closest-hit kernel launch_trace_stage picks: every
// block the SMs hold at once (blocks beyond that would only start once others
// have drained the queue).
template <class K>
int resident_blocks_per_sm(K kernel)
{
    int n = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, kernel, 128, 0) != cudaSuccess || n < 1)
        n = 6;
    return n;
}

template <class Src, int kQ>
int trace_grid_of(bool perLane, bool watertight, int smCount)
{
    static const int lane[2] = {resident_blocks_per_sm(k_trace_lane<Src, false, kQ>),
        resident_blocks_per_sm(k_trace_lane<Src, true, kQ>)};
    static const int warp[2] = {resident_blocks_per_sm(k_trace<Src, false, kQ>),
        resident_blocks_per_sm(k_trace<Src, true, kQ>)};
    return smCount * (perLane ? lane[watertight ? 1 : 0] : warp[watertight ? 1 : 0]);
}

// quads: the node width every scene of the launch uses (2: 8-wide, 1: 4-wide), 0: mixed
template <class Src>
int trace_grid(bool perLane, bool watertight, uint32_t quads, int smCount)
{
    return quads == 2 ? trace_grid_of<Src, 2>(perLane, watertight, smCount)
                      : trace_grid_of<Src, 0>(perLane, watertight, smCount);
}

template <class Src, bool kWT, int kQ>
void launch_trace_kernel(bool perLane, int grid, cudaStream_t s, const Src &src, const float4 *qO,
    const float4 *qD, const unsigned int *queueCount, int4 *hitA, int *hitInst, unsigned int *ctl,
    unsigned long long *counters, uint32_t *status)
{
    if (perLane)
        launch_next(k_trace_lane<Src, kWT, kQ>, grid, kLaneThreads, s, src, qO, qD, queueCount, hitA,
            hitInst, ctl, counters, status);
    else
        launch_next(k_trace<Src, kWT, kQ>, grid, 128, s, src, qO, qD, queueCount, hitA, hitInst, ctl,
            counters, status);
}

// Launches the closest-hit kernel of one bounce: per-warp or per-lane
// scheduling, reference MT or watertight triangle test, 8-wide nodes or a
// width read from the scene (template arguments, so no choice costs another
// anything).
template <class Src>
void launch_trace_stage(bool perLane, bool watertight, uint32_t quads, int grid, cudaStream_t s,
    const Src &src, const float4 *qO, const float4 *qD, const unsigned int *queueCount, int4 *hitA,
    int *hitInst, unsigned int *ctl, unsigned long long *counters, uint32_t *status)
{
    auto launch = quads == 2 ? (watertight ? launch_trace_kernel<Src, true, 2>
                                           : launch_trace_kernel<Src, false, 2>)
                             : (watertight ? launch_trace_kernel<Src, true, 0>
                                           : launch_trace_kernel<Src, false, 0>);
    launch(perLane, grid, s, src, qO, qD, queueCount, hitA, hitInst, ctl, counters, status);
}

}  // namespace gbsp
