// Batched closest-hit ray casting (config 2 and sp_RayIntersectScene batches).
//
// Small batches: k_intersect, one launch that takes the rays, walks them and
// writes the outputs.  Large batches of (typically incoherent) rays go through
// the wavefront's per-lane closest-hit kernel instead, where a lane fetches its
// next ray as soon as its current one is done: the rays are split into the
// queue layout, traced, and the queue-ordered hits turned into the requested
// outputs, three chained launches.

#include <algorithm>

#include "gbsp_internal.h"
#include "traverse.cuh"
#include "wavefront.cuh"

namespace gbsp {

constexpr int kWarpsPerSm = 7;  // k_intersect, see there


struct QueryOutputs {
    float *t;
    int32_t *tri, *obj;
    float *attr;  // 6 per ray: t, normal, uv
    uint32_t *mat;
};

__device__ __forceinline__ void write_outputs(const SceneView &sv, const RayHit &h, uint32_t i,
    const QueryOutputs &out)
{
    const bool hit = h.prim >= 0;
    if (out.t) out.t[i] = hit ? h.t : -1.0f;
    if (out.tri) out.tri[i] = hit ? (int32_t)__ldg(sv.triIds + h.prim) : -1;
    const Instance *in = hit ? sv.instances + h.inst : nullptr;
    if (out.obj) out.obj[i] = hit ? (int32_t)__ldg(&in->objectIndex) : -1;
    if (out.attr) {
        float *a = out.attr + 6 * (size_t)i;
        if (hit) {
            V3 n;
            float ux, uy;
            hit_surface(sv, h, n, ux, uy);
            a[0] = h.t;
            a[1] = n.x;
            a[2] = n.y;
            a[3] = n.z;
            a[4] = ux;
            a[5] = uy;
        } else {
            a[0] = -1.0f;
            a[1] = a[2] = a[3] = a[4] = a[5] = 0.0f;
        }
    }
    if (out.mat) out.mat[i] = hit ? __ldg(&in->materialId) : 0u;
}

// Ray i of a batch: (origin, pad, direction, pad) float4 pairs, or six packed
// floats as the host API takes them (4-byte aligned).
template <bool kPacked>
__device__ __forceinline__ void load_ray(const float *rays, size_t i, V3 &o, V3 &d)
{
    if (kPacked) {
        const float *r = rays + 6 * i;
        o = v3(__ldg(r), __ldg(r + 1), __ldg(r + 2));
        d = v3(__ldg(r + 3), __ldg(r + 4), __ldg(r + 5));
    } else {
        const float4 *r = reinterpret_cast<const float4 *>(rays) + 2 * i;
        const float4 a = __ldg(r), b = __ldg(r + 1);
        o = v3(a.x, a.y, a.z);
        d = v3(b.x, b.y, b.z);
    }
}

// One ray per lane, `lanes` lanes of a warp.
//
// Bound: the latency of the longest walk, and the host around it.  Up to 7
// warps per SM share a batch before a warp takes a second ray.  4,096, 20,011
// and 65,535 rays against 24 spheres of 1,280 triangles: 27.2, 34.9 and 38.9 us
// on the device (39.2, 40.9 and 43.9 with full warps taken from a counter and
// general node visits); at 4 warps per SM 30.0, 40.4 and 41.3, at 14 27.1, 35.8
// and 40.2, at 28 37.4, 44.6 and 45.6 us.  The per-lane path's three launches
// cost 35 us for one ray where this takes 8.
// 7 blocks per SM (72 registers) are for 8-wide nodes; walks of a width read from the
// scene take 88 to 92 without a bound: 40,000 watertight rays over 4-wide nodes
// 50.2 us with it, 48.5 without.
template <bool kWT, int kQ, bool kPacked>
__global__ void __launch_bounds__(128, kQ == 2 ? 7 : 1) k_intersect(SceneView sv, const float *__restrict__ rays,
    uint32_t count, uint32_t lanes, QueryOutputs out, unsigned long long *counters, uint32_t *status)
{
    const uint32_t lane = threadIdx.x & 31, warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const uint32_t i = warp * lanes + lane;
    TraceCounters cnt = {0, 0, 0, 0, 0};
    uint32_t done = 0, hits = 0;
    if (lane < lanes && i < count) {
        V3 o, d;
        load_ray<kPacked>(rays, i, o, d);
        const RayHit h = trace_closest<true, kWT, kQ>(sv, o, d, status, cnt);
        write_outputs(sv, h, i, out);
        done = 1;
        hits = h.prim >= 0 ? 1u : 0u;
    }
    __syncwarp();
    uint32_t v[7] = {done, hits, cnt.topNodes, cnt.meshNodes, cnt.triTests, cnt.boxTests, cnt.meshTests};
#pragma unroll
    for (int k = 0; k < 7; k++) v[k] = __reduce_add_sync(0xFFFFFFFFu, v[k]);
    if (lane == 0 && v[0]) {
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

// Rays -> queue layout (origin with path id 0, direction).
template <bool kPacked>
__global__ void __launch_bounds__(256) k_split_rays(const float *__restrict__ rays, uint32_t count,
    float4 *__restrict__ qo, float4 *__restrict__ qd, unsigned int *ctl)
{
    uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i == 0) reset_wave_ctl(ctl, count);
    if (i >= count) return;
    V3 o, d;
    load_ray<kPacked>(rays, i, o, d);
    qo[i] = make_float4(o.x, o.y, o.z, 0.0f);
    qd[i] = make_float4(d.x, d.y, d.z, 0.0f);
}

// Queue-ordered hits -> the per-ray outputs asked for.
__global__ void __launch_bounds__(256) k_intersect_outputs(SceneView sv, const int4 *hitA,
    const int *hitInst, uint32_t count, QueryOutputs out)
{
    stage_begin();
    uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= count) return;
    int4 hA = hitA[i];
    RayHit h;
    h.t = __int_as_float(hA.x);
    h.u = __int_as_float(hA.y);
    h.v = __int_as_float(hA.z);
    h.prim = hA.w;
    h.inst = hitInst[i];
    write_outputs(sv, h, i, out);
}

// Batches from this size on take the per-lane path (which counts as hits those
// in front of the origin only, as frames do): it is the faster one where many
// rays per lane differ in length, 2^20 rays against 2^18 triangles, and costs
// two launches more, 55 against 39 us at this size on the scene above.
constexpr uint32_t kPerLaneBatch = 1u << 16;

template <bool kPacked>
static int launch_small(cudaStream_t s, const SceneView &sv, uint32_t count, const float *rays,
    const QueryOutputs &out, int smCount, unsigned long long *counters, uint32_t *status)
{
    auto kern = sv.nodeQuads == 2 ? (sv.watertight ? k_intersect<true, 2, kPacked> : k_intersect<false, 2, kPacked>)
                                  : (sv.watertight ? k_intersect<true, 0, kPacked> : k_intersect<false, 0, kPacked>);
    const uint32_t warps = (uint32_t)smCount * kWarpsPerSm;
    const uint32_t lanes = std::min(32u, (count + warps - 1) / warps);
    const uint32_t used = (count + lanes - 1) / lanes;
    kern<<<(used + 3) / 4, 128, 0, s>>>(sv, rays, count, lanes, out, counters, status);
    GBSP_CUDA_TRY(cudaGetLastError());
    return GBSP_OK;
}

int launch_intersect(gbsp_runtime *rt, const SceneView &sv, uint32_t count, const float *rays, bool packed,
    float *tOut, int32_t *triOut, int32_t *objOut, float *attrOut, uint32_t *matOut)
{
    if (!count) return GBSP_OK;
    cudaStream_t s = rt->stream;
    const bool watertight = sv.watertight != 0;
    if (count < kPerLaneBatch) {
        const QueryOutputs out = {tOut, triOut, objOut, attrOut, matOut};
        auto launch = packed ? launch_small<true> : launch_small<false>;
        return launch(s, sv, count, rays, out, rt->smCount, rt->dCounters, rt->dStatus);
    }
    // One block holds a piece of the batch: origins, directions, hits (16 bytes each),
    // object ids, and the queue's control words, so that a call shares nothing with a
    // render but the metrics.  A call that is being captured brings its own block: a
    // graph must not refer to one that a later call may replace.
    const size_t ctlQuads = kCtlCount * sizeof(unsigned int) / sizeof(float4);
    const auto quads_for = [&](size_t n) { return 3 * n + (n + 3) / 4 + ctlQuads; };
    const size_t most = (kQueueKeep / sizeof(float4) - ctlQuads - 1) * 4 / 13;
    const size_t pieces = (count + most - 1) / most, piece = (count + pieces - 1) / pieces;
    cudaStreamCaptureStatus capture = cudaStreamCaptureStatusNone;
    GBSP_CUDA_TRY(cudaStreamIsCapturing(s, &capture));
    std::lock_guard<std::mutex> lock(rt->queryLaunch);
    DeviceBuffer<float4> ownQueue;
    DeviceBuffer<float4> &queue = capture != cudaStreamCaptureStatusNone ? ownQueue : rt->queryQueue;
    if (int rc = queue.reserve(quads_for(piece), s)) return rc;
    OneScene one = {};
    one.sv = sv;
    for (size_t first = 0; first < count; first += piece) {
        const uint32_t n = (uint32_t)std::min<size_t>(piece, count - first);
        float4 *o = queue.ptr, *d = o + n;
        int4 *hits = reinterpret_cast<int4 *>(d + n);
        int *inst = reinterpret_cast<int *>(hits + n);
        unsigned int *ctl = reinterpret_cast<unsigned int *>(queue.ptr + quads_for(n) - ctlQuads);
        const QueryOutputs at = {tOut ? tOut + first : nullptr, triOut ? triOut + first : nullptr,
            objOut ? objOut + first : nullptr, attrOut ? attrOut + 6 * first : nullptr,
            matOut ? matOut + first : nullptr};
        const int blocks = (int)((n + 255) / 256);
        (packed ? k_split_rays<true> : k_split_rays<false>)<<<blocks, 256, 0, s>>>(
            rays + (packed ? 6 : 8) * first, n, o, d, ctl);
        launch_trace_stage(true, watertight, sv.nodeQuads,
            trace_grid<OneScene>(true, watertight, sv.nodeQuads, rt->smCount), s, one, o, d,
            ctl + queue_word(0), hits, inst, ctl, rt->dCounters, rt->dStatus);
        launch_next(k_intersect_outputs, blocks, 256, s, sv, hits, inst, n, at);
    }
    GBSP_CUDA_TRY(cudaGetLastError());
    return GBSP_OK;
}

}  // namespace gbsp
