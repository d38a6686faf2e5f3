// Learned denoiser kernels: a kernel-predicting CNN (8 conv3x3 layers of 48
// channels, ReLU, a 5x5 per-pixel filter from a softmax over 25 logits),
// trained on pairs of low-spp frames (radiance + albedo, normal, depth
// G-buffers) and high-spp targets rendered by this path tracer.  No
// reference counterpart: vk_cinematic has no denoiser.
//
// Tensors are NHWC.  Activations and weights are BF16, accumulation FP32.
//  * conv3x3 forward / data gradient: implicit GEMM on the tensor cores,
//    M = pixels, N = output channels, K = 9 taps x input channels, with
//    mma.sync m16n8k16 BF16.  CTAs are persistent: each loads the layer's
//    weights into shared memory once (padded rows, conflict-free fragment
//    loads) and then walks 64-pixel row segments.
//  * weight gradient: FP32 outer products over pixel chunks, one tap per
//    CTA, reduced with atomics.
//  * filter, loss and Adam: elementwise FP32.

#include <cstdint>

#include <cuda.h>
#include <cuda_bf16.h>
#include <cudaTypedefs.h>
#include <algorithm>
#include <atomic>
#include <mutex>

#include "gbsp_internal.h"
#include "launch.cuh"

namespace gbsp {
namespace dn {

constexpr int kTileP = 64;   // pixels per row segment
constexpr int kThreads = 128;

__device__ __forceinline__ void mma_bf16_16816(float *c, uint32_t a0, uint32_t a1, uint32_t a2,
    uint32_t a3, uint32_t b0, uint32_t b1)
{
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 "
        "{%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

__device__ __forceinline__ uint32_t pack_bf16(float lo, float hi)
{
    __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<uint32_t *>(&v);
}

// Activations and their gradients use a channel-group-planar layout,
// [B][H][C/8][W][8]: each 8-channel group of an image row is a contiguous
// plane of W x 16 bytes (BF16), so that a row segment's pixels are one
// contiguous read per group.  Element (row = b H + y, x, c):
__device__ __forceinline__ size_t cg_index(size_t row, int x, int c, int W, int C)
{
    return ((row * (size_t)(C / 8) + (size_t)(c / 8)) * (size_t)W + (size_t)x) * 8 + (size_t)(c % 8);
}

// 3: FP32 logits + bias fed straight into the 5x5 kernel-prediction filter
// 4: data gradient times the ReLU mask of the activations it is taken at, BF16
// (apart, the FP32 gradient went through memory twice: 32 + 49 us per 48 -> 48
// layer of a 16 x 128^2 batch, 27 us in one)
enum Epilogue : int { kEpiBf16BiasRelu = 0, kEpiF32Bias = 1, kEpiF32 = 2, kEpiFilter = 3, kEpiReluGrad = 4 };

// out[p][co] = sum_{tap, ci} in[p + off(tap)][ci] * w[tap][co][ci] (+ bias, ReLU)
template <int CIN, int COUT, int EPI>
__global__ void __launch_bounds__(kThreads) k_conv3x3(const __nv_bfloat16 *__restrict__ in, int B,
    int H, int W, const __nv_bfloat16 *__restrict__ w, const float *__restrict__ bias,
    __nv_bfloat16 *__restrict__ outB, float *__restrict__ outF)
{
    static_assert(CIN % 16 == 0 && COUT % 8 == 0, "channel padding");
    constexpr int SIN = CIN + 8;  // padded element stride per pixel (bank-conflict free)
    constexpr int SPX = kTileP + 2;
    extern __shared__ __align__(128) unsigned char smemRaw[];
    __nv_bfloat16 *sW = reinterpret_cast<__nv_bfloat16 *>(smemRaw);   // [9][COUT][SIN]
    __nv_bfloat16 *sIn = sW + 9 * COUT * SIN;                          // [3][SPX][SIN]
    const int tid = threadIdx.x;
    for (int i = tid; i < 9 * COUT * (CIN / 2); i += kThreads) {
        int row = i / (CIN / 2), c2 = i % (CIN / 2);
        reinterpret_cast<uint32_t *>(sW + row * SIN)[c2] =
            reinterpret_cast<const uint32_t *>(w)[(size_t)row * (CIN / 2) + c2];
    }
    const int warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
    const int tilesPerRow = (W + kTileP - 1) / kTileP;
    const int numTiles = tilesPerRow * B * H;
    for (int tile = blockIdx.x; tile < numTiles; tile += gridDim.x) {
        const int row = tile / tilesPerRow;  // b * H + y
        const int x0 = (tile % tilesPerRow) * kTileP;
        const int b = row / H, y = row % H;
        __syncthreads();  // previous tile's reads of sIn are done (and sW is loaded)
        for (int i = tid; i < 3 * SPX * (CIN / 2); i += kThreads) {
            int c2 = i % (CIN / 2);
            int px = (i / (CIN / 2)) % SPX;
            int ry = i / ((CIN / 2) * SPX);
            int gy = y + ry - 1, gx = x0 + px - 1;
            uint32_t v = 0;
            if (gy >= 0 && gy < H && gx >= 0 && gx < W)
                v = reinterpret_cast<const uint32_t *>(in)[cg_index((size_t)(b * H + gy), gx, 2 * c2, W, CIN) / 2];
            reinterpret_cast<uint32_t *>(sIn + (ry * SPX + px) * SIN)[c2] = v;
        }
        __syncthreads();
        float acc[COUT / 8][4];
#pragma unroll
        for (int n = 0; n < COUT / 8; n++) acc[n][0] = acc[n][1] = acc[n][2] = acc[n][3] = 0.0f;
        const int m0 = warp * 16;
#pragma unroll 1
        for (int tap = 0; tap < 9; tap++) {
            const int ty = tap / 3, tx = tap % 3;
            const __nv_bfloat16 *aBase = sIn + (ty * SPX + m0 + tx) * SIN;
            const __nv_bfloat16 *bBase = sW + tap * COUT * SIN;
#pragma unroll
            for (int kc = 0; kc < CIN; kc += 16) {
                uint32_t a0 = *reinterpret_cast<const uint32_t *>(aBase + g * SIN + kc + 2 * t);
                uint32_t a1 = *reinterpret_cast<const uint32_t *>(aBase + (g + 8) * SIN + kc + 2 * t);
                uint32_t a2 = *reinterpret_cast<const uint32_t *>(aBase + g * SIN + kc + 2 * t + 8);
                uint32_t a3 = *reinterpret_cast<const uint32_t *>(aBase + (g + 8) * SIN + kc + 2 * t + 8);
#pragma unroll
                for (int n = 0; n < COUT / 8; n++) {
                    const __nv_bfloat16 *bp = bBase + (n * 8 + g) * SIN + kc + 2 * t;
                    uint32_t b0 = *reinterpret_cast<const uint32_t *>(bp);
                    uint32_t b1 = *reinterpret_cast<const uint32_t *>(bp + 8);
                    mma_bf16_16816(acc[n], a0, a1, a2, a3, b0, b1);
                }
            }
        }
        // epilogue: rows g and g+8 of the warp's slab, columns 2t, 2t+1 of each n tile
#pragma unroll
        for (int half = 0; half < 2; half++) {
            int x = x0 + m0 + g + 8 * half;
            if (x >= W) continue;
            size_t p = (size_t)row * W + x;  // logits (FP32, NHWC)
#pragma unroll
            for (int n = 0; n < COUT / 8; n++) {
                int co = n * 8 + 2 * t;
                float v0 = acc[n][2 * half], v1 = acc[n][2 * half + 1];
                if (EPI != kEpiF32) {
                    v0 += bias[co];
                    v1 += bias[co + 1];
                }
                if (EPI == kEpiBf16BiasRelu) {
                    v0 = fmaxf(v0, 0.0f);
                    v1 = fmaxf(v1, 0.0f);
                    reinterpret_cast<uint32_t *>(outB)[cg_index(row, x, co, W, COUT) / 2] =
                        pack_bf16(v0, v1);
                } else if (EPI == kEpiF32Bias) {
                    *reinterpret_cast<float2 *>(outF + p * COUT + co) = make_float2(v0, v1);
                } else {
                    *reinterpret_cast<float2 *>(outF + cg_index(row, x, co, W, COUT)) =
                        make_float2(v0, v1);
                }
            }
        }
    }
}

template <int CIN, int COUT, int EPI>
int launch_conv(cudaStream_t s, int smCount, const void *in, int B, int H, int W, const void *w,
    const float *bias, void *outB, float *outF)
{
    constexpr int SIN = CIN + 8;
    size_t smem = (size_t)(9 * COUT + 3 * (kTileP + 2)) * SIN * 2;
    auto kern = k_conv3x3<CIN, COUT, EPI>;
    GBSP_CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    int tiles = ((W + kTileP - 1) / kTileP) * B * H;
    int grid = smCount * 3;
    if (grid > tiles) grid = tiles;
    kern<<<grid, kThreads, smem, s>>>(reinterpret_cast<const __nv_bfloat16 *>(in), B, H, W,
        reinterpret_cast<const __nv_bfloat16 *>(w), bias, reinterpret_cast<__nv_bfloat16 *>(outB),
        outF);
    GBSP_CUDA_TRY(cudaGetLastError());
    return GBSP_OK;
}

// ---------------------------------------------------------------------------
// conv3x3 on the 5th-generation tensor cores (tcgen05).
//
// GEMM: M = 128 pixels of one image row, K = 9 taps x CIN, and the G =
// kTcGroupRows output rows y .. y + G - 1 of a group side by side along N
// (row y + j in accumulator columns [j COUT, (j + 1) COUT)).  One elected
// thread issues tcgen05.mma.cta_group::1.kind::f16 (BF16 x BF16 -> FP32) per
// (input row, horizontal tap, 16-channel slice): input row y - 1 + k feeds
// every output row j of the group with k - j in 0..2 at once, with the
// matching tap rows of the [ty 2 | ty 1 | ty 0] weight stack as a
// contiguous B slice (N = COUT, 2 COUT or 3 COUT).  An M = 128 MMA costs
// about the same up to N = 96 and runs at the dense rate from N = 128, so
// G = 4 takes 6 instead of 12 MMAs per (tap, slice) for 4 rows.  Both
// operands are read straight from shared memory through matrix descriptors,
// so the 3x3 neighbourhood is never expanded: a horizontal tap is a
// 16-byte-granular offset of the A descriptor into a staged input row.
//
// Shared memory holds the operands in the canonical no-swizzle K-major
// layout: 8 x 16-byte core matrices (8 rows of 8 BF16 channels), rows
// contiguous.  Input rows: ring slots of two rows, each [CIN/8 channel
// groups][kTcSpx pixels][16 B] (a core matrix = 8 consecutive pixels of one
// channel group, so a pixel shift moves the start by 16 B); weights: [3
// taps][CIN/8 groups][3 tap rows x COUT][16 B].  Descriptor strides: leading
// (K) = next channel group, stride (M or N) = next 8 rows = 128 B.
//
// One persistent CTA per SM walks vertical strips (one 128-pixel column
// segment, a run of rows) with its warps specialised and coupled only by
// mbarriers:
//   * warp 1 (producer) loads input rows in pairs into a ring of kTcRing slots,
//     one lane per channel plane of a pair (cp.async.bulk of the plane's 130
//     pixels, one contiguous run of the planar layout; pixels outside the image
//     are zeroed by the warp), as many pairs in flight as the ring allows; a
//     pair lands on its rowFull barrier by transaction count, and its slot is
//     reused once the MMAs of the last row group that reads it have completed
//     (rowEmpty, signalled by tcgen05.commit);
//   * lane 0 of warp 0 issues, per group of kTcGroupRows output rows, the
//     (kTcGroupRows + 2) x 3 x CIN/16 MMAs reading its input rows into one
//     TMEM accumulator, then commits to that accumulator's accFull and to the
//     rowEmpty of the input rows no later group reads;
//   * warps 4-11 are two epilogue groups taking alternate row groups (warp
//     w owns TMEM lanes 32 (w % 4) .. + 31 = pixels): wait on accFull, read
//     the accumulator with tcgen05.ld, apply bias / ReLU / BF16 packing (or
//     the fused filter), and release it on accEmpty, while the tensor core
//     already works on the next group.
// Every wait is bounded; a timeout raises a shared abort flag that ends the
// other roles' waits, and sets g_dnStatus.
//
// What bounds it (48 -> 48 at 1080p, 85.9 GFLOP, 398 MB in and out): memory, 69
// us by itself = 5.8 TB/s (79 before strip_rows), with the MMAs behind it (54 per
// row group, of about 70 cycles each: 49 us).  Before, 99 us: the issuing thread
// waited on six row barriers per group at about 340 cycles each, none of it hidden
// (without loads, stores and
// eight ninths of the MMAs 47 us; with one wait per group 29); and TMA boxes of
// [group][130 pixels][8 channels] move 16 bytes per request (loads alone 60
// us, 49 as runs).  Two epilogue groups per accumulator: 79 us, the same.
// ---------------------------------------------------------------------------
constexpr int kTcTileP = 128;
// One CTA per SM: warp 0 issues the MMAs, warp 1 loads rows (a lane per channel plane
// of a row pair), warps 4-11 are two epilogue groups that take alternate row groups.
constexpr int kTcThreads = 384;
constexpr int kTcEpiGroups = 2;
constexpr int kTcAccSlots = 4;  // at most; accumulator a is drained by epilogue group a % 2
constexpr int kTcSpx = kTcTileP + 2;     // staged pixels per row: x0 - 1 .. x0 + 128
constexpr int kTcGroupRows = 4;  // output rows per accumulator
// Input rows travel in pairs: one full and one empty barrier per two rows.  A row
// group reads three pairs, two of them new, so its issuing thread waits twice for
// rows and releases two slots.
constexpr int kTcRing = 7;  // row pairs in shared memory: 3 read by a group's MMAs, the rest in flight
constexpr uint32_t kTcWaitLimit = 1u << 26;

__device__ uint32_t g_dnStatus;

__device__ __forceinline__ uint32_t smem_u32(const void *p)
{
    return (uint32_t)__cvta_generic_to_shared(p);
}

// Bounded mbarrier wait (at most kTcWaitLimit polls and kTcWaitNs of
// wall time) that also gives up when another role has aborted.
constexpr uint64_t kTcWaitNs = 2000000000ull;

__device__ __forceinline__ uint64_t global_ns()
{
    uint64_t t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

__device__ __forceinline__ bool tc_wait(uint32_t bar, uint32_t parity, volatile uint32_t *abortFlag)
{
    const uint64_t t0 = global_ns();
    for (uint32_t it = 0; it < kTcWaitLimit; it++) {
        uint32_t done;
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}"
            : "=r"(done) : "r"(bar), "r"(parity) : "memory");
        if (done) return true;
        if (*abortFlag) return false;
        if ((it & 255u) == 255u && global_ns() - t0 > kTcWaitNs) break;
    }
    *abortFlag = 1u;
    return false;
}

__device__ __forceinline__ void mbar_arrive(uint32_t bar)
{
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" :: "r"(bar) : "memory");
}

__device__ __forceinline__ void tc_commit(uint32_t bar)
{
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];"
                 :: "r"(bar) : "memory");
}

// Shared-memory matrix descriptor: start >> 4 (bits 0-13), leading-dimension
// byte offset >> 4 (16-29), stride-dimension byte offset >> 4 (32-45),
// descriptor version 1 (bits 46-47), base offset 0, no swizzle (bits 61-63 = 0).
__device__ __forceinline__ uint64_t smem_desc(uint32_t addr, uint32_t lbo, uint32_t sbo)
{
    return (uint64_t)((addr & 0x3FFFFu) >> 4) | ((uint64_t)((lbo >> 4) & 0x3FFFu) << 16) |
        ((uint64_t)((sbo >> 4) & 0x3FFFu) << 32) | (1ull << 46);
}

// Instruction descriptor of kind::f16: D FP32 (bits 4-5 = 1), A and B BF16
// (bits 7-9 = 1, 10-12 = 1), both K-major, N >> 3 at bits 17-22, M >> 4 at 24-28.
template <int M, int N>
__device__ __forceinline__ uint32_t instr_desc_bf16()
{
    return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(N >> 3) << 17) |
        ((uint32_t)(M >> 4) << 24);
}

__device__ __forceinline__ void softmax25(const float *l, float *w)
{
    float m = l[0];
#pragma unroll
    for (int k = 1; k < 25; k++) m = fmaxf(m, l[k]);
    float s = 0.0f;
#pragma unroll
    for (int k = 0; k < 25; k++) {
        w[k] = __expf(l[k] - m);
        s += w[k];
    }
    float inv = 1.0f / s;
#pragma unroll
    for (int k = 0; k < 25; k++) w[k] *= inv;
}

__device__ __forceinline__ uint64_t tap_pixel(uint64_t p, int x, int y, int W, int H, int k)
{
    int gx = min(max(x + k % 5 - 2, 0), W - 1), gy = min(max(y + k / 5 - 2, 0), H - 1);
    return p - (uint64_t)x - (uint64_t)y * W + (uint64_t)gy * W + gx;
}

// 16 consecutive FP32 accumulator columns of this thread's TMEM lane.
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t (&r)[16])
{
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
        "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
          "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]),
          "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr));
}

// One tcgen05.mma.cta_group::1.kind::f16 (BF16 x BF16 -> FP32 in tensor
// memory); accumulate = 0 overwrites the accumulator.
__device__ __forceinline__ void tc_mma(uint32_t dTmem, uint64_t aDesc, uint64_t bDesc,
    uint32_t idesc, uint32_t accumulate)
{
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
        :: "r"(dTmem), "l"(aDesc), "l"(bDesc), "r"(idesc), "r"(accumulate));
}

// Bias / ReLU / BF16 packing of one pixel's COUT accumulators and the store:
// BF16 activations and FP32 gradients channel-group-planar, FP32 logits NHWC.
template <int COUT, int EPI>
__device__ __forceinline__ void conv_store(const uint32_t (&r)[COUT], size_t row, int x, int W,
    const float *__restrict__ bias, __nv_bfloat16 *__restrict__ outB, float *__restrict__ outF,
    const uint4 (&act)[COUT / 8])
{
#pragma unroll
    for (int c = 0; c < COUT; c += 8) {
        float v[8];
        const __nv_bfloat16 *a = reinterpret_cast<const __nv_bfloat16 *>(&act[c / 8]);
#pragma unroll
        for (int k = 0; k < 8; k++) {
            v[k] = __uint_as_float(r[c + k]);
            if (EPI == kEpiBf16BiasRelu || EPI == kEpiF32Bias) v[k] += bias[c + k];
            if (EPI == kEpiBf16BiasRelu) v[k] = fmaxf(v[k], 0.0f);
            if (EPI == kEpiReluGrad) v[k] = __bfloat162float(a[k]) > 0.0f ? v[k] : 0.0f;
        }
        if (EPI == kEpiBf16BiasRelu || EPI == kEpiReluGrad) {
            *reinterpret_cast<uint4 *>(outB + cg_index(row, x, c, W, COUT)) = make_uint4(
                pack_bf16(v[0], v[1]), pack_bf16(v[2], v[3]), pack_bf16(v[4], v[5]),
                pack_bf16(v[6], v[7]));
        } else {
            float4 *o = reinterpret_cast<float4 *>(
                EPI == kEpiF32Bias ? outF + (row * W + x) * COUT + c : outF + cg_index(row, x, c, W, COUT));
            o[0] = make_float4(v[0], v[1], v[2], v[3]);
            o[1] = make_float4(v[4], v[5], v[6], v[7]);
        }
    }
}

// Softmax of the 25 kernel logits (accumulators + bias) and the 5x5 filter of
// the noisy radiance around pixel p = (x, y): the same arithmetic as k_filter
// on stored logits, so the fused and unfused results are bit-identical.  The
// clamped columns and rows are computed once each (25 clamped tap indices had
// cost more than the filter: 160 -> 117 us at 1080p).  Loading the 25 taps
// ahead of the accumulators spills and was slower (129 us), as were twice the
// epilogue warps (129 us).  All of the filter's arithmetic and loads now cost 22
// of a whole inference's 548 us; four rows of a group sharing their taps 562
// (168 registers, spills), two rows 548.
template <int COUT>
__device__ __forceinline__ void conv_filter_store(const uint32_t (&r)[COUT], size_t p, int x, int y,
    int W, int H, const float *__restrict__ bias, const float4 *noisy, float4 *out)
{
    static_assert(COUT >= 25, "kernel logits");
    float wk[25];
#pragma unroll
    for (int k = 0; k < 25; k++) wk[k] = __uint_as_float(r[k]) + bias[k];
    softmax25(wk, wk);
    int dx[5];
#pragma unroll
    for (int i = 0; i < 5; i++) dx[i] = min(max(x + i - 2, 0), W - 1);
    const float4 *image = noisy + (p - (size_t)x - (size_t)y * W);
    float3 o = make_float3(0, 0, 0);
#pragma unroll
    for (int j = 0; j < 5; j++) {
        const float4 *line = image + (size_t)min(max(y + j - 2, 0), H - 1) * W;
#pragma unroll
        for (int i = 0; i < 5; i++) {
            const float4 c = line[dx[i]];
            o.x += wk[5 * j + i] * c.x;
            o.y += wk[5 * j + i] * c.y;
            o.z += wk[5 * j + i] * c.z;
        }
    }
    out[p] = make_float4(o.x, o.y, o.z, 1.0f);
}

// A chained kernel: what it reads may be what the launch before it writes, so
// no operand is __restrict__ or read with __ldg (launch.cuh).
template <int CIN, int COUT, int EPI>
__global__ void __launch_bounds__(kTcThreads, 1) k_conv3x3_tc(const __nv_bfloat16 *in, int B, int H, int W,
    int rowsPerStrip, int reverse, const __nv_bfloat16 *w, const float *bias, __nv_bfloat16 *outB,
    float *outF, const float4 *noisy, float4 *outFilt, const __nv_bfloat16 *act)
{
    constexpr int G = kTcGroupRows;
    static_assert(CIN % 16 == 0 && COUT % 16 == 0 && 3 * COUT <= 256, "tcgen05 tile shape");
    constexpr int KG = CIN / 8;  // 16-byte channel groups
    constexpr int ACC_COLS = G * COUT <= 128 ? 128 : 256;  // G output rows side by side
    static_assert(G * COUT <= ACC_COLS, "accumulator");
    // an even number of accumulators: accumulator a is always drained by epilogue group a % 2
    constexpr int SLOTS = 512 / ACC_COLS >= kTcAccSlots ? kTcAccSlots : 512 / ACC_COLS;
    static_assert(SLOTS % kTcEpiGroups == 0, "accumulator slots");
    constexpr int TMEM_COLS = 512;
    extern __shared__ __align__(128) unsigned char smemRaw[];
    uint4 *sW = reinterpret_cast<uint4 *>(smemRaw);  // [3][KG][3 COUT]
    // ring slots of [2 rows][KG][kTcSpx] 16-byte pixels, each slot 128-byte aligned
    constexpr uint32_t kRowUnits = (uint32_t)(KG * kTcSpx);  // 16-byte units
    constexpr uint32_t kSlotBytes = (2 * kRowUnits * 16 + 127) / 128 * 128;
    const uint32_t ringAddr = (smem_u32(sW + 9 * KG * COUT) + 127u) & ~127u;
    __shared__ __align__(8) uint64_t rowFull[kTcRing], rowEmpty[kTcRing];
    __shared__ __align__(8) uint64_t accFull[SLOTS], accEmpty[SLOTS], drain;
    __shared__ uint32_t tmemBase;
    __shared__ volatile uint32_t abortFlag;
    __shared__ __align__(16) float sBias[COUT];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
                     :: "r"(smem_u32(&tmemBase)), "r"(TMEM_COLS));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    if (tid == 0) {
        for (int i = 0; i < kTcRing; i++) {
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" :: "r"(smem_u32(&rowFull[i])));
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" :: "r"(smem_u32(&rowEmpty[i])));
        }
        for (int i = 0; i < SLOTS; i++) {
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" :: "r"(smem_u32(&accFull[i])));
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 128;" :: "r"(smem_u32(&accEmpty[i])));
        }
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" :: "r"(smem_u32(&drain)));
        abortFlag = 0u;
        asm volatile("fence.mbarrier_init.release.cluster;");
    }
    asm volatile("tcgen05.fence::before_thread_sync;");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;");
    const uint32_t tmem = tmemBase;
    // Barriers and tensor memory are set up while the kernel before this one
    // drains: with it eight layers at 1080p take 626 us instead of 638, and a
    // training step of 16 crops of 128 x 128 496 instead of 545.  The producer
    // warp starts its rows without waiting for the other warps' weights; started
    // before its own share of them it cost 649 us at 1080p (488 a step).
    stage_begin();
    if (tid < COUT) sBias[tid] = EPI != kEpiF32 && EPI != kEpiReluGrad ? bias[tid] : 0.0f;
    // weights -> stacked canonical layout: block (tx, kg) holds 3 COUT rows of 16 B, the
    // tap rows ty = 2, 1, 0 one after the other, each row w[3 ty + tx][co][8 kg .. 8 kg + 7]
    for (int i = tid; i < 9 * KG * COUT; i += kTcThreads) {
        const int r = i % (3 * COUT), blk = i / (3 * COUT);
        const int kg = blk % KG, tx = blk / KG;
        const int ty = 2 - r / COUT, co = r % COUT;
        if (EPI == kEpiReluGrad) {
            // w holds the layer's forward weights [tap][CIN][COUT]: this convolution's are
            // w'[tap][co][ci] = w[8 - tap][ci][co] (neighbouring threads, neighbouring co)
            const uint16_t *src = reinterpret_cast<const uint16_t *>(w) +
                ((8 - 3 * ty - tx) * CIN + 8 * kg) * COUT + co;
            uint16_t e[8];
#pragma unroll
            for (int k = 0; k < 8; k++) e[k] = src[k * COUT];
            sW[i] = make_uint4(e[0] | (uint32_t)e[1] << 16, e[2] | (uint32_t)e[3] << 16,
                e[4] | (uint32_t)e[5] << 16, e[6] | (uint32_t)e[7] << 16);
        } else {
            sW[i] = reinterpret_cast<const uint4 *>(w)[((size_t)(3 * ty + tx) * COUT + co) * KG + kg];
        }
    }
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    if (warp == 1)
        asm volatile("bar.arrive 1, %0;" :: "n"(kTcThreads) : "memory");
    else
        asm volatile("bar.sync 1, %0;" :: "n"(kTcThreads) : "memory");

    const int segs = (W + kTcTileP - 1) / kTcTileP;
    const int stripsPerCol = (H + rowsPerStrip - 1) / rowsPerStrip;
    const int numStrips = B * segs * stripsPerCol;
    // strip geometry: segment origin x0, output rows [y0, y1) in P groups of G rows
    // (the last group may reach past the image); staged input rows y0 - 1 .. y0 + G P
#define GBSP_STRIP_GEOMETRY(strip)                                                       \
    const int st = reverse ? numStrips - 1 - (strip) : (strip);                     \
    const int sy = st % stripsPerCol, seg = (st / stripsPerCol) % segs;                  \
    const int b = st / (stripsPerCol * segs);                                             \
    const int x0 = seg * kTcTileP, y0 = sy * rowsPerStrip;                                \
    const int y1 = min(H, y0 + rowsPerStrip);                                             \
    const int P = (y1 - y0 + G - 1) / G;                                                  \
    (void)b;                                                                              \
    (void)x0;                                                                             \
    (void)y1

    if (warp == 0) {
        if (lane == 0) {
            // ---- MMA issue.  Input row gy of a strip has sequence number qBase + gy - y0 + 1.
            // Group (y .. y + G - 1) accumulates its G output rows side by side (row y + j in
            // columns [j COUT, (j + 1) COUT)).  Input row y - 1 + k feeds output rows
            // j = max(0, k - 2) .. min(G - 1, k) through tap rows ty = k - j: one MMA whose
            // B operand is the contiguous slice of the [ty 2 | ty 1 | ty 0] weight stack.
            uint32_t idesc[4];
            idesc[1] = instr_desc_bf16<kTcTileP, COUT>();
            idesc[2] = instr_desc_bf16<kTcTileP, 2 * COUT>();
            idesc[3] = instr_desc_bf16<kTcTileP, 3 * COUT>();
            const uint64_t aDesc0 = smem_desc(ringAddr, kTcSpx * 16, 128);
            const uint64_t bDesc0 = smem_desc(smem_u32(sW), 3 * COUT * 16, 128);
            // issue order per (tx, kc): k = 2 and k = G + 1 first (their outputs tile all G
            // rows, so they can start the accumulator), then the rest
            static_assert(G == 4, "issue order below is for groups of 4 rows");
            constexpr int kOrder[G + 2] = {2, 5, 0, 1, 3, 4};
            uint32_t groupCount = 0;
            uint32_t pos = 0;    // ring slot of the group's first row pair
            uint32_t phase = 0;  // parity of the next wait on each slot (bit per slot)
            bool ok = true;
            const auto next_slot = [](uint32_t v) { return v + 1u == (uint32_t)kTcRing ? 0u : v + 1u; };
            const auto wait_pair = [&](uint32_t slot) {
                const bool r = tc_wait(smem_u32(&rowFull[slot]), phase >> slot & 1u, &abortFlag);
                phase ^= 1u << slot;
                return r;
            };
            for (int strip = blockIdx.x; strip < numStrips && ok; strip += gridDim.x) {
                GBSP_STRIP_GEOMETRY(strip);
                ok = wait_pair(pos);
                for (int p = 0; p < P && ok; p++) {
                    // input rows y - 1 .. y + G: the pairs in slots pos, pos + 1 and pos + 2
                    // (from the bottom up when reversed)
                    const uint32_t slot1 = next_slot(pos), slot2 = next_slot(slot1);
                    ok = wait_pair(slot1);
                    ok = ok && wait_pair(slot2);
                    if (!ok) break;
                    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                    const uint32_t acc = groupCount % SLOTS, use = groupCount / SLOTS;
                    if (use > 0 && !tc_wait(smem_u32(&accEmpty[acc]), (use - 1u) & 1u, &abortFlag)) {
                        ok = false;
                        break;
                    }
                    asm volatile("tcgen05.fence::after_thread_sync;");
                    const uint32_t dAcc = tmem + acc * (uint32_t)ACC_COLS;
                    // A descriptors of the three pairs: only the low word's address field differs
                    const uint32_t aHi = (uint32_t)(aDesc0 >> 32);
                    const uint32_t top = reverse ? slot2 : pos, bottom = reverse ? pos : slot2;
                    const uint32_t aLo[3] = {(uint32_t)aDesc0 + top * (kSlotBytes / 16),
                        (uint32_t)aDesc0 + slot1 * (kSlotBytes / 16),
                        (uint32_t)aDesc0 + bottom * (kSlotBytes / 16)};
#pragma unroll
                    for (int tx = 0; tx < 3; tx++) {
#pragma unroll
                        for (int kc = 0; kc < CIN / 16; kc++) {
#pragma unroll
                            for (int o = 0; o < G + 2; o++) {
                                const int k = kOrder[o];
                                const int jlo = k - 2 > 0 ? k - 2 : 0, jhi = k < G - 1 ? k : G - 1;
                                // 16-byte units: row of the pair, channel group 2 kc, pixel tx
                                const uint64_t aDesc = (uint64_t)aHi << 32 |
                                    (aLo[k / 2] + (k % 2) * kRowUnits + 2 * kc * kTcSpx + tx);
                                // weight block (tx, 2 kc), starting at tap row ty = k - jlo
                                const uint64_t bDesc = bDesc0 +
                                    (uint64_t)((tx * KG + 2 * kc) * 3 * COUT + (2 - k + jlo) * COUT);
                                const uint32_t accumulate = (tx | kc) || o >= 2 ? 1u : 0u;
                                tc_mma(dAcc + (uint32_t)(jlo * COUT), aDesc, bDesc,
                                    idesc[jhi - jlo + 1], accumulate);
                            }
                        }
                    }
                    tc_commit(smem_u32(&accFull[acc]));
                    // the group's first two pairs have no later reader
                    tc_commit(smem_u32(&rowEmpty[pos]));
                    tc_commit(smem_u32(&rowEmpty[slot1]));
                    pos = slot2;
                    groupCount++;
                }
                if (!ok) break;
                // the strip's last row pair is free once its last MMAs finish
                tc_commit(smem_u32(&rowEmpty[pos]));
                pos = next_slot(pos);
            }
            // every MMA issued has finished before the accumulators are freed
            // (waited for even after an abort: the tensor memory is freed below)
            tc_commit(smem_u32(&drain));
            volatile uint32_t never = 0u;
            if (!tc_wait(smem_u32(&drain), 0u, &never)) abortFlag = 1u;
            if (!ok) abortFlag = 1u;
        }
        __syncwarp();
    } else if (warp < 4) {
        // ---- producer (warp 1): row pairs (y0 - 1, y0), ..., (y0 + G P - 1, y0 + G P) of
        // every strip.  Lane l copies plane l % KG of row l / KG of a pair: its pixels
        // x0 - 1 .. x0 + 128 are one contiguous run of the planar layout, so the copy is one
        // cp.async.bulk of up to 2,080 bytes; what lies outside the image is zeroed by the
        // warp before the pair's barrier is armed.
        if (warp == 1) {
            constexpr int kPlanes = 2 * KG;
            static_assert(kPlanes <= 32, "a lane per plane");
            uint32_t q = 0, slot = 0, use = 0;  // row pair q goes to slot q % kTcRing for the use-th time
            bool ok = true;
            for (int strip = blockIdx.x; strip < numStrips && ok; strip += gridDim.x) {
                GBSP_STRIP_GEOMETRY(strip);
                // pixels [first, last) of the 130 lie inside the image
                const int first = x0 == 0 ? 1 : 0;
                const int last = min(kTcSpx, W - x0 + 1);
                for (int k = 0; k <= G / 2 * P; k++, q++) {
                    const int gy = y0 - 1 + 2 * (reverse ? G / 2 * P - k : k);
                    if (use > 0)
                        ok = tc_wait(smem_u32(&rowEmpty[slot]), (use - 1u) & 1u, &abortFlag);
                    if (!__all_sync(0xFFFFFFFFu, ok)) {
                        ok = false;
                        break;
                    }
                    const uint32_t dst = ringAddr + slot * kSlotBytes;
                    const bool in0 = gy >= 0 && gy < H, in1 = gy + 1 < H;  // gy + 1 >= 0
                    const int border = first + kTcSpx - last;  // pixels of a row outside the image
                    if (!(in0 && in1) || border > 0) {
                        const auto zero = [&](int plane, int px) {
                            asm volatile("st.shared.v4.u32 [%0], {%1, %1, %1, %1};"
                                         :: "r"(dst + 16u * (uint32_t)(plane * kTcSpx + px)), "r"(0u) : "memory");
                        };
                        for (int i = lane; i < kPlanes * border; i += 32) {
                            const int px = i / kPlanes;
                            zero(i % kPlanes, px < first ? px : last + px - first);
                        }
                        if (!in0)
                            for (int i = lane; i < KG * kTcSpx; i += 32) zero(i / kTcSpx, i % kTcSpx);
                        if (!in1)
                            for (int i = lane; i < KG * kTcSpx; i += 32) zero(KG + i / kTcSpx, i % kTcSpx);
                        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                    }
                    __syncwarp();
                    const uint32_t bar = smem_u32(&rowFull[slot]);
                    const uint32_t bytes = (uint32_t)(last - first) * 16u;
                    if (lane == 0)
                        asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;"
                                     :: "r"(bar), "r"(bytes * (uint32_t)(KG * ((in0 ? 1 : 0) + (in1 ? 1 : 0))))
                                     : "memory");
                    __syncwarp();
                    if (lane < kPlanes && (lane < KG ? in0 : in1)) {
                        const size_t row = (size_t)b * H + (size_t)(gy + lane / KG);
                        const __nv_bfloat16 *src = in + cg_index(row, x0 - 1 + first, 8 * (lane % KG), W, CIN);
                        asm volatile(
                            "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes"
                            " [%0], [%1], %2, [%3];"
                            :: "r"(dst + 16u * (uint32_t)(lane * kTcSpx + first)), "l"(src), "r"(bytes), "r"(bar)
                            : "memory");
                    }
                    if (++slot == (uint32_t)kTcRing) {
                        slot = 0;
                        use++;
                    }
                }
            }
            // every copy issued has landed before the CTA's shared memory is released
            if (lane == 0) {
                volatile uint32_t never = 0u;
                for (uint32_t s0 = 0; s0 < kTcRing && s0 < q; s0++) {
                    const uint32_t lastUse = (q - 1u - ((q - 1u - s0) % kTcRing)) / kTcRing;
                    if (!tc_wait(smem_u32(&rowFull[s0]), lastUse & 1u, &never)) abortFlag = 1u;
                }
                if (!ok) abortFlag = 1u;
            }
        }
        __syncwarp();
    } else {
        // ---- epilogue: group g = (warp - 4) / 4 takes the row groups with groupCount % 2 == g;
        // warp w reads TMEM lanes 32 (w % 4) .. + 31 (pixels)
        const int quarter = warp & 3, group = (warp - 4) >> 2;
        uint32_t groupCount = 0;
        bool ok = true;
        for (int strip = blockIdx.x; strip < numStrips && ok; strip += gridDim.x) {
            GBSP_STRIP_GEOMETRY(strip);
            for (int p = 0; p < P; p++, groupCount++) {
                if ((int)(groupCount % kTcEpiGroups) != group) continue;
                const uint32_t acc = groupCount % SLOTS, use = groupCount / SLOTS;
                if (EPI == kEpiReluGrad) {
                    // the group's mask rows are on their way from memory while its MMAs run: G
                    // rows of COUT / 8 planes, four 128-byte lines of eight pixels each (a
                    // training step of 16 crops of 128 x 128 489 -> 469 us; one or two groups
                    // further ahead they hold up the input rows, 481)
                    const int yg = y0 + G * (reverse ? P - 1 - p : p);
                    for (int i = lane; i < G * (COUT / 8) * 4; i += 32) {
                        const int y = yg + i / (COUT / 2), px = x0 + quarter * 32 + 8 * (i & 3);
                        if (y < y1 && px < W)
                            asm volatile("prefetch.global.L2 [%0];"
                                         :: "l"(act + cg_index((size_t)(b * H + y), px, 8 * (i / 4 % (COUT / 8)), W, COUT)));
                    }
                }
                ok = tc_wait(smem_u32(&accFull[acc]), use & 1u, &abortFlag);
                __syncwarp();
                if (!__all_sync(0xFFFFFFFFu, ok)) {
                    ok = false;
                    break;
                }
                asm volatile("tcgen05.fence::after_thread_sync;");
                const uint32_t cols = tmem + ((uint32_t)(quarter * 32) << 16) + acc * (uint32_t)ACC_COLS;
                const int x = x0 + quarter * 32 + lane;
#pragma unroll 1
                for (int j = 0; j < G; j++) {
                    const int y = y0 + G * (reverse ? P - 1 - p : p) + j;
                    // the ReLU mask is asked for before the accumulators
                    uint4 mask[COUT / 8] = {};
                    if (EPI == kEpiReluGrad && x < W && y < y1) {
#pragma unroll
                        for (int c = 0; c < COUT; c += 8)
                            mask[c / 8] = *reinterpret_cast<const uint4 *>(
                                act + cg_index((size_t)(b * H + y), x, c, W, COUT));
                    }
                    uint32_t r[COUT];
#pragma unroll
                    for (int c = 0; c < COUT; c += 16)
                        tmem_ld16(cols + (uint32_t)(j * COUT + c), *reinterpret_cast<uint32_t(*)[16]>(r + c));
                    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
                    if (x < W && y < y1) {
                        const size_t row = (size_t)(b * H + y);
                        if constexpr (EPI == kEpiFilter)
                            conv_filter_store<COUT>(r, row * W + x, x, y, W, H, sBias, noisy,
                                outFilt);
                        else
                            conv_store<COUT, EPI>(r, row, x, W, sBias, outB, outF, mask);
                    }
                }
                asm volatile("tcgen05.fence::before_thread_sync;");
                mbar_arrive(smem_u32(&accEmpty[acc]));
            }
        }
    }
#undef GBSP_STRIP_GEOMETRY
    asm volatile("tcgen05.fence::before_thread_sync;");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;");
    if (tid == 0 && abortFlag) atomicOr(&g_dnStatus, 1u);
    if (warp == 0)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;"
                     :: "r"(tmem), "r"(TMEM_COLS));
}

// Rate probe for the MMA shape the convolutions use: one CTA, `issuers`
// threads (lane 0 of warps 0..issuers-1) each issue `iters` back-to-back
// 128 x N x 16 BF16 MMAs from zeroed shared memory into their own TMEM
// accumulator, then wait for completion.  The A operand starts aOff16 16-byte
// units past a 1,024-byte boundary (a pixel-shifted view of a staged row).
// cycles[k] = clock64 cycles of issuer k from its first issue to the
// completion of its last MMA.
template <int N>
__global__ void __launch_bounds__(64) k_tc_rate(int iters, int issuers, int aOff16,
    unsigned long long *cycles)
{
    __shared__ __align__(1024) uint4 sA[2 * 128 + 64];
    __shared__ __align__(1024) uint4 sB[2 * 256];
    __shared__ __align__(8) uint64_t bar[2];
    __shared__ uint32_t tmemBase;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    for (int i = tid; i < 2 * 128 + 64; i += 64) sA[i] = make_uint4(0, 0, 0, 0);
    for (int i = tid; i < 2 * 256; i += 64) sB[i] = make_uint4(0, 0, 0, 0);
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
                     :: "r"(smem_u32(&tmemBase)), "r"(512));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    if (tid == 0) {
        for (int i = 0; i < 2; i++)
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" :: "r"(smem_u32(&bar[i])));
        asm volatile("fence.mbarrier_init.release.cluster;");
    }
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    asm volatile("tcgen05.fence::before_thread_sync;");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;");
    const uint32_t tmem = tmemBase;
    if (lane == 0 && warp < issuers) {
        const uint32_t idesc = instr_desc_bf16<128, N>();
        const uint64_t a = smem_desc(smem_u32(sA + aOff16), 128 * 16, 128);
        const uint64_t b = smem_desc(smem_u32(sB), N * 16, 128);
        const uint32_t d = tmem + (uint32_t)(256 * warp);
        const long long t0 = clock64();
        for (int i = 0; i < iters; i++) {
            asm volatile(
                "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
                "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
                :: "r"(d), "l"(a), "l"(b), "r"(idesc), "r"(i ? 1u : 0u));
        }
        tc_commit(smem_u32(&bar[warp]));
        volatile uint32_t never = 0u;
        const bool done = tc_wait(smem_u32(&bar[warp]), 0u, &never);
        cycles[warp] = done ? (unsigned long long)(clock64() - t0) : 0ull;
    }
    asm volatile("tcgen05.fence::before_thread_sync;");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;");
    if (warp == 0)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" :: "r"(tmem), "r"(512));
}

// Raises a kernel's dynamic shared memory limit once per device (the call costs
// as much as a launch).
struct SmemLimit {
    std::atomic<uint64_t> done{0};  // bit per device
    int operator()(const void *kernel, size_t bytes)
    {
        int dev = 0;
        GBSP_CUDA_TRY(cudaGetDevice(&dev));
        const uint64_t bit = 1ull << (dev & 63);
        if (dev < 64 && (done.load(std::memory_order_acquire) & bit)) return GBSP_OK;
        GBSP_CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes));
        if (dev < 64) done.fetch_or(bit, std::memory_order_release);
        return GBSP_OK;
    }
};

// tcgen05 convolutions launched so far (all shapes): its parity picks the strip order.
static std::atomic<unsigned> g_convLaunches{0};

// cuTensorMapEncodeTiled from the driver, looked up once through the runtime
// (no link-time dependency on libcuda).
static PFN_cuTensorMapEncodeTiled_v12000 tensor_map_encoder()
{
    static PFN_cuTensorMapEncodeTiled_v12000 fn = nullptr;
    static std::once_flag once;
    std::call_once(once, [] {
        void *p = nullptr;
        cudaDriverEntryPointQueryResult q = cudaDriverEntryPointSymbolNotFound;
        if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault,
                &q) == cudaSuccess && q == cudaDriverEntryPointSuccess)
            fn = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(p);
    });
    return fn;
}

// TMA map of a channel-group-planar BF16 activation tensor [B][H][cin/8][W][8]
// seen as 32-bit words [B][H][cin/8][W * 4] (dimension order:
// word, channel group, row, image): one box = boxPixels * 4 words (boxPixels
// <= 64) of every channel group of one row, landing as [group][pixel][8
// channels] in one 16 boxPixels-byte run per group, zero outside the tensor.
// x coordinates are pixel * 4 (16-byte aligned, negative allowed).
static int planar_words_tensor_map(CUtensorMap *map, const void *in, int B, int H, int W, int cin,
    int boxPixels)
{
    PFN_cuTensorMapEncodeTiled_v12000 encode = tensor_map_encoder();
    if (!encode) return set_error(GBSP_ERR_CUDA, "cuTensorMapEncodeTiled is not available");
    if (boxPixels < 1 || boxPixels > 64)
        return set_error(GBSP_ERR_INVALID_ARGUMENT, "box of %d pixels", boxPixels);
    const cuuint64_t dims[4] = {(cuuint64_t)W * 4, (cuuint64_t)cin / 8, (cuuint64_t)H,
        (cuuint64_t)B};
    const cuuint64_t strides[3] = {(cuuint64_t)W * 16, (cuuint64_t)W * cin * 2,
        (cuuint64_t)H * W * cin * 2};
    const cuuint32_t box[4] = {(cuuint32_t)boxPixels * 4, (cuuint32_t)cin / 8, 1, 1};
    const cuuint32_t elem[4] = {1, 1, 1, 1};
    CUresult r = encode(map, CU_TENSOR_MAP_DATA_TYPE_UINT32, 4, const_cast<void *>(in), dims,
        strides, box, elem, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
        CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS)
        return set_error(GBSP_ERR_CUDA, "cuTensorMapEncodeTiled failed (%d)", (int)r);
    return GBSP_OK;
}

// Rows per strip for `cols` columns of H rows on `ctas` CTAs: strips go
// round-robin, so a launch takes as long as the CTA with the most rows, `rounds`
// strips of `rows` and about one row's time per strip for its halo.  Eight
// layers at 1080p (15 columns): strips of 20 rows, "about six per CTA", which
// left the last of six rounds a third full, 626 us; 12, 16, 28, 36 and 56 rows
// 583, 591, 591, 571 and 580; 108, one strip for each of 150 CTAs, 555.
inline int strip_rows(int cols, int H, int ctas)
{
    const auto whole = [](int64_t rows) {
        return (int)((rows + kTcGroupRows - 1) / kTcGroupRows * kTcGroupRows);  // whole row groups
    };
    const int first = (cols + ctas - 1) / ctas;
    int best = whole(H);
    int64_t bestCost = (int64_t)first * (best + 1);
    for (int r = first; r < first + 8; r++) {
        const int64_t perCol = (int64_t)r * ctas / cols;  // strips a column may have in r rounds
        const int rows = whole((H + perCol - 1) / perCol);
        const int64_t strips = (int64_t)cols * ((H + rows - 1) / rows);
        const int64_t cost = (strips + ctas - 1) / ctas * (rows + 1);
        if (cost < bestCost) {
            bestCost = cost;
            best = rows;
        }
    }
    return best;
}

template <int CIN, int COUT, int EPI>
int launch_conv_tc(cudaStream_t s, int smCount, const void *in, int B, int H, int W, const void *w,
    const float *bias, void *outB, float *outF, const float4 *noisy = nullptr,
    float4 *outFilt = nullptr, const void *act = nullptr)
{
    // weights, then the ring (rounded up to a 128-byte boundary inside the kernel)
    size_t smem = (size_t)9 * (CIN / 8) * COUT * 16 +
        (size_t)kTcRing * ((2 * (CIN / 8) * kTcSpx * 16 + 127) / 128 * 128) + 128;
    auto kern = k_conv3x3_tc<CIN, COUT, EPI>;
    static SmemLimit limit;
    if (int rc = limit((const void *)kern, smem)) return rc;
    const int ctas = smCount;  // one CTA per SM (the row ring takes most of shared memory)
    const int cols = B * ((W + kTcTileP - 1) / kTcTileP);
    const int rows = strip_rows(cols, H, ctas);
    const int strips = cols * ((H + rows - 1) / rows);
    int grid = strips < ctas ? strips : ctas;
    // consecutive convolutions walk the strips, and the rows of a strip, in
    // opposite orders, so a layer starts on the rows its predecessor wrote last
    // (still in L2): eight layers at 1080p 548 us, with the strips alone 555
    const int reverse = (int)(g_convLaunches.fetch_add(1, std::memory_order_relaxed) & 1u);
    launch_next_smem(kern, grid, kTcThreads, smem, s, reinterpret_cast<const __nv_bfloat16 *>(in), B, H, W, rows,
        reverse, reinterpret_cast<const __nv_bfloat16 *>(w), bias, reinterpret_cast<__nv_bfloat16 *>(outB),
        outF, noisy, outFilt, reinterpret_cast<const __nv_bfloat16 *>(act));
    GBSP_CUDA_TRY(cudaGetLastError());
    return GBSP_OK;
}

// Input features: log(1 + radiance), albedo, normal, depth/(1 + depth),
// zero-padded to 16 channels.
__global__ void k_features(const float4 *__restrict__ rad, const float4 *__restrict__ aov,
    uint64_t n, int W, __nv_bfloat16 *__restrict__ out)
{
    stage_begin();
    uint64_t p = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
    if (p >= n) return;
    float4 r = rad[p];
    float4 a = aov[2 * p], nn = aov[2 * p + 1];
    float d = fmaxf(a.w, 0.0f);
    float f[16] = {log1pf(fmaxf(r.x, 0.0f)), log1pf(fmaxf(r.y, 0.0f)), log1pf(fmaxf(r.z, 0.0f)),
        a.x, a.y, a.z, nn.x, nn.y, nn.z, d / (1.0f + d), 0, 0, 0, 0, 0, 0};
    const size_t row = p / (uint64_t)W;
    const int x = (int)(p % (uint64_t)W);
#pragma unroll
    for (int g = 0; g < 2; g++)
        *reinterpret_cast<uint4 *>(out + cg_index(row, x, 8 * g, W, 16)) = make_uint4(
            pack_bf16(f[8 * g], f[8 * g + 1]), pack_bf16(f[8 * g + 2], f[8 * g + 3]),
            pack_bf16(f[8 * g + 4], f[8 * g + 5]), pack_bf16(f[8 * g + 6], f[8 * g + 7]));
}

// w'[8 - tap][ci][co] = w[tap][co][ci]: weights of the data-gradient conv.
__global__ void k_flip_transpose(const __nv_bfloat16 *w, int cout, int cin, __nv_bfloat16 *wt)
{
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= 9 * cout * cin) return;
    int tap = i / (cout * cin), r = i % (cout * cin), co = r / cin, ci = r % cin;
    wt[((8 - tap) * cin + ci) * cout + co] = w[i];
}

// d = dAct * (act > 0) as BF16 (ReLU backward).
__global__ void k_relu_bwd(const float *__restrict__ dAct, const __nv_bfloat16 *__restrict__ act,
    uint64_t n, __nv_bfloat16 *__restrict__ out)
{
    uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
    if (i >= n) return;
    float a = __bfloat162float(act[i]);
    out[i] = __float2bfloat16_rn(a > 0.0f ? dAct[i] : 0.0f);
}

// dW[tap][co][ci] += sum_p d[p][co] * in[p + off(tap)][ci]; dBias[co] += sum_p d[p][co].
// CTA = (pixel chunk, tap); 128 threads, each owns a (COUT/8 x CIN/16) block.
template <int CIN, int COUT>
__global__ void __launch_bounds__(128) k_conv3x3_wgrad(const __nv_bfloat16 *__restrict__ in,
    const __nv_bfloat16 *__restrict__ d, int B, int H, int W, int chunk, float *dW, float *dBias)
{
    constexpr int TC = COUT / 8, TI = CIN / 16;  // 8 x 16 thread grid
    constexpr int STAGE = 32;                    // pixels staged per iteration
    __shared__ float sD[STAGE][COUT];
    __shared__ float sI[STAGE][CIN];
    const int tap = blockIdx.y, dy = tap / 3 - 1, dx = tap % 3 - 1;
    const uint64_t N = (uint64_t)B * H * W;
    const uint64_t p0 = (uint64_t)blockIdx.x * chunk;
    const int tco = threadIdx.x / 16, tci = threadIdx.x % 16;
    float acc[TC][TI];
#pragma unroll
    for (int a = 0; a < TC; a++)
#pragma unroll
        for (int c = 0; c < TI; c++) acc[a][c] = 0.0f;
    float bacc = 0.0f;
    for (int base = 0; base < chunk; base += STAGE) {
        __syncthreads();
        for (int i = threadIdx.x; i < STAGE * COUT; i += 128) {
            int k = i / COUT, co = i % COUT;
            uint64_t p = p0 + base + k;
            sD[k][co] = p < N ? __bfloat162float(d[cg_index(p / W, (int)(p % W), co, W, COUT)]) : 0.0f;
        }
        for (int i = threadIdx.x; i < STAGE * CIN; i += 128) {
            int k = i / CIN, ci = i % CIN;
            uint64_t p = p0 + base + k;
            float v = 0.0f;
            if (p < N) {
                int x = (int)(p % W), y = (int)((p / W) % H);
                int gx = x + dx, gy = y + dy;
                if (gx >= 0 && gx < W && gy >= 0 && gy < H)
                    v = __bfloat162float(in[cg_index(p / W + dy, gx, ci, W, CIN)]);
            }
            sI[k][ci] = v;
        }
        __syncthreads();
        for (int k = 0; k < STAGE; k++) {
            float dv[TC], iv[TI];
#pragma unroll
            for (int a = 0; a < TC; a++) dv[a] = sD[k][tco * TC + a];
#pragma unroll
            for (int c = 0; c < TI; c++) iv[c] = sI[k][tci * TI + c];
#pragma unroll
            for (int a = 0; a < TC; a++)
#pragma unroll
                for (int c = 0; c < TI; c++) acc[a][c] += dv[a] * iv[c];
            if (tap == 4 && threadIdx.x < COUT) bacc += sD[k][threadIdx.x];
        }
    }
#pragma unroll
    for (int a = 0; a < TC; a++)
#pragma unroll
        for (int c = 0; c < TI; c++)
            atomicAdd(&dW[((size_t)tap * COUT + tco * TC + a) * CIN + tci * TI + c], acc[a][c]);
    if (tap == 4 && threadIdx.x < COUT) atomicAdd(&dBias[threadIdx.x], bacc);
}

// Weight gradient on the tensor cores (mma.sync m16n8k16, BF16 in, FP32
// accumulate): per tap, dW[tap][co][ci] = sum_p d[p][co] * x[p + off(tap)][ci]
// is a GEMM with M = COUT, N = CIN and K = pixels.  A CTA of 9 warps (warp =
// tap) walks 64-pixel row segments: it stages d transposed ([co][pixel]) and
// the three input rows around the segment transposed ([row][ci][pixel], one
// pixel of halo on each side), then every warp multiplies its tap's shifted
// view, holding all COUT/16 x CIN/8 accumulator tiles in registers.  Each CTA
// writes its partial sums (and the bias gradient sum_p d[p][co]) to its own
// slice of a scratch buffer; k_wgrad_reduce adds the slices in a fixed order,
// so the result is deterministic.
constexpr int kWgTile = 64;
constexpr int kWgStride = kWgTile + 8;  // padded pixel stride of the staged rows

template <int CIN, int COUT>
__global__ void __launch_bounds__(288) k_conv3x3_wgrad_tc(const __nv_bfloat16 *__restrict__ in,
    const __nv_bfloat16 *__restrict__ d, int B, int H, int W, float *__restrict__ partial)
{
    static_assert(CIN % 8 == 0 && COUT % 16 == 0, "tile shape");
    constexpr int MT = COUT / 16, NT = CIN / 8;
    __shared__ __align__(16) __nv_bfloat16 sD[COUT][kWgStride];
    __shared__ __align__(16) __nv_bfloat16 sX[3][CIN][kWgStride];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
    const int tap = warp, ty = tap / 3, tx = tap % 3;
    float acc[MT][NT][4];
#pragma unroll
    for (int m = 0; m < MT; m++)
#pragma unroll
        for (int n = 0; n < NT; n++) acc[m][n][0] = acc[m][n][1] = acc[m][n][2] = acc[m][n][3] = 0.0f;
    float bacc = 0.0f;  // threads 0..COUT-1: bias gradient of channel tid
    const int segs = (W + kWgTile - 1) / kWgTile;
    const int tiles = segs * B * H;
    for (int tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
        const int row = tile / segs, x0 = (tile % segs) * kWgTile;
        const int b = row / H, y = row % H;
        __syncthreads();
        // staging: one 16-byte load per (pixel, 8-channel group) of the planar
        // tensors (consecutive threads take consecutive pixels of one plane),
        // spread over the transposed [channel][pixel] tiles
        for (int i = tid; i < kWgTile * (COUT / 8); i += 288) {
            const int k = i % kWgTile, cg = i / kWgTile, x = x0 + k;
            uint4 v = make_uint4(0, 0, 0, 0);
            if (x < W) v = *reinterpret_cast<const uint4 *>(d + cg_index((size_t)row, x, 8 * cg, W, COUT));
            const __nv_bfloat16 *e = reinterpret_cast<const __nv_bfloat16 *>(&v);
#pragma unroll
            for (int j = 0; j < 8; j++) sD[8 * cg + j][k] = e[j];
        }
        for (int i = tid; i < 3 * (kWgTile + 2) * (CIN / 8); i += 288) {
            const int px = i % (kWgTile + 2), cg = (i / (kWgTile + 2)) % (CIN / 8);
            const int ry = i / ((kWgTile + 2) * (CIN / 8));
            const int gy = y + ry - 1, gx = x0 + px - 1;
            uint4 v = make_uint4(0, 0, 0, 0);
            if (gy >= 0 && gy < H && gx >= 0 && gx < W)
                v = *reinterpret_cast<const uint4 *>(in + cg_index((size_t)(b * H + gy), gx, 8 * cg, W, CIN));
            const __nv_bfloat16 *e = reinterpret_cast<const __nv_bfloat16 *>(&v);
#pragma unroll
            for (int j = 0; j < 8; j++) sX[ry][8 * cg + j][px] = e[j];
        }
        __syncthreads();
        if (tid < COUT) {
            for (int k = 0; k < kWgTile; k++) bacc += __bfloat162float(sD[tid][k]);
        }
#pragma unroll
        for (int k0 = 0; k0 < kWgTile; k0 += 16) {
            uint32_t a[MT][4];
#pragma unroll
            for (int m = 0; m < MT; m++) {
                const __nv_bfloat16 *r0 = &sD[m * 16 + g][k0 + 2 * t];
                const __nv_bfloat16 *r1 = &sD[m * 16 + g + 8][k0 + 2 * t];
                a[m][0] = *reinterpret_cast<const uint32_t *>(r0);
                a[m][1] = *reinterpret_cast<const uint32_t *>(r1);
                a[m][2] = *reinterpret_cast<const uint32_t *>(r0 + 8);
                a[m][3] = *reinterpret_cast<const uint32_t *>(r1 + 8);
            }
#pragma unroll
            for (int n = 0; n < NT; n++) {
                // B[k][ci] = x[pixel k + tx - 1 of the segment][ci]: the staged row ty
                // at halo index k + tx (odd for tx = 1: two 16-bit loads per pair)
                const __nv_bfloat16 *c = &sX[ty][n * 8 + g][k0 + 2 * t + tx];
                __nv_bfloat162 p0, p1;
                p0.x = c[0];
                p0.y = c[1];
                p1.x = c[8];
                p1.y = c[9];
                uint32_t b0 = *reinterpret_cast<uint32_t *>(&p0);
                uint32_t b1 = *reinterpret_cast<uint32_t *>(&p1);
#pragma unroll
                for (int m = 0; m < MT; m++)
                    mma_bf16_16816(acc[m][n], a[m][0], a[m][1], a[m][2], a[m][3], b0, b1);
            }
        }
    }
    // C fragment: rows g / g + 8 (co), columns 2t, 2t + 1 (ci) of each tile
    float *out = partial + (size_t)blockIdx.x * (9 * COUT * CIN + COUT);
#pragma unroll
    for (int m = 0; m < MT; m++)
#pragma unroll
        for (int n = 0; n < NT; n++)
#pragma unroll
            for (int h = 0; h < 2; h++) {
                int co = m * 16 + g + 8 * h, ci = n * 8 + 2 * t;
                float *o = out + ((size_t)tap * COUT + co) * CIN + ci;
                o[0] = acc[m][n][2 * h];
                o[1] = acc[m][n][2 * h + 1];
            }
    if (tid < COUT) out[9 * COUT * CIN + tid] = bacc;
}

// dW[i] += sum over CTA slices of partial[slice][i], added from the first slice
// to the last, for one or several layers, a thread per entry; the last COUT
// entries of a slice are the bias gradient.  A bias gradient is a small sum of
// large terms, so the order of its additions shows (1e-5 for a sum in eight
// groups).
// Bound: the loads (12.6 MB at 152 slices of 48 x 48 weights), latency for a layer
// by itself (13 us), memory for the eight layers of the network in one launch (88
// MB, 19 us; 27 with eight groups of threads, 37 through shared memory).
constexpr int kReduceThreads = 128;
constexpr int kWgLayers = 8;  // layers per launch

struct ReduceJobs {
    struct Layer {
        const float *partial;
        float *dW, *dBias;
        int perSlice, wCount;
        uint32_t firstBlock;
    } l[kWgLayers];
    int count, slices;
};

__global__ void __launch_bounds__(kReduceThreads) k_wgrad_reduce(const __grid_constant__ ReduceJobs jobs)
{
    stage_begin();
    int layer = 0;
    while (layer + 1 < jobs.count && blockIdx.x >= jobs.l[layer + 1].firstBlock) layer++;
    const ReduceJobs::Layer &l = jobs.l[layer];
    const int i = (int)(blockIdx.x - l.firstBlock) * kReduceThreads + threadIdx.x;
    if (i >= l.perSlice) return;
    const float *partial = l.partial + i;  // plain loads: the kernel before this one writes it
    float sum = 0.0f;
#pragma unroll 8
    for (int k = 0; k < jobs.slices; k++) sum += partial[(size_t)k * l.perSlice];
    if (i < l.wCount)
        l.dW[i] += sum;
    else
        l.dBias[i - l.wCount] += sum;
}

// ---------------------------------------------------------------------------
// Weight gradient on the 5th-generation tensor cores (tcgen05), fed by TMA.
//
// dW[ty 3 + tx][co][ci] = sum_p d[y][p][co] x[y + ty - 1][p + tx - 1][ci] over
// every output pixel (b, y, p).  Substituting the input pixel q = p + tx - 1,
// one GEMM per input-row chunk gives all nine taps at once:
//   D[(ty, ci)][(tx, co)] = sum_q x[y + ty - 1][q][ci] d[y][q - tx + 1][co],
// M = 3 CIN rows (two M = 128 MMAs when CIN = 48, one when CIN = 16), N = 3
// COUT, K = 64 input pixels q of a chunk (4 MMAs of K = 16 per M block).
//
// Both operands are MN-major, which is the channel-group-planar layout
// itself: a core matrix (8 pixels along K x 8 channels along M or N, one
// 16-byte row per pixel) is 128 contiguous bytes of one channel group, so the
// leading (K) byte offset is 128 and the stride (M / N) byte offset is one
// 8-channel block.  A chunk's operands are six TMA boxes of [group][64
// pixels][8 channels] (the tensor seen as 32-bit words, so that a box is one
// 1 KB run per channel group): the three input rows (A, one 1 KB block per
// (ty, group)) and three copies of the output-gradient row shifted by one pixel
// each (B, one block per (tx, group)), zero outside the tensor; nothing is
// transposed in registers.  A block of ones after the input rows makes
// accumulator row 3 CIN the sum of d over the chunk: with column block
// tx = 1, the bias gradient.
//
// One launch takes up to kWgLayers layers of one shape.  One persistent CTA per
// SM walks its chunks (b, y, 64-pixel segment), layer after layer, through a
// ring of kWtStages stages: lane 0 of the producer warp waits for a free stage
// (its `empty` barrier, committed by the MMAs that read it) and issues the six
// loads against the stage's `full` transaction count, into the next layer
// without a stop; lane 0 of the MMA warp waits on `full` and issues the MMAs
// into FP32 accumulators in tensor memory that persist over all of the CTA's
// chunks of a layer.  At a layer's end (`done`) the other warps read the
// accumulators, write the CTA's partial sums to its slice of a scratch buffer
// and hand the accumulators back (`drained`); k_wgrad_reduce adds the slices in
// a fixed order (deterministic).  Every wait is bounded and raises g_dnStatus
// on timeout.
//
// Bound: the loads (each input row three times, from L2) and, with a launch, an
// allocation and a reduction per layer, the host: a training step of 16 crops
// of 128 x 128 took 585 us around 485 us on the device, with 16 launches for
// its weight gradients; with four 550 around 490, and 364 us of the host
// instead of 570.  The six 48 x 48 layers: 99 us together, 112 one by one.
// ---------------------------------------------------------------------------
constexpr int kWtPx = 64;
constexpr int kWtStages = 4;
constexpr int kWtThreads = 320;  // eight epilogue warps, the producer, the MMA issuer

struct WtMaps {
    CUtensorMap x[kWgLayers], d[kWgLayers];
};

template <int CIN, int COUT>
struct WtShape {
    static constexpr int KGI = CIN / 8, KGO = COUT / 8;
    static constexpr int MROWS = 3 * CIN, N = 3 * COUT;
    static constexpr int MB = (MROWS + 8 + 127) / 128;          // M = 128 blocks, with the ones
    static constexpr uint32_t kBlock = kWtPx * 16;              // 8 rows x 64 pixels: 1 KB
    static constexpr uint32_t kBOff = (3 * KGI + 1) * kBlock;   // input rows, then the ones
    static constexpr uint32_t kBBytes = 3 * KGO * kBlock;
    static constexpr uint32_t kAExtent = MB * 16 * kBlock;      // what the M = 128 MMAs read
    static constexpr uint32_t kStage =
        ((kBOff + kBBytes > kAExtent ? kBOff + kBBytes : kAExtent) + 1023u) / 1024u * 1024u;
    static constexpr uint32_t kTxBytes = (uint32_t)(3 * KGI + 3 * KGO) * kBlock;
    static constexpr int TMEM_COLS = MB * N <= 256 ? 256 : 512;
    static_assert(CIN % 8 == 0 && COUT % 16 == 0 && N <= 256 && MB * N <= 512, "tile shape");
};

template <int CIN, int COUT>
__global__ void __launch_bounds__(kWtThreads, 1) k_conv3x3_wgrad_tma(
    const __grid_constant__ WtMaps maps, int layers, int B, int H, int W, float *__restrict__ partial)
{
    using S = WtShape<CIN, COUT>;
    constexpr int N = S::N, MB = S::MB, MROWS = S::MROWS;
    // the ring starts at the first 1 KB boundary (the launch adds 1 KB of slack)
    extern __shared__ __align__(128) unsigned char smemRaw[];
    const uint32_t base = (smem_u32(smemRaw) + 1023u) & ~1023u;
    __shared__ __align__(8) uint64_t full[kWtStages], empty[kWtStages], done, drained;
    __shared__ uint32_t tmemBase;
    __shared__ volatile uint32_t abortFlag;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    // the ones block of every stage (BF16 1.0 pairs), written once
    for (int k = tid; k < kWtStages * (int)(S::kBlock / 4); k += kWtThreads) {
        const uint32_t st = (uint32_t)k / (S::kBlock / 4), w = (uint32_t)k % (S::kBlock / 4);
        asm volatile("st.shared.u32 [%0], %1;" :: "r"(base + st * S::kStage + (uint32_t)(3 * S::KGI) *
            S::kBlock + 4u * w), "r"(0x3F803F80u) : "memory");
    }
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
                     :: "r"(smem_u32(&tmemBase)), "r"(S::TMEM_COLS));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    if (tid == 0) {
        for (int i = 0; i < kWtStages; i++) {
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" :: "r"(smem_u32(&full[i])));
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" :: "r"(smem_u32(&empty[i])));
        }
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" :: "r"(smem_u32(&done)));
        asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" :: "r"(smem_u32(&drained)), "r"(4 * MB));
        abortFlag = 0u;
        asm volatile("fence.mbarrier_init.release.cluster;");
    }
    asm volatile("tcgen05.fence::before_thread_sync;");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;");
    const uint32_t tmem = tmemBase;
    stage_begin();
    const int segs = (W + kWtPx - 1) / kWtPx;
    const int chunks = B * H * segs;

    // the launch sizes the grid so that every CTA has a chunk
    if (warp == 8) {
        if (lane == 0) {
            uint32_t i = 0;
            bool ok = true;
            for (int l = 0; l < layers && ok; l++) {
                const uint64_t mapX = reinterpret_cast<uint64_t>(&maps.x[l]),
                               mapD = reinterpret_cast<uint64_t>(&maps.d[l]);
                for (int c = blockIdx.x; c < chunks; c += gridDim.x, i++) {
                    const uint32_t st = i % kWtStages, use = i / kWtStages;
                    if (use > 0 && !(ok = tc_wait(smem_u32(&empty[st]), (use - 1u) & 1u, &abortFlag)))
                        break;
                    const int seg = c % segs, row = c / segs;
                    const int b = row / H, y = row % H, x0 = seg * kWtPx;
                    const uint32_t bar = smem_u32(&full[st]), sb = base + st * S::kStage;
                    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;"
                                 :: "r"(bar), "r"(S::kTxBytes) : "memory");
                    // word coordinates: pixel * 4 (a 16-byte multiple)
#pragma unroll
                    for (int t = 0; t < 3; t++) {
                        asm volatile(
                            "cp.async.bulk.tensor.4d.shared::cluster.global.mbarrier::complete_tx::bytes"
                            " [%0], [%1, {%2, %3, %4, %5}], [%6];"
                            :: "r"(sb + (uint32_t)(t * S::KGI) * S::kBlock), "l"(mapX), "r"(4 * x0), "r"(0),
                               "r"(y + t - 1), "r"(b), "r"(bar)
                            : "memory");
                        asm volatile(
                            "cp.async.bulk.tensor.4d.shared::cluster.global.mbarrier::complete_tx::bytes"
                            " [%0], [%1, {%2, %3, %4, %5}], [%6];"
                            :: "r"(sb + S::kBOff + (uint32_t)(t * S::KGO) * S::kBlock), "l"(mapD),
                               "r"(4 * (x0 + 1 - t)), "r"(0), "r"(y), "r"(b), "r"(bar)
                            : "memory");
                    }
                }
            }
            // every box issued has landed before the CTA's shared memory is released
            volatile uint32_t never = 0u;
            for (uint32_t s0 = 0; s0 < (uint32_t)kWtStages && s0 < i; s0++) {
                const uint32_t lastUse = (i - 1u - ((i - 1u - s0) % kWtStages)) / kWtStages;
                if (!tc_wait(smem_u32(&full[s0]), lastUse & 1u, &never)) abortFlag = 1u;
            }
            if (!ok) abortFlag = 1u;
        }
        __syncwarp();
    } else if (warp == 9) {
        if (lane == 0) {
            // A and B MN-major (instruction descriptor bits 15 and 16)
            const uint32_t idesc = instr_desc_bf16<128, N>() | (1u << 15) | (1u << 16);
            uint32_t i = 0;
            bool ok = true;
            for (int l = 0; l < layers && ok; l++) {
                if (l > 0) {
                    if (!(ok = tc_wait(smem_u32(&drained), (uint32_t)(l - 1) & 1u, &abortFlag))) break;
                    asm volatile("tcgen05.fence::after_thread_sync;");
                }
                bool first = true;
                for (int c = blockIdx.x; c < chunks; c += gridDim.x, i++) {
                    const uint32_t st = i % kWtStages, use = i / kWtStages;
                    if (!(ok = tc_wait(smem_u32(&full[st]), use & 1u, &abortFlag))) break;
                    asm volatile("tcgen05.fence::after_thread_sync;");
                    const uint32_t aAddr = base + st * S::kStage, bAddr = aAddr + S::kBOff;
#pragma unroll
                    for (int kk = 0; kk < kWtPx / 16; kk++) {
                        // K-adjacent core matrices (8 pixels) 128 B apart, M- or N-adjacent
                        // ones (8 channels) one block apart
                        const uint64_t bDesc = smem_desc(bAddr + (uint32_t)kk * 256u, 128, S::kBlock);
#pragma unroll
                        for (int mb = 0; mb < MB; mb++) {
                            const uint64_t aDesc = smem_desc(aAddr + (uint32_t)(mb * 16) * S::kBlock +
                                (uint32_t)kk * 256u, 128, S::kBlock);
                            tc_mma(tmem + (uint32_t)(mb * N), aDesc, bDesc, idesc,
                                (!first || kk > 0) ? 1u : 0u);
                        }
                    }
                    first = false;
                    tc_commit(smem_u32(&empty[st]));
                }
                // every MMA issued has finished before the accumulators are read
                // or freed (waited for even after an abort)
                tc_commit(smem_u32(&done));
                volatile uint32_t never = 0u;
                if (!tc_wait(smem_u32(&done), (uint32_t)l & 1u, &never)) abortFlag = 1u;
            }
            if (!ok) abortFlag = 1u;
        }
        __syncwarp();
    } else if (warp < 4 * MB) {
        // ---- epilogue: warp w reads TMEM lanes 32 (w % 4) .. + 31 of M block w / 4:
        // accumulator row R = (ty, ci), or MROWS for the bias; column n = (tx, co)
        const int mb = warp >> 2, quarter = warp & 3;
        const int R = mb * 128 + quarter * 32 + lane;
        const int ty = R / CIN, ci = R % CIN;
        for (int l = 0; l < layers; l++) {
            uint32_t ok = lane == 0 ? (uint32_t)tc_wait(smem_u32(&done), (uint32_t)l & 1u, &abortFlag) : 0u;
            if (!__shfl_sync(0xFFFFFFFFu, ok, 0)) break;
            asm volatile("tcgen05.fence::after_thread_sync;");
            float *out = partial + ((size_t)l * gridDim.x + blockIdx.x) * (9 * COUT * CIN + COUT);
#pragma unroll 1
            for (int c0 = 0; c0 < N; c0 += 16) {
                uint32_t v[16];
                tmem_ld16(tmem + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(mb * N + c0), v);
                asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
                if (R < MROWS) {
#pragma unroll
                    for (int k = 0; k < 16; k++) {
                        const int n = c0 + k, tx = n / COUT, co = n % COUT;
                        out[((size_t)(3 * ty + tx) * COUT + co) * CIN + ci] = __uint_as_float(v[k]);
                    }
                } else if (R == MROWS) {
#pragma unroll
                    for (int k = 0; k < 16; k++) {
                        const int n = c0 + k;
                        if (n / COUT == 1) out[9 * COUT * CIN + n % COUT] = __uint_as_float(v[k]);
                    }
                }
            }
            asm volatile("tcgen05.fence::before_thread_sync;");
            __syncwarp();
            if (lane == 0) mbar_arrive(smem_u32(&drained));
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;");
    if (tid == 0 && abortFlag) atomicOr(&g_dnStatus, 1u);
    if (warp == 0)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;"
                     :: "r"(tmem), "r"(S::TMEM_COLS));
}

// Per-pixel 5x5 filter from softmax(logits[0..24]) applied to the noisy
// radiance (clamped to the image edge).
__global__ void k_filter(const float *__restrict__ logits, const float4 *__restrict__ noisy, int B,
    int H, int W, float4 *__restrict__ out)
{
    uint64_t p = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
    if (p >= (uint64_t)B * H * W) return;
    int x = (int)(p % W), y = (int)((p / W) % H);
    float l[25], w[25];
#pragma unroll
    for (int k = 0; k < 25; k++) l[k] = logits[p * 32 + k];
    softmax25(l, w);
    float3 o = make_float3(0, 0, 0);
#pragma unroll
    for (int k = 0; k < 25; k++) {
        float4 c = noisy[tap_pixel(p, x, y, W, H, k)];
        o.x += w[k] * c.x;
        o.y += w[k] * c.y;
        o.z += w[k] * c.z;
    }
    out[p] = make_float4(o.x, o.y, o.z, 1.0f);
}

// Per-tile error check of a denoised frame against the plain path tracer.
// A (the denoiser's input) and C are two independent plain renders with the
// same spp, D the denoised A.  For unbiased plain estimates with variance s^2,
// E[(D - C)^2] = (D - mu)^2 + s^2 and E[(A - C)^2] = 2 s^2, so per pixel and
// channel (D - C)^2 - (A - C)^2 / 2 estimates the denoiser's squared error;
// divided by D^2 + 0.01 and averaged over a tile it estimates the tile's
// relMSE.  The per-pixel terms are noisy at low spp, so a tile falls back
// only when the bound lies below the estimate by more than kFallbackZ
// standard errors of the tile mean (a one-sided test at about 98%): then it
// is served from the plain samples, (A + C) / 2; the others keep D.  One CTA of 256 threads per tile
// (tile <= 16 x 16).  tileErr[t] receives the estimate, flags[t] 1 when the
// tile fell back.
constexpr float kFallbackZ = 2.0f;

__global__ void __launch_bounds__(256) k_tile_fallback(const float4 *__restrict__ D,
    const float4 *__restrict__ A, const float4 *__restrict__ C, int B, int H, int W, int tile,
    float bound, float4 *__restrict__ out, float *__restrict__ tileErr, uint32_t *__restrict__ flags)
{
    const int tilesX = (W + tile - 1) / tile, tilesY = (H + tile - 1) / tile;
    const int t = blockIdx.x;
    const int b = t / (tilesX * tilesY), ty = (t / tilesX) % tilesY, tx = t % tilesX;
    const int lx = threadIdx.x % tile, ly = threadIdx.x / tile;
    const int x = tx * tile + lx, y = ty * tile + ly;
    const bool in = threadIdx.x < tile * tile && x < W && y < H;
    const size_t p = ((size_t)b * H + y) * W + x;
    float e = 0.0f, e2 = 0.0f, n = 0.0f;
    float4 d = make_float4(0, 0, 0, 0), a = d, c = d;
    if (in) {
        d = D[p];
        a = A[p];
        c = C[p];
        float dv[3] = {d.x, d.y, d.z}, av[3] = {a.x, a.y, a.z}, cv[3] = {c.x, c.y, c.z};
#pragma unroll
        for (int k = 0; k < 3; k++) {
            float dc = dv[k] - cv[k], ac = av[k] - cv[k];
            const float term = (dc * dc - 0.5f * ac * ac) / (dv[k] * dv[k] + 0.01f);
            e += term;
            e2 += term * term;
        }
        n = 3.0f;
    }
    __shared__ float sE[8], sE2[8], sN[8];
    for (int off = 16; off; off >>= 1) {
        e += __shfl_xor_sync(0xFFFFFFFFu, e, off);
        e2 += __shfl_xor_sync(0xFFFFFFFFu, e2, off);
        n += __shfl_xor_sync(0xFFFFFFFFu, n, off);
    }
    if ((threadIdx.x & 31) == 0) {
        sE[threadIdx.x >> 5] = e;
        sE2[threadIdx.x >> 5] = e2;
        sN[threadIdx.x >> 5] = n;
    }
    __syncthreads();
    float te = 0.0f, te2 = 0.0f, tn = 0.0f;
    for (int k = 0; k < 8; k++) {
        te += sE[k];
        te2 += sE2[k];
        tn += sN[k];
    }
    const float est = tn > 0.0f ? te / tn : 0.0f;
    // standard error of the tile mean from the spread of its per-pixel terms
    const float var = tn > 1.0f ? fmaxf(te2 - te * est, 0.0f) / (tn - 1.0f) : 0.0f;
    const float se = tn > 0.0f ? sqrtf(var / tn) : 0.0f;
    const bool fallback = est - kFallbackZ * se > bound;
    if (threadIdx.x == 0) {
        tileErr[t] = est;
        flags[t] = fallback ? 1u : 0u;
    }
    if (in)
        out[p] = fallback ? make_float4(0.5f * (a.x + c.x), 0.5f * (a.y + c.y), 0.5f * (a.z + c.z), 1.0f)
                          : d;
}

// Served-output check of a denoised frame D against the plain path tracer,
// per tile x tile block.  A: the plain render D was denoised from (sppA
// samples per pixel); C: an independent plain render (sppC).  Per value v
// (pixel and RGB channel), with sigma^2 the per-sample variance of the
// pixel's estimator:
//   E[(D - C)^2] = (D - mu)^2 + sigma^2 / sppC,
//   E[(A - C)^2] = sigma^2 (1 / sppA + 1 / sppC),
// so (D - C)^2 - (A - C)^2 * sppA / (sppA + sppC) estimates D's squared error
// without bias, and (A - C)^2 * sppA * sppC / (sppA + sppC) estimates
// sigma^2.  tileErr = the tile mean of the first over (D^2 + 0.01); the tile
// is flagged when that estimate exceeds `bound` by more than kFallbackZ
// standard errors of the mean.  needSpp = the plain samples per pixel that
// reach `bound` on the tile, margin x mean(sigma^2 / (M^2 + 0.01)) / bound
// with M the pooled plain mean (margin > 1 covers the noise of the variance
// estimate), at least 1 and at most maxSpp.
__global__ void __launch_bounds__(256) k_tile_check(const float4 *__restrict__ D,
    const float4 *__restrict__ A, float sppA, const float4 *__restrict__ C, float sppC, int B,
    int H, int W, int tile, float bound, float margin, uint32_t maxSpp, float *__restrict__ tileErr,
    uint32_t *__restrict__ flags, uint32_t *__restrict__ needSpp)
{
    const int tilesX = (W + tile - 1) / tile, tilesY = (H + tile - 1) / tile;
    const int t = blockIdx.x;
    const int b = t / (tilesX * tilesY), ty = (t / tilesX) % tilesY, tx = t % tilesX;
    const int lx = threadIdx.x % tile, ly = threadIdx.x / tile;
    const int x = tx * tile + lx, y = ty * tile + ly;
    const bool in = threadIdx.x < tile * tile && x < W && y < H;
    const float wVarC = sppA / (sppA + sppC), wVar = sppA * sppC / (sppA + sppC);
    const float wA = sppA / (sppA + sppC), wC = sppC / (sppA + sppC);
    float e = 0.0f, e2 = 0.0f, n = 0.0f, r1 = 0.0f;
    if (in) {
        const size_t p = ((size_t)b * H + y) * W + x;
        const float4 d = D[p], a = A[p], c = C[p];
        float dv[3] = {d.x, d.y, d.z}, av[3] = {a.x, a.y, a.z}, cv[3] = {c.x, c.y, c.z};
#pragma unroll
        for (int k = 0; k < 3; k++) {
            const float dc = dv[k] - cv[k], ac = av[k] - cv[k];
            const float term = (dc * dc - wVarC * ac * ac) / (dv[k] * dv[k] + 0.01f);
            e += term;
            e2 += term * term;
            const float m = wA * av[k] + wC * cv[k];
            r1 += wVar * ac * ac / (m * m + 0.01f);
        }
        n = 3.0f;
    }
    __shared__ float sE[8], sE2[8], sN[8], sR[8];
    for (int off = 16; off; off >>= 1) {
        e += __shfl_xor_sync(0xFFFFFFFFu, e, off);
        e2 += __shfl_xor_sync(0xFFFFFFFFu, e2, off);
        n += __shfl_xor_sync(0xFFFFFFFFu, n, off);
        r1 += __shfl_xor_sync(0xFFFFFFFFu, r1, off);
    }
    if ((threadIdx.x & 31) == 0) {
        sE[threadIdx.x >> 5] = e;
        sE2[threadIdx.x >> 5] = e2;
        sN[threadIdx.x >> 5] = n;
        sR[threadIdx.x >> 5] = r1;
    }
    __syncthreads();
    if (threadIdx.x != 0) return;
    float te = 0.0f, te2 = 0.0f, tn = 0.0f, tr = 0.0f;
    for (int k = 0; k < 8; k++) {
        te += sE[k];
        te2 += sE2[k];
        tn += sN[k];
        tr += sR[k];
    }
    const float est = tn > 0.0f ? te / tn : 0.0f;
    const float var = tn > 1.0f ? fmaxf(te2 - te * est, 0.0f) / (tn - 1.0f) : 0.0f;
    const float se = tn > 0.0f ? sqrtf(var / tn) : 0.0f;
    tileErr[t] = est;
    flags[t] = est - kFallbackZ * se > bound ? 1u : 0u;
    const float need = tn > 0.0f ? margin * (tr / tn) / bound : 1.0f;
    needSpp[t] = need >= (float)maxSpp ? maxSpp : (uint32_t)fmaxf(1.0f, ceilf(need));
}

// Served frame: D on unflagged tiles; on flagged tiles the mean of every
// plain sample of the pixel, (sppA A + sppC C + sppF[t] F) / (sppA + sppC +
// sppF[t]) with F the fallback render of the tile (sppF[t] = 0: none).
__global__ void __launch_bounds__(256) k_tile_merge(const float4 *__restrict__ D,
    const float4 *__restrict__ A, float sppA, const float4 *__restrict__ C, float sppC,
    const float4 *__restrict__ F, const uint32_t *__restrict__ sppF, int B, int H, int W,
    int tile, const uint32_t *__restrict__ flags, float4 *__restrict__ out)
{
    const size_t p = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= (size_t)B * H * W) return;
    const int x = (int)(p % W), y = (int)((p / W) % H), b = (int)(p / ((size_t)W * H));
    const int tilesX = (W + tile - 1) / tile, tilesY = (H + tile - 1) / tile;
    const int t = (b * tilesY + y / tile) * tilesX + x / tile;
    if (!flags[t]) {
        out[p] = D[p];
        return;
    }
    const float f = F ? (float)sppF[t] : 0.0f;
    const float inv = 1.0f / (sppA + sppC + f);
    const float4 a = A[p], c = C[p];
    const float4 g = f > 0.0f ? F[p] : make_float4(0, 0, 0, 0);
    out[p] = make_float4((sppA * a.x + sppC * c.x + f * g.x) * inv,
        (sppA * a.y + sppC * c.y + f * g.y) * inv, (sppA * a.z + sppC * c.z + f * g.z) * inv, 1.0f);
}

// relMSE = mean over pixels and channels of (out - ref)^2 / (ref^2 + 0.01);
// writes dLogits (BF16, 32 channels, zeros beyond 25) and adds the loss sum.
// A pixel's logits are one 128-byte line, read with 128-bit loads (25 scalar
// loads looked up 32 lines each), and a block adds its loss with one atomic.
// 16 x 128^2 pixels: 38 -> 22 us.
constexpr int kRelmseThreads = 128;

// Sum of the blocks' losses and how many have added theirs; zero before a launch.
struct LossTotal {
    double sum;
    unsigned long long blocks;
};

// kVec: logits and dLogits 16-byte aligned (else 32-bit accesses)
template <bool kVec>
__global__ void __launch_bounds__(kRelmseThreads) k_relmse_bwd(const float *__restrict__ logits,
    const float4 *__restrict__ noisy, const float4 *__restrict__ target, int B, int H, int W,
    float invCount, __nv_bfloat16 *__restrict__ dLogits, float *lossSum, LossTotal *total)
{
    stage_begin();
    uint64_t p = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
    float loss = 0.0f;
    if (p < (uint64_t)B * H * W) {
        const uint64_t row = p / (uint64_t)W;
        const int x = (int)(p - row * (uint64_t)W), y = (int)(row % (uint64_t)H);
        float w[28];
#pragma unroll
        for (int k = 0; k < 7; k++) {
            const float *l = logits + p * 32 + 4 * k;
            const float4 v = kVec ? __ldg(reinterpret_cast<const float4 *>(l))
                                  : make_float4(__ldg(l), __ldg(l + 1), __ldg(l + 2), __ldg(l + 3));
            w[4 * k] = v.x;
            w[4 * k + 1] = v.y;
            w[4 * k + 2] = v.z;
            w[4 * k + 3] = v.w;
        }
        softmax25(w, w);
        float3 o = make_float3(0, 0, 0);
        const float4 *image = noisy + (p - (uint64_t)x - (uint64_t)y * W);
        int dx[5], dy[5];
#pragma unroll
        for (int i = 0; i < 5; i++) {
            dx[i] = min(max(x + i - 2, 0), W - 1);
            dy[i] = min(max(y + i - 2, 0), H - 1);
        }
#pragma unroll
        for (int k = 0; k < 25; k++) {
            const float4 c = __ldg(image + (size_t)dy[k / 5] * W + dx[k % 5]);
            o.x += w[k] * c.x;
            o.y += w[k] * c.y;
            o.z += w[k] * c.z;
        }
        float4 r = target[p];
        float ex = o.x - r.x, ey = o.y - r.y, ez = o.z - r.z;
        float nx = 1.0f / (r.x * r.x + 0.01f), ny = 1.0f / (r.y * r.y + 0.01f),
              nz = 1.0f / (r.z * r.z + 0.01f);
        loss = ex * ex * nx + ey * ey * ny + ez * ez * nz;
        float gx = 2.0f * ex * nx * invCount, gy = 2.0f * ey * ny * invCount,
              gz = 2.0f * ez * nz * invCount;
        float gk[25], dot = 0.0f;
#pragma unroll
        for (int k = 0; k < 25; k++) {
            const float4 c = __ldg(image + (size_t)dy[k / 5] * W + dx[k % 5]);
            gk[k] = gx * c.x + gy * c.y + gz * c.z;
            dot += w[k] * gk[k];
        }
#pragma unroll
        for (int c = 0; c < 32; c += 8) {
            uint32_t q[4];
#pragma unroll
            for (int j = 0; j < 4; j++) {
                const int k = c + 2 * j;
                float v0 = k < 25 ? w[k < 25 ? k : 0] * (gk[k < 25 ? k : 0] - dot) : 0.0f;
                float v1 = k + 1 < 25 ? w[k + 1 < 25 ? k + 1 : 0] * (gk[k + 1 < 25 ? k + 1 : 0] - dot) : 0.0f;
                q[j] = pack_bf16(v0, v1);
            }
            __nv_bfloat16 *out = dLogits + cg_index(row, x, c, W, 32);
            if (kVec)
                *reinterpret_cast<uint4 *>(out) = make_uint4(q[0], q[1], q[2], q[3]);
            else
#pragma unroll
                for (int j = 0; j < 4; j++) reinterpret_cast<uint32_t *>(out)[j] = q[j];
        }
    }
    for (int off = 16; off; off >>= 1) loss += __shfl_xor_sync(0xFFFFFFFFu, loss, off);
    __shared__ float sums[kRelmseThreads / 32];
    if ((threadIdx.x & 31) == 0) sums[threadIdx.x >> 5] = loss;
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int k = 1; k < kRelmseThreads / 32; k++) loss += sums[k];
        if (!total) {
            atomicAdd(lossSum, loss);
        } else {
            // the blocks' sums in double precision, rounded once by the last of them: what
            // float sums in the order of arrival are off by, 1e-6 and another value in
            // each run, is gone (4e-8 from the sum in 64 bits of the same logits)
            atomicAdd(&total->sum, (double)loss);
            __threadfence();
            if (atomicAdd(&total->blocks, 1ull) == gridDim.x - 1u) {
                __threadfence();
                *lossSum += (float)atomicAdd(&total->sum, 0.0);
            }
        }
    }
}

__global__ void k_adam(float *param, __nv_bfloat16 *paramBf16, const float *grad, float *m,
    float *v, uint64_t n, float lr, float b1, float b2, float eps, float c1, float c2)
{
    uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
    if (i >= n) return;
    float g = grad[i];
    float mi = b1 * m[i] + (1.0f - b1) * g;
    float vi = b2 * v[i] + (1.0f - b2) * g * g;
    m[i] = mi;
    v[i] = vi;
    float p = param[i] - lr * (mi / c1) / (sqrtf(vi / c2) + eps);
    param[i] = p;
    if (paramBf16) paramBf16[i] = __float2bfloat16_rn(p);
}

// The same step over several tensors in one launch: blocks are dealt out to the
// tensors by firstBlock.  16 launches of a network's tensors took 56 us of the
// GPU, one takes 5 us.
constexpr int kAdamTensors = 32;
struct AdamTensors {
    gbsp_dn_adam_tensor t[kAdamTensors];
    uint32_t firstBlock[kAdamTensors + 1];
};

__global__ void __launch_bounds__(256) k_adam_all(const __grid_constant__ AdamTensors a, int count,
    float lr, float b1, float b2, float eps, float c1, float c2)
{
    int k = 0;
    while (k + 1 < count && blockIdx.x >= a.firstBlock[k + 1]) k++;
    const gbsp_dn_adam_tensor &t = a.t[k];
    const uint64_t i = (uint64_t)(blockIdx.x - a.firstBlock[k]) * 256 + threadIdx.x;
    if (i >= t.n) return;
    float g = t.grad[i];
    float mi = b1 * t.m[i] + (1.0f - b1) * g;
    float vi = b2 * t.v[i] + (1.0f - b2) * g * g;
    t.m[i] = mi;
    t.v[i] = vi;
    float p = t.param[i] - lr * (mi / c1) / (sqrtf(vi / c2) + eps);
    t.param[i] = p;
    if (t.paramBf16) reinterpret_cast<__nv_bfloat16 *>(t.paramBf16)[i] = __float2bfloat16_rn(p);
}

inline unsigned blocks(uint64_t n, unsigned t) { return (unsigned)((n + t - 1) / t); }

int sm_count()
{
    int dev = 0, n = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
    return n > 0 ? n : 1;
}

}  // namespace dn
}  // namespace gbsp

using namespace gbsp;
using namespace gbsp::dn;

// Appends a layer's slices to a reduction; returns its blocks so far.
static uint32_t add_reduce(ReduceJobs &jobs, uint32_t blocks, const float *partial, int cout, int cin,
    float *dW, float *dBias)
{
    const int wCount = 9 * cout * cin, perSlice = wCount + cout;
    jobs.l[jobs.count++] = {partial, dW, dBias, perSlice, wCount, blocks};
    return blocks + (uint32_t)((perSlice + kReduceThreads - 1) / kReduceThreads);
}

static cudaError_t launch_reduce(cudaStream_t s, const ReduceJobs &jobs, uint32_t blocks)
{
    launch_next(k_wgrad_reduce, (int)blocks, kReduceThreads, s, jobs);
    return cudaGetLastError();
}

template <int CIN, int COUT>
static int launch_wgrad_tc(cudaStream_t s, const __nv_bfloat16 *in, const __nv_bfloat16 *d, int B,
    int H, int W, float *dW, float *dBias)
{
    const int tiles = ((W + kWgTile - 1) / kWgTile) * B * H;
    int perSm = 1;
    GBSP_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&perSm,
        k_conv3x3_wgrad_tc<CIN, COUT>, 288, 0));
    int grid = sm_count() * (perSm > 0 ? perSm : 1);
    if (grid > tiles) grid = tiles;
    const int perSlice = 9 * COUT * CIN + COUT;
    float *partial = nullptr;
    GBSP_CUDA_TRY(cudaMallocAsync((void **)&partial, sizeof(float) * (size_t)grid * perSlice, s));
    k_conv3x3_wgrad_tc<CIN, COUT><<<grid, 288, 0, s>>>(in, d, B, H, W, partial);
    cudaError_t e = cudaGetLastError();
    if (e == cudaSuccess) {
        ReduceJobs jobs = {};
        jobs.slices = grid;
        e = launch_reduce(s, jobs, add_reduce(jobs, 0, partial, COUT, CIN, dW, dBias));
    }
    cudaFreeAsync(partial, s);
    if (e != cudaSuccess) return cuda_error(e, "weight gradient");
    return GBSP_OK;
}

// The layers of shape CIN x COUT among `layers`: one launch, partial sums of the
// k-th of them at partial + k * grid * perSlice; the reduction jobs are added.
template <int CIN, int COUT>
static int launch_wgrad_tma(cudaStream_t s, const gbsp_dn_weight_grad_layer *layers, uint32_t count, int B,
    int H, int W, int grid, float *&partial, ReduceJobs &jobs, uint32_t &blocks)
{
    using S = WtShape<CIN, COUT>;
    const size_t smem = 1024 + (size_t)kWtStages * S::kStage;
    auto kern = k_conv3x3_wgrad_tma<CIN, COUT>;
    WtMaps maps;
    int n = 0, rc;
    float *const first = partial;
    for (uint32_t k = 0; k < count; k++) {
        const gbsp_dn_weight_grad_layer &l = layers[k];
        if (l.cin != CIN || l.cout != COUT) continue;
        if ((rc = planar_words_tensor_map(&maps.x[n], l.in, B, H, W, CIN, kWtPx)) ||
            (rc = planar_words_tensor_map(&maps.d[n], l.dOut, B, H, W, COUT, kWtPx)))
            return rc;
        blocks = add_reduce(jobs, blocks, partial, COUT, CIN, l.dW, l.dBias);
        partial += (size_t)grid * (9 * COUT * CIN + COUT);
        n++;
    }
    if (!n) return GBSP_OK;
    static SmemLimit limit;
    if ((rc = limit((const void *)kern, smem))) return rc;
    launch_next_smem(kern, grid, kWtThreads, smem, s, maps, n, B, H, W, first);
    GBSP_CUDA_TRY(cudaGetLastError());
    return GBSP_OK;
}

static int wgrad_grid(int B, int H, int W)
{
    const int64_t chunks = (int64_t)((W + kWtPx - 1) / kWtPx) * B * H;
    return (int)std::min<int64_t>(sm_count(), chunks);
}

static size_t wgrad_scratch_floats(const gbsp_dn_weight_grad_layer *layers, uint32_t count, int grid)
{
    size_t floats = 0;
    for (uint32_t k = 0; k < count; k++)
        floats += (size_t)grid * (9 * layers[k].cout * layers[k].cin + layers[k].cout);
    return floats;
}

static int weight_grads(cudaStream_t s, const gbsp_dn_weight_grad_layer *layers, uint32_t count, int B, int H,
    int W, float *scratch)
{
    const int grid = wgrad_grid(B, H, W);
    float *own = nullptr;
    if (!scratch) {
        GBSP_CUDA_TRY(cudaMallocAsync((void **)&own, sizeof(float) * wgrad_scratch_floats(layers, count, grid), s));
        scratch = own;
    }
    float *partial = scratch;
    ReduceJobs jobs = {};
    jobs.slices = grid;
    uint32_t blocks = 0;
    int rc = launch_wgrad_tma<16, 48>(s, layers, count, B, H, W, grid, partial, jobs, blocks);
    if (!rc) rc = launch_wgrad_tma<48, 48>(s, layers, count, B, H, W, grid, partial, jobs, blocks);
    if (!rc) rc = launch_wgrad_tma<48, 32>(s, layers, count, B, H, W, grid, partial, jobs, blocks);
    if (!rc) {
        const cudaError_t e = launch_reduce(s, jobs, blocks);
        if (e != cudaSuccess) rc = cuda_error(e, "TMA-fed weight gradient");
    }
    if (own) cudaFreeAsync(own, s);
    return rc;
}

extern "C" {

int gbsp_dn_features(void *stream, const float *radiance, const float *aov, uint64_t pixels,
    uint32_t width, uint16_t *out)
{
    if (!radiance || !aov || !out) return set_error(GBSP_ERR_INVALID_ARGUMENT, "NULL argument");
    if (!pixels) return GBSP_OK;
    if (!width || pixels % width)
        return set_error(GBSP_ERR_INVALID_ARGUMENT, "pixels must be whole rows of `width`");
    k_features<<<blocks(pixels, 256), 256, 0, (cudaStream_t)stream>>>(
        reinterpret_cast<const float4 *>(radiance), reinterpret_cast<const float4 *>(aov), pixels,
        (int)width, reinterpret_cast<__nv_bfloat16 *>(out));
    GBSP_CUDA_TRY(cudaGetLastError());
    return GBSP_OK;
}

int gbsp_dn_conv3x3_forward(void *stream, const uint16_t *in, uint32_t B, uint32_t H, uint32_t W,
    uint32_t cin, const uint16_t *weights, const float *bias, uint32_t cout, int epilogue,
    uint16_t *outBf16, float *outF32)
{
    cudaStream_t s = (cudaStream_t)stream;
    if (!in || !weights || !B || !H || !W) return set_error(GBSP_ERR_INVALID_ARGUMENT, "bad conv args");
    int sm = sm_count();
    if (epilogue == kEpiBf16BiasRelu && !outBf16) return set_error(GBSP_ERR_INVALID_ARGUMENT, "outBf16");
    if (epilogue != kEpiBf16BiasRelu && !outF32) return set_error(GBSP_ERR_INVALID_ARGUMENT, "outF32");
    if (epilogue != kEpiF32 && !bias) return set_error(GBSP_ERR_INVALID_ARGUMENT, "bias");
#define GBSP_CONV_CASE(CI, CO, EP)                                                               \
    if (cin == CI && cout == CO && epilogue == EP)                                               \
        return launch_conv<CI, CO, EP>(s, sm, in, B, H, W, weights, bias, outBf16, outF32);
    GBSP_CONV_CASE(16, 48, kEpiBf16BiasRelu)
    GBSP_CONV_CASE(48, 48, kEpiBf16BiasRelu)
    GBSP_CONV_CASE(48, 32, kEpiF32Bias)
    GBSP_CONV_CASE(48, 48, kEpiF32)
    GBSP_CONV_CASE(32, 48, kEpiF32)
#undef GBSP_CONV_CASE
    return set_error(GBSP_ERR_INVALID_ARGUMENT, "conv3x3 %u->%u epilogue %d not instantiated", cin,
        cout, epilogue);
}

int gbsp_dn_conv3x3_forward_tc(void *stream, const uint16_t *in, uint32_t B, uint32_t H,
    uint32_t W, uint32_t cin, const uint16_t *weights, const float *bias, uint32_t cout,
    int epilogue, uint16_t *outBf16, float *outF32)
{
    cudaStream_t s = (cudaStream_t)stream;
    if (!in || !weights || !B || !H || !W) return set_error(GBSP_ERR_INVALID_ARGUMENT, "bad conv args");
    int sm = sm_count();
    if (epilogue == kEpiBf16BiasRelu && !outBf16) return set_error(GBSP_ERR_INVALID_ARGUMENT, "outBf16");
    if (epilogue != kEpiBf16BiasRelu && !outF32) return set_error(GBSP_ERR_INVALID_ARGUMENT, "outF32");
    if (epilogue != kEpiF32 && !bias) return set_error(GBSP_ERR_INVALID_ARGUMENT, "bias");
    if (((uintptr_t)in | (uintptr_t)weights | (uintptr_t)outBf16 | (uintptr_t)outF32) & 15u)
        return set_error(GBSP_ERR_INVALID_ARGUMENT, "conv tensors must be 16-byte aligned");
#define GBSP_CONV_CASE(CI, CO, EP)                                                               \
    if (cin == CI && cout == CO && epilogue == EP)                                               \
        return launch_conv_tc<CI, CO, EP>(s, sm, in, B, H, W, weights, bias, outBf16, outF32);
    GBSP_CONV_CASE(16, 48, kEpiBf16BiasRelu)
    GBSP_CONV_CASE(48, 48, kEpiBf16BiasRelu)
    GBSP_CONV_CASE(48, 32, kEpiF32Bias)
    GBSP_CONV_CASE(48, 48, kEpiF32)
    GBSP_CONV_CASE(32, 48, kEpiF32)
#undef GBSP_CONV_CASE
    return set_error(GBSP_ERR_INVALID_ARGUMENT, "conv3x3 %u->%u epilogue %d not instantiated", cin,
        cout, epilogue);
}

int gbsp_dn_conv3x3_filter_tc(void *stream, const uint16_t *in, uint32_t B, uint32_t H,
    uint32_t W, uint32_t cin, const uint16_t *weights, const float *bias, const float *noisy,
    float *out)
{
    cudaStream_t s = (cudaStream_t)stream;
    if (!in || !weights || !bias || !noisy || !out || !B || !H || !W)
        return set_error(GBSP_ERR_INVALID_ARGUMENT, "bad fused conv/filter args");
    if (((uintptr_t)in | (uintptr_t)weights | (uintptr_t)noisy | (uintptr_t)out) & 15u)
        return set_error(GBSP_ERR_INVALID_ARGUMENT, "conv tensors must be 16-byte aligned");
    if (cin != 48)
        return set_error(GBSP_ERR_INVALID_ARGUMENT, "fused conv/filter %u->32 not instantiated", cin);
    return launch_conv_tc<48, 32, kEpiFilter>(s, sm_count(), in, (int)B, (int)H, (int)W, weights,
        bias, nullptr, nullptr, reinterpret_cast<const float4 *>(noisy),
        reinterpret_cast<float4 *>(out));
}

int gbsp_dn_conv3x3_data_grad_relu_tc(void *stream, const uint16_t *dOut, uint32_t B, uint32_t H,
    uint32_t W, uint32_t cout, const uint16_t *weights, uint32_t cin, const uint16_t *act, uint16_t *dIn)
{
    cudaStream_t s = (cudaStream_t)stream;
    if (!dOut || !weights || !act || !dIn || !B || !H || !W)
        return set_error(GBSP_ERR_INVALID_ARGUMENT, "bad data-gradient args");
    if (((uintptr_t)dOut | (uintptr_t)weights | (uintptr_t)act | (uintptr_t)dIn) & 15u)
        return set_error(GBSP_ERR_INVALID_ARGUMENT, "conv tensors must be 16-byte aligned");
    if (cin == 48 && cout == 48)
        return launch_conv_tc<48, 48, kEpiReluGrad>(s, sm_count(), dOut, (int)B, (int)H, (int)W, weights,
            nullptr, dIn, nullptr, nullptr, nullptr, act);
    if (cin == 48 && cout == 32)
        return launch_conv_tc<32, 48, kEpiReluGrad>(s, sm_count(), dOut, (int)B, (int)H, (int)W, weights,
            nullptr, dIn, nullptr, nullptr, nullptr, act);
    return set_error(GBSP_ERR_INVALID_ARGUMENT, "data gradient %u->%u not instantiated", cin, cout);
}

int gbsp_dn_tc_rate(uint32_t n, uint32_t iters, uint32_t issuers, uint32_t aOffset16,
    double *cyclesPerMma)
{
    if (!cyclesPerMma || !iters || issuers < 1 || issuers > 2 || aOffset16 > 64)
        return set_error(GBSP_ERR_INVALID_ARGUMENT, "bad MMA rate probe args");
    unsigned long long *d = nullptr;
    GBSP_CUDA_TRY(cudaMalloc((void **)&d, 2 * sizeof(unsigned long long)));
    cudaMemset(d, 0, 2 * sizeof(unsigned long long));
    switch (n) {
    case 16: k_tc_rate<16><<<1, 64>>>((int)iters, (int)issuers, (int)aOffset16, d); break;
    case 32: k_tc_rate<32><<<1, 64>>>((int)iters, (int)issuers, (int)aOffset16, d); break;
    case 48: k_tc_rate<48><<<1, 64>>>((int)iters, (int)issuers, (int)aOffset16, d); break;
    case 64: k_tc_rate<64><<<1, 64>>>((int)iters, (int)issuers, (int)aOffset16, d); break;
    case 96: k_tc_rate<96><<<1, 64>>>((int)iters, (int)issuers, (int)aOffset16, d); break;
    case 128: k_tc_rate<128><<<1, 64>>>((int)iters, (int)issuers, (int)aOffset16, d); break;
    case 144: k_tc_rate<144><<<1, 64>>>((int)iters, (int)issuers, (int)aOffset16, d); break;
    case 256: k_tc_rate<256><<<1, 64>>>((int)iters, (int)issuers, (int)aOffset16, d); break;
    default:
        cudaFree(d);
        return set_error(GBSP_ERR_INVALID_ARGUMENT, "MMA rate probe: N = %u not instantiated", n);
    }
    cudaError_t e = cudaDeviceSynchronize();
    unsigned long long h[2] = {0, 0};
    if (e == cudaSuccess) e = cudaMemcpy(h, d, sizeof(h), cudaMemcpyDeviceToHost);
    cudaFree(d);
    GBSP_CUDA_TRY(e);
    for (uint32_t k = 0; k < issuers; k++) cyclesPerMma[k] = (double)h[k] / (double)iters;
    return h[0] ? GBSP_OK : set_error(GBSP_ERR_DEVICE_STATUS, "MMA rate probe timed out");
}

int gbsp_dn_status(uint32_t *status)
{
    if (!status) return set_error(GBSP_ERR_INVALID_ARGUMENT, "status is NULL");
    GBSP_CUDA_TRY(cudaMemcpyFromSymbol(status, g_dnStatus, sizeof(uint32_t)));
    uint32_t zero = 0;
    GBSP_CUDA_TRY(cudaMemcpyToSymbol(g_dnStatus, &zero, sizeof(uint32_t)));
    return *status ? set_error(GBSP_ERR_DEVICE_STATUS, "denoiser device status 0x%x", *status)
                   : GBSP_OK;
}

int gbsp_dn_flip_transpose(void *stream, const uint16_t *w, uint32_t cout, uint32_t cin,
    uint16_t *wt)
{
    uint32_t n = 9 * cout * cin;
    k_flip_transpose<<<blocks(n, 256), 256, 0, (cudaStream_t)stream>>>(
        reinterpret_cast<const __nv_bfloat16 *>(w), (int)cout, (int)cin,
        reinterpret_cast<__nv_bfloat16 *>(wt));
    GBSP_CUDA_TRY(cudaGetLastError());
    return GBSP_OK;
}

int gbsp_dn_relu_backward(void *stream, const float *dAct, const uint16_t *act, uint64_t n,
    uint16_t *out)
{
    if (!n) return GBSP_OK;
    k_relu_bwd<<<blocks(n, 256), 256, 0, (cudaStream_t)stream>>>(dAct,
        reinterpret_cast<const __nv_bfloat16 *>(act), n, reinterpret_cast<__nv_bfloat16 *>(out));
    GBSP_CUDA_TRY(cudaGetLastError());
    return GBSP_OK;
}

int gbsp_dn_conv3x3_weight_grad_tc(void *stream, const uint16_t *in, const uint16_t *dOut,
    uint32_t B, uint32_t H, uint32_t W, uint32_t cin, uint32_t cout, float *dW, float *dBias)
{
    cudaStream_t s = (cudaStream_t)stream;
    if (!in || !dOut || !dW || !dBias || !B || !H || !W)
        return set_error(GBSP_ERR_INVALID_ARGUMENT, "bad weight-gradient args");
    const __nv_bfloat16 *i16 = reinterpret_cast<const __nv_bfloat16 *>(in);
    const __nv_bfloat16 *d16 = reinterpret_cast<const __nv_bfloat16 *>(dOut);
    if (cin == 16 && cout == 48) return launch_wgrad_tc<16, 48>(s, i16, d16, B, H, W, dW, dBias);
    if (cin == 48 && cout == 48) return launch_wgrad_tc<48, 48>(s, i16, d16, B, H, W, dW, dBias);
    if (cin == 48 && cout == 32) return launch_wgrad_tc<48, 32>(s, i16, d16, B, H, W, dW, dBias);
    return set_error(GBSP_ERR_INVALID_ARGUMENT, "weight grad %u->%u not instantiated", cin, cout);
}

uint64_t gbsp_dn_weight_grads_scratch(const gbsp_dn_weight_grad_layer *layers, uint32_t count, uint32_t B,
    uint32_t H, uint32_t W)
{
    return layers ? sizeof(float) * wgrad_scratch_floats(layers, count, wgrad_grid((int)B, (int)H, (int)W)) : 0;
}

int gbsp_dn_weight_grads_tcgen05(void *stream, const gbsp_dn_weight_grad_layer *layers, uint32_t count,
    uint32_t B, uint32_t H, uint32_t W, float *scratch)
{
    if (!layers || !count || count > (uint32_t)kWgLayers || !B || !H || !W)
        return set_error(GBSP_ERR_INVALID_ARGUMENT, "bad weight-gradient args");
    for (uint32_t k = 0; k < count; k++) {
        const gbsp_dn_weight_grad_layer &l = layers[k];
        if (!l.in || !l.dOut || !l.dW || !l.dBias)
            return set_error(GBSP_ERR_INVALID_ARGUMENT, "bad weight-gradient args");
        if (((uintptr_t)l.in | (uintptr_t)l.dOut) & 15u)
            return set_error(GBSP_ERR_INVALID_ARGUMENT, "weight-gradient tensors must be 16-byte aligned");
        if (!((l.cin == 16 && l.cout == 48) || (l.cin == 48 && (l.cout == 48 || l.cout == 32))))
            return set_error(GBSP_ERR_INVALID_ARGUMENT, "weight grad %u->%u not instantiated", l.cin, l.cout);
    }
    return weight_grads((cudaStream_t)stream, layers, count, (int)B, (int)H, (int)W, scratch);
}

int gbsp_dn_conv3x3_weight_grad_tcgen05(void *stream, const uint16_t *in, const uint16_t *dOut,
    uint32_t B, uint32_t H, uint32_t W, uint32_t cin, uint32_t cout, float *dW, float *dBias)
{
    const gbsp_dn_weight_grad_layer l = {in, dOut, dW, dBias, cin, cout};
    return gbsp_dn_weight_grads_tcgen05(stream, &l, 1, B, H, W, nullptr);
}

int gbsp_dn_conv3x3_weight_grad(void *stream, const uint16_t *in, const uint16_t *dOut,
    uint32_t B, uint32_t H, uint32_t W, uint32_t cin, uint32_t cout, float *dW, float *dBias)
{
    cudaStream_t s = (cudaStream_t)stream;
    uint64_t n = (uint64_t)B * H * W;
    int chunk = 2048;
    dim3 grid(blocks(n, chunk), 9);
    const __nv_bfloat16 *i16 = reinterpret_cast<const __nv_bfloat16 *>(in);
    const __nv_bfloat16 *d16 = reinterpret_cast<const __nv_bfloat16 *>(dOut);
    if (cin == 16 && cout == 48)
        k_conv3x3_wgrad<16, 48><<<grid, 128, 0, s>>>(i16, d16, B, H, W, chunk, dW, dBias);
    else if (cin == 48 && cout == 48)
        k_conv3x3_wgrad<48, 48><<<grid, 128, 0, s>>>(i16, d16, B, H, W, chunk, dW, dBias);
    else if (cin == 48 && cout == 32)
        k_conv3x3_wgrad<48, 32><<<grid, 128, 0, s>>>(i16, d16, B, H, W, chunk, dW, dBias);
    else
        return set_error(GBSP_ERR_INVALID_ARGUMENT, "weight grad %u->%u not instantiated", cin, cout);
    GBSP_CUDA_TRY(cudaGetLastError());
    return GBSP_OK;
}

int gbsp_dn_filter(void *stream, const float *logits, const float *noisy, uint32_t B, uint32_t H,
    uint32_t W, float *out)
{
    uint64_t n = (uint64_t)B * H * W;
    k_filter<<<blocks(n, 128), 128, 0, (cudaStream_t)stream>>>(logits,
        reinterpret_cast<const float4 *>(noisy), B, H, W, reinterpret_cast<float4 *>(out));
    GBSP_CUDA_TRY(cudaGetLastError());
    return GBSP_OK;
}

int gbsp_dn_tile_check(void *stream, const float *denoised, const float *plainA, uint32_t sppA,
    const float *plainC, uint32_t sppC, uint32_t B, uint32_t H, uint32_t W, uint32_t tile,
    float bound, float margin, uint32_t maxSpp, float *tileErr, uint32_t *flags, uint32_t *needSpp)
{
    if (!denoised || !plainA || !plainC || !tileErr || !flags || !needSpp || !B || !H || !W ||
        !sppA || !sppC || !maxSpp || !(bound > 0.0f) || !(margin > 0.0f))
        return set_error(GBSP_ERR_INVALID_ARGUMENT, "bad tile check args");
    if (tile < 1 || tile > 16) return set_error(GBSP_ERR_INVALID_ARGUMENT, "tile must be 1..16");
    const uint64_t tiles = (uint64_t)B * ((H + tile - 1) / tile) * ((W + tile - 1) / tile);
    if (tiles > 0x7FFFFFFFull) return set_error(GBSP_ERR_CAPACITY, "too many tiles");
    k_tile_check<<<(unsigned)tiles, 256, 0, (cudaStream_t)stream>>>(
        reinterpret_cast<const float4 *>(denoised), reinterpret_cast<const float4 *>(plainA),
        (float)sppA, reinterpret_cast<const float4 *>(plainC), (float)sppC, (int)B, (int)H, (int)W,
        (int)tile, bound, margin, maxSpp, tileErr, flags, needSpp);
    GBSP_CUDA_TRY(cudaGetLastError());
    return GBSP_OK;
}

int gbsp_dn_tile_merge(void *stream, const float *denoised, const float *plainA, uint32_t sppA,
    const float *plainC, uint32_t sppC, const float *fallback, const uint32_t *sppF, uint32_t B,
    uint32_t H, uint32_t W, uint32_t tile, const uint32_t *flags, float *out)
{
    if (!denoised || !plainA || !plainC || !flags || !out || !B || !H || !W || !sppA || !sppC ||
        (fallback && !sppF))
        return set_error(GBSP_ERR_INVALID_ARGUMENT, "bad tile merge args");
    if (tile < 1 || tile > 16) return set_error(GBSP_ERR_INVALID_ARGUMENT, "tile must be 1..16");
    const uint64_t n = (uint64_t)B * H * W;
    k_tile_merge<<<(unsigned)((n + 255) / 256), 256, 0, (cudaStream_t)stream>>>(
        reinterpret_cast<const float4 *>(denoised), reinterpret_cast<const float4 *>(plainA),
        (float)sppA, reinterpret_cast<const float4 *>(plainC), (float)sppC,
        reinterpret_cast<const float4 *>(fallback), sppF, (int)B, (int)H, (int)W, (int)tile, flags,
        reinterpret_cast<float4 *>(out));
    GBSP_CUDA_TRY(cudaGetLastError());
    return GBSP_OK;
}

int gbsp_dn_tile_fallback(void *stream, const float *denoised, const float *plainA,
    const float *plainC, uint32_t B, uint32_t H, uint32_t W, uint32_t tile, float bound,
    float *out, float *tileErr, uint32_t *flags)
{
    if (!denoised || !plainA || !plainC || !out || !tileErr || !flags || !B || !H || !W)
        return set_error(GBSP_ERR_INVALID_ARGUMENT, "bad fallback args");
    if (tile < 1 || tile > 16) return set_error(GBSP_ERR_INVALID_ARGUMENT, "tile must be 1..16");
    uint64_t tiles = (uint64_t)B * ((H + tile - 1) / tile) * ((W + tile - 1) / tile);
    k_tile_fallback<<<(unsigned)tiles, 256, 0, (cudaStream_t)stream>>>(
        reinterpret_cast<const float4 *>(denoised), reinterpret_cast<const float4 *>(plainA),
        reinterpret_cast<const float4 *>(plainC), (int)B, (int)H, (int)W, (int)tile, bound,
        reinterpret_cast<float4 *>(out), tileErr, flags);
    GBSP_CUDA_TRY(cudaGetLastError());
    return GBSP_OK;
}

static int relmse_backward(void *stream, const float *logits, const float *noisy, const float *target,
    uint32_t B, uint32_t H, uint32_t W, uint16_t *dLogits, float *lossSum, LossTotal *total)
{
    uint64_t n = (uint64_t)B * H * W;
    auto kern = (((uintptr_t)logits | (uintptr_t)dLogits) & 15u) ? k_relmse_bwd<false> : k_relmse_bwd<true>;
    kern<<<blocks(n, kRelmseThreads), kRelmseThreads, 0, (cudaStream_t)stream>>>(logits,
        reinterpret_cast<const float4 *>(noisy), reinterpret_cast<const float4 *>(target), B, H, W,
        1.0f / (3.0f * (float)n), reinterpret_cast<__nv_bfloat16 *>(dLogits), lossSum, total);
    GBSP_CUDA_TRY(cudaGetLastError());
    return GBSP_OK;
}

int gbsp_dn_relmse_backward(void *stream, const float *logits, const float *noisy,
    const float *target, uint32_t B, uint32_t H, uint32_t W, uint16_t *dLogits, float *lossSum)
{
    return relmse_backward(stream, logits, noisy, target, B, H, W, dLogits, lossSum, nullptr);
}

int gbsp_dn_relmse_backward_f64(void *stream, const float *logits, const float *noisy,
    const float *target, uint32_t B, uint32_t H, uint32_t W, uint16_t *dLogits, float *lossSum, void *scratch)
{
    if (!scratch || ((uintptr_t)scratch & 7u))
        return set_error(GBSP_ERR_INVALID_ARGUMENT, "scratch must be 8-byte aligned");
    return relmse_backward(stream, logits, noisy, target, B, H, W, dLogits, lossSum,
        static_cast<LossTotal *>(scratch));
}

int gbsp_dn_adam(void *stream, float *param, uint16_t *paramBf16, const float *grad, float *m,
    float *v, uint64_t n, float lr, float beta1, float beta2, float eps, uint32_t step)
{
    float c1 = 1.0f - powf(beta1, (float)step), c2 = 1.0f - powf(beta2, (float)step);
    k_adam<<<blocks(n, 256), 256, 0, (cudaStream_t)stream>>>(param,
        reinterpret_cast<__nv_bfloat16 *>(paramBf16), grad, m, v, n, lr, beta1, beta2, eps, c1, c2);
    GBSP_CUDA_TRY(cudaGetLastError());
    return GBSP_OK;
}

int gbsp_dn_adam_all(void *stream, const gbsp_dn_adam_tensor *tensors, uint32_t count, float lr,
    float beta1, float beta2, float eps, uint32_t step)
{
    if (count && !tensors) return set_error(GBSP_ERR_INVALID_ARGUMENT, "tensors is NULL");
    for (uint32_t k = 0; k < count; k++) {  // all of them before the first is updated
        const gbsp_dn_adam_tensor &t = tensors[k];
        if (t.n && (!t.param || !t.grad || !t.m || !t.v))
            return set_error(GBSP_ERR_INVALID_ARGUMENT, "Adam tensor %u has a NULL pointer", k);
        if ((t.n + 255) / 256 > 0x7FFFFFFFull) return set_error(GBSP_ERR_CAPACITY, "too many parameters");
    }
    float c1 = 1.0f - powf(beta1, (float)step), c2 = 1.0f - powf(beta2, (float)step);
    for (uint32_t k0 = 0; k0 < count;) {
        AdamTensors a = {};
        int n = 0;
        uint64_t block = 0;
        for (; k0 < count && n < kAdamTensors; k0++) {
            const gbsp_dn_adam_tensor &t = tensors[k0];
            if (!t.n) continue;
            if (block + (t.n + 255) / 256 > 0x7FFFFFFFull) break;  // in a launch of its own
            a.t[n] = t;
            a.firstBlock[n++] = (uint32_t)block;
            block += (t.n + 255) / 256;
        }
        if (!n) break;
        a.firstBlock[n] = (uint32_t)block;
        k_adam_all<<<(unsigned)block, 256, 0, (cudaStream_t)stream>>>(a, n, lr, beta1, beta2, eps, c1, c2);
        GBSP_CUDA_TRY(cudaGetLastError());
    }
    return GBSP_OK;
}

}  // extern "C"
