// Cube maps from an equirectangular HDR image: the reference's CreateCubeMap
// and CreateIrradianceCubeMap (src/cubemap.cpp:106-291) as CUDA kernels.
//
// CreateCubeMap: one thread per output texel (6 faces x height x width),
// face direction -> (azimuth, inclination) -> clamp-to-edge bilinear sample.
//
// CreateIrradianceCubeMap, uniform mode (the application's setting): the
// (phi, theta) grid of step 0.1 is accumulated in float exactly as the
// reference's loops do (63 x 16 = 1,008 samples) and its tangent-space
// directions and cos(theta) sin(theta) weights are tabulated once per block
// in shared memory; one warp integrates one texel, lane l taking samples l,
// l + 32, ..., then a shuffle tree sums the lanes.  The 32 MB source image
// stays L2-resident (129 MB L2), so the kernel is bound by texel fetches from
// L2 and the per-sample atan2/sqrt.
//
// Random mode: the reference draws 3 numbers per sample from ONE XorShift32
// stream for the whole cube (face, row, column, sample order).  Every texel
// draws exactly 3 * samplesPerPixel numbers, so sample k of texel i starts at
// state M^(3 (i samplesPerPixel + k)) * s0, M the 32 x 32 GF(2) matrix of one
// XorShift32 step.  One warp integrates one texel: it jumps to the texel's
// state with the matrices J^(2^b), J = M^(3 samplesPerPixel), of the set bits b
// of i (lane c holds column c, one xor reduction per product), and lane l to
// its run of samples with a matrix of its own.  The host makes both tables and
// passes them with the launch.
//
// Transcendentals are CUDA's sinf/cosf/atan2f (their last bits differ from
// glibc's), so results match the reference to within those differences;
// everything else follows the reference's operation order without
// contraction.

#include <algorithm>
#include <vector>

#include "gbsp_internal.h"

namespace gbsp {
namespace cube {

constexpr float kRadianceClamp = 10.0f;  // RADIANCE_CLAMP, src/config.h:37
constexpr int kMaxGridSamples = 1024;
constexpr float kGridDelta = 0.1f;
constexpr int kIrrWarps = 8;

struct Basis {
    V3 forward, up, right;
};

// MapCubeMapLayerIndexToBasisVectors (src/cubemap.cpp:56-103)
__device__ __forceinline__ Basis face_basis(uint32_t layer)
{
    switch (layer) {
    case 0: return Basis{v3(1, 0, 0), v3(0, 1, 0), v3(0, 0, -1)};
    case 1: return Basis{v3(-1, 0, 0), v3(0, 1, 0), v3(0, 0, 1)};
    case 2: return Basis{v3(0, 1, 0), v3(0, 0, -1), v3(1, 0, 0)};
    case 3: return Basis{v3(0, -1, 0), v3(0, 0, 1), v3(1, 0, 0)};
    case 4: return Basis{v3(0, 0, 1), v3(0, 1, 0), v3(1, 0, 0)};
    default: return Basis{v3(0, 0, -1), v3(0, 1, 0), v3(-1, 0, 0)};
    }
}

struct Image {
    const float4 *pixels;
    uint32_t width, height;
};

__device__ __forceinline__ float4 lerp4(float4 a, float4 b, float t)
{
    float s = 1.0f - t;
    return make_float4(a.x * s + b.x * t, a.y * s + b.y * t, a.z * s + b.z * t, a.w * s + b.w * t);
}

// SampleImageBilinear (src/image.h:34-73), clamp-to-edge
__device__ __forceinline__ float4 sample_bilinear(const Image &im, float u, float v)
{
    float px = (u * (float)im.width) - 0.5f;
    float py = (v * (float)im.height) - 0.5f;
    px = rmax(px, 0.0f);
    py = rmax(py, 0.0f);
    uint32_t x0 = (uint32_t)floorf(px), x1 = x0 + 1;
    uint32_t y0 = (uint32_t)floorf(py), y1 = y0 + 1;
    float fx = px - (float)x0, fy = py - (float)y0;
    x1 = min(x1, im.width - 1);
    y1 = min(y1, im.height - 1);
    x0 = min(x0, im.width - 1);  // u <= 1 keeps the reference's x0 in range too
    y0 = min(y0, im.height - 1);
    float4 a = __ldg(&im.pixels[(size_t)y0 * im.width + x0]);
    float4 b = __ldg(&im.pixels[(size_t)y0 * im.width + x1]);
    float4 c = __ldg(&im.pixels[(size_t)y1 * im.width + x0]);
    float4 d = __ldg(&im.pixels[(size_t)y1 * im.width + x1]);
    return lerp4(lerp4(a, b, fx), lerp4(c, d, fx), fy);
}

// ToSphericalCoordinates + MapToEquirectangular + y flip
// (src/math_lib.h:849-884, src/cubemap.cpp:176-178)
__device__ __forceinline__ void direction_uv(V3 d, float &u, float &v)
{
    float inc = atan2f(sqrtf(d.x * d.x + d.z * d.z), d.y);
    float az = atan2f(d.z, d.x);
    if (az < 0.0f) az += 2.0f * kPi;
    u = az / (2.0f * kPi);
    v = 1.0f - (cosf(inc) * 0.5f + 0.5f);
}

__device__ __forceinline__ V3 face_direction(const Basis &b, uint32_t x, uint32_t y,
    uint32_t width, uint32_t height)
{
    float fx = (float)x / (float)width;
    float fy = (float)y / (float)height;
    fy = 1.0f - fy;
    fx = fx * 2.0f - 1.0f;
    fy = fy * 2.0f - 1.0f;
    return normalize(add(add(b.forward, mul(b.right, fx)), mul(b.up, fy)));
}

// Bound: instructions of the lookup (two atan2f, a cosf, a square root and
// four divisions per texel), about 40 us of them at 6 x 1024^2 texels; 134 MB
// of traffic would take 20.  Texel coordinates come from a 3-d grid: three
// 64-bit divisions of a flat index had cost a fifth of the kernel.  6 x 1024^2
// from 2048 x 1024: 78 -> 64 us, 90 % of the issue slots busy.  A thread takes
// up to four rows of a column (the column's division and products once) while
// that leaves two waves of blocks: with the irradiance map 162.4 -> 156.3 us (two
// rows 158.9, eight 158.6).
//
// Blocks are kX = 32 texels wide, or where that pads the rows by more than a quarter
// as wide as pads them least (below 16 texels down to one; from there on blocks of 4
// lose 0.3 us on small maps).  6 x 1 x 4096 texels 9.7 -> 2.2 us, 6 x 33 x 4000 16.1
// -> 11.2; a flat index took 2.6 and 11.9.
constexpr uint32_t kCubeThreads = 256;

static uint32_t cube_block_width(uint32_t width)
{
    uint32_t best = 32;
    const auto padded = [&](uint32_t x) { return ((uint64_t)width + x - 1) / x * x; };
    if (4 * padded(32) <= 5 * (uint64_t)width) return 32;
    for (uint32_t x = 16; x; x >>= 1)
        if ((x >= 8 || width < 16) && padded(x) < padded(best)) best = x;
    return best;
}

template <int kX>
__global__ void __launch_bounds__(kCubeThreads) k_cube_map(Image im, uint32_t width, uint32_t height,
    float4 *__restrict__ out)
{
    constexpr uint32_t kY = kCubeThreads / kX;
    const uint32_t x = blockIdx.x * kX + threadIdx.x, layer = blockIdx.z;
    if (x >= width) return;
    const Basis b = face_basis(layer);
    for (uint32_t y = blockIdx.y * kY + threadIdx.y; y < height; y += gridDim.y * kY) {
        V3 dir = face_direction(b, x, y, width, height);
        float u, v;
        direction_uv(dir, u, v);
        out[((size_t)layer * height + y) * width + x] = sample_bilinear(im, u, v);
    }
}

// Uniform grid of nPhi x nTheta samples, theta fastest: table entries (t.x,
// t.y = cos(theta), t.z, sin(theta)) of MapSphericalToCartesianCoordinates
// (src/math_lib.h:864-871) at phi and theta as the reference's loops reach
// them (additions of 0.1f, src/cubemap.cpp:155-160).
//
// Bound: the gathers, four texels per sample that no neighbouring lane shares
// (L1 86 % busy, issue 63 %): 95 us for 6 x 32^2 texels, with or without 32-byte
// loads of texel pairs.  Every block fills its own table, so a call needs no
// allocation and no upload: 2.9 + 13 us of the call before.  Two samples in
// flight 162 us for a bake of both maps; one 166, four 163.
__global__ void __launch_bounds__(32 * kIrrWarps) k_irradiance_uniform(Image im, uint32_t width,
    uint32_t height, uint32_t nPhi, uint32_t nTheta, float4 *__restrict__ out)
{
    __shared__ float4 table[kMaxGridSamples];
    const uint32_t gridCount = nPhi * nTheta;
    for (uint32_t k = threadIdx.x; k < gridCount; k += blockDim.x) {
        float phi = 0.0f, theta = 0.0f;
        for (uint32_t i = k / nTheta; i; i--) phi += kGridDelta;
        for (uint32_t i = k % nTheta; i; i--) theta += kGridDelta;
        float st = sinf(theta);
        float4 e;
        e.x = st * cosf(phi);
        e.z = st * sinf(phi);
        e.y = cosf(theta);
        e.w = st;
        table[k] = e;
    }
    __syncthreads();
    const int lane = threadIdx.x & 31;
    const uint32_t total = 6u * width * height;  // checked to fit
    const uint32_t warps = gridDim.x * kIrrWarps;
    for (uint64_t i64 = blockIdx.x * kIrrWarps + (threadIdx.x >> 5); i64 < total; i64 += warps) {
        const uint32_t i = (uint32_t)i64, x = i % width, y = i / width % height, layer = i / width / height;
        Basis b = face_basis(layer);
        V3 normal = face_direction(b, x, y, width, height);
        V3 tangent = normalize(cross(b.up, normal));
        V3 bitangent = normalize(cross(normal, tangent));
        V3 irr = v3(0.0f, 0.0f, 0.0f);
#pragma unroll 2
        for (uint32_t k = lane; k < gridCount; k += 32) {
            float4 e = table[k];
            V3 w = add(add(mul(normal, e.y), mul(tangent, e.x)), mul(bitangent, e.z));
            float u, v;
            direction_uv(w, u, v);
            float4 s = sample_bilinear(im, u, v);
            V3 rad = v3(rclamp(s.x, 0.0f, kRadianceClamp), rclamp(s.y, 0.0f, kRadianceClamp),
                rclamp(s.z, 0.0f, kRadianceClamp));
            irr = add(irr, mul(mul(rad, e.y), e.w));  // radiance * Cos(theta) * Sin(theta)
        }
#pragma unroll
        for (int off = 16; off; off >>= 1) {
            irr.x += __shfl_xor_sync(0xFFFFFFFFu, irr.x, off);
            irr.y += __shfl_xor_sync(0xFFFFFFFFu, irr.y, off);
            irr.z += __shfl_xor_sync(0xFFFFFFFFu, irr.z, off);
        }
        if (lane == 0) {
            float invCount = 1.0f / (float)gridCount;
            out[i] = make_float4((kPi * irr.x) * invCount, (kPi * irr.y) * invCount,
                (kPi * irr.z) * invCount, 1.0f);
        }
    }
}

struct JumpTables {
    uint32_t texel[32][32];  // texel[b][c]: column c of J^(2^b)
    uint32_t lane[32][32];   // lane[l][c]: column c of M^(3 step l), lane l's first sample
    uint32_t step;           // samples between the lanes' first ones
};

// The tables in shared memory, and the state of lane l of a warp whose first
// sample is that of texel i.
struct SharedJumps {
    uint32_t texelCols[32][32], laneCols[32][33];  // laneCols[c][l]
    __device__ __forceinline__ void load(const JumpTables &jumps)
    {
        for (uint32_t k = threadIdx.x; k < 1024; k += blockDim.x) {
            texelCols[k >> 5][k & 31] = jumps.texel[k >> 5][k & 31];
            laneCols[k & 31][k >> 5] = jumps.lane[k >> 5][k & 31];
        }
        __syncthreads();
    }
    __device__ __forceinline__ uint32_t state(uint32_t seed, uint32_t i, uint32_t lane) const
    {
        uint32_t state = seed;
        for (uint32_t bits = i; bits; bits &= bits - 1)
            state = __reduce_xor_sync(0xFFFFFFFFu, state >> lane & 1u ? texelCols[__ffs(bits) - 1][lane] : 0u);
        uint32_t rng = 0;
        for (uint32_t bits = state; bits; bits &= bits - 1) rng ^= laneCols[__ffs(bits) - 1][lane];
        return rng;
    }
};

// irr plus `count` samples around dir, one after another.
__device__ __forceinline__ V3 add_samples(V3 irr, const Image &im, V3 dir, uint64_t count, float contribution,
    uint32_t &rng)
{
    for (uint64_t k = 0; k < count; k++) {
        // Vec3(RandomBilateral() x3) with GCC's right-to-left argument order
        float oz = random_bilateral(rng);
        float oy = random_bilateral(rng);
        float ox = random_bilateral(rng);
        V3 sd = normalize(add(dir, v3(ox, oy, oz)));
        if (dot(sd, dir) < 0.0f) sd = neg(sd);
        float cosine = rmax(dot(dir, sd), 0.0f);
        float u, v;
        direction_uv(sd, u, v);
        float4 s = sample_bilinear(im, u, v);
        V3 rad = v3(rclamp(s.x * cosine, 0.0f, kRadianceClamp),
            rclamp(s.y * cosine, 0.0f, kRadianceClamp), rclamp(s.z * cosine, 0.0f, kRadianceClamp));
        irr = add(irr, mul(rad, contribution));
    }
    return irr;
}

// Bound: latency of the samples' dependent chains (random numbers, direction,
// lookup).  A thread per texel walked all of its samples one after another,
// with at most 24,576 threads for a 6 x 64^2 map, and the call waited for its
// table's upload.  6 x 8^2 texels of 128 samples 394 -> 47 us for the call, 6 x
// 64^2 of 8 300 -> 96, of 128 401 -> 122; the host's tables take 25 us of it.
__global__ void __launch_bounds__(32 * kIrrWarps) k_irradiance_random(Image im, uint32_t width,
    uint32_t height, uint32_t spp, const __grid_constant__ JumpTables jumps, uint32_t seed,
    float4 *__restrict__ out)
{
    __shared__ SharedJumps shared;
    shared.load(jumps);
    const uint32_t lane = threadIdx.x & 31;
    const uint32_t total = 6u * width * height;  // checked to fit
    const uint32_t warps = gridDim.x * kIrrWarps;
    const float contribution = 1.0f / (float)spp;
    // 64 bits: step * lane may pass 2^32
    const uint64_t first = min((uint64_t)spp, (uint64_t)jumps.step * lane),
                   count = min((uint64_t)spp - first, (uint64_t)jumps.step);
    for (uint64_t i64 = blockIdx.x * kIrrWarps + (threadIdx.x >> 5); i64 < total; i64 += warps) {
        const uint32_t i = (uint32_t)i64, x = i % width, y = i / width % height, layer = i / width / height;
        uint32_t rng = shared.state(seed, i, lane);
        const V3 dir = face_direction(face_basis(layer), x, y, width, height);
        V3 irr = add_samples(v3(0.0f, 0.0f, 0.0f), im, dir, count, contribution, rng);
#pragma unroll
        for (int off = 16; off; off >>= 1) {
            irr.x += __shfl_xor_sync(0xFFFFFFFFu, irr.x, off);
            irr.y += __shfl_xor_sync(0xFFFFFFFFu, irr.y, off);
            irr.z += __shfl_xor_sync(0xFFFFFFFFu, irr.z, off);
        }
        if (lane == 0) out[i] = make_float4(irr.x, irr.y, irr.z, 1.0f);
    }
}

// Whether a lane takes a whole texel.  A warp per texel jumps for each of them and
// leaves lanes idle below 32 samples and behind 33 (0.67 + 0.28 run ns a texel); a
// lane per texel takes 0.035 + 0.011 spp ns but at least 0.73 us a sample, its chain.
// The line is where the chain is 1.2 times shorter than the warps' work; from 257
// samples on the jump no longer shows and the warps' finer grain wins (256^2 of 512:
// 2,217 us, 2,345 with lanes).  Calls in us, warp and lane per texel, maps of 6 x:
//   32^2   1 sample  46  40;    8  49  51;  128  67  143
//   64^2   8 samples 90  51;   33  99  74;  128 116  145
//   128^2  8 samples 150 65;   33 183 102;  128 243  221
//   512^2  8 samples 1,509 254;  33 1,904 710;  128 2,800 2,291
// (a thread per texel that jumped by itself, with an upload per call: 512^2 543, 956
// and 2,562).
static bool lane_per_texel(uint64_t texels, uint32_t spp, uint32_t run)
{
    return run <= 8 && texels * (12 + 5 * run) >= 16000ull * spp;
}

// The same values with a lane per texel: a warp jumps once for 32 texels, and a
// lane adds the sums of the runs in the order of the warp's reduction above.
__global__ void __launch_bounds__(32 * kIrrWarps) k_irradiance_random_wide(Image im, uint32_t width,
    uint32_t height, uint32_t spp, uint32_t run, const __grid_constant__ JumpTables jumps, uint32_t seed,
    float4 *__restrict__ out)
{
    __shared__ SharedJumps shared;
    shared.load(jumps);
    const uint32_t lane = threadIdx.x & 31;
    const uint32_t total = 6u * width * height;  // checked to fit
    const uint64_t texels = 32ull * kIrrWarps * gridDim.x;
    const float contribution = 1.0f / (float)spp;
    const int runs = (int)((spp + (uint64_t)run - 1) / run);  // at most 32
    for (uint64_t base = 32ull * (blockIdx.x * kIrrWarps + (threadIdx.x >> 5)); base < total; base += texels) {
        uint32_t rng = shared.state(seed, (uint32_t)base, lane);
        const uint64_t i64 = base + lane;
        if (i64 >= total) continue;
        const uint32_t i = (uint32_t)i64, x = i % width, y = i / width % height, layer = i / width / height;
        const V3 dir = face_direction(face_basis(layer), x, y, width, height);
        V3 sums[16];
        for (int r = 0; r < runs; r++) {
            const uint64_t first = (uint64_t)run * r;
            const V3 sum = add_samples(v3(0.0f, 0.0f, 0.0f), im, dir, min((uint64_t)run, spp - first),
                contribution, rng);
            sums[r & 15] = r < 16 ? sum : add(sums[r & 15], sum);
        }
        for (int off = 8; off; off >>= 1)
            for (int r = 0; r < off && r + off < runs; r++) sums[r] = add(sums[r], sums[r + off]);
        out[i] = make_float4(sums[0].x, sums[0].y, sums[0].z, 1.0f);
    }
}

// ---- host: GF(2) jump-ahead of XorShift32 --------------------------------
using Mat = std::vector<uint32_t>;  // 32 columns

static uint32_t apply(const Mat &m, uint32_t s)
{
    uint32_t r = 0;
    for (; s; s &= s - 1) r ^= m[__builtin_ctz(s)];
    return r;
}

static Mat multiply(const Mat &a, const Mat &b)
{
    Mat r(32);
    for (int c = 0; c < 32; c++) r[c] = apply(a, b[c]);
    return r;
}

static Mat step_matrix()
{
    Mat m(32);
    for (int c = 0; c < 32; c++) {
        uint32_t s = 1u << c;
        m[c] = xorshift32(s);
    }
    return m;
}

static Mat power(Mat base, uint64_t n)
{
    Mat r(32);
    for (int c = 0; c < 32; c++) r[c] = 1u << c;
    while (n) {
        if (n & 1) r = multiply(r, base);
        base = multiply(base, base);
        n >>= 1;
    }
    return r;
}

}  // namespace cube
}  // namespace gbsp

using namespace gbsp;

static int check_image(const float *equirect, uint32_t eqW, uint32_t eqH, uint32_t w, uint32_t h,
    const float *faces)
{
    if (!eqW || !eqH || !w || !h) return set_error(GBSP_ERR_INVALID_ARGUMENT, "empty image");
    if (!equirect || !faces) return set_error(GBSP_ERR_INVALID_ARGUMENT, "NULL image");
    if (((uintptr_t)equirect | (uintptr_t)faces) & 15u)
        return set_error(GBSP_ERR_INVALID_ARGUMENT, "images must be 16-byte aligned");
    return GBSP_OK;
}

static int sm_count()
{
    int dev = 0, sms = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    return sms > 0 ? sms : 1;
}

static int grid_for(uint64_t work, int block)
{
    uint64_t want = (work + block - 1) / block;
    uint64_t cap = (uint64_t)sm_count() * 16;
    return (int)(want < cap ? (want ? want : 1) : cap);
}

extern "C" {

uint32_t gbsp_xorshift32_jump(uint32_t state, uint64_t steps)
{
    return cube::apply(cube::power(cube::step_matrix(), steps), state);
}

int gbsp_create_cube_map(void *stream, const float *equirect, uint32_t eqWidth, uint32_t eqHeight,
    uint32_t width, uint32_t height, float *faces)
{
    int rc = check_image(equirect, eqWidth, eqHeight, width, height, faces);
    if (rc) return rc;
    cube::Image im{reinterpret_cast<const float4 *>(equirect), eqWidth, eqHeight};
    const dim3 block(cube::cube_block_width(width), cube::kCubeThreads / cube::cube_block_width(width));
    const uint32_t cols = (width + block.x - 1) / block.x, bands = (height + block.y - 1) / block.y;
    // two waves of 8 blocks per SM
    const uint64_t rows = std::min<uint64_t>(4, std::max<uint64_t>(1, 6ull * cols * bands / (16ull * sm_count())));
    const dim3 grid(cols, (uint32_t)std::min<uint64_t>((bands + rows - 1) / rows, 65535u), 6);
    auto kern = block.x == 32 ? cube::k_cube_map<32>
        : block.x == 16       ? cube::k_cube_map<16>
        : block.x == 8        ? cube::k_cube_map<8>
        : block.x == 4        ? cube::k_cube_map<4>
        : block.x == 2        ? cube::k_cube_map<2>
                              : cube::k_cube_map<1>;
    kern<<<grid, block, 0, (cudaStream_t)stream>>>(im, width, height,
        reinterpret_cast<float4 *>(faces));
    GBSP_CUDA_TRY(cudaGetLastError());
    return GBSP_OK;
}

int gbsp_create_irradiance_cube_map(void *stream, const float *equirect, uint32_t eqWidth,
    uint32_t eqHeight, uint32_t width, uint32_t height, uint32_t samplesPerPixel, uint32_t mode,
    float *faces)
{
    int rc = check_image(equirect, eqWidth, eqHeight, width, height, faces);
    if (rc) return rc;
    if (mode != GBSP_IRRADIANCE_UNIFORM && mode != GBSP_IRRADIANCE_RANDOM)
        return set_error(GBSP_ERR_INVALID_ARGUMENT, "unknown irradiance mode %u", mode);
    if (mode == GBSP_IRRADIANCE_RANDOM && samplesPerPixel == 0)
        return set_error(GBSP_ERR_INVALID_ARGUMENT, "samplesPerPixel must be positive");
    cudaStream_t s = (cudaStream_t)stream;
    cube::Image im{reinterpret_cast<const float4 *>(equirect), eqWidth, eqHeight};
    uint64_t total = 6ull * width * height;
    if (total >> 32) return set_error(GBSP_ERR_CAPACITY, "cube map too large");
    if (mode == GBSP_IRRADIANCE_UNIFORM) {
        // the lengths of the reference's loops: phi, theta += 0.1f in float (src/cubemap.cpp:155-160)
        uint32_t nPhi = 0, nTheta = 0;
        for (float phi = 0.0f; phi < 2.0f * kPi; phi += cube::kGridDelta) nPhi++;
        for (float theta = 0.0f; theta < 0.5f * kPi; theta += cube::kGridDelta) nTheta++;
        if (nPhi * nTheta > (uint32_t)cube::kMaxGridSamples)
            return set_error(GBSP_ERR_CAPACITY, "sample grid too large");
        int block = 32 * cube::kIrrWarps;
        uint64_t blocks = (total + cube::kIrrWarps - 1) / cube::kIrrWarps;
        cube::k_irradiance_uniform<<<grid_for(blocks * block, block), block, 0, s>>>(im, width, height, nPhi,
            nTheta, reinterpret_cast<float4 *>(faces));
        GBSP_CUDA_TRY(cudaGetLastError());
        return GBSP_OK;
    }
    // random mode: a texel's sum is that of up to 32 runs of `run` samples each
    const uint32_t run = (uint32_t)(((uint64_t)samplesPerPixel + 31) / 32);
    const bool wide = cube::lane_per_texel(total, samplesPerPixel, run);
    cube::JumpTables jumps = {};
    jumps.step = wide ? samplesPerPixel : run;
    const auto copy = [](uint32_t *dst, const cube::Mat &m) { std::copy(m.begin(), m.end(), dst); };
    cube::Mat j = cube::power(cube::step_matrix(), 3ull * samplesPerPixel);
    for (int b = 0; b < 32 && total >> b; b++) {
        copy(jumps.texel[b], j);
        j = cube::multiply(j, j);
    }
    const cube::Mat step = cube::power(cube::step_matrix(), 3ull * jumps.step);
    j = cube::power(step, 0);
    for (uint64_t l = 0; l < 32 && (wide || l * run < samplesPerPixel); l++) {
        copy(jumps.lane[l], j);
        j = cube::multiply(j, step);
    }
    const uint64_t warps = wide ? (total + 31) / 32 : total;
    const uint64_t blocks = (warps + cube::kIrrWarps - 1) / cube::kIrrWarps;
    const int block = 32 * cube::kIrrWarps, grid = grid_for(blocks * block, block);
    if (wide)
        cube::k_irradiance_random_wide<<<grid, block, 0, s>>>(im, width, height, samplesPerPixel, run, jumps,
            0x45BA12F3u, reinterpret_cast<float4 *>(faces));
    else
        cube::k_irradiance_random<<<grid, block, 0, s>>>(im, width, height, samplesPerPixel, jumps,
            0x45BA12F3u, reinterpret_cast<float4 *>(faces));
    GBSP_CUDA_TRY(cudaGetLastError());
    return GBSP_OK;
}

}  // extern "C"
