#include "sah_build.h"

#include <algorithm>
#include <cstring>
#include <vector>

namespace gbsp {
namespace {

// 64 bins: on the 1080p benchmark scene 16, 32, 64 and 128 bins gave 6.71,
// 6.48, 6.45 and 6.44 node visits per ray (1,518, 1,542, 1,547 and 1,550
// Msamples/s) for a host build time that grows with the bin count.
constexpr int kSahBins = 64;

// Four floats in one register of either host's vector unit.
typedef float F4 __attribute__((vector_size(16)));

F4 load(const float4 &v)
{
    F4 r;
    memcpy(&r, &v, 16);
    return r;
}
void store(float4 &v, F4 r) { memcpy(&v, &r, 16); }
// keep a where b is not smaller (larger), also where b is NaN
F4 min_of(F4 a, F4 b) { return b < a ? b : a; }
F4 max_of(F4 a, F4 b) { return b > a ? b : a; }
// a node's box: rmin and rmax per lane
F4 box_min(F4 a, F4 b) { return a < b ? a : b; }
F4 box_max(F4 a, F4 b) { return a > b ? a : b; }

float half_area(F4 lo, F4 hi)
{
    const F4 d = hi - lo;
    return d[0] * d[1] + d[1] * d[2] + d[2] * d[0];
}

// Bins along one axis; a bin is set up by its first primitive, `used` marks
// the bins that hold one.
struct Bins {
    uint64_t used;
    uint32_t cnt[kSahBins];
    F4 lo[kSahBins], hi[kSahBins];
};
static_assert(kSahBins == 64, "one bit of Bins::used per bin");

int bin_of(float scaled) { return std::min(kSahBins - 1, std::max(0, (int)scaled)); }

}  // namespace

// Cost: most nodes of a binary tree hold a few primitives, so the sweeps visit
// the occupied bins only.  A split behind an empty bin has the cost of the one
// before it and never wins (the first of equal costs does), so the tree is the
// one that sweeps over all bins give.  A scene build of 257 objects took 739 us
// with full sweeps and scalar boxes (446 of them outside the collapse's waits),
// 195 with occupied bins, 127 with vector boxes and the axes binned together.
void sah_binary_tree(const float4 *plo, const float4 *phi, uint32_t n,
    const BinaryTree<float4, uint32_t> &t)
{
    std::copy(plo, plo + n, t.primLo);
    std::copy(phi, phi + n, t.primHi);
    std::vector<F4> cen(n);
    for (uint32_t i = 0; i < n; i++) {
        t.order[i] = i;
        cen[i] = (load(plo[i]) + load(phi[i])) * 0.5f;
    }
    struct Job {
        uint32_t node, begin, end;
    };
    std::vector<Job> jobs;
    jobs.push_back({0, 0, n});
    uint32_t next = 1;
    const float inf = 3.0e38f;
    const F4 emptyLo = {inf, inf, inf, 0.0f}, emptyHi = {-inf, -inf, -inf, 0.0f};
    static thread_local Bins bins[3];
    while (!jobs.empty()) {
        const Job j = jobs.back();
        jobs.pop_back();
        F4 blo = emptyLo, bhi = emptyHi, cmin = emptyLo, cmax = emptyHi;
        for (uint32_t k = j.begin; k < j.end; k++) {
            const uint32_t p = t.order[k];
            blo = box_min(blo, load(plo[p]));
            bhi = box_max(bhi, load(phi[p]));
            cmin = min_of(cmin, cen[p]);
            cmax = max_of(cmax, cen[p]);
        }
        store(t.nodeLo[j.node], blo);
        store(t.nodeHi[j.node], bhi);
        t.first[j.node] = j.begin;
        t.last[j.node] = j.end - 1;
        const F4 ext = cmax - cmin;
        F4 scale = {};
        for (int a = 0; a < 3; a++) {
            bins[a].used = 0;
            if (ext[a] > 0.0f) scale[a] = (float)kSahBins / ext[a];
        }
        for (uint32_t k = j.begin; k < j.end; k++) {
            const uint32_t p = t.order[k];
            const F4 at = (cen[p] - cmin) * scale, lo = load(plo[p]), hi = load(phi[p]);
            for (int a = 0; a < 3; a++) {
                Bins &bin = bins[a];
                const int b = bin_of(at[a]);
                if (!(bin.used >> b & 1u)) {
                    bin.used |= 1ull << b;
                    bin.cnt[b] = 1;
                    bin.lo[b] = min_of(emptyLo, lo);
                    bin.hi[b] = max_of(emptyHi, hi);
                } else {
                    bin.cnt[b]++;
                    bin.lo[b] = min_of(bin.lo[b], lo);
                    bin.hi[b] = max_of(bin.hi[b], hi);
                }
            }
        }
        int bestAxis = -1, bestBin = 0;
        float bestCost = inf;
        for (int a = 0; a < 3; a++) {
            if (!(ext[a] > 0.0f)) continue;
            const Bins &bin = bins[a];
            // suffix areas and counts behind each occupied bin, then a prefix sweep
            uint8_t at[kSahBins];
            int m = 0;
            for (uint64_t rest = bin.used; rest; rest &= rest - 1) at[m++] = (uint8_t)__builtin_ctzll(rest);
            float rArea[kSahBins];
            uint32_t rCnt[kSahBins];
            F4 lo = emptyLo, hi = emptyHi;
            uint32_t count = 0;
            for (int k = m - 1; k > 0; k--) {
                count += bin.cnt[at[k]];
                lo = min_of(lo, bin.lo[at[k]]);
                hi = max_of(hi, bin.hi[at[k]]);
                rCnt[k] = count;
                rArea[k] = half_area(lo, hi);
            }
            lo = emptyLo, hi = emptyHi;
            count = 0;
            for (int k = 0; k + 1 < m; k++) {
                count += bin.cnt[at[k]];
                lo = min_of(lo, bin.lo[at[k]]);
                hi = max_of(hi, bin.hi[at[k]]);
                const float cost = half_area(lo, hi) * (float)count + rArea[k + 1] * (float)rCnt[k + 1];
                if (cost < bestCost) {
                    bestCost = cost;
                    bestAxis = a;
                    bestBin = at[k];
                }
            }
        }
        uint32_t mid = j.begin + (j.end - j.begin) / 2;
        if (bestAxis >= 0) {
            const float s = scale[bestAxis], c0 = cmin[bestAxis];
            uint32_t *it = std::partition(t.order + j.begin, t.order + j.end,
                [&](uint32_t p) { return bin_of((cen[p][bestAxis] - c0) * s) <= bestBin; });
            const uint32_t m = (uint32_t)(it - t.order);
            if (m > j.begin && m < j.end) mid = m;
        }
        const uint32_t ranges[2][2] = {{j.begin, mid}, {mid, j.end}};
        for (int side = 0; side < 2; side++) {
            const uint32_t b = ranges[side][0], e = ranges[side][1];
            uint32_t ref;
            if (e - b == 1) {
                ref = kBinLeaf | b;
            } else {
                ref = next++;
                jobs.push_back({ref, b, e});
            }
            (side ? t.right : t.left)[j.node] = ref;
        }
    }
}

}  // namespace gbsp
