// The SAH build against a plain restatement that sweeps every bin of every
// axis: the same tree, order and boxes, bit for bit.
#include <algorithm>
#include <cstdio>
#include <cstring>
#include <random>
#include <vector>

#include "sah_build.h"

using namespace gbsp;
typedef BinaryTree<float4, uint32_t> Tree;
static const float inf = 3.0e38f;

struct Box {
    float lo[3], hi[3];
    Box() { for (int a = 0; a < 3; a++) lo[a] = inf, hi[a] = -inf; }
    void add(const Box &b)
    {
        for (int a = 0; a < 3; a++) lo[a] = std::min(lo[a], b.lo[a]), hi[a] = std::max(hi[a], b.hi[a]);
    }
    float area() const
    {
        const float x = hi[0] - lo[0], y = hi[1] - lo[1], z = hi[2] - lo[2];
        return x * y + y * z + z * x;
    }
};

struct Plain {
    const std::vector<Box> &prim;
    const Tree &t;
    uint32_t next = 1;
    float cen(uint32_t p, int a) const { return (prim[p].lo[a] + prim[p].hi[a]) * 0.5f; }
    struct Job { uint32_t node, b, e; };
    void run(uint32_t n)
    {
        for (uint32_t i = 0; i < n; i++) t.order[i] = i;
        std::vector<Job> jobs{{0, 0, n}};
        while (!jobs.empty()) {
            const Job j = jobs.back();
            jobs.pop_back();
            Box all;
            float c0[3] = {inf, inf, inf}, c1[3] = {-inf, -inf, -inf};
            for (uint32_t k = j.b; k < j.e; k++) {
                all.add(prim[t.order[k]]);
                for (int a = 0; a < 3; a++) {
                    c0[a] = std::min(c0[a], cen(t.order[k], a));
                    c1[a] = std::max(c1[a], cen(t.order[k], a));
                }
            }
            t.nodeLo[j.node] = float4{all.lo[0], all.lo[1], all.lo[2], 0.0f};
            t.nodeHi[j.node] = float4{all.hi[0], all.hi[1], all.hi[2], 0.0f};
            t.first[j.node] = j.b;
            t.last[j.node] = j.e - 1;
            int axis = -1, split = 0;
            float best = inf;
            auto bin = [&](uint32_t p, int a) {
                return std::min(63, (int)((cen(p, a) - c0[a]) * (64.0f / (c1[a] - c0[a]))));
            };
            for (int a = 0; a < 3; a++) {
                if (!(c1[a] > c0[a])) continue;
                for (int s = 0; s < 63; s++) {
                    Box l, r;
                    uint32_t nl = 0, nr = 0;
                    for (uint32_t k = j.b; k < j.e; k++) {
                        const uint32_t p = t.order[k];
                        if (bin(p, a) <= s) l.add(prim[p]), nl++;
                        else r.add(prim[p]), nr++;
                    }
                    if (!nl || !nr) continue;
                    const float cost = l.area() * (float)nl + r.area() * (float)nr;
                    if (cost < best) best = cost, axis = a, split = s;
                }
            }
            uint32_t mid = j.b + (j.e - j.b) / 2;
            if (axis >= 0) {
                uint32_t *it = std::partition(t.order + j.b, t.order + j.e,
                    [&](uint32_t p) { return bin(p, axis) <= split; });
                if (it > t.order + j.b && it < t.order + j.e) mid = (uint32_t)(it - t.order);
            }
            const uint32_t r[2][2] = {{j.b, mid}, {mid, j.e}};
            for (int s = 0; s < 2; s++) {
                uint32_t ref = kBinLeaf | r[s][0];
                if (r[s][1] - r[s][0] > 1) {
                    ref = next++;
                    jobs.push_back({ref, r[s][0], r[s][1]});
                }
                (s ? t.right : t.left)[j.node] = ref;
            }
        }
    }
};

int main()
{
    std::mt19937 rng(7);
    std::uniform_real_distribution<float> u(-1.0f, 1.0f);
    int bad = 0;
    for (const uint32_t n : {2u, 3u, 4u, 7u, 64u, 65u, 257u, 900u})
        for (int kind = 0; kind < 5; kind++) {
            std::vector<Box> prim(n);
            std::vector<float4> lo(n), hi(n);
            for (uint32_t i = 0; i < n; i++) {
                for (int a = 0; a < 3; a++) {
                    float c = 10.0f * u(rng), h = 0.2f + 0.1f * u(rng);
                    if (kind == 1) c = (float)((i >> (3 * a)) & 7u);            // a grid: equal costs
                    if (kind == 2) c = a == 1 ? c : 0.0f;                       // one axis only
                    if (kind == 3) c = 2.0f;                                    // every centroid equal
                    if (kind == 4) c = i ? 1.0e-3f * u(rng) : 1.0e4f, h = 0.0f; // one far away, no extent
                    prim[i].lo[a] = c - h, prim[i].hi[a] = c + h;
                }
                lo[i] = float4{prim[i].lo[0], prim[i].lo[1], prim[i].lo[2], 0.0f};
                hi[i] = float4{prim[i].hi[0], prim[i].hi[1], prim[i].hi[2], 0.0f};
            }
            std::vector<float4> ma(Tree::size(n)), mb(Tree::size(n));
            const Tree a(ma.data(), n), b(mb.data(), n);
            sah_binary_tree(lo.data(), hi.data(), n, a);
            Plain{prim, b}.run(n);
            bool same = !memcmp(a.order, b.order, 4 * n);
            for (uint32_t k = 0; k + 1 < n; k++)
                same = same && a.left[k] == b.left[k] && a.right[k] == b.right[k] && a.first[k] == b.first[k] &&
                    a.last[k] == b.last[k] && !memcmp(&a.nodeLo[k], &b.nodeLo[k], 16) &&
                    !memcmp(&a.nodeHi[k], &b.nodeHi[k], 16);
            same = same && !memcmp(a.primLo, lo.data(), 16 * n) && !memcmp(a.primHi, hi.data(), 16 * n);
            if (!same) bad++, printf("n %u kind %d differs\n", n, kind);
        }
    printf("%d differ\n", bad);
    return bad != 0;
}
