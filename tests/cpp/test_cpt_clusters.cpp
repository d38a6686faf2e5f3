// CPU check of the compute path tracer's cluster rejection: for many meshes and
// rays (edge-on ones among them) no triangle of a rejected cluster is accepted
// by the triangle test.  Prints the share of rejected clusters per set.
#include <cstdio>
#include <cstdlib>
#include <random>

#include "cpt_clusters.h"

using namespace gbsp;
using namespace gbsp::cpt;

static std::mt19937 g_rng(7);
static float uni(float a, float b) { return std::uniform_real_distribution<float>(a, b)(g_rng); }
static V3 unit()
{
    std::normal_distribution<float> n;
    V3 v = v3(n(g_rng), n(g_rng), n(g_rng));
    float inv = 1.0f / sqrtf(cdot(v, v));
    return v3(v.x * inv, v.y * inv, v.z * inv);
}
static V3 shader_normalize(V3 v)
{
    float inv = 1.0f / sqrtf(cdot(v, v));
    return v3(v.x * inv, v.y * inv, v.z * inv);
}

struct Mesh {
    std::vector<V3> a, e1, e2;
    void tri(V3 p, V3 q, V3 r)
    {
        a.push_back(p);
        e1.push_back(sub(q, p));
        e2.push_back(sub(r, p));
    }
};

// latitude-longitude sphere: slivers and (at the poles) degenerate triangles
static Mesh sphere(int rows, float radius, V3 at)
{
    Mesh m;
    const auto p = [&](int i, int j) {
        float th = 3.14159265f * i / rows, ph = 6.2831853f * j / (2 * rows);
        return v3(at.x + radius * sinf(th) * cosf(ph), at.y + radius * cosf(th),
            at.z + radius * sinf(th) * sinf(ph));
    };
    for (int i = 0; i < rows; i++)
        for (int j = 0; j < 2 * rows; j++) {
            m.tri(p(i, j), p(i + 1, j), p(i, j + 1));
            m.tri(p(i + 1, j), p(i + 1, j + 1), p(i, j + 1));
        }
    return m;
}
static Mesh soup(int n, float size, float spread, float sliver)
{
    Mesh m;
    for (int k = 0; k < n; k++) {
        V3 c = mul(unit(), uni(0, spread)), u = mul(unit(), size), v = mul(unit(), size * sliver);
        m.tri(c, add(c, u), add(add(c, mul(u, uni(0, 1))), v));
    }
    return m;
}
static Mesh grid(int n, float step, float tilt)  // one plane
{
    Mesh m;
    const auto p = [&](int i, int j) { return v3(i * step, (i + 0.3f * j) * step * tilt, j * step); };
    for (int i = 0; i < n; i++)
        for (int j = 0; j < n; j++) {
            m.tri(p(i, j), p(i + 1, j), p(i, j + 1));
            m.tri(p(i + 1, j), p(i + 1, j + 1), p(i, j + 1));
        }
    return m;
}

static long long run(const char *name, const Mesh &m, int rays, float dist)
{
    std::vector<Cluster> cl;
    std::vector<uint32_t> order;
    build_clusters({m.a.data(), m.e1.data(), m.e2.data(), (uint32_t)m.a.size()}, cl, order);
    std::vector<int> seen(m.a.size(), 0);
    for (uint32_t k : order)
        if (k != 0xFFFFFFFFu) seen[k]++;
    for (int s : seen)
        if (s != 1) {
            printf("%s: order is not a permutation\n", name);
            return 1;
        }
    long long wrong = 0, rejected = 0, accepted = 0, total = 0;
    for (int r = 0; r < rays; r++) {
        V3 o, d;
        const uint32_t k = g_rng() % m.a.size();
        const float eps = powf(10.0f, uni(-9, -2)) * (g_rng() % 4 ? 1.0f : 0.0f);
        const V3 n = ccross(m.e1[k], m.e2[k]);
        switch (r % 4) {
        case 0:  // anything
            o = mul(unit(), dist * uni(0.2f, 1));
            d = unit();
            break;
        case 1:  // at a triangle
            o = mul(unit(), dist * uni(0.2f, 1));
            d = sub(add(m.a[k], mul(m.e1[k], uni(0, 0.5f))), o);
            break;
        case 2:  // in a triangle's plane, up to eps, from afar
            o = add(add(m.a[k], mul(m.e1[k], dist * uni(-1, 1) / sqrtf(cdot(m.e1[k], m.e1[k]) + 1e-30f))),
                mul(m.e2[k], uni(-3, 3)));
            d = add(add(mul(m.e1[k], uni(-1, 1)), mul(m.e2[k], uni(-1, 1))),
                mul(n, eps / sqrtf(cdot(n, n) + 1e-30f)));
            break;
        default:  // leaving a triangle along its plane
            o = add(add(m.a[k], mul(m.e1[k], uni(0, 1))), mul(shader_normalize(n), 0.001f * (g_rng() % 2)));
            d = add(add(mul(m.e1[k], uni(-1, 1)), mul(m.e2[k], uni(-1, 1))), mul(unit(), eps));
        }
        d = shader_normalize(d);
        for (size_t c = 0; c < cl.size(); c++) {
            const bool may = cluster_may_hit(cl[c].sphere, cl[c].cone, cl[c].edge, o, d);
            total++;
            rejected += !may;
            for (uint32_t j = 0; j < kClusterTris; j++) {
                const uint32_t t = order[c * kClusterTris + j];
                if (t == 0xFFFFFFFFu) continue;
                if (!mt_test(o, d, m.a[t], m.e1[t], m.e2[t], 3.402823466e+38f).ok) continue;
                accepted++;
                wrong += !may;
            }
        }
    }
    printf("%-16s %6zu triangles: %5.1f%% of clusters rejected, %lld accepted tests, %lld in rejected clusters\n",
        name, m.a.size(), 100.0 * rejected / total, accepted, wrong);
    return wrong;
}

int main(int argc, char **argv)
{
    const int rays = argc > 1 ? atoi(argv[1]) : 4000;
    long long wrong = 0;
    wrong += run("sphere", sphere(16, 1, v3(0, 0, 0)), rays, 30);
    wrong += run("sphere far", sphere(16, 1, v3(0, 0, 0)), rays, 3000);
    wrong += run("sphere offset", sphere(12, 1, v3(500, -200, 80)), rays, 900);
    wrong += run("fine sphere", sphere(40, 5, v3(0, 1, 0)), rays / 8, 60);
    wrong += run("soup", soup(600, 0.1f, 3, 1), rays, 20);
    wrong += run("slivers", soup(600, 0.5f, 3, 1e-4f), rays, 20);
    wrong += run("needles", soup(600, 2, 3, 1e-7f), rays, 20);
    wrong += run("plane", grid(12, 1, 0), rays, 50);
    wrong += run("tilted plane", grid(12, 1, 0.37f), rays, 50);
    wrong += run("quad", grid(1, 50, 0), rays, 50);
    return wrong ? 1 : 0;
}
