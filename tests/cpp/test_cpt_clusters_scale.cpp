// CPU check of the compute path tracer's cluster rejection where floats run out
// of exponent: rays whose direction comes out of a normalisation that underflows,
// meshes so small or large that products of their edges under- or overflow.  No
// triangle of a rejected cluster is accepted by the triangle test, and what the
// bound does not cover has no finite sphere.
#include <cstdio>
#include <random>

#include "cpt_clusters.h"

using namespace gbsp;
using namespace gbsp::cpt;

static std::mt19937 g_rng(11);
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
    std::vector<Cluster> clusters;
    std::vector<uint32_t> order;
    void tri(V3 p, V3 q, V3 r)
    {
        a.push_back(p);
        e1.push_back(sub(q, p));
        e2.push_back(sub(r, p));
    }
};

// a sphere (size > 0) or a soup of small triangles (size < 0) across `scale`
static Mesh mesh(float scale, float size)
{
    Mesh m;
    if (size > 0.0f) {
        const int rows = 12;
        const auto p = [&](int i, int j) {
            float th = 3.14159265f * i / rows, ph = 6.2831853f * j / (2 * rows);
            return mul(v3(sinf(th) * cosf(ph), cosf(th), sinf(th) * sinf(ph)), scale);
        };
        for (int i = 0; i < rows; i++)
            for (int j = 0; j < 2 * rows; j++) {
                m.tri(p(i, j), p(i + 1, j), p(i, j + 1));
                m.tri(p(i + 1, j), p(i + 1, j + 1), p(i, j + 1));
            }
    } else {
        for (int k = 0; k < 400; k++) {
            V3 c = mul(unit(), scale * uni(0, 1)), u = mul(unit(), -size * scale), v = mul(unit(), -size * scale);
            m.tri(c, add(c, u), add(c, v));
        }
    }
    build_clusters({m.a.data(), m.e1.data(), m.e2.data(), (uint32_t)m.a.size()}, m.clusters, m.order);
    return m;
}

// an entity's inverse matrix: rotated axes scaled by `length`, up to 2, or with
// `flat` one axis up to 1e-12 of that
struct Inverse {
    float m[16] = {}, s[3];
    V3 axis[3];
    Inverse(float length, bool flat)
    {
        axis[0] = unit();
        axis[2] = shader_normalize(ccross(axis[0], unit()));
        axis[1] = ccross(axis[2], axis[0]);
        s[0] = 1.0f, s[1] = uni(1, 2), s[2] = flat ? powf(10.0f, uni(-12, 0)) : uni(1, 2);
        for (int c = 0; c < 3; c++) {
            m[4 * c] = axis[c].x * (length * s[c]);
            m[4 * c + 1] = axis[c].y * (length * s[c]);
            m[4 * c + 2] = axis[c].z * (length * s[c]);
        }
        m[15] = 1.0f;
    }
    // the world direction that becomes t
    V3 world(V3 t) const
    {
        return shader_normalize(v3(cdot(axis[0], t) / s[0], cdot(axis[1], t) / s[1], cdot(axis[2], t) / s[2]));
    }
    V3 direction(V3 d) const
    {
        return shader_normalize(v3((m[0] * d.x + m[4] * d.y) + m[8] * d.z, (m[1] * d.x + m[5] * d.y) + m[9] * d.z,
            (m[2] * d.x + m[6] * d.y) + m[10] * d.z));
    }
};

// rays among and around the mesh, out of the spaces of entities
static long long run(const Mesh &m, float scale, float length, int rays, long long &accepted, long long &rejected)
{
    long long wrong = 0;
    for (int r = 0; r < rays; r++) {
        const uint32_t k = g_rng() % m.a.size();
        const V3 o = mul(unit(), scale * (r % 3 ? uni(0, 2) : uni(0, 40)));
        V3 d = unit();
        if (r % 2) d = shader_normalize(mul(sub(add(m.a[k], mul(m.e1[k], uni(0, 0.5f))), o), 1.0f / scale));
        if (r % 4 == 2)  // along a triangle's plane
            d = shader_normalize(mul(add(mul(m.e1[k], uni(-1, 1)), mul(m.e2[k], uni(-1, 1))), 1.0f / scale));
        bool apply = true;
        if (length != 1.0f) {
            const Inverse inverse(length, r % 5 == 0);
            d = inverse.direction(inverse.world(d));
            apply = unit_directions(inverse.m);
            wrong += apply && !(fabsf(cdot(d, d) - 1.0f) <= 1e-6f);
        }
        for (size_t c = 0; c < m.clusters.size(); c++) {
            const Cluster &cl = m.clusters[c];
            const bool may = !apply || cluster_may_hit(cl.sphere, cl.cone, cl.edge, o, d);
            rejected += !may;
            for (uint32_t j = 0; j < kClusterTris; j++) {
                const uint32_t t = m.order[c * kClusterTris + j];
                if (t == 0xFFFFFFFFu) continue;
                if (!mt_test(o, d, m.a[t], m.e1[t], m.e2[t], 3.402823466e+38f).ok) continue;
                accepted++;
                wrong += !may;
            }
        }
    }
    return wrong;
}

int main(int, char **)
{
    long long all = 0;
    for (float size : {1.0f, -0.3f, -0.02f}) {
        const Mesh m = mesh(1.0f, size);
        for (int e = 0; e <= 23; e++) {
            long long accepted = 0, rejected = 0;
            const float length = 0.999f * powf(10.0f, (float)-e);
            const long long wrong = run(m, 1.0f, length, 1500, accepted, rejected);
            printf("size %5.2f direction %g: %lld accepted, %lld clusters rejected, %lld wrong\n", size, length,
                accepted, rejected, wrong);
            all += wrong;
            // the rejection still has to reject where it applies
            if (e <= 15 && rejected == 0) all++;
        }
    }
    for (float size : {1.0f, -0.3f, -0.02f})
        for (int e = -22; e <= 20; e++) {
            long long accepted = 0, rejected = 0;
            const float scale = powf(10.0f, (float)e);
            const Mesh m = mesh(scale, size);
            const long long wrong = run(m, scale, 1.0f, 600, accepted, rejected);
            int open = 0;
            for (const Cluster &c : m.clusters) open += std::isinf(c.sphere.w);
            printf("size %5.2f scale %g: %lld accepted, %lld clusters rejected, %d of %zu open, %lld wrong\n", size,
                scale, accepted, rejected, open, m.clusters.size(), wrong);
            all += wrong;
            // the longest edge is below 0.6 of the scale, the shortest above 1e-6 of it
            // (without area: pole triangles, always tested)
            if (e <= -15 || e >= 17) all += open != (int)m.clusters.size();
            if (e >= -12 && e <= 14 && size < 0.0f) all += open != 0 || rejected == 0;
        }
    return all ? 1 : 0;
}
