// Triangle clusters of the compute-shader path tracer, and the test that lets
// a ray skip one without changing any result.
//
// The shader tests every triangle with a Moller-Trumbore test in float, no
// box and no culling, so which triangles count as hit is decided by rounding
// too: a ray that runs almost inside a triangle's plane can be accepted
// although it passes far beside the triangle.  cluster_may_hit therefore
// rejects a cluster only where no such rounding is possible.
//
// Bound.  With T = o - a, unit roundoff u = 2^-24 and |d| = 1 (unit_directions
// says for which entities that holds; the others test all clusters), the computed
// numerators and determinant of the test are off by at most 8 u times the
// product of the vectors in them (7 u counted, no contraction; with edges of
// 1e-15 to 1e15 what underflow adds, 2^-147 at most, is below u |e| (|T| + L), and
// no determinant is so large that its reciprocal is denormal; a cluster with any
// other edge is always tested).  Let the test
// accept with barycentrics (x, y), p = a + x e1 + y e2 (within a few u of the
// triangle), r = o - p, and r' its part perpendicular to d.  Then
//     |r' . (d x e_i)| <= h |e_i|,   h = 8 u (|T| + L),  L = max |e_i|,
// and with n = e1 x e2, k = |e1||e2| / |n| and c = |d . n| / |n|:
//   (1) |r'| <= 2 h k / c            (solve the two equations for r')
//   (2) |r' . n| / |n| <= 2 h k      (expand n in the e_i)
// So a triangle that the ray passes at more than m = 1e-3 (|T| + L) can only
// be accepted if c < 2 h k / m <= 1e-3 k (edge-on) AND its plane passes
// within 2 h k of the ray's line.  A cluster keeps bounds of its triangles'
// positions (sphere), normals (cone), k, L and plane offsets; it is rejected
// when the ray misses the sphere by more than m and no normal in the cone
// meets both conditions: with q the perpendicular from the line to the centre
// they say |d . n| <= D1 and |q . n| <= D2, so n lies within asin(x), x = D1 +
// D2 / |q|, of the axis +-(d x q), and the cone (axis A, half angle y) holds
// no such n if 1 - (A . (d x q) / |q|)^2 = (A . d)^2 + (A . q)^2 / |q|^2 exceeds
// (sin y + x)^2.  Every quantity is rounded towards keeping the cluster, and
// anything not finite keeps it.
#pragma once

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <vector>

#include "gbsp_common.cuh"

namespace gbsp {
namespace cpt {

constexpr uint32_t kClusterTris = 16;  // triangles per cluster at most: half a warp

// 48 bytes, read as three 128-bit loads.
struct __align__(16) Cluster {
    float4 sphere;  // centre, radius (infinite: always tested)
    float4 cone;    // axis, sine of the half angle + 1.01e-3 k (rounded up)
    float4 edge;    // plane offset, 1.01e-6 k + 1e-5, L, unused
};

GBSP_HD float cdot(V3 a, V3 b) { return (a.x * b.x + a.y * b.y) + a.z * b.z; }
GBSP_HD V3 ccross(V3 a, V3 b)
{
    return v3(a.y * b.z - a.z * b.y, a.z * b.x - a.x * b.z, a.x * b.y - a.y * b.x);
}

// The shader's triangle test (src/shaders/test_compute.comp.glsl:320-430).
struct MtHit {
    float t, u, v;
    bool ok;
};
GBSP_HD MtHit mt_test(V3 lo, V3 ld, V3 a, V3 e1, V3 e2, float tMax)
{
    MtHit r;
    V3 T = v3(lo.x - a.x, lo.y - a.y, lo.z - a.z);
    V3 p = ccross(ld, e2);
    V3 q = ccross(T, e1);
    float mx = cdot(q, e2), my = cdot(p, T), mz = cdot(q, ld);
    float det = 1.0f / cdot(p, e1);
    r.t = det * mx;
    r.u = det * my;
    r.v = det * mz;
    float w = 1.0f - r.u - r.v;
    r.ok = r.u >= 0.0f && r.u <= 1.0f && r.v >= 0.0f && r.v <= 1.0f && w >= 0.0f && w <= 1.0f &&
        r.t >= 0.0f && r.t < tMax;
    return r;
}

// Products added without a rounding in between: for the bounds below, not for
// the shader's own arithmetic.
GBSP_HD float fdot(V3 a, V3 b) { return fmaf(a.z, b.z, fmaf(a.y, b.y, a.x * b.x)); }

GBSP_HD float inverse_sqrt(float x)
{
#ifdef __CUDA_ARCH__
    return rsqrtf(x);  // 2 ulp, covered by the margins below
#else
    return 1.0f / sqrtf(x);
#endif
}

// False only if mt_test accepts none of the cluster's triangles for the ray
// (lo, ld), ld of unit length up to rounding.
GBSP_HD bool cluster_may_hit(float4 sphere, float4 cone, float4 edge, V3 lo, V3 ld)
{
    const V3 w = v3(sphere.x - lo.x, sphere.y - lo.y, sphere.z - lo.z);
    const float s = fdot(w, ld);
    // from the line to the centre
    const V3 q = v3(fmaf(-ld.x, s, w.x), fmaf(-ld.y, s, w.y), fmaf(-ld.z, s, w.z));
    const float q2 = fdot(q, q), iq = inverse_sqrt(q2), ql = q2 * iq;
    // >= |T| + L: |w| is at most |s| + |q|
    const float far = fmaf(fabsf(s) + ql, 1.0001f, sphere.w + edge.z);
    const float c = fdot(ld, v3(cone.x, cone.y, cone.z));
    const float e = fdot(q, v3(cone.x, cone.y, cone.z)) * iq;
    const float reach = fmaf(fmaf(edge.y, far, edge.x), iq, cone.w);  // sin y + x
    const bool outside = ql > fmaf(1.01e-3f, far, sphere.w);
    const bool away = fmaf(c, c, e * e) > fmaf(reach * reach, 1.0001f, 1e-5f);
    return !(outside && away);
}

// Whether every unit direction d comes out of an entity's space with unit length:
// v / |v| in floats, v = R d with R the upper 3 x 3 of inv (column-major 4 x 4), has
// unit length up to 12 u unless the squares in |v| are denormal, |v| below 1e-18.
// |v| is at least the smallest singular value of R, itself at least 1 / |R^-1|, less
// the rounding of the product, 3 u |R|.
inline bool unit_directions(const float *inv)
{
    double r[9], norm = 0.0, adj = 0.0;
    for (int k = 0; k < 9; k++) {
        r[k] = inv[4 * (k / 3) + k % 3];
        norm += r[k] * r[k];
    }
    double det = 0.0;
    for (int i = 0; i < 3; i++)
        for (int j = 0; j < 3; j++) {
            const double c = r[3 * ((i + 1) % 3) + (j + 1) % 3] * r[3 * ((i + 2) % 3) + (j + 2) % 3] -
                r[3 * ((i + 1) % 3) + (j + 2) % 3] * r[3 * ((i + 2) % 3) + (j + 1) % 3];
            adj += c * c;
            if (i == 0) det += r[j] * c;
        }
    const double smallest = std::fabs(det) / std::sqrt(adj);
    return smallest >= 1e-16 && smallest >= 1e-6 * std::sqrt(norm) && std::isfinite(norm);
}

// Builds the clusters of one mesh: triangle k has vertex a[k] and edges e1[k],
// e2[k] (floats as the test uses them).  order receives the triangles cluster
// by cluster, cluster c holding order[16 c ..] (the last places of a cluster
// may be ~0: empty).  Clusters come from median splits along the widest axis
// of the triangles' centres (in units of the mesh's extent) or normals.
struct ClusterTriangles {
    const V3 *a, *e1, *e2;
    uint32_t count;
};

inline void build_clusters(const ClusterTriangles &t, std::vector<Cluster> &clusters,
    std::vector<uint32_t> &order)
{
    struct D3 {
        double x, y, z;
    };
    const auto sub3 = [](D3 p, D3 q) { return D3{p.x - q.x, p.y - q.y, p.z - q.z}; };
    const auto dot3 = [](D3 p, D3 q) { return p.x * q.x + p.y * q.y + p.z * q.z; };
    const auto cross3 = [](D3 p, D3 q) {
        return D3{p.y * q.z - p.z * q.y, p.z * q.x - p.x * q.z, p.x * q.y - p.y * q.x};
    };
    const auto d3 = [](V3 p) { return D3{p.x, p.y, p.z}; };
    const uint32_t n = t.count;
    std::vector<float> key(6 * (size_t)n);
    double lo[3] = {1e300, 1e300, 1e300}, hi[3] = {-1e300, -1e300, -1e300};
    for (uint32_t k = 0; k < n; k++) {
        const D3 a = d3(t.a[k]), e1 = d3(t.e1[k]), e2 = d3(t.e2[k]);
        const double c[3] = {a.x + (e1.x + e2.x) / 3, a.y + (e1.y + e2.y) / 3, a.z + (e1.z + e2.z) / 3};
        const D3 m = cross3(e1, e2);
        const double len = std::sqrt(dot3(m, m));
        const double v[3] = {m.x, m.y, m.z};
        for (int j = 0; j < 3; j++) {
            const double x = std::isfinite(c[j]) ? c[j] : 0.0;
            key[6 * (size_t)k + j] = (float)x;
            key[6 * (size_t)k + 3 + j] = len > 0.0 && std::isfinite(len) ? (float)(v[j] / len) : 0.0f;
            lo[j] = std::min(lo[j], x);
            hi[j] = std::max(hi[j], x);
        }
    }
    const double extent = std::max({hi[0] - lo[0], hi[1] - lo[1], hi[2] - lo[2]});
    for (uint32_t k = 0; k < n; k++)
        for (int j = 0; j < 3; j++)
            key[6 * (size_t)k + j] = extent > 0.0 ? (float)((key[6 * (size_t)k + j] - lo[j]) / extent * 2.0) : 0.0f;
    std::vector<uint32_t> idx(n);
    for (uint32_t k = 0; k < n; k++) idx[k] = k;
    std::vector<std::pair<uint32_t, uint32_t>> jobs;
    if (n) jobs.push_back({0u, n});
    while (!jobs.empty()) {
        const auto [b, e] = jobs.back();
        jobs.pop_back();
        if (e - b > kClusterTris) {
            int axis = 0;
            float widest = -1.0f;
            for (int j = 0; j < 6; j++) {
                float mn = 3e38f, mx = -3e38f;
                for (uint32_t k = b; k < e; k++) {
                    mn = std::min(mn, key[6 * (size_t)idx[k] + j]);
                    mx = std::max(mx, key[6 * (size_t)idx[k] + j]);
                }
                if (mx - mn > widest) {
                    widest = mx - mn;
                    axis = j;
                }
            }
            const uint32_t half = ((e - b) / 2 + kClusterTris - 1) / kClusterTris * kClusterTris;
            std::nth_element(idx.begin() + b, idx.begin() + b + half, idx.begin() + e,
                [&](uint32_t p, uint32_t q) {
                    const float kp = key[6 * (size_t)p + axis], kq = key[6 * (size_t)q + axis];
                    return kp < kq || (kp == kq && p < q);
                });
            jobs.push_back({b + half, e});
            jobs.push_back({b, b + half});
            continue;
        }
        // bounds of the cluster, in double, then rounded outward
        D3 bl{1e300, 1e300, 1e300}, bh{-1e300, -1e300, -1e300}, mean{0, 0, 0};
        bool bad = false;
        double k1 = 0.0, edgeMax = 0.0;
        for (uint32_t k = b; k < e; k++) {
            const D3 a = d3(t.a[idx[k]]), e1 = d3(t.e1[idx[k]]), e2 = d3(t.e2[idx[k]]);
            const D3 v[3] = {a, {a.x + e1.x, a.y + e1.y, a.z + e1.z}, {a.x + e2.x, a.y + e2.y, a.z + e2.z}};
            for (const D3 &p : v) {
                bad = bad || !(std::isfinite(p.x) && std::isfinite(p.y) && std::isfinite(p.z));
                bl = {std::min(bl.x, p.x), std::min(bl.y, p.y), std::min(bl.z, p.z)};
                bh = {std::max(bh.x, p.x), std::max(bh.y, p.y), std::max(bh.z, p.z)};
            }
            const D3 m = cross3(e1, e2);
            const double len = std::sqrt(dot3(m, m)), l1 = std::sqrt(dot3(e1, e1)), l2 = std::sqrt(dot3(e2, e2));
            if (!(len > 1e-9 * l1 * l2) || !(std::min(l1, l2) >= 1e-15 && std::max(l1, l2) <= 1e15)) {
                bad = true;
                continue;
            }
            k1 = std::max(k1, l1 * l2 / len);
            edgeMax = std::max({edgeMax, l1, l2});
            mean = {mean.x + m.x / len, mean.y + m.y / len, mean.z + m.z / len};
        }
        Cluster c = {};
        const float cx = (float)((bl.x + bh.x) / 2), cy = (float)((bl.y + bh.y) / 2),
                    cz = (float)((bl.z + bh.z) / 2);
        const D3 centre{cx, cy, cz};
        double meanLen = std::sqrt(dot3(mean, mean));
        const D3 axisD = meanLen > 1e-6 ? D3{mean.x / meanLen, mean.y / meanLen, mean.z / meanLen} : D3{0, 0, 1};
        const float ax = (float)axisD.x, ay = (float)axisD.y, az = (float)axisD.z;
        double rho = 0.0, cosMin = 1.0, offset = 0.0;
        for (uint32_t k = b; k < e && !bad; k++) {
            const D3 a = d3(t.a[idx[k]]), e1 = d3(t.e1[idx[k]]), e2 = d3(t.e2[idx[k]]);
            const D3 v[3] = {a, {a.x + e1.x, a.y + e1.y, a.z + e1.z}, {a.x + e2.x, a.y + e2.y, a.z + e2.z}};
            for (const D3 &p : v) rho = std::max(rho, std::sqrt(dot3(sub3(p, centre), sub3(p, centre))));
            const D3 m = cross3(e1, e2);
            const double len = std::sqrt(dot3(m, m));
            cosMin = std::min(cosMin, (m.x * ax + m.y * ay + m.z * az) / len);
            offset = std::max(offset, std::fabs(dot3(m, sub3(a, centre)) / len));
        }
        // a cone of more than 80 degrees bounds nothing useful
        if (cosMin < 0.17) cosMin = -1.0;
        if (bad || !std::isfinite(rho)) {
            c.sphere = make_float4(0, 0, 0, INFINITY);
        } else {
            const double r = rho * 1.0001 + 1e-6 * edgeMax;
            const double sinA = cosMin < 0 ? 1.0 :
                std::min(1.0, std::sqrt(1.0 - std::min(1.0, cosMin * cosMin)) + 1e-3);
            c.sphere = make_float4(cx, cy, cz, (float)r);
            c.cone = make_float4(ax, ay, az, (float)((sinA + 1.01e-3 * k1) * 1.0001));
            c.edge = make_float4((float)((offset + r * 1.01e-3 * k1) * 1.0001), (float)(1.01e-6 * k1 + 1e-5),
                (float)(edgeMax * 1.0001), 0);
        }
        clusters.push_back(c);
        for (uint32_t k = 0; k < kClusterTris; k++) order.push_back(b + k < e ? idx[b + k] : 0xFFFFFFFFu);
    }
}

}  // namespace cpt
}  // namespace gbsp
