// CPU check of the cull's margins themselves (bvhtracer_gb300/csrc/cull.cuh): for single triangles
// that the reference's float test accepts, the exact intersection (long double) must lie within the
// margins leaf_cull computes -- |u* - u| + |v* - v| <= duv and |t* - t| <= dt0 + t dt1 -- with and
// without a normal cone.  Rays are aimed at interiors, edges and vertices, from near and far,
// grazing the plane so that |det| comes down to the acceptance threshold, axis-aligned and scaled.
// Usage: cull_margins <iterations> <margin scale>; a scale well below 1 shrinks the margins on
// purpose (violations must then appear).  Prints the largest error / margin ratios.
#include <cfloat>
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <random>

#include "cull.cuh"
using namespace bvhgpu;

struct V { float x, y, z; };
static inline V sub(V a, V b) { return {a.x - b.x, a.y - b.y, a.z - b.z}; }
static inline V cross(V a, V b) { return {a.y * b.z - a.z * b.y, a.z * b.x - a.x * b.z, a.x * b.y - a.y * b.x}; }
static inline float dot(V a, V b) { return (a.x * b.x + a.y * b.y) + a.z * b.z; }

int main(int argc, char** argv) {
    const long iters = argc > 1 ? atol(argv[1]) : 1000000;
    const double scale_margin = argc > 2 ? atof(argv[2]) : 1.0;
    std::mt19937_64 rng(99);
    std::uniform_real_distribution<double> U(0.0, 1.0);
    auto ur = [&](double a, double b) { return (float)(a + (b - a) * U(rng)); };
    long accepted = 0, low_det = 0, coned = 0, violations = 0;
    double worst_uv = 0.0, worst_t = 0.0;
    for (long it = 0; it < iters; ++it) {
        const double size = std::pow(10.0, ur(-1.7, 3.0));
        const float off = (float)(size * std::pow(10.0, ur(-1, 2)));
        V v0 = {ur(-1, 1) * off, ur(-1, 1) * off, ur(-1, 1) * off};
        const float es = (float)size, th = (float)std::pow(10.0, ur(-3, 0));
        V v1 = {v0.x + ur(-1, 1) * es, v0.y + ur(-1, 1) * es, v0.z + ur(-1, 1) * es};
        V v2 = {v0.x + ur(-1, 1) * es * th, v0.y + ur(-1, 1) * es, v0.z + ur(-1, 1) * es * th};
        const V e1 = sub(v1, v0), e2 = sub(v2, v0), nn = cross(e1, e2);
        double a = U(rng), b = U(rng) * (1 - a);
        const int mode = (int)(U(rng) * 4);
        if (mode == 0) b = 0;
        if (mode == 1) b = 1 - a;
        V d;
        if (U(rng) < 0.6) {  // grazing: in the plane, with a small normal part
            const float g = (float)std::pow(10.0, ur(-7, 0)) / std::sqrt(dot(nn, nn));
            const float w1 = ur(-1, 1) / es, w2 = ur(-1, 1) / es;
            d = {e1.x * w1 + e2.x * w2 + g * nn.x, e1.y * w1 + e2.y * w2 + g * nn.y, e1.z * w1 + e2.z * w2 + g * nn.z};
        } else {
            d = {ur(-1, 1), ur(-1, 1), ur(-1, 1)};
        }
        const float dl = std::sqrt(dot(d, d)) * (U(rng) < 0.2 ? ur(0.2, 5.0) : 1.0f);
        if (!(dl > 0.0f)) continue;
        d = {d.x / dl, d.y / dl, d.z / dl};
        if (U(rng) < 0.1) (&d.x)[(int)(U(rng) * 3)] = 0.0f;
        const float back = (float)(size * std::pow(10.0, ur(-2, 2)));
        V o = {(float)(v0.x + a * e1.x + b * e2.x) - d.x * back, (float)(v0.y + a * e1.y + b * e2.y) - d.y * back,
               (float)(v0.z + a * e1.z + b * e2.z) - d.z * back};
        // the reference's test (triangle.rs:42-72), float, unfused
        const V n = cross(d, e2);
        const float det = dot(e1, n);
        if (std::fabs(det) < 0.0001f) continue;
        const float f = 1.0f / det;
        const V s = sub(o, v0);
        const float u = f * dot(s, n);
        if (u < 0.0f || u > 1.0f) continue;
        const V q = cross(s, e1);
        const float v = f * dot(d, q);
        if (v < 0.0f || u + v > 1.0f) continue;
        const float t = f * dot(e2, q);
        if (!(t > 0.0001f)) continue;
        ++accepted;
        low_det += std::fabs(det) < 1e-3f;
        // the margins of a leaf holding just this triangle
        const V p1 = {v0.x + e1.x, v0.y + e1.y, v0.z + e1.z}, p2 = {v0.x + e2.x, v0.y + e2.y, v0.z + e2.z};
        float lo[3], hi[3];
        for (int i = 0; i < 3; ++i) {
            lo[i] = std::fmin((&v0.x)[i], std::fmin((&p1.x)[i], (&p2.x)[i]));
            hi[i] = std::fmax((&v0.x)[i], std::fmax((&p1.x)[i], (&p2.x)[i]));
        }
        const float m1 = std::fmax(std::fabs(e1.x), std::fmax(std::fabs(e1.y), std::fabs(e1.z)));
        const float m2 = std::fmax(std::fabs(e2.x), std::fmax(std::fabs(e2.y), std::fabs(e2.z)));
        const GroupSeal g = group_seal(lo, hi, m1, m2, true);
        LeafCone cone{nn.x, nn.y, nn.z, 0.0f, 0.0f, 0.0f};
        if (U(rng) < 0.5) {
            const float ca[3] = {e1.x, e1.y, e1.z}, cb[3] = {e2.x, e2.y, e2.z};
            cone_terms(ca, cb, cone.ax, cone.ay, cone.az, cone.cos_phi, cone.nmin);
            cone.sin_phi = cone_sin(cone.cos_phi);
            ++coned;
        }
        const LeafCull lc = leaf_cull(cull_ray(o.x, o.y, o.z, d.x, d.y, d.z), g.q, g.b, t, 1e30f, cone);
        if (!lc.on) continue;
        typedef long double L;
        const L sx = (L)o.x - v0.x, sy = (L)o.y - v0.y, sz = (L)o.z - v0.z;
        const L nx = (L)d.y * e2.z - (L)d.z * e2.y, ny = (L)d.z * e2.x - (L)d.x * e2.z, nz = (L)d.x * e2.y - (L)d.y * e2.x;
        const L D = e1.x * nx + e1.y * ny + e1.z * nz;
        const L qx = sy * e1.z - sz * e1.y, qy = sz * e1.x - sx * e1.z, qz = sx * e1.y - sy * e1.x;
        const L us = (sx * nx + sy * ny + sz * nz) / D, vs = (d.x * qx + d.y * qy + d.z * qz) / D;
        const L ts = (e2.x * qx + e2.y * qy + e2.z * qz) / D;
        const double ruv = (double)((fabsl(us - u) + fabsl(vs - v)) / (L)lc.duv) / scale_margin;
        const double rt = (double)(fabsl(ts - t) / ((L)lc.dt0 + (L)t * lc.dt1)) / scale_margin;
        worst_uv = std::fmax(worst_uv, ruv);
        worst_t = std::fmax(worst_t, rt);
        if (!(ruv <= 1.0) || !(rt <= 1.0)) ++violations;
    }
    printf("accepted %ld low-det %ld coned %ld violations %ld worst uv %.4f worst t %.4f\n", accepted, low_det, coned, violations,
           worst_uv, worst_t);
    return violations ? 1 : 0;
}
