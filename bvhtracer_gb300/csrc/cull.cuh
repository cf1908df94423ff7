// Conservative culling of groups of triangles inside a leaf, with results identical to testing
// every triangle.
//
// The reference tests every triangle of a leaf with its float Moeller-Trumbore test
// (triangle.rs:42-72); its BVHs are nearly flat, so leaves hold thousands of triangles.  The
// library puts a hidden tree of boxes over the triangles of each large leaf, and a box is skipped
// for a ray only when no triangle in it can be accepted by that float test with a t at or below the
// ray's current closest t -- so the closest hit (and its ties, decided by triangle index) is
// unchanged.
//
// Why skipping is safe.  For float inputs o, d, v0, e1, e2 the test computes (each step rounded,
// no fused multiply-add) n = d x e2, det = e1.n, s = o - v0, u = (s.n)/det, q = s x e1,
// v = (d.q)/det, t = (e2.q)/det and accepts when |det| >= 1e-4, 0 <= u <= 1, 0 <= v, u + v <= 1
// and t > 1e-4.  Stars are the same quantities in exact arithmetic: the exact intersection of the
// ray's line with the plane of the triangle v0 + a e1 + b e2, P* = o + t* d = v0 + u* e1 + v* e2.
// u0 = 2^-24 is the unit roundoff and perm(a, b, c) = sum over the six orders (i, j, k) of
// |a_i| |b_j| |c_k|, the sum of the absolute terms of a . (b x c).  Counting roundings per term
// (a product, a difference of products, the product and two sums of the dot product, and one for
// the rounded s), to first order:
//   |det - det*| <= 5 u0 perm(e1, d, e2)       |s.n - (s.n)*| <= 6 u0 perm(s, d, e2)
//   |d.q - (d.q)*| <= 6 u0 perm(d, s, e1)      |e2.q - (e2.q)*| <= 6 u0 perm(e2, s, e1)
// With E1 / E2 bounding |e1_i| / |e2_i|, S_i bounding |s_i| over the triangles of the leaf, |x|_1 the
// sum of absolute components and W = sum over i != j of S_i |d_j|:
//   perm(s, d, e2) <= W E2,  perm(d, s, e1) <= W E1,
//   perm(e1, d, e2) <= 2 E1 E2 |d|_1,  perm(e2, s, e1) <= 2 E1 E2 |S|_1.
// The code takes 8 and 7 for the 6 and 5 (E_uv = 8 u0 W per unit of edge, E_det = 14 u0 E1 E2 |d|_1,
// E_t = 16 u0 E1 E2 |S|_1), which covers the higher orders and the rounding of the bounds
// themselves.  An accepted triangle has |det| >= 1e-4, so |det*| >= Dlo = 1e-4 - E_det, and with
// u, v in [0, 1]
//   |u* - u| <= Du = (E_uv E2 + E_det) / Dlo + 2 u0,   |v* - v| <= Dv = (E_uv E1 + E_det) / Dlo + 2 u0,
//   |t* - t| <= Dt(t) = (E_t + t E_det) / Dlo + 2 u0 t
// (the code adds a few u0 to each).  (u, v) itself lies in the parameter triangle up to u0 (u + v <= 1
// is tested on a rounded sum), so every coordinate of P* is within
//   R = Du E1 + Dv E2 + 2 u0 (E1 + E2) <= (2 E_uv E1 E2 + E_det (E1 + E2)) / Dlo + 4 u0 (E1 + E2)
// of the triangle.  P* is on the ray's line: if the line, up to t_best + Dt(t_best), misses a box of
// triangles grown by R, no triangle in it is accepted at or below t_best.  Underflow adds at most
// a few 2^-149 S to a triple product, far below the u0 terms kept; the bounds on the triple
// products are checked to be below 1e30, so nothing in the float test overflows.
//
// The bound on t is symmetric, so an accepted hit (t > 1e-4) also has t* > 1e-4 - Dt(1e-4): parts of
// the line behind that need no test either.
//
// The same bounds hold with any other lower bound of |det*| for Dlo.  A leaf also keeps a cone of its
// triangles' normal lines (an axis A with every |N_k . A| >= cos_phi |N_k| |A|, N_k = e1 x e2) and a
// lower bound nmin of |N_k|; det* = -d . N_k, so for a ray whose line makes an angle theta with A's,
// |det*| >= nmin |d| cos(theta + phi) when theta + phi < 90 degrees -- for triangles facing the ray
// this is far above 1e-4, and the margins shrink by the same factor.  The cone is only evaluated
// where the margin from 1e-4 alone is not narrow already (kNarrowDuv).
//
// The leaf keeps Q >= E1 + E2 (so E1 E2 <= P = Q^2 / 4) and B >= every |coordinate| of its boxes
// (S_i = |o_i| + B); the margins are computed once per ray and leaf (leaf_cull) and each box then
// costs one slab test (box_live).  Every bound is rounded outward, the stored boxes are widened
// outward by a relative 4 u0 (they are computed from the rounded vertices v0 + e1, v0 + e2), and
// the grown box gets an extra slack of 8 u0 (2 B + |o_i| + R) per axis, which exceeds the rounding of
// the slab arithmetic fma(lo, 1 / d, -(o + g) / d) with the IEEE reciprocal
// (<= 5.1 u0 R + 4.1 u0 |o| + 2.1 u0 |lo|).  Leaves with a non-finite or huge coordinate (Q = +inf),
// rays with a non-finite or huge component or a tiny non-zero d_i (|1 / d_i| >= 1e20), and leaves
// without a positive Dlo are never culled.  Audited on the CPU against the float test on
// adversarial rays (aimed at edges and vertices, grazing the plane, axis-aligned): no culled box
// held an accepted hit at or below t_best, and the largest measured error was 0.21 of its margin (11.9 M hits).
//
// Counting the roundings term by term, instead of bounding each triple product by its largest
// factors with a further factor 4 on every term, makes R 50 to 100 times and Du + Dv 3 to 9 times
// narrower: hidden trees pay for far rays too.
#pragma once

#include <cfloat>
#include <cmath>
#include <cstdint>

#ifdef __CUDACC__
#define BVHGPU_HD __host__ __device__ __forceinline__
#else
#define BVHGPU_HD inline
#endif

namespace bvhgpu {

constexpr float kCullUnit = 5.9604645e-8f;  // u0 = 2^-24
// A barycentric margin Du + Dv below which the bound from |det| >= 1e-4 is used as it is: the cone
// would cost more to evaluate than its narrower margin saves (at 0.5 | 0.05: animated instanced frame 1,546 | 1,562 us,
// scene image 326 | 330, others the same).
constexpr float kNarrowDuv = 0.5f;
constexpr float kCullHuge = 1e15f;

BVHGPU_HD float cull_fmax(float a, float b) { return a > b ? a : b; }
BVHGPU_HD float cull_fmin(float a, float b) { return a < b ? a : b; }
BVHGPU_HD float cull_abs(float a) { return a < 0.0f ? -a : a; }
BVHGPU_HD float cull_down(float t) { return t < 0.0f ? t * (1.0f + 4.0f * kCullUnit) : t * (1.0f - 4.0f * kCullUnit); }
BVHGPU_HD float cull_up(float t) { return t < 0.0f ? t * (1.0f - 4.0f * kCullUnit) : t * (1.0f + 4.0f * kCullUnit); }
#ifdef __CUDACC__
BVHGPU_HD float cull_fma(float a, float b, float c) { return fmaf(a, b, c); }
#else
BVHGPU_HD float cull_fma(float a, float b, float c) { return std::fma(a, b, c); }
#endif

// A group of triangles sealed for the cull: its box widened outward, and its contributions to the
// leaf's Q (E1 + E2, rounded up; +inf for a non-finite or huge group) and B (largest |coordinate|).
struct GroupSeal {
    float lo[3], hi[3];
    float q, b;
};

// From the raw min / max of a group's vertices v0, v0 + e1, v0 + e2 (as computed in float) and
// the raw largest |e1_i|, |e2_i|.  `finite` is false when any input was non-finite.
BVHGPU_HD GroupSeal group_seal(const float lo[3], const float hi[3], float e1max, float e2max, bool finite) {
    GroupSeal c;
    bool ok = finite && e1max < kCullHuge && e2max < kCullHuge;
    float b = 0.0f;
    for (int i = 0; i < 3; ++i) {
        ok = ok && cull_abs(lo[i]) < kCullHuge && cull_abs(hi[i]) < kCullHuge;
        c.lo[i] = cull_down(lo[i]);
        c.hi[i] = cull_up(hi[i]);
        b = cull_fmax(b, cull_fmax(cull_abs(c.lo[i]), cull_abs(c.hi[i])));
    }
    c.q = ok ? (e1max + e2max) * (1.0f + 4.0f * kCullUnit) : INFINITY;
    c.b = ok ? b : 0.0f;
    if (!ok)  // keep the box finite: the leaf is never culled anyway (q = inf)
        for (int i = 0; i < 3; ++i) c.lo[i] = c.hi[i] = 0.0f;
    return c;
}

// The per-ray part of the cull.
struct CullRay {
    float o[3], d[3], rd[3];
    bool ok;
};

// rx, ry, rz: the IEEE reciprocals 1 / dx, 1 / dy, 1 / dz (the traversal's own).
BVHGPU_HD CullRay cull_ray_rd(float ox, float oy, float oz, float dx, float dy, float dz, float rx, float ry,
                              float rz) {
    CullRay r;
    r.o[0] = ox; r.o[1] = oy; r.o[2] = oz;
    r.d[0] = dx; r.d[1] = dy; r.d[2] = dz;
    r.rd[0] = rx; r.rd[1] = ry; r.rd[2] = rz;
    bool ok = true;
    for (int i = 0; i < 3; ++i) {
        // a zero component is handled exactly; any other needs |1 / d_i| < 1e20 (with |o|, B below
        // 1e15 no product of the slab arithmetic can overflow)
        ok = ok && cull_abs(r.o[i]) < kCullHuge && cull_abs(r.d[i]) < kCullHuge &&
             (r.d[i] == 0.0f || cull_abs(r.rd[i]) < 1e20f);
    }
    r.ok = ok;
    return r;
}

BVHGPU_HD CullRay cull_ray(float ox, float oy, float oz, float dx, float dy, float dz) {
    return cull_ray_rd(ox, oy, oz, dx, dy, dz, 1.0f / dx, 1.0f / dy, 1.0f / dz);
}

// The normal cone of a group of triangles (see above); nmin = 0 or cos_phi <= 0: none.  sin_phi is
// an upper bound of sqrt(1 - cos_phi^2) (cone_sin).
struct LeafCone {
    float ax, ay, az;
    float cos_phi, sin_phi, nmin;
};

BVHGPU_HD float cone_sin(float cos_phi) {
    return sqrtf(cull_fmax(0.0f, 1.0f - cos_phi * cos_phi * (1.0f - 4.0f * kCullUnit))) * (1.0f + 4.0f * kCullUnit);
}

// One triangle's contribution to a cone around axis (ax, ay, az): a lower bound of
// |N . A| / (|N| |A|) and of |N| for the exact N = e1 x e2, from the float edges.
BVHGPU_HD void cone_terms(const float e1[3], const float e2[3], float ax, float ay, float az, float& cos_lo,
                          float& n_lo) {
    const float u0 = kCullUnit;
    // N = e1 x e2 in float, each component within eN of the exact one
    const float n[3] = {e1[1] * e2[2] - e1[2] * e2[1], e1[2] * e2[0] - e1[0] * e2[2], e1[0] * e2[1] - e1[1] * e2[0]};
    const float en[3] = {3.0f * u0 * (cull_abs(e1[1] * e2[2]) + cull_abs(e1[2] * e2[1])),
                         3.0f * u0 * (cull_abs(e1[2] * e2[0]) + cull_abs(e1[0] * e2[2])),
                         3.0f * u0 * (cull_abs(e1[0] * e2[1]) + cull_abs(e1[1] * e2[0]))};
    const float a[3] = {ax, ay, az};
    float dot = 0.0f, dot_err = 0.0f, nn = 0.0f, n_err = 0.0f, aa = 0.0f;
    for (int i = 0; i < 3; ++i) {
        dot += n[i] * a[i];
        dot_err += (en[i] + 4.0f * u0 * cull_abs(n[i])) * cull_abs(a[i]);
        nn += n[i] * n[i];
        n_err += en[i];
        aa += a[i] * a[i];
    }
    const float nlen = sqrtf(nn), alen = sqrtf(aa);
    n_lo = (nlen * (1.0f - 8.0f * u0) - n_err) * (1.0f - 4.0f * u0);
    const float num = cull_abs(dot) - dot_err;
    const float den = (nlen * (1.0f + 8.0f * u0) + n_err) * alen * (1.0f + 8.0f * u0);
    cos_lo = (num > 0.0f && den > 0.0f && n_lo > 0.0f) ? num / den * (1.0f - 8.0f * u0) : -1.0f;
    if (!(n_lo > 0.0f)) n_lo = 0.0f;
}

// A lower bound of |d . N_k| for every triangle of a leaf with cone c (0 when it gives none).
BVHGPU_HD float cone_det_lo(const float d[3], const LeafCone& c) {
    const float u0 = kCullUnit;
    if (!(c.nmin > 0.0f) || !(c.cos_phi > 0.0f) || !(c.cos_phi <= 1.0f) || !(c.sin_phi >= 0.0f)) return 0.0f;
    const float a = d[0] * c.ax + d[1] * c.ay + d[2] * c.az;
    const float a_err = 4.0f * u0 * (cull_abs(d[0] * c.ax) + cull_abs(d[1] * c.ay) + cull_abs(d[2] * c.az));
    const float dd = d[0] * d[0] + d[1] * d[1] + d[2] * d[2];
    const float AA = c.ax * c.ax + c.ay * c.ay + c.az * c.az;
    const float dlen = sqrtf(dd), alen = sqrtf(AA);
    const float cos_t = (cull_abs(a) - a_err) / (dlen * alen * (1.0f + 8.0f * u0)) * (1.0f - 4.0f * u0);
    if (!(cos_t > 0.0f)) return 0.0f;
    const float sin_t = sqrtf(cull_fmax(0.0f, 1.0f - cos_t * cos_t * (1.0f - 4.0f * u0))) * (1.0f + 4.0f * u0);
    const float sin_p = c.sin_phi;
    const float cs = (cos_t * c.cos_phi * (1.0f - 4.0f * u0) - sin_t * sin_p * (1.0f + 4.0f * u0)) * (1.0f - 4.0f * u0);
    if (!(cs > 0.0f)) return 0.0f;
    const float lo = c.nmin * dlen * (1.0f - 4.0f * u0) * cs * (1.0f - 64.0f * u0);
    return lo < FLT_MAX ? lo : 0.0f;
}

// The per-(ray, leaf) part: the grown slab planes folded with the origin, c_lo = o + g and
// c_hi = o - g per axis, pre-scaled by -1 / d where d is not zero (slab t = fma(x, 1/d, s)), the
// largest t that still matters (thi, from the ray's closest t) and the smallest (tlo: accepted hits
// have t > 1e-4, so t* > 1e-4 - Dt(1e-4)).  thi follows the closest t through leaf_thi.
// on = false: nothing of this leaf is culled for this ray.  zero: bit i set when d_i == 0.
struct LeafCull {
    float slo[3], shi[3];
    float thi, tlo;
    float dt0, dt1;  // Dt(t) <= dt0 + t dt1 (rounded up)
    float duv;       // the barycentric margin Du + Dv the planes were grown for
    bool on;
    uint32_t zero;
};

BVHGPU_HD float leaf_thi(const LeafCull& lc, float t_best) {
    if (!(t_best < FLT_MAX)) return INFINITY;
    return (t_best + (lc.dt0 + t_best * lc.dt1)) * (1.0f + 8.0f * kCullUnit) + 1e-30f;
}

// max_duv: the largest barycentric margin (Du + Dv) worth culling with; on = false above it.
BVHGPU_HD LeafCull leaf_cull(const CullRay& r, float Q, float B, float t_best, float max_duv, const LeafCone& cone) {
    const float u0 = kCullUnit;
    LeafCull lc;
    lc.on = false;
    lc.zero = 0u;
    for (int i = 0; i < 3; ++i) {
        if (r.d[i] == 0.0f) lc.zero |= 1u << i;
        lc.slo[i] = lc.shi[i] = 0.0f;
    }
    lc.thi = INFINITY;
    lc.tlo = -INFINITY;
    lc.dt0 = lc.dt1 = 0.0f;
    lc.duv = INFINITY;
    if (!r.ok || !(Q < kCullHuge) || !(B < kCullHuge)) return lc;
    const float up = 1.0f + 16.0f * u0;  // covers the rounding of a short chain of positive terms
    const float s0 = cull_abs(r.o[0]) + B, s1 = cull_abs(r.o[1]) + B, s2 = cull_abs(r.o[2]) + B;
    const float d0 = cull_abs(r.d[0]), d1 = cull_abs(r.d[1]), d2 = cull_abs(r.d[2]);
    const float W = (s0 * (d1 + d2) + s1 * (d0 + d2) + s2 * (d0 + d1)) * up;
    const float D1 = (d0 + d1 + d2) * up, S1 = (s0 + s1 + s2) * up;
    const float P = 0.25f * Q * Q * up;  // >= E1 E2
    if (!(W * Q < 1e30f) || !(D1 * P < 1e30f) || !(S1 * P < 1e30f)) return lc;
    const float e_det = 14.0f * u0 * P * D1 * up;
    const float e_uv = 8.0f * u0 * W * up;  // times E2 for u, E1 for v
    // |det*| >= Dlo: accepted |det| >= 1e-4 (the float 0.0001f, triangle.rs:47), or the cone's bound
    const float e_sum = (e_uv * Q + 2.0f * e_det) * up;  // (Du + Dv - 4 u0) Dlo
    float Dlo = 0.0001f * (1.0f - 4.0f * u0) - e_det;
    if (!(e_sum < kNarrowDuv * Dlo)) Dlo = cull_fmax(Dlo, cone_det_lo(r.d, cone));
    if (!(Dlo > 0.0f)) return lc;
    const float KD = 1.0f / Dlo * (1.0f + 4.0f * u0);  // >= 1 / Dlo
    if (!(KD < kCullHuge)) return lc;
    const float duv = (e_sum * KD + 16.0f * u0) * up;
    // margins of half a triangle or more cull little: the caller tests the leaf in order instead
    lc.duv = duv;
    if (!(duv < max_duv)) return lc;
    const float R = ((2.0f * e_uv * P + e_det * Q) * KD + 16.0f * u0 * Q) * up + 1e-30f;
    if (!(R < kCullHuge)) return lc;
    const float e_t = 16.0f * u0 * P * S1 * up;
    // Dt(t) = (E_t + t E_det) / Dlo + 2 u0 t <= dt0 + t dt1
    lc.dt0 = e_t * KD * up;
    lc.dt1 = (e_det * KD + 4.0f * u0) * up;
    lc.thi = leaf_thi(lc, t_best);
    const float th = 0.0001f;  // the test's threshold (triangle.rs:47)
    lc.tlo = cull_down(th - (lc.dt0 + th * lc.dt1) * (1.0f + 8.0f * u0)) - 1e-30f;
    for (int i = 0; i < 3; ++i) {
        const float g = R + 8.0f * u0 * (2.0f * B + cull_abs(r.o[i]) + R) + 1e-30f;
        const float clo = r.o[i] + g, chi = r.o[i] - g;
        if (lc.zero & (1u << i)) {  // the line keeps o_i: culled when the grown slab does not contain it
            lc.slo[i] = clo;
            lc.shi[i] = chi;
        } else {                    // t = (lo - c_lo) / d = fma(lo, 1/d, -c_lo / d)
            lc.slo[i] = -(clo * r.rd[i]);
            lc.shi[i] = -(chi * r.rd[i]);
        }
    }
    lc.on = true;
    return lc;
}

// Whether the line of the ray, between lc.tlo and lc.thi, meets the box [lo, hi] grown by the
// leaf's margins (always true when !lc.on); t_enter: where it enters (for near-first order).
BVHGPU_HD bool box_live(const float lo[3], const float hi[3], const float rd[3], const LeafCull& lc, float& t_enter) {
    t_enter = 0.0f;
    if (!lc.on) return true;
    float tlo = lc.tlo, thi = lc.thi;
    bool out = false;
    for (int i = 0; i < 3; ++i) {
        if (lc.zero & (1u << i)) {
            out = out || lo[i] > lc.slo[i] || hi[i] < lc.shi[i];
        } else {
            const float t1 = cull_fma(lo[i], rd[i], lc.slo[i]);
            const float t2 = cull_fma(hi[i], rd[i], lc.shi[i]);
            tlo = cull_fmax(tlo, cull_fmin(t1, t2));
            thi = cull_fmin(thi, cull_fmax(t1, t2));
        }
    }
    t_enter = tlo;
    return !out && !(tlo > thi);
}

}  // namespace bvhgpu
