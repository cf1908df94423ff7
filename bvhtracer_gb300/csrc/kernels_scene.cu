// BLAS vertex upload + refit, TLAS rebuild and instanced (two-level) traversal.
//
// Refit (Bvh::refit, bvh.rs:469-493): leaf boxes by a reduction over the triangles (exact
// order-preserving keys, so the min/max and its ties are the reference's), then the inner
// nodes bottom-up with one arrival counter per node: the second child to finish computes its
// parent with the reference's min/max order (left child first).
//
// TLAS rebuild (Tlas::rebuild, tlas.rs:204-250): the reference's agglomerative clustering by one block
// that keeps the list in registers (see k_tlas_rebuild).
#include <cuda_runtime.h>

#include <algorithm>
#include <vector>

#include "common.cuh"
#include "internal.hpp"
#include "persistent.cuh"
#include "render.cuh"
#include "variants.cuh"
#include "wide.cuh"

namespace bvhgpu {
namespace {

constexpr int kBlock = 128;
constexpr uint32_t kNone = 0xFFFFFFFFu;
constexpr unsigned kFull = 0xFFFFFFFFu;

// Writes the traversal layout {v0, e1 = v1 - v0, e2 = v2 - v0} (the subtractions of
// triangle.rs:44-45, so no bit changes) and the raw vertices used by refit.
__global__ void k_write_tris(const float* __restrict__ tris9, uint32_t n, float4* __restrict__ out,
                             float4* __restrict__ verts, float* __restrict__ pairs) {
    uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float* t = tris9 + 9ull * i;
    float4 v0 = make_float4(t[0], t[1], t[2], 0.0f);
    float4 v1 = make_float4(t[3], t[4], t[5], 0.0f);
    float4 v2 = make_float4(t[6], t[7], t[8], 0.0f);
    out[3ull * i] = v0;
    out[3ull * i + 1] = make_float4(fsub(v1.x, v0.x), fsub(v1.y, v0.y), fsub(v1.z, v0.z), 0.0f);
    out[3ull * i + 2] = make_float4(fsub(v2.x, v0.x), fsub(v2.y, v0.y), fsub(v2.z, v0.z), 0.0f);
    verts[3ull * i] = v0;
    verts[3ull * i + 1] = v1;
    verts[3ull * i + 2] = v2;
    // pair layout: component c of triangle i at float 20 * (i / 2) + 2c + (i & 1)
    float c[9] = {v0.x, v0.y, v0.z, fsub(v1.x, v0.x), fsub(v1.y, v0.y), fsub(v1.z, v0.z),
                  fsub(v2.x, v0.x), fsub(v2.y, v0.y), fsub(v2.z, v0.z)};
    float* P = pairs + 20ull * (i >> 1) + (i & 1u);
#pragma unroll
    for (int k = 0; k < 9; ++k) P[2 * k] = c[k];
}

// ---- hidden trees of the large leaves, refreshed after every triangle write -----------------
// One launch, bottom-up: four lanes per hidden leaf (one per triangle pair; membership fixed at
// upload) copy its triangles into the packed pairs and fold their bounds, edge sizes and normals;
// then, as in the refit, the last child of a node to arrive (one counter per block of siblings,
// reset by it) folds the siblings' aggregates in child order, writes the node's box and its cone
// record, and climbs on.
//  - Boxes, Q and B are minima and maxima of the triangles' own values: the same in any order.
//  - A node's normal cone is built from its grandchildren's cones: the axis is the sum of the children's
//    folded unit-normal sums (any axis is valid), and normals within phi_c of the line of a grandchild's
//    axis are within theta_c + phi_c of the line of the node's axis (theta_c between the axes).  That loosens
//    with every level (roots over 3,400 triangles: 47 degrees where the normals span 40).  In models so large
//    that a root's cone decides whether its leaf can be walked at all (cones_decide), the roots' cones are
//    measured over their triangles instead (fold_root_cones).
// The quad of lanes climbs together, a child per lane.  What bounds it: the climb's dependent hops (a
// counter, a fence and up to four 128-B records each).
// Against two passes of every node over all its triangles (a warp per 256 pairs), which read each
// pair twice per tree level, together with the triangle rewrite before it: 327,680-triangle mesh
// 240 -> 87 us, 20,480 triangles 98 -> 57 us.  Building each cone from the children alone loosened the
// roots (a sphere of radius 100 seen from 3,000: 1,126 -> 1,464 us, more leaves tested in order).
struct HiddenAgg {
    float lo[3], hi[3];  // raw bounds of v0, v0 + e1, v0 + e2
    float e1m, e2m;      // largest |e1_i|, |e2_i|
    float s[3];          // sum of the unit normals, each turned towards the others
    float cphi, nmin;    // the cone around s: least |N . s| / (|N| |s|) (<= 0: none) and |N|
    float finite;        // 1: every input was finite
};
constexpr float kNoEntry = 2.0f;  // cphi of a missing child

// An aggregate is 8 float4: the node's own four, then its children's cones {s, cphi} (a leaf's first is
// its own).
__device__ __forceinline__ HiddenAgg load_agg(const float4* a) {
    const float4 x = __ldcg(a), y = __ldcg(a + 1), z = __ldcg(a + 2), w = __ldcg(a + 3);
    return HiddenAgg{{x.x, x.y, x.z}, {y.x, y.y, y.z}, x.w, y.w, {z.x, z.y, z.z}, z.w, w.x, w.y};
}
__device__ __forceinline__ HiddenAgg empty_agg() {
    return HiddenAgg{{FLT_MAX, FLT_MAX, FLT_MAX}, {-FLT_MAX, -FLT_MAX, -FLT_MAX}, 0.0f, 0.0f, {0.0f, 0.0f, 0.0f}, kNoEntry,
                     FLT_MAX, 1.0f};
}

// Adds b's normals to a's, turned towards them.
__device__ __forceinline__ void fold_normals(float* a, const float* b) {
    const float sg = (a[0] * b[0] + a[1] * b[1] + a[2] * b[2]) < 0.0f ? -1.0f : 1.0f;
    for (int i = 0; i < 3; ++i) a[i] += sg * b[i];
}

__device__ __forceinline__ void fold_bounds(HiddenAgg& a, const HiddenAgg& b) {
    for (int i = 0; i < 3; ++i) {
        a.lo[i] = fminf(a.lo[i], b.lo[i]);
        a.hi[i] = fmaxf(a.hi[i], b.hi[i]);
    }
    a.e1m = fmaxf(a.e1m, b.e1m);
    a.e2m = fmaxf(a.e2m, b.e2m);
    a.finite = fminf(a.finite, b.finite);
}

// The fold of the four lanes' aggregates, the same in all four (a lower lane's normals before a higher
// one's); cphi is left alone.
__device__ __forceinline__ void quad_fold(HiddenAgg& g, unsigned quad) {
#pragma unroll
    for (int off = 1; off <= 2; off <<= 1) {
        HiddenAgg o;
        for (int j = 0; j < 3; ++j) {
            o.lo[j] = __shfl_xor_sync(quad, g.lo[j], off);
            o.hi[j] = __shfl_xor_sync(quad, g.hi[j], off);
            o.s[j] = __shfl_xor_sync(quad, g.s[j], off);
        }
        o.e1m = __shfl_xor_sync(quad, g.e1m, off);
        o.e2m = __shfl_xor_sync(quad, g.e2m, off);
        o.finite = __shfl_xor_sync(quad, g.finite, off);
        g.nmin = fminf(g.nmin, __shfl_xor_sync(quad, g.nmin, off));
        fold_bounds(g, o);
        if (threadIdx.x & off) {
            fold_normals(o.s, g.s);
            for (int j = 0; j < 3; ++j) g.s[j] = o.s[j];
        } else {
            fold_normals(g.s, o.s);
        }
    }
}
__device__ __forceinline__ float quad_min(float v, unsigned quad) {
    v = fminf(v, __shfl_xor_sync(quad, v, 1));
    return fminf(v, __shfl_xor_sync(quad, v, 2));
}

// A lower bound of |cos| between normals within phi_c (cphi) of the line of axis s, and the line of axis a
// (cos(theta + phi), rounded down as in cone_det_lo); <= 0 where it gives none.
__device__ __forceinline__ float wider_cone(const float* a, const float* s, float cphi) {
    const float u0 = kCullUnit;
    if (!(cphi > 0.0f) || !(cphi <= 1.0f)) return -1.0f;
    const float dot = a[0] * s[0] + a[1] * s[1] + a[2] * s[2];
    const float err = 4.0f * u0 * (fabsf(a[0] * s[0]) + fabsf(a[1] * s[1]) + fabsf(a[2] * s[2]));
    const float la = sqrtf(a[0] * a[0] + a[1] * a[1] + a[2] * a[2]), ls = sqrtf(s[0] * s[0] + s[1] * s[1] + s[2] * s[2]);
    float ct = (fabsf(dot) - err) / (la * ls * (1.0f + 8.0f * u0)) * (1.0f - 4.0f * u0);
    if (!(ct > 0.0f)) return -1.0f;
    ct = fminf(ct, 1.0f);
    const float st = cone_sin(ct), sp = cone_sin(cphi);
    const float c = (ct * cphi * (1.0f - 4.0f * u0) - st * sp * (1.0f + 4.0f * u0)) * (1.0f - 4.0f * u0);
    return c > 0.0f ? c : -1.0f;
}

// Whether the plain margin (leaf_cull) of a tree with bounds Q, B is too wide to walk it (2, the default limit)
// already for rays from within 2 B of the origin: its cone alone then decides.  Below, the looser roots cost
// nothing measurable, and the second pass over the triangles would (update of 20,480 triangles 25 -> 32 us,
// with a refit 43 -> 46).
__device__ __forceinline__ bool cones_decide(float Q, float B) {
    const float w = 2.0f * 1.7320508f * 3.0f * B;  // W of a unit direction along the diagonal
    return !(8.0f * kCullUnit * w * Q + 28.0f * kCullUnit * 1.7320508f * 0.25f * Q * Q < 2.0f * 0.0001f);
}

// up[i] of hidden node i (both counted from the first hidden node): {first node of its sibling block,
// siblings, parent node (kNoRefresh: a hidden root), the parent's cone record}.  measured: fold_root_cones
// follows and makes the roots' cones.  decide (may be null): set to 1 where cones_decide.
__global__ void __launch_bounds__(256) k_hidden_refresh(const float4* __restrict__ tris, const uint2* __restrict__ slots,
                                                        uint32_t p0, float4* __restrict__ pairs,
                                                        float4* nodes, uint32_t nhid, const uint4* __restrict__ up,
                                                        float4* agg, uint32_t* arrivals, float4* __restrict__ cones, bool measured,
                                                        uint32_t* decide) {
    const uint32_t i = (blockIdx.x * blockDim.x + threadIdx.x) >> 2, q = threadIdx.x & 3u;
    uint32_t first = 0u, count = 0u;
    if (i < nhid) {
        first = __float_as_uint(nodes[2ull * i].w);
        count = __float_as_uint(nodes[2ull * i + 1].w);
    }
    const bool leaf = (count & kHiddenLeaf) != 0u;
    HiddenAgg g = empty_agg();
    float c[2][9];
    bool have[2] = {false, false};
    if (leaf && q < (count & ~kHiddenLeaf)) {
        const uint32_t p = first + q;
        const uint2 idx = slots[p - p0];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const uint32_t k = h ? idx.y : idx.x;
            have[h] = k != kMiss;
            float4 v0 = make_float4(0.0f, 0.0f, 0.0f, 0.0f), e1 = v0, e2 = v0;
            if (have[h]) {
                v0 = tris[3ull * k];
                e1 = tris[3ull * k + 1];
                e2 = tris[3ull * k + 2];
            }
            const float t[9] = {v0.x, v0.y, v0.z, e1.x, e1.y, e1.z, e2.x, e2.y, e2.z};
            for (int j = 0; j < 9; ++j) c[h][j] = t[j];
        }
        // the packed pair, its triangles' indices in the last two words
        float4* P = pairs + 5ull * p;
#pragma unroll
        for (int j = 0; j < 4; ++j) P[j] = make_float4(c[0][2 * j], c[1][2 * j], c[0][2 * j + 1], c[1][2 * j + 1]);
        P[4] = make_float4(c[0][8], c[1][8], __uint_as_float(idx.x), __uint_as_float(idx.y));
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            if (!have[h]) continue;
            bool fin = true;
            for (int j = 0; j < 3; ++j) {
                const float v = c[h][j], a = c[h][3 + j], b = c[h][6 + j], p1 = fadd(v, a), p2 = fadd(v, b);
                fin = fin && isfinite(v) && isfinite(a) && isfinite(b) && isfinite(p1) && isfinite(p2);
                g.lo[j] = fminf(g.lo[j], fminf(v, fminf(p1, p2)));
                g.hi[j] = fmaxf(g.hi[j], fmaxf(v, fmaxf(p1, p2)));
                g.e1m = fmaxf(g.e1m, fabsf(a));
                g.e2m = fmaxf(g.e2m, fabsf(b));
            }
            if (!fin) g.finite = 0.0f;
            const float* a = c[h] + 3;
            const float* b = c[h] + 6;
            float n[3] = {a[1] * b[2] - a[2] * b[1], a[2] * b[0] - a[0] * b[2], a[0] * b[1] - a[1] * b[0]};
            const float len = sqrtf(n[0] * n[0] + n[1] * n[1] + n[2] * n[2]);
            if (len > 0.0f && isfinite(len)) {
                for (int j = 0; j < 3; ++j) n[j] /= len;
                fold_normals(g.s, n);
            }
        }
    }
    if (!leaf) return;  // whole quads leave together
    const unsigned quad = 0xFu << (threadIdx.x & 28u);
    quad_fold(g, quad);
    g.nmin = FLT_MAX;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        if (!have[h]) continue;
        float cl, nl;
        cone_terms(c[h] + 3, c[h] + 6, g.s[0], g.s[1], g.s[2], cl, nl);
        g.cphi = cl < g.cphi ? cl : (cl == cl ? g.cphi : -1.0f);  // NaN: no cone
        g.nmin = nl < g.nmin ? nl : (nl == nl ? g.nmin : 0.0f);
    }
    g.cphi = quad_min(g.cphi, quad);
    g.nmin = quad_min(g.nmin, quad);
    float4 entry = make_float4(g.s[0], g.s[1], g.s[2], q == 0u ? g.cphi : kNoEntry);  // cone of the node's child q
    uint32_t cur = i;
    for (;;) {
        const GroupSeal box = group_seal(g.lo, g.hi, g.e1m, g.e2m, g.finite != 0.0f);
        if (q < 3u) {  // first and count stay
            reinterpret_cast<float*>(nodes + 2ull * cur)[q] = box.lo[q];
            reinterpret_cast<float*>(nodes + 2ull * cur + 1)[q] = box.hi[q];
        }
        float4* a = agg + 8ull * cur;
        __stcg(a + q, q == 0u   ? make_float4(g.lo[0], g.lo[1], g.lo[2], g.e1m)
                      : q == 1u ? make_float4(g.hi[0], g.hi[1], g.hi[2], g.e2m)
                      : q == 2u ? make_float4(g.s[0], g.s[1], g.s[2], g.cphi)
                                : make_float4(g.nmin, g.finite, kNoEntry, 0.0f));
        __stcg(a + 4u + q, entry);
        const uint4 u = up[cur];
        __threadfence();
        __syncwarp(quad);
        uint32_t arrived = 0u;
        if (q == 0u) arrived = atomicAdd(arrivals + u.x, 1u);
        arrived = __shfl_sync(quad, arrived, (int)(threadIdx.x & 28u));
        if (arrived != u.y - 1u) return;        // a sibling is still to come
        if (q == 0u) arrivals[u.x] = 0u;        // ready for the next refresh
        __threadfence();
        // lane q: child q and its children's cones
        g = empty_agg();
        float4 below[4];
        const float4* ch = agg + 8ull * (u.x + q);
        if (q < u.y) {
            g = load_agg(ch);
#pragma unroll
            for (int j = 0; j < 4; ++j) below[j] = __ldcg(ch + 4 + j);
        }
        entry = make_float4(g.s[0], g.s[1], g.s[2], g.cphi);
        quad_fold(g, quad);
        float cphi = kNoEntry;
        if (q < u.y) {
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const float s[3] = {below[j].x, below[j].y, below[j].z};
                if (below[j].w != kNoEntry) cphi = fminf(cphi, wider_cone(g.s, s, below[j].w));
            }
        }
        g.cphi = quad_min(cphi, quad);
        const GroupSeal seal = group_seal(g.lo, g.hi, g.e1m, g.e2m, g.finite != 0.0f);
        if (u.z == kNoRefresh) {
            if (decide != nullptr && q == 0u && cones_decide(seal.q, seal.b)) *decide = 1u;
            if (measured) {  // the axis and the bounds
                if (q == 0u) cones[2ull * u.w] = make_float4(g.s[0], g.s[1], g.s[2], -1.0f);
                if (q == 1u) cones[2ull * u.w + 1] = make_float4(1.0f, g.nmin, seal.q, seal.b);
                return;
            }
        }
        const bool ok = isfinite(g.s[0]) && isfinite(g.s[1]) && isfinite(g.s[2]) && g.cphi > 0.0f && g.cphi <= 1.0f &&
                        g.nmin > 0.0f && g.nmin < FLT_MAX;
        if (!ok) g.cphi = -1.0f;
        if (q == 0u) cones[2ull * u.w] = make_float4(ok ? g.s[0] : 0.0f, ok ? g.s[1] : 0.0f, ok ? g.s[2] : 0.0f, g.cphi);
        if (q == 1u) cones[2ull * u.w + 1] = make_float4(ok ? cone_sin(g.cphi) : 1.0f, ok ? g.nmin : 0.0f, seal.q, seal.b);
        if (u.z == kNoRefresh) return;
        cur = u.z;
    }
}

// The hidden roots' normal cones, measured: the least |cos| between any of a root's triangles' normals and its axis.
// links[li] of reference leaf li: {first node of the root's children's block (kNone: no hidden tree), cone
// record, triangles}.  Every lane brings one triangle (link: its leaf's; a leaf's triangles are consecutive,
// so a warp's are mostly of one root); the warp folds them into the root's word, which the refresh left at
// kNoEntry, and the last triangles to arrive finish the record.  Primaries of 400 x 400 from 3 radii, roots from
// their grandchildren's cones | measured: 81,920-triangle sphere of radius 100 1,651 | 1,270 us, 20,480
// triangles 465 | 360 us.
__device__ __forceinline__ void fold_root_cones(uint4 link, const float* e1, const float* e2, float4* agg, uint32_t* arrivals,
                                                float4* cones) {
    const unsigned lane = threadIdx.x & 31u;
    int cosine = 0x7FFFFFFF;  // a float's bits: they order as signed integers, and -1 is below all
    if (link.x != kNone) {
        const float4 a = __ldcg(cones + 2ull * link.y);
        float cl, nl;
        cone_terms(e1, e2, a.x, a.y, a.z, cl, nl);
        cosine = __float_as_int(cl == cl ? cl : -1.0f);
    }
    unsigned todo = __ballot_sync(kFull, link.x != kNone);
    while (todo) {
        const int leader = __ffs(todo) - 1;
        const uint32_t root = __shfl_sync(kFull, link.x, leader);
        const unsigned group = __ballot_sync(kFull, link.x == root);
        const int least = __reduce_min_sync(kFull, link.x == root ? cosine : 0x7FFFFFFF);
        todo &= ~group;
        if ((int)lane != leader) continue;
        int* word = reinterpret_cast<int*>(agg + 8ull * root + 3u) + 2;
        atomicMin(word, least);
        __threadfence();
        if (atomicAdd(arrivals + root, (uint32_t)__popc(group)) + (uint32_t)__popc(group) != link.z) continue;
        __threadfence();
        arrivals[root] = 0u;  // ready for the next refresh
        const float c = __int_as_float(__ldcg(word));
        const float4 a = __ldcg(cones + 2ull * link.y), b = __ldcg(cones + 2ull * link.y + 1);
        const bool ok = isfinite(a.x) && isfinite(a.y) && isfinite(a.z) && c > 0.0f && c <= 1.0f && b.y > 0.0f && b.y < FLT_MAX;
        cones[2ull * link.y] = ok ? make_float4(a.x, a.y, a.z, c) : make_float4(0.0f, 0.0f, 0.0f, -1.0f);
        cones[2ull * link.y + 1] = make_float4(ok ? cone_sin(c) : 1.0f, ok ? b.y : 0.0f, b.z, b.w);
    }
}

__global__ void __launch_bounds__(256) k_hidden_root_cones(const float4* __restrict__ tris, uint32_t ntris,
                                                           const uint32_t* __restrict__ tri_leaf,
                                                           const uint4* __restrict__ links, float4* agg, uint32_t* arrivals,
                                                           float4* cones) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    uint4 link = make_uint4(kNone, 0u, 0u, 0u);
    float e1[3] = {0.0f, 0.0f, 0.0f}, e2[3] = {0.0f, 0.0f, 0.0f};
    if (i < ntris) {
        const float4 a = tris[3ull * i + 1], b = tris[3ull * i + 2];
        const uint32_t li = tri_leaf[i];
        if (li != kNone) link = links[li];
        e1[0] = a.x; e1[1] = a.y; e1[2] = a.z;
        e2[0] = b.x; e2[1] = b.y; e2[2] = b.z;
    }
    fold_root_cones(link, e1, e2, agg, arrivals, cones);
}

// ---- refit, parallel over triangles --------------------------------------------------------
// update_node_bounds (bvh.rs:317-330) folds a leaf's vertices in order v0, v1, v2 of triangle
// first, first+1, ... with f32::min / f32::max.  The fold's result is the minimum (maximum)
// value, and among equal values (only +0 / -0 differ in bits) the first one in that order.  The
// same result is computed in parallel with 64-bit keys: an order-preserving map of the value
// with both zeros mapped to one rank, then the position in the fold order (lower wins on a tie).
// NaNs are skipped, as f32::min skips them.  The reduced key names the winning vertex, whose
// actual bits are read back.

// Segmented min of 64-bit keys over consecutive lanes with the same segment id (leaf): the
// first lane of each segment ends up holding the segment's minimum.
__device__ __forceinline__ unsigned long long seg_min(unsigned long long k, uint32_t seg) {
    const unsigned lane = threadIdx.x & 31u;
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
        unsigned long long o = __shfl_down_sync(kFull, k, off);
        uint32_t os = __shfl_down_sync(kFull, seg, off);
        if (lane + off < 32u && os == seg && o < k) k = o;
    }
    return k;
}
__device__ __forceinline__ unsigned long long seg_max(unsigned long long k, uint32_t seg) {
    const unsigned lane = threadIdx.x & 31u;
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
        unsigned long long o = __shfl_down_sync(kFull, k, off);
        uint32_t os = __shfl_down_sync(kFull, seg, off);
        if (lane + off < 32u && os == seg && o > k) k = o;
    }
    return k;
}

constexpr unsigned long long kKeyMinIdentity = 0xFFFFFFFFFFFFFFFFull;
constexpr unsigned long long kKeyMaxIdentity = 0ull;

// One thread per triangle: keys of its three vertices per axis, reduced over the warp's lanes of
// the same leaf, then one atomicMin / atomicMax per (leaf, axis) from the segment's first lane.
// keys: 6 per leaf slot (min x y z, max x y z), at the identity before the launch.
// ROOTS: the hidden roots' cones too (fold_root_cones; the refresh before this launch left them out).
template <bool ROOTS>
__global__ void __launch_bounds__(256) k_refit_tris(const float4* __restrict__ verts, uint32_t ntris,
                                                    const uint32_t* __restrict__ tri_leaf,
                                                    unsigned long long* keys, const uint4* __restrict__ links,
                                                    float4* agg, uint32_t* arrivals, float4* cones) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    const unsigned lane = threadIdx.x & 31u;
    uint32_t slot = kNone;
    float4 v[3];
    if (i < ntris) {
        slot = tri_leaf[i];
        v[0] = verts[3ull * i];
        v[1] = verts[3ull * i + 1];
        v[2] = verts[3ull * i + 2];
    }
    const uint32_t prev = __shfl_up_sync(kFull, slot, 1);
    const bool head = slot != kNone && (lane == 0u || prev != slot);
#pragma unroll
    for (int axis = 0; axis < 3; ++axis) {
        unsigned long long kmin = kKeyMinIdentity, kmax = kKeyMaxIdentity;
        if (slot != kNone) {
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                const float x = axis == 0 ? v[c].x : (axis == 1 ? v[c].y : v[c].z);
                if (x != x) continue;
                const uint32_t pos = 3u * i + (uint32_t)c;
                const unsigned long long r = (unsigned long long)ordered(x) << 32;
                const unsigned long long a = r | pos, b = r | (0xFFFFFFFFu - pos);
                if (a < kmin) kmin = a;
                if (b > kmax) kmax = b;
            }
        }
        kmin = seg_min(kmin, slot);
        kmax = seg_max(kmax, slot);
        if (head) {
            if (kmin != kKeyMinIdentity) atomicMin(&keys[6ull * slot + axis], kmin);
            if (kmax != kKeyMaxIdentity) atomicMax(&keys[6ull * slot + 3 + axis], kmax);
        }
    }
    if (ROOTS) {
        uint4 link = make_uint4(kNone, 0u, 0u, 0u);
        if (slot != kNone) link = links[slot];
        // the subtractions of the triangle write
        const float e1[3] = {fsub(v[1].x, v[0].x), fsub(v[1].y, v[0].y), fsub(v[1].z, v[0].z)};
        const float e2[3] = {fsub(v[2].x, v[0].x), fsub(v[2].y, v[0].y), fsub(v[2].z, v[0].z)};
        fold_root_cones(link, e1, e2, agg, arrivals, cones);
    }
}

// One thread per leaf: decode the keys into the winning vertices' values (identity = the fold's
// start value FLT_MAX / -FLT_MAX), reset the keys, write the leaf, then walk up: the second child
// to arrive at a parent computes it (bvh.rs:490-491: min(left, right), max(left, right)).
__global__ void __launch_bounds__(kBlock) k_refit_leaves(float4* nodes, const float4* __restrict__ verts,
                                                         const uint32_t* __restrict__ leaves, uint32_t nleaves,
                                                         const uint32_t* __restrict__ parent, uint32_t* counters,
                                                         unsigned long long* keys) {
    uint32_t li = blockIdx.x * blockDim.x + threadIdx.x;
    if (li >= nleaves) return;
    const uint32_t ni = leaves[li];
    float b[6];
    for (int k = 0; k < 6; ++k) {
        const unsigned long long key = keys[6ull * li + k];
        const bool is_min = k < 3;
        keys[6ull * li + k] = is_min ? kKeyMinIdentity : kKeyMaxIdentity;
        if (key == (is_min ? kKeyMinIdentity : kKeyMaxIdentity)) {
            b[k] = is_min ? FLT_MAX : -FLT_MAX;
            continue;
        }
        uint32_t pos = (uint32_t)(key & 0xFFFFFFFFull);
        if (!is_min) pos = 0xFFFFFFFFu - pos;
        const float4 vv = verts[pos];  // pos = 3 * triangle + vertex indexes the float4 vertex array
        const int axis = k % 3;
        b[k] = axis == 0 ? vv.x : (axis == 1 ? vv.y : vv.z);
    }
    const float4 lo = nodes[2ull * ni], hi = nodes[2ull * ni + 1];
    nodes[2ull * ni] = make_float4(b[0], b[1], b[2], lo.w);
    nodes[2ull * ni + 1] = make_float4(b[3], b[4], b[5], hi.w);
    __threadfence();
    uint32_t p = parent[ni];
    while (p != kNone) {
        uint32_t old = atomicAdd(&counters[p], 1u);
        if (old == 0u) return;  // the sibling subtree is not done yet; it will continue
        counters[p] = 0u;
        __threadfence();
        float4 plo = __ldcg(&nodes[2ull * p]);
        float4 phi = __ldcg(&nodes[2ull * p + 1]);
        uint32_t l = __float_as_uint(plo.w);
        float4 llo = __ldcg(&nodes[2ull * l]), lhi = __ldcg(&nodes[2ull * l + 1]);
        float4 rlo = __ldcg(&nodes[2ull * l + 2]), rhi = __ldcg(&nodes[2ull * l + 3]);
        __stcg(&nodes[2ull * p], make_float4(min_ni(llo.x, rlo.x), min_ni(llo.y, rlo.y), min_ni(llo.z, rlo.z), plo.w));
        __stcg(&nodes[2ull * p + 1],
               make_float4(max_ni(lhi.x, rhi.x), max_ni(lhi.y, rhi.y), max_ni(lhi.z, rhi.z), phi.w));
        __threadfence();
        p = parent[p];
    }
}

// ---- TLAS ------------------------------------------------------------------------------------
// Tlas::rebuild (tlas.rs:204-250) walks nearest neighbours over a list of node indices and
// calls find_best_match (tlas.rs:179-202) -- a full scan of the list -- at every step, about three
// times per merge.  The scans follow one another, so the rebuild's time is their number times the
// latency of one.  Here one block keeps the list in registers (k_tlas_rebuild): thread t owns
// clusters t, t + B, ..., a scan is one area per owned cluster, a warp minimum and a minimum over
// the warps behind a single barrier, and a merge needs no barrier of its own.  A candidate is one
// 64-bit key: the area's order-preserving rank (both zeros one rank) above the position, so the
// smallest key is the smallest area with ties to the lower position, as the reference's strict `<`
// scan from FLT_MAX keeps it; areas not below FLT_MAX (and NaN) are never keys.  The TLAS is bit for
// bit Tlas::rebuild's, including the case where position a itself leaves the list.
constexpr unsigned long long kNoKey = 0xFFFFFFFFFFFFFFFFull;

struct Box6 {
    float lx, ly, lz, hx, hy, hz;
};

// find_best_match's area (tlas.rs:184-193): component_max / component_min, then
// ex*ey + ey*ez + ez*ex.  The area is only compared (as a key rank), never stored, so fmaxf /
// fminf stand in for the first-operand-on-ties f32::max / f32::min: they ignore NaN the same way
// and can differ only in the sign of a zero coordinate, which changes at most the sign of a zero
// area -- the same rank.
__device__ __forceinline__ float sa_merge(const Box6& a, const Box6& b) {
    float ex = fsub(fmaxf(a.hx, b.hx), fminf(a.lx, b.lx));
    float ey = fsub(fmaxf(a.hy, b.hy), fminf(a.ly, b.ly));
    float ez = fsub(fmaxf(a.hz, b.hz), fminf(a.lz, b.lz));
    return fadd(fadd(fmul(ex, ey), fmul(ey, ez)), fmul(ez, ex));
}

// The key of candidate r for query box P (kNoKey where the reference would not take it).
__device__ __forceinline__ unsigned long long sa_key(const Box6& P, const Box6& R, int r) {
    const float s = sa_merge(P, R);
    return s < FLT_MAX ? (((unsigned long long)ordered(s) << 32) | (uint32_t)r) : kNoKey;
}

__device__ __forceinline__ int key_pos(unsigned long long k) { return k == kNoKey ? -1 : (int)(uint32_t)k; }

// Warp minimum of 64-bit keys as two 32-bit warp reductions: the smallest high half (area rank),
// then the smallest low half (position) among the lanes holding that high half.
__device__ __forceinline__ unsigned long long warp_min_key(unsigned long long k) {
    const uint32_t hi = __reduce_min_sync(kFull, (uint32_t)(k >> 32));
    const uint32_t lo = __reduce_min_sync(kFull, (uint32_t)(k >> 32) == hi ? (uint32_t)k : 0xFFFFFFFFu);
    return ((unsigned long long)hi << 32) | lo;
}

__device__ __forceinline__ void xf_point_g(const float* m, float x, float y, float z, float* out) {
    out[0] = fadd(fadd(fadd(fmul(m[0], x), fmul(m[4], y)), fmul(m[8], z)), fmul(m[12], 1.0f));
    out[1] = fadd(fadd(fadd(fmul(m[1], x), fmul(m[5], y)), fmul(m[9], z)), fmul(m[13], 1.0f));
    out[2] = fadd(fadd(fadd(fmul(m[2], x), fmul(m[6], y)), fmul(m[10], z)), fmul(m[14], 1.0f));
}

__device__ __forceinline__ void store_tlas_node(float4* out, uint32_t i, const Box6& b, uint32_t left_right,
                                                uint32_t blas) {
    out[2ull * i] = make_float4(b.lx, b.ly, b.lz, __uint_as_float(left_right));
    out[2ull * i + 1] = make_float4(b.hx, b.hy, b.hz, __uint_as_float(blas));
}

// Object i's world bounds (SceneObject::set_transform, scene_object.rs:60-75).
__device__ __forceinline__ Box6 object_bounds(const GBlas& b, const float* m) {
    const float4 rlo = b.nodes[0], rhi = b.nodes[1];  // Bvh::bounds = nodes[0].aabb (bvh.rs:499-501)
    float lo[3] = {FLT_MAX, FLT_MAX, FLT_MAX};
    float hi[3] = {-FLT_MAX, -FLT_MAX, -FLT_MAX};
    for (int c = 0; c < 8; ++c) {
        float p[3];
        xf_point_g(m, (c & 1) ? rhi.x : rlo.x, (c & 2) ? rhi.y : rlo.y, (c & 4) ? rhi.z : rlo.z, p);
        for (int k = 0; k < 3; ++k) {
            lo[k] = min_ni(lo[k], p[k]);
            hi[k] = max_ni(hi[k], p[k]);
        }
    }
    return Box6{lo[0], lo[1], lo[2], hi[0], hi[1], hi[2]};
}

__device__ __forceinline__ Box6 merged_box(const Box6& a, const Box6& b) {  // Aabb::new of positions a and b
    return Box6{min_ni(a.lx, b.lx), min_ni(a.ly, b.ly), min_ni(a.lz, b.lz),
                max_ni(a.hx, b.hx), max_ni(a.hy, b.hy), max_ni(a.hz, b.hz)};
}

// An object or merged cluster in shared memory: its box and node index.
struct Cluster {
    Box6 box;
    int node;
};
__device__ __forceinline__ Cluster load_cluster(const float4* sm, int slot) {
    const float4 x = sm[2 * slot], y = sm[2 * slot + 1];
    return Cluster{Box6{x.x, x.y, x.z, x.w, y.x, y.y}, __float_as_int(y.z)};
}
__device__ __forceinline__ void store_cluster(float4* sm, int slot, const Box6& b, int node) {
    sm[2 * slot] = make_float4(b.lx, b.ly, b.lz, b.hx);
    sm[2 * slot + 1] = make_float4(b.hy, b.hz, __int_as_float(node), 0.0f);
}

// The whole rebuild of up to B * K objects by one block.  A cluster keeps its slot for life (thread
// slot % B owns it: box and list position in registers, a copy of the box in shared memory for the
// queries); the reference's list moves are changes of positions only.  The walk is followed by every
// thread (a, b and their clusters are block-uniform).  A shared cluster is read only between a scan's
// barrier and the next one; a merge writes one, between the same barriers and without another
// reader: the clusters at a and b are already in registers and the next query is the merged one.
// status[0] gets nodes_used, status[1] an error (the reference would panic).
template <int B, int K>
__global__ void __launch_bounds__(B) k_tlas_rebuild(const GBlas* __restrict__ blas_table,
                                                    const uint32_t* __restrict__ obj_blas,
                                                    const float* __restrict__ xf, uint32_t nobj,
                                                    float4* __restrict__ tlas_out, uint32_t* status) {
    static_assert(B % 32 == 0 && B / 32 <= 32, "one lane per warp in the second reduction");
    static_assert(B * K <= 65536, "16-bit positions and slots in a key");
    constexpr uint32_t kNobody = 0xFFFFFFFFu, kRankMax = 0xFF7FFFFFu;  // kRankMax: FLT_MAX's rank
    extern __shared__ float4 tsm[];
    __shared__ unsigned long long s_best[2][B / 32];
    const int n = (int)nobj, tid = (int)threadIdx.x, warp = tid >> 5, lane = tid & 31;
    Box6 own[K];
    uint32_t ps[K];  // list position << 16 | slot
#pragma unroll
    for (int j = 0; j < K; ++j) {
        const int i = tid + j * B;
        // no cluster (also after a merge): areas with this box are infinite or NaN
        own[j] = Box6{0.0f, 0.0f, 0.0f, INFINITY, INFINITY, INFINITY};
        ps[j] = 0xFFFF0000u | (uint32_t)i;
        if (i < n) {
            ps[j] = ((uint32_t)i << 16) | (uint32_t)i;
            own[j] = object_bounds(blas_table[obj_blas[i]], xf + 16ull * i);
            store_cluster(tsm, i, own[j], 1 + i);  // leaves at 1..nobj (tlas.rs:210-218)
            store_tlas_node(tlas_out, 1u + (uint32_t)i, own[j], 0u, (uint32_t)i);
        }
    }
    __syncthreads();
    int count = n, used = 1 + n, buf = 0;
    uint32_t err = 0;
    uint64_t steps = 0;
    const uint64_t max_steps = 4ull * nobj * nobj + 64;
    // find_best_match with box P, leaving out the cluster whose (position, slot) is `self`: the
    // candidate's (position, slot), kNobody if there is none
    auto best = [&](const Box6& P, uint32_t self) {
        unsigned long long k[K];
#pragma unroll
        for (int j = 0; j < K; ++j) {
            // the order-preserving rank of the area, both zeros one rank (-0 + 0 = +0); an area that is
            // not below FLT_MAX ranks at or above kRankMax, NaN too (the canonical one, positive)
            const int bits = __float_as_int(fadd(sa_merge(P, own[j]), 0.0f));
            const uint32_t rank = (uint32_t)(bits ^ ((bits >> 31) | (int)0x80000000));
            k[j] = ((unsigned long long)(ps[j] == self ? 0xFFFFFFFFu : rank) << 32) | ps[j];
        }
#pragma unroll
        for (int s = 1; s < K; s *= 2)
#pragma unroll
            for (int j = 0; j + s < K; j += 2 * s) k[j] = k[j + s] < k[j] ? k[j + s] : k[j];
        unsigned long long m = warp_min_key(k[0]);
        if (lane == 0) s_best[buf][warp] = m;
        __syncthreads();
        m = warp_min_key(lane < B / 32 ? s_best[buf][lane] : kNoKey);
        buf ^= 1;  // the other slots are free: every thread read them before this scan's barrier
        return (uint32_t)(m >> 32) < kRankMax ? (uint32_t)m : kNobody;
    };
    // a and b are (position << 16 | slot); the position of a goes stale when a itself was the last
    uint32_t a = 0u;
    Cluster A = load_cluster(tsm, 0);
    uint32_t b = best(A.box, a);
    while (count > 1) {
        if (b == kNobody || ++steps > max_steps) {
            err = 1;
            break;
        }
        const Cluster C = load_cluster(tsm, (int)(b & 0xFFFFu));
        const uint32_t c = best(C.box, b);
        if (a != c) {
            a = b;
            A = C;
            b = c;
            continue;
        }
        // node `used` = Aabb::new of a and b, LeftRightIndex::new(node a, node b) = a + (b << 16)
        // (tlas.rs:18-22, 234-236); position a then holds it and position b the last one
        // (tlas.rs:238-240), also when a itself is the last
        const int last = count - 1, a_slot = (int)(a & 0xFFFFu), b_slot = (int)(b & 0xFFFFu);
        const Box6 m = merged_box(A.box, C.box);
        if (tid == 0) store_tlas_node(tlas_out, (uint32_t)used, m, (uint32_t)A.node + ((uint32_t)C.node << 16), 0u);
        if (tid == a_slot % B) store_cluster(tsm, a_slot, m, used);
#pragma unroll
        for (int j = 0; j < K; ++j) {
            const int slot = tid + j * B;
            if (slot == a_slot) own[j] = m;
            if (slot == b_slot) own[j] = Box6{0.0f, 0.0f, 0.0f, INFINITY, INFINITY, INFINITY};
            if ((ps[j] >> 16) == (uint32_t)last) ps[j] = (b & 0xFFFF0000u) | (uint32_t)slot;
        }
        A = Cluster{m, used};
        count = last;
        used += 1;
        b = best(m, a);  // its barrier publishes the merged cluster
    }
    if (tid == 0) {
        if (err == 0) {  // nodes[0] = nodes[list[a]] (tlas.rs:248); thread 0 wrote every inner node itself
            const float4 r0 = tlas_out[2ull * A.node], r1 = tlas_out[2ull * A.node + 1];
            tlas_out[0] = r0;
            tlas_out[1] = r1;
        }
        status[0] = (uint32_t)used;
        status[1] = err;
    }
}

// Larger scenes: the same walk with the list in global memory (`work`), every scan by a block of 512.
constexpr int kTlasThreads = 512;

struct TlasList {  // one entry per list position
    float *lx, *ly, *lz, *hx, *hy, *hz;  // node bounds (nodes[list[p]].aabb)
    int* node;                            // list[p]: node index
};

__device__ __forceinline__ Box6 load_box(const TlasList& S, int p) {
    return Box6{S.lx[p], S.ly[p], S.lz[p], S.hx[p], S.hy[p], S.hz[p]};
}

// One merge of the walk by warp 0's lanes 0-6 (each touches only its own array): lane c < 6 the
// c-th coordinate array, lane 6 the node list.
__device__ __forceinline__ void tlas_merge(const TlasList& S, int n, float4* tlas_out, int a, int b, int last, int used,
                                           int lane) {
    if (lane >= 7) return;
    // node `used` as 8 floats: lo.xyz, left_right, hi.xyz, blas (0 for an inner node)
    float* out = reinterpret_cast<float*>(tlas_out) + 8ull * (uint32_t)used;
    if (lane < 6) {
        float* arr = S.lx + lane * n;  // lx, ly, lz, hx, hy, hz are consecutive arrays
        const float va = arr[a], vb = arr[b];
        const float m = lane < 3 ? min_ni(va, vb) : max_ni(va, vb);
        arr[a] = m;
        arr[b] = arr[last];
        out[lane < 3 ? lane : lane + 1] = m;
    } else {
        out[3] = __uint_as_float((uint32_t)S.node[a] + ((uint32_t)S.node[b] << 16));
        out[7] = __uint_as_float(0u);
        S.node[a] = used;
        S.node[b] = S.node[last];
    }
}

__global__ void __launch_bounds__(kTlasThreads) k_tlas_rebuild_large(const GBlas* __restrict__ blas_table,
                                                                     const uint32_t* __restrict__ obj_blas,
                                                                     const float* __restrict__ xf, uint32_t nobj,
                                                                     float4* __restrict__ tlas_out, uint32_t* status,
                                                                     float* work) {
    __shared__ unsigned long long s_key;
    const int n = (int)nobj;
    const TlasList S = {work,         work + n,     work + 2 * n, work + 3 * n,
                        work + 4 * n, work + 5 * n, reinterpret_cast<int*>(work + 6 * n)};
    const int tid = (int)threadIdx.x;
    const int warp = tid >> 5, lane = tid & 31, nwarps = (int)(blockDim.x >> 5);
    for (int i = tid; i < n; i += (int)blockDim.x) {
        const Box6 o = object_bounds(blas_table[obj_blas[i]], xf + 16ull * i);
        S.lx[i] = o.lx;
        S.ly[i] = o.ly;
        S.lz[i] = o.lz;
        S.hx[i] = o.hx;
        S.hy[i] = o.hy;
        S.hz[i] = o.hz;
        S.node[i] = 1 + i;
        store_tlas_node(tlas_out, 1u + (uint32_t)i, o, 0u, (uint32_t)i);
    }
    __syncthreads();
    int count = n, used = 1 + n, a = 0;
    uint32_t err = 0;
    uint64_t steps = 0;
    const uint64_t max_steps = 4ull * nobj * nobj + 64;
    auto best = [&](int p) {
        if (tid == 0) s_key = kNoKey;
        __syncthreads();
        const int chunk = (count + nwarps - 1) / nwarps;
        const int r0 = warp * chunk, r1 = min(count, r0 + chunk);
        if (r0 < r1) {
            const Box6 P = load_box(S, p);
            unsigned long long k = kNoKey;
            for (int r = r0 + lane; r < r1; r += 32) {
                if (r == p) continue;
                const unsigned long long kr = sa_key(P, load_box(S, r), r);
                k = kr < k ? kr : k;
            }
            k = warp_min_key(k);
            if (lane == 0 && k != kNoKey) atomicMin(&s_key, k);
        }
        __syncthreads();
        const int r = key_pos(s_key);
        __syncthreads();
        return r;
    };
    int b = best(0);
    while (count > 1) {
        if (b < 0 || ++steps > max_steps) {
            err = 1;
            break;
        }
        const int c = best(b);
        if (a != c) {
            a = b;
            b = c;
            continue;
        }
        if (warp == 0) tlas_merge(S, n, tlas_out, a, b, count - 1, used, lane);
        count -= 1;
        used += 1;
        __syncthreads();
        b = best(a);
    }
    __syncthreads();  // the inner nodes written by warp 0's lanes are visible to thread 0
    if (tid == 0) {
        if (err == 0) {  // nodes[0] = nodes[list[a]] (tlas.rs:248)
            const uint32_t r = (uint32_t)S.node[a];
            const float4 r0 = tlas_out[2ull * r], r1 = tlas_out[2ull * r + 1];
            tlas_out[0] = r0;
            tlas_out[1] = r1;
        }
        status[0] = (uint32_t)used;
        status[1] = err;
    }
}

// ---- two-level traversal ------------------------------------------------------------------
// Tlas::intersect (tlas.rs:123-177) with SceneObject::intersect (scene_object.rs:78-89) at the
// leaves: the ray goes to model space through the cached inverse, 1/d' is recomputed (Ray::new)
// and the BLAS traversal (Trav, the same as for a single BLAS) shares the TLAS's closest t.  The
// LaneRay holds the model-space ray while a BLAS is traversed; the world ray is kept here.  Big
// BLAS leaves are handed to the warp-cooperative leaf phase, keyed by (BLAS, leaf), so rays in
// different instances of the same BLAS share the loaded triangle pairs.
struct SceneData {
    const float4* tlas;
    const GBlas* blas_table;
    const uint32_t* obj_blas;
    const float* inv;
    uint32_t tlas_nodes;
};

// SceneObject::intersect's ray: world ray (wo, wd) through the cached inverse m, 1/d' recomputed.
__device__ __forceinline__ void to_model(const float* m, float3 wo, float3 wd, LaneRay& r) {
    r.o.x = fadd(fadd(fadd(fmul(__ldg(m + 0), wo.x), fmul(__ldg(m + 4), wo.y)), fmul(__ldg(m + 8), wo.z)),
                 fmul(__ldg(m + 12), 1.0f));
    r.o.y = fadd(fadd(fadd(fmul(__ldg(m + 1), wo.x), fmul(__ldg(m + 5), wo.y)), fmul(__ldg(m + 9), wo.z)),
                 fmul(__ldg(m + 13), 1.0f));
    r.o.z = fadd(fadd(fadd(fmul(__ldg(m + 2), wo.x), fmul(__ldg(m + 6), wo.y)), fmul(__ldg(m + 10), wo.z)),
                 fmul(__ldg(m + 14), 1.0f));
    r.d.x = fadd(fadd(fadd(fmul(__ldg(m + 0), wd.x), fmul(__ldg(m + 4), wd.y)), fmul(__ldg(m + 8), wd.z)),
                 fmul(__ldg(m + 12), 0.0f));
    r.d.y = fadd(fadd(fadd(fmul(__ldg(m + 1), wd.x), fmul(__ldg(m + 5), wd.y)), fmul(__ldg(m + 9), wd.z)),
                 fmul(__ldg(m + 13), 0.0f));
    r.d.z = fadd(fadd(fadd(fmul(__ldg(m + 2), wd.x), fmul(__ldg(m + 6), wd.y)), fmul(__ldg(m + 10), wd.z)),
                 fmul(__ldg(m + 14), 0.0f));
    r.rd = recip3(r.d);
}

template <class STK, int TSTACK>
struct SceneTrav {
    TravT<STK> bt;
    GBlas blas;
    uint2 tstack[TSTACK];  // pending far TLAS nodes: (left_right, blas)
    int tsp;
    uint32_t lr, bl, tsteps;
    bool in_blas;
    float3 wo, wd, wrd;

    __device__ __forceinline__ void init(const SceneData& sd, LaneRay& r) {
        const float4 lo = __ldg(sd.tlas), hi = __ldg(sd.tlas + 1);
        lr = __float_as_uint(lo.w);
        bl = __float_as_uint(hi.w);
        tsp = 0;
        tsteps = 0;
        in_blas = false;
        wo = r.o;
        wd = r.d;
        wrd = r.rd;
        blas.nodes = nullptr;
        blas.tris = nullptr;
        blas.pairs = nullptr;
        blas.hx = nullptr;
        blas.cones = nullptr;
        blas.nodes_used = blas.ntris = blas.root_count = blas.root_first = 0;
    }

    __device__ __forceinline__ bool tpop() {
        if (tsp == 0) return true;
        --tsp;
        lr = tstack[tsp].x;
        bl = tstack[tsp].y;
        return false;
    }

    // After the cooperative test of the current big BLAS leaf.
    __device__ __forceinline__ StepResult after_leaf() {
        if (!bt.pop()) return kStepContinue;
        in_blas = false;
        return tpop() ? kStepFinished : kStepContinue;
    }

    __device__ __forceinline__ StepResult advance(const SceneData& sd, LaneRay& r, LeafPolicy pol, uint32_t* err) {
        for (;;) {
            if (in_blas) {
                const StepResult st = bt.step(blas, r, pol, err);
                if (st == kStepContinue) continue;
                if (st == kStepBigLeaf) return st;
                in_blas = false;
                if (tpop()) return kStepFinished;
                continue;
            }
            if (++tsteps > 2u * sd.tlas_nodes + 16u) {
                atomicOr(err, kErrSteps);
                return kStepFinished;
            }
            if (lr == 0u) {  // TLAS leaf: SceneObject::intersect
                to_model(sd.inv + 16ull * bl, wo, wd, r);
                r.inst_cur = bl;
                blas = sd.blas_table[__ldg(sd.obj_blas + bl)];
                bt.init(blas);
                in_blas = true;
                continue;
            }
            // LeftRightIndex getters are swapped (tlas.rs:24-32): left() is the high half.
            const uint32_t li = (lr & 0xFFFF0000u) >> 16, ri = lr & 0xFFFFu;
            const float4 l0 = __ldg(sd.tlas + 2ull * li), l1 = __ldg(sd.tlas + 2ull * li + 1);
            const float4 r0 = __ldg(sd.tlas + 2ull * ri), r1 = __ldg(sd.tlas + 2ull * ri + 1);
            float dl, dr;
            const bool hl = slab(l0, l1, wo, wrd, r.ct, dl);
            const bool hr = slab(r0, r1, wo, wrd, r.ct, dr);
            const float kl = hl ? dl : FLT_MAX;
            const float kr = hr ? dr : FLT_MAX;
            const bool left_near = kl < kr;
            const bool near_hit = left_near ? hl : hr;
            const bool far_hit = left_near ? hr : hl;
            if (near_hit) {
                if (far_hit) {
                    if (tsp >= TSTACK) {
                        atomicOr(err, kErrStack);
                        return kStepFinished;
                    }
                    tstack[tsp++] = left_near ? make_uint2(ubits(r0.w), ubits(r1.w)) : make_uint2(ubits(l0.w), ubits(l1.w));
                }
                lr = left_near ? ubits(l0.w) : ubits(r0.w);
                bl = left_near ? ubits(l1.w) : ubits(r1.w);
                continue;
            }
            if (tpop()) return kStepFinished;
        }
    }
};

// Cooperative phase of the two-level traversal (same grouping as the single-BLAS kernels).
template <class STK, int TSTACK>
__device__ __forceinline__ void scene_coop_phase(unsigned pend, SceneTrav<STK, TSTACK>& tr, LaneRay& r,
                                                 StepResult& st) {
    const unsigned lane = threadIdx.x & 31u;
    const unsigned long long key = reinterpret_cast<unsigned long long>(tr.blas.pairs);
    while (pend) {
        const int leader = __ffs(pend) - 1;
        const uint32_t f = __shfl_sync(kFull, tr.bt.first, leader);
        const uint32_t c = __shfl_sync(kFull, tr.bt.cnt, leader);
        const unsigned long long lk = __shfl_sync(kFull, key, leader);
        const ulonglong2* P = reinterpret_cast<const ulonglong2*>(lk);
        unsigned group = __ballot_sync(kFull, ((pend >> lane) & 1u) && tr.bt.first == f && key == lk);
        pend &= ~group;
        while (group) {
            const int a = __ffs(group) - 1;
            group &= group - 1u;
            if (group) {
                const int b = __ffs(group) - 1;
                group &= group - 1u;
                coop_leaf2(P, f, c, a, b, r);
                if ((int)lane == a || (int)lane == b) st = tr.after_leaf();
            } else {
                coop_leaf(P, f, c, a, r);
                if ((int)lane == a) st = tr.after_leaf();
            }
        }
    }
}

constexpr int kTlasStack = 64;

template <int BLOCK, int MINB, class STK>
__global__ void __launch_bounds__(BLOCK, MINB) k_trace_scene(SceneData sd, const float4* __restrict__ rays,
                                                             uint32_t n, GHit* __restrict__ hits, LeafPolicy pol,
                                                             uint32_t* err) {
    extern __shared__ uint2 stack_smem[];
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (__all_sync(kFull, i >= n)) return;
    const bool active = i < n;
    LaneRay r;
    SceneTrav<STK, kTlasStack> tr;
    tr.bt.stk.bind(stack_smem);
    StepResult st = kStepFinished;
    if (active) {
        float3 o, d;
        float t0;
        load_ray(rays, i, o, d, t0);
        r.o = o;
        r.d = d;
        r.rd = recip3(d);
        r.ct = t0;
        r.hu = r.hv = 0.0f;
        r.hp = 0;
        r.hit = false;
        r.inst = r.inst_cur = 0;
        tr.init(sd, r);
        st = kStepContinue;
    }
    for (;;) {
        if (st == kStepContinue) st = tr.advance(sd, r, pol, err);
        const unsigned pend = __ballot_sync(kFull, st == kStepBigLeaf);
        if (pend == 0u) break;
        scene_coop_phase(pend, tr, r, st);
    }
    if (active) store_hit(hits, i, r.hit && r.ct < FLT_MAX, r.ct, r.hu, r.hv, r.hp, r.inst);
}

// The accumulator and shader of a render over a scene.  The normal and texture accumulators
// look up `scene.get_unchecked(instance_index)` (renderer.rs:258-263, 312-317): with lookup 0 the
// reference's packed index -- instance 0, because Bvh::intersect packs instance 0
// (InstancePrimitiveIndex::from_primitive, bvh.rs:296), and the primitive's low 20 bits
// (intersection.rs:57-60) -- with lookup 1 the hit's own object.  A primitive outside the looked-up
// model's data (where the reference's slice indexing panics) or missing shading data sets kErrLookup
// and the pixel's radiance is zero.
__device__ __forceinline__ void shade_scene_pixel(const SceneData& sd, const RenderParams& P,
                                                  const ShadeEntry* __restrict__ shade_tab,
                                                  const float* __restrict__ xf, int lookup, const LaneRay& r, int x, int y,
                                                  uint8_t* __restrict__ rgba, uint32_t* err) {
    const bool hit = r.hit && r.ct < FLT_MAX;
    const float* nrm = nullptr;
    const float* tc = nullptr;
    const uint8_t* tex = nullptr;
    uint32_t tw = 0, th = 0, prim = r.hp;
    const float* oxf = xf;
    bool ok = true;
    if (hit && (P.acc_kind == BVHGPU_ACC_NORMAL || P.acc_kind == BVHGPU_ACC_TEXTURE)) {
        const uint32_t obj = lookup ? r.inst : 0u;
        prim = lookup ? r.hp : (r.hp & 0x000FFFFFu);
        const ShadeEntry e = shade_tab[__ldg(sd.obj_blas + obj)];
        oxf = xf + 16ull * obj;
        nrm = e.normals;
        tc = e.tex_coords;
        tex = e.texels;
        tw = e.tex_w;
        th = e.tex_h;
        ok = prim < e.ntris && (P.acc_kind == BVHGPU_ACC_NORMAL ? nrm != nullptr
                                                                : (tc != nullptr && tex != nullptr && tw && th));
        if (!ok) atomicOr(err, kErrLookup);
    }
    const float3 rad = ok ? accumulate(P, hit, r.ct, r.hu, r.hv, prim, nrm, oxf, tc, tex, tw, th)
                          : make_float3(0.0f, 0.0f, 0.0f);
    reinterpret_cast<uchar4*>(rgba)[(size_t)y * P.width + x] = shade(P, rad);
}

// PathTracer::evaluate over a whole scene (renderer.rs:345-384 -> Scene::intersect, scene.rs:32-34):
// one 64-thread block per 8x8 tile, the camera ray through the pixel's top-left corner, the two-level
// traversal of k_trace_scene, then the accumulator and shader.
template <int STACK>
__global__ void __launch_bounds__(64) k_render_scene(SceneData sd, RenderParams P,
                                                     const ShadeEntry* __restrict__ shade_tab,
                                                     const float* __restrict__ xf, int lookup,
                                                     uint8_t* __restrict__ rgba, LeafPolicy pol, uint32_t* err) {
    const int tiles_x = (P.width + 7) / 8;
    const int tile = blockIdx.x;
    const int x = (tile % tiles_x) * 8 + (threadIdx.x & 7);
    const int y = (tile / tiles_x) * 8 + (threadIdx.x >> 3);
    const bool active = x < P.width && y < P.height;  // all lanes stay for the cooperative leaf steps
    LaneRay r;
    SceneTrav<LocalStack<STACK>, kTlasStack> tr;
    tr.bt.stk.bind(nullptr);
    StepResult st = kStepFinished;
    if (active) {
        float3 o, d;
        camera_ray(P, x, y, o, d);
        r.o = o;
        r.d = d;
        r.rd = recip3(d);
        r.ct = FLT_MAX;
        r.hu = r.hv = 0.0f;
        r.hp = 0;
        r.hit = false;
        r.inst = r.inst_cur = 0;
        tr.init(sd, r);
        st = kStepContinue;
    }
    for (;;) {
        if (st == kStepContinue) st = tr.advance(sd, r, pol, err);
        const unsigned pend = __ballot_sync(kFull, st == kStepBigLeaf);
        if (pend == 0u) break;
        scene_coop_phase(pend, tr, r, st);
    }
    if (!active) return;
    shade_scene_pixel(sd, P, shade_tab, xf, lookup, r, x, y, rgba, err);
}

// ---- one warp per ray (wide.cuh) over a scene ----------------------------------------------------
struct WideSceneSmem {
    WideSmem blas;
    uint2 tlas[kWideTlas];
};

// The closest hit of world ray r (every lane the same) in the scene; r ends in the last visited object's
// model space.  False: stopped, as wide_blas.
__device__ __forceinline__ bool wide_scene(const SceneData& sd, LaneRay& r, LeafPolicy pol, WideSceneSmem& sm,
                                           const Deadline& deadline, uint32_t* err) {
    const unsigned lane = threadIdx.x & 31u;
    const float3 wo = r.o, wd = r.d, wrd = r.rd;
    uint32_t lr = __float_as_uint(__ldg(sd.tlas).w), bl = __float_as_uint(__ldg(sd.tlas + 1).w), tsteps = 0u, tsp = 0u;
    for (;;) {
        if (++tsteps > 2u * sd.tlas_nodes + 16u) {
            if (lane == 0u) atomicOr(err, kErrSteps);
            return false;
        }
        bool pop = true;
        if (lr == 0u) {
            to_model(sd.inv + 16ull * bl, wo, wd, r);
            r.inst_cur = bl;
            const GBlas b = sd.blas_table[__ldg(sd.obj_blas + bl)];
            if (!wide_blas(b, r, pol, sm.blas, deadline, err)) return false;
        } else {
            const uint32_t li = (lr & 0xFFFF0000u) >> 16, ri = lr & 0xFFFFu;  // the swapped getters (tlas.rs:24-32)
            const float4 l0 = __ldg(sd.tlas + 2ull * li), l1 = __ldg(sd.tlas + 2ull * li + 1);
            const float4 r0 = __ldg(sd.tlas + 2ull * ri), r1 = __ldg(sd.tlas + 2ull * ri + 1);
            float dl, dr;
            const bool hl = slab(l0, l1, wo, wrd, r.ct, dl);
            const bool hr = slab(r0, r1, wo, wrd, r.ct, dr);
            const bool left_near = (hl ? dl : FLT_MAX) < (hr ? dr : FLT_MAX);
            if (left_near ? hl : hr) {
                if (left_near ? hr : hl) {
                    if (tsp >= kWideTlas) {
                        if (lane == 0u) atomicOr(err, kErrStack);
                        return false;
                    }
                    if (lane == 0u)
                        sm.tlas[tsp] = left_near ? make_uint2(ubits(r0.w), ubits(r1.w)) : make_uint2(ubits(l0.w), ubits(l1.w));
                    ++tsp;
                    __syncwarp();
                }
                lr = left_near ? ubits(l0.w) : ubits(r0.w);
                bl = left_near ? ubits(l1.w) : ubits(r1.w);
                pop = false;
            }
        }
        if (pop) {
            if (tsp == 0u) return true;
            const uint2 e = sm.tlas[--tsp];
            lr = e.x;
            bl = e.y;
            __syncwarp();
        }
    }
}

__device__ __forceinline__ void init_scene_ray(LaneRay& r, float3 o, float3 d, float t) {
    init_lane_ray(r, o, d, t);
    r.inst = r.inst_cur = 0;
}

__global__ void __launch_bounds__(32 * kWideWarps) k_trace_scene_wide(SceneData sd, const float4* __restrict__ rays, uint32_t n,
                                                                      GHit* __restrict__ hits, LeafPolicy pol, uint32_t* err) {
    __shared__ WideSceneSmem smem[kWideWarps];
    const uint32_t i = blockIdx.x * kWideWarps + (threadIdx.x >> 5);
    if (i >= n) return;
    LaneRay r;
    float3 o, d;
    float t0;
    load_ray(rays, i, o, d, t0);
    init_scene_ray(r, o, d, t0);
    wide_scene(sd, r, pol, smem[threadIdx.x >> 5], Deadline{0ull}, err);
    if ((threadIdx.x & 31u) == 0u) store_hit(hits, i, r.hit && r.ct < FLT_MAX, r.ct, r.hu, r.hv, r.hp, r.inst);
}

__global__ void __launch_bounds__(32 * kWideWarps) k_render_scene_wide(SceneData sd, RenderParams P,
                                                                       const ShadeEntry* __restrict__ shade_tab,
                                                                       const float* __restrict__ xf, int lookup,
                                                                       uint8_t* __restrict__ rgba, LeafPolicy pol, uint32_t* err) {
    __shared__ WideSceneSmem smem[kWideWarps];
    const uint32_t i = blockIdx.x * kWideWarps + (threadIdx.x >> 5);
    if (i >= (uint32_t)P.width * (uint32_t)P.height) return;
    const int x = (int)(i % (uint32_t)P.width), y = (int)(i / (uint32_t)P.width);
    float3 o, d;
    camera_ray(P, x, y, o, d);
    LaneRay r;
    init_scene_ray(r, o, d, FLT_MAX);
    wide_scene(sd, r, pol, smem[threadIdx.x >> 5], Deadline{0ull}, err);
    if ((threadIdx.x & 31u) == 0u) shade_scene_pixel(sd, P, shade_tab, xf, lookup, r, x, y, rgba, err);
}

__global__ void __launch_bounds__(32 * kWideWarps) k_scene_bounce_wide(SceneData sd, const float4* __restrict__ rays, uint32_t n,
                                                                       uint32_t seed, GHit* __restrict__ hits0,
                                                                       GHit* __restrict__ hits1, LeafPolicy pol, uint32_t* err,
                                                                       unsigned long long* began) {
    __shared__ WideSceneSmem smem[kWideWarps];
    WideSceneSmem& sm = smem[threadIdx.x >> 5];
    const uint32_t i = blockIdx.x * kWideWarps + (threadIdx.x >> 5);
    const bool first = (threadIdx.x & 31u) == 0u;
    if (i >= n) return;
    Deadline deadline;
    deadline.start(err, began);
    LaneRay r;
    float3 o, d;
    float t0;
    load_ray(rays, i, o, d, t0);
    init_scene_ray(r, o, d, t0);
    wide_scene(sd, r, pol, sm, deadline, err);
    const bool h = r.hit && r.ct < FLT_MAX;
    if (first) store_hit(hits0, i, h, r.ct, r.hu, r.hv, r.hp, r.inst);
    float3 po, pd;
    bool have = false;
    if (h) {
        const float4* T = sd.blas_table[__ldg(sd.obj_blas + r.inst)].tris + 3ull * r.hp;
        have = bounce_dir_instanced(o, d, r.ct, __ldg(T + 1), __ldg(T + 2), sd.inv + 16ull * r.inst, seed, i, po, pd);
    }
    if (!have) {
        if (first) store_hit(hits1, i, false, 0, 0, 0, 0, 0);
        return;
    }
    init_scene_ray(r, po, pd, FLT_MAX);
    wide_scene(sd, r, pol, sm, deadline, err);
    if (first) store_hit(hits1, i, r.hit && r.ct < FLT_MAX, r.ct, r.hu, r.hv, r.hp, r.inst);
}

// Persistent primary + bounce over a scene (the instanced frame): idle lanes are refilled from
// the queue; a primary that hits continues in its lane with the bounce ray of its hit.
template <int BLOCK, int MINB, class STK>
__global__ void __launch_bounds__(BLOCK, MINB) k_scene_persistent_bounce(SceneData sd, const float4* __restrict__ rays,
                                                                         uint32_t n, uint32_t seed,
                                                                         GHit* __restrict__ hits0,
                                                                         GHit* __restrict__ hits1, uint32_t* queue,
                                                                         LeafPolicy pol, uint32_t refill,
                                                                         uint32_t* err) {
    extern __shared__ uint2 stack_smem[];
    const unsigned lane = threadIdx.x & 31u;
    int phase = 0;  // 0 needs work, 1 primary, 2 bounce, 3 retired
    uint32_t idx = 0;
    LaneRay r;
    SceneTrav<STK, kTlasStack> tr;
    tr.bt.stk.bind(stack_smem);
    StepResult st = kStepFinished;
    bool queue_open = true;
    Deadline dl;
    dl.start(err);
    for (;;) {
        if (dl.expired(err)) return;
        const unsigned need = __ballot_sync(kFull, phase == 0);
        const unsigned busy = __ballot_sync(kFull, phase == 1 || phase == 2);
        if (need != 0u && ((uint32_t)__popc(need) >= refill || busy == 0u)) {
            const int leader = __ffs(need) - 1;
            uint32_t base = 0;
            if ((int)lane == leader) base = atomicAdd(queue, (uint32_t)__popc(need));
            base = __shfl_sync(kFull, base, leader);
            if (base + (uint32_t)__popc(need) >= n) queue_open = false;
            if (phase == 0) {
                const uint32_t my = base + __popc(need & ((1u << lane) - 1u));
                if (my < n) {
                    idx = my;
                    float3 o, d;
                    float t0;
                    load_ray(rays, idx, o, d, t0);
                    r.o = o;
                    r.d = d;
                    r.rd = recip3(d);
                    r.ct = t0;
                    r.hu = r.hv = 0.0f;
                    r.hp = 0;
                    r.hit = false;
                    r.inst = r.inst_cur = 0;
                    tr.init(sd, r);
                    st = kStepContinue;
                    phase = 1;
                } else {
                    phase = 3;
                }
            }
        }
        while (phase == 1 || phase == 2) {
            if (st == kStepContinue) st = tr.advance(sd, r, pol, err);
            if (st != kStepFinished) break;
            const bool h = r.hit && r.ct < FLT_MAX;
            if (phase == 2) {
                store_hit(hits1, idx, h, r.ct, r.hu, r.hv, r.hp, r.inst);
                phase = 0;
                break;
            }
            store_hit(hits0, idx, h, r.ct, r.hu, r.hv, r.hp, r.inst);
            float3 po, pd;
            bool have = false;
            if (h) {
                const GBlas hb = sd.blas_table[__ldg(sd.obj_blas + r.inst)];
                const float4* T = hb.tris + 3ull * r.hp;
                have = bounce_dir_instanced(tr.wo, tr.wd, r.ct, __ldg(T + 1), __ldg(T + 2), sd.inv + 16ull * r.inst,
                                            seed, idx, po, pd);
            }
            if (!have) {
                store_hit(hits1, idx, false, 0, 0, 0, 0, 0);
                phase = 0;
                break;
            }
            r.o = po;
            r.d = pd;
            r.rd = recip3(pd);
            r.ct = FLT_MAX;
            r.hu = r.hv = 0.0f;
            r.hp = 0;
            r.hit = false;
            r.inst = r.inst_cur = 0;
            tr.init(sd, r);
            st = kStepContinue;
            phase = 2;
        }
        const unsigned pend = __ballot_sync(kFull, (phase == 1 || phase == 2) && st == kStepBigLeaf);
        if (pend == 0u) {
            if (!queue_open && __ballot_sync(kFull, phase == 0 || phase == 1 || phase == 2) == 0u) break;
            continue;
        }
        scene_coop_phase(pend, tr, r, st);
    }
}

// Bounce rays of an instanced frame in pixel order (for checking against the oracle).
__global__ void k_scene_bounce_rays(SceneData sd, const float4* __restrict__ rays, const GHit* __restrict__ hits0,
                                    uint32_t n, uint32_t seed, float4* __restrict__ out, uint8_t* __restrict__ valid) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const GHit h = hits0[i];
    bool have = false;
    float3 po = make_float3(0, 0, 0), pd = po;
    if (h.prim != kMiss) {
        float3 o, d;
        float t0;
        load_ray(rays, i, o, d, t0);
        const GBlas hb = sd.blas_table[sd.obj_blas[h.inst]];
        const float4* T = hb.tris + 3ull * h.prim;
        have = bounce_dir_instanced(o, d, h.t, T[1], T[2], sd.inv + 16ull * h.inst, seed, i, po, pd);
    }
    out[2ull * i] = make_float4(po.x, po.y, po.z, FLT_MAX);
    out[2ull * i + 1] = make_float4(pd.x, pd.y, pd.z, 0.0f);
    valid[i] = have ? 1 : 0;
}

// ---- animation (the frame pattern of the reference's demos, closed form) --------------------
// Radial vertex wobble: v = dir * (r0 + amp * sin(freq * t + phase)), t read from device memory
// so that a captured frame graph replays with the current time.
__global__ void k_wobble(float* __restrict__ verts, const float* __restrict__ dirs, const float* __restrict__ r0,
                         const float* __restrict__ phase, uint32_t nv, float amp, float freq,
                         const float* __restrict__ time) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= nv) return;
    const float t = *time;
    const float r = r0[i] + amp * sinf(freq * t + phase[i]);
    verts[3ull * i] = dirs[3ull * i] * r;
    verts[3ull * i + 1] = dirs[3ull * i + 1] * r;
    verts[3ull * i + 2] = dirs[3ull * i + 2] * r;
}

// Instance i at time t: rotation R_i = R0_i * Rot(axis_i, omega_i t) (Rodrigues), uniform scale
// s_i, translation T_i; xf = [s R | T] and its inverse [R^T / s | -R^T T / s], column-major.
__global__ void k_animate_instances(float* __restrict__ xf, float* __restrict__ inv, const float* __restrict__ rot0,
                                    const float* __restrict__ axis, const float* __restrict__ omega,
                                    const float* __restrict__ scale, const float* __restrict__ trans, uint32_t n,
                                    const float* __restrict__ time) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float t = *time;
    const float ang = omega[i] * t;
    float sn, cs;
    sincosf(ang, &sn, &cs);
    const float kx = axis[3 * i], ky = axis[3 * i + 1], kz = axis[3 * i + 2];
    const float oc = 1.0f - cs;
    // Rot(axis, ang), row-major A[r][c]
    float A[3][3] = {{cs + kx * kx * oc, kx * ky * oc - kz * sn, kx * kz * oc + ky * sn},
                     {ky * kx * oc + kz * sn, cs + ky * ky * oc, ky * kz * oc - kx * sn},
                     {kz * kx * oc - ky * sn, kz * ky * oc + kx * sn, cs + kz * kz * oc}};
    const float* B = rot0 + 9ull * i;  // row-major R0
    float R[3][3];
    for (int r = 0; r < 3; ++r)
        for (int c = 0; c < 3; ++c) R[r][c] = B[3 * r] * A[0][c] + B[3 * r + 1] * A[1][c] + B[3 * r + 2] * A[2][c];
    const float s = scale[i], is = 1.0f / s;
    const float tx = trans[3 * i], ty = trans[3 * i + 1], tz = trans[3 * i + 2];
    float* X = xf + 16ull * i;
    float* I = inv + 16ull * i;
    for (int c = 0; c < 3; ++c)
        for (int r = 0; r < 3; ++r) {
            X[4 * c + r] = s * R[r][c];
            I[4 * c + r] = is * R[c][r];
        }
    X[3] = X[7] = X[11] = 0.0f;
    X[12] = tx; X[13] = ty; X[14] = tz; X[15] = 1.0f;
    I[3] = I[7] = I[11] = 0.0f;
    for (int r = 0; r < 3; ++r) I[12 + r] = -(is * (R[0][r] * tx + R[1][r] * ty + R[2][r] * tz));
    I[15] = 1.0f;
}

__global__ void k_advance_time(float* time, float dt) { *time += dt; }

inline unsigned grid_for(uint32_t n, int block) { return (unsigned)((n + block - 1) / block); }

}  // namespace

cudaError_t launch_write_tris(bvhgpu_ctx* ctx, DeviceBlas& b, const float* d_tris9, cudaStream_t s, uint32_t* decide) {
    if (b.ntris == 0) return cudaSuccess;
    LaunchScope scope(ctx, BVHGPU_K_OTHER, s);
    k_write_tris<<<grid_for(b.ntris, 256), 256, 0, s>>>(d_tris9, b.ntris, b.tris, b.verts,
                                                        reinterpret_cast<float*>(b.pairs));
    g_launches++;
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    return launch_hidden_refresh(ctx, b, s, false, decide);
}

cudaError_t launch_hidden_refresh(bvhgpu_ctx* ctx, DeviceBlas& b, cudaStream_t s, bool refit_follows, uint32_t* decide) {
    if (b.nhid == 0) return cudaSuccess;
    LaunchScope scope(ctx, BVHGPU_K_OTHER, s);
    k_hidden_refresh<<<grid_for(4u * b.nhid, 256), 256, 0, s>>>(
        b.tris, b.hx + hidden_table_u2(b.ntris), pairs_in_order(b.ntris), reinterpret_cast<float4*>(b.pairs),
        b.nodes + 2ull * b.nodes_used, b.nhid, b.hup, b.hagg, b.harrivals, b.cones, b.measured_roots, decide);
    g_launches++;
    if (b.measured_roots && !refit_follows) {
        k_hidden_root_cones<<<grid_for(b.ntris, 256), 256, 0, s>>>(b.tris, b.ntris, b.tri_leaf, b.hup + b.nhid, b.hagg,
                                                                  b.harrivals, b.cones);
        g_launches++;
    }
    return cudaGetLastError();
}

cudaError_t launch_refit(bvhgpu_ctx* ctx, DeviceBlas& b, cudaStream_t s, bool after_refresh) {
    if (b.nleaves == 0) return cudaSuccess;
    LaunchScope scope(ctx, BVHGPU_K_REFIT, s);
    auto* tris = after_refresh && b.measured_roots ? k_refit_tris<true> : k_refit_tris<false>;
    tris<<<grid_for(b.ntris, 256), 256, 0, s>>>(b.verts, b.ntris, b.tri_leaf, b.leaf_keys, b.hup + b.nhid, b.hagg, b.harrivals,
                                                b.cones);
    k_refit_leaves<<<grid_for(b.nleaves, kBlock), kBlock, 0, s>>>(b.nodes, b.verts, b.leaves, b.nleaves, b.parent,
                                                                  b.counters, b.leaf_keys);
    g_launches += 2;
    return cudaGetLastError();
}

size_t tlas_work_bytes(uint32_t nobj) { return 7ull * sizeof(float) * nobj; }

template <int B, int K>
static cudaError_t tlas_rebuild_block(bvhgpu_ctx* ctx, DeviceScene& sc, cudaStream_t s) {
    const size_t smem = 32ull * sc.nobjects;
    // the default limit covers the kernel's static shared memory (s_best) too
    constexpr size_t kStatic = 2 * sizeof(unsigned long long) * (B / 32);
    if (smem + kStatic > 48u * 1024u) {
        const cudaError_t e = cudaFuncSetAttribute(k_tlas_rebuild<B, K>, cudaFuncAttributeMaxDynamicSharedMemorySize, 32 * B * K);
        if (e != cudaSuccess) return e;
    }
    k_tlas_rebuild<B, K><<<1, B, smem, s>>>(static_cast<const GBlas*>(sc.blas_table), sc.obj_blas, sc.xf, sc.nobjects,
                                            sc.tlas, ctx->d_scratch + 8);
    return cudaGetLastError();
}

cudaError_t launch_tlas_rebuild(bvhgpu_ctx* ctx, DeviceScene& sc, cudaStream_t s) {
    LaunchScope scope(ctx, BVHGPU_K_TLAS_BUILD, s);
    g_launches++;
    const uint32_t n = sc.nobjects;
    // The fewest threads that hold the list in 2, 4 or 8 clusters each: fewer warps make the barrier
    // and the reductions of a scan shorter, more than 8 clusters a thread make the scan itself
    // longer.  In us, at 256 objects: 32 x 8 295, 64 x 4 218, 128 x 2 184, 256 x 1 197 (every find_best_match
    // as a scan of global memory 703; the block of 512 that cached each position's best 524); at 512: 128 x 4 433,
    // 256 x 2 589, 512 x 1 805; at 1,000: 128 x 8 1,158, 256 x 4 1,124, 512 x 2 1,309, 1024 x 1 1,583 (scans of shared
    // memory 2,913); at 4,096: 256 x 16 11,540, 512 x 8 11,590, 1024 x 4 12,980 (19,530).
    if (n <= 256u) return tlas_rebuild_block<128, 2>(ctx, sc, s);
    if (n <= 512u) return tlas_rebuild_block<128, 4>(ctx, sc, s);
    if (n <= 1024u) return tlas_rebuild_block<256, 4>(ctx, sc, s);
    if (n <= 2048u) return tlas_rebuild_block<256, 8>(ctx, sc, s);
    static_assert(kTlasBlockObjects == 512u * 8u, "the largest block's list");
    if (n <= kTlasBlockObjects) return tlas_rebuild_block<512, 8>(ctx, sc, s);
    k_tlas_rebuild_large<<<1, kTlasThreads, 0, s>>>(static_cast<const GBlas*>(sc.blas_table), sc.obj_blas, sc.xf, n,
                                                    sc.tlas, ctx->d_scratch + 8, static_cast<float*>(sc.tlas_work));
    return cudaGetLastError();
}

static SceneData scene_data(bvhgpu_ctx* ctx, DeviceScene& sc, uint32_t* depth) {
    SceneData sd;
    sd.tlas = sc.tlas;
    sd.blas_table = static_cast<const GBlas*>(sc.blas_table);
    sd.obj_blas = sc.obj_blas;
    sd.inv = sc.inv;
    sd.tlas_nodes = 2 * sc.nobjects;
    uint32_t d = 1;
    for (uint32_t id : sc.table_blas) d = std::max(d, ctx->blas[id].depth);
    *depth = d;
    return sd;
}

cudaError_t launch_trace_scene(bvhgpu_ctx* ctx, DeviceScene& sc, const float4* rays, uint32_t n, void* hits,
                               cudaStream_t s) {
    if (n == 0) return cudaSuccess;
    uint32_t depth = 1;
    SceneData sd = scene_data(ctx, sc, &depth);
    LaunchScope scope(ctx, BVHGPU_K_TRACE_SCENE, s);
    const Variant v = resolve(ctx->tune[BVHGPU_K_TRACE_SCENE], depth);
    if (n <= wide_rays(ctx, BVHGPU_K_TRACE_SCENE, sc)) {
        k_trace_scene_wide<<<grid_for(n, kWideWarps), 32 * kWideWarps, 0, s>>>(sd, rays, n, static_cast<GHit*>(hits), v.pol,
                                                                               ctx->d_err);
        g_launches++;
        return cudaGetLastError();
    }
    cudaError_t e = with_variant(v.shape, v.stack, [&](auto sh, auto tg) {
        using SH = decltype(sh);
        using STK = typename decltype(tg)::type;
        k_trace_scene<SH::block, SH::minb, STK><<<grid_for(n, SH::block), SH::block,
                                                  stack_smem_bytes<STK>(SH::block), s>>>(
            sd, rays, n, static_cast<GHit*>(hits), v.pol, ctx->d_err);
        return cudaGetLastError();
    });
    g_launches++;
    return e;
}

cudaError_t launch_render_scene(bvhgpu_ctx* ctx, DeviceScene& sc, const bvhgpu_camera& cam, int w, int h, int acc,
                                const float* acc_params, int shader, const float* shader_params,
                                const ShadeEntry* d_shade, int lookup, uint8_t* d_rgba, cudaStream_t s) {
    uint32_t depth = 1;
    SceneData sd = scene_data(ctx, sc, &depth);
    const RenderParams P = make_render_params(cam, w, h, acc, acc_params, shader, shader_params);
    const LeafPolicy pol = resolve(ctx->tune[BVHGPU_K_TRACE_SCENE], depth).pol;
    const unsigned tiles = (unsigned)(((w + 7) / 8) * ((h + 7) / 8));
    LaunchScope scope(ctx, BVHGPU_K_RENDER, s);
    const uint64_t px = (uint64_t)w * (uint64_t)h;
    if (px <= wide_rays(ctx, BVHGPU_K_TRACE_SCENE, sc)) {
        k_render_scene_wide<<<grid_for((uint32_t)px, kWideWarps), 32 * kWideWarps, 0, s>>>(sd, P, d_shade, sc.xf, lookup, d_rgba,
                                                                                           pol, ctx->d_err);
        g_launches++;
        return cudaGetLastError();
    }
    // the smallest local stack that holds the deepest BLAS's pending far children
    if (depth <= 33)
        k_render_scene<32><<<tiles, 64, 0, s>>>(sd, P, d_shade, sc.xf, lookup, d_rgba, pol, ctx->d_err);
    else if (depth <= 65)
        k_render_scene<64><<<tiles, 64, 0, s>>>(sd, P, d_shade, sc.xf, lookup, d_rgba, pol, ctx->d_err);
    else if (depth <= 129)
        k_render_scene<128><<<tiles, 64, 0, s>>>(sd, P, d_shade, sc.xf, lookup, d_rgba, pol, ctx->d_err);
    else
        k_render_scene<256><<<tiles, 64, 0, s>>>(sd, P, d_shade, sc.xf, lookup, d_rgba, pol, ctx->d_err);
    g_launches++;
    return cudaGetLastError();
}

cudaError_t launch_scene_bounce(bvhgpu_ctx* ctx, DeviceScene& sc, const float4* rays, uint32_t n, uint32_t seed,
                                void* hits0, void* hits1, cudaStream_t s) {
    if (n == 0) return cudaSuccess;
    uint32_t depth = 1;
    SceneData sd = scene_data(ctx, sc, &depth);
    const Variant v = resolve(ctx->tune[BVHGPU_K_SCENE_BOUNCE], depth);
    if (n <= wide_rays(ctx, BVHGPU_K_SCENE_BOUNCE, sc)) {
        unsigned long long* began;
        const cudaError_t e = launch_start(ctx, s, &began);
        if (e != cudaSuccess) return e;
        LaunchScope scope(ctx, BVHGPU_K_SCENE_BOUNCE, s);
        k_scene_bounce_wide<<<grid_for(n, kWideWarps), 32 * kWideWarps, 0, s>>>(sd, rays, n, seed, static_cast<GHit*>(hits0),
                                                                                static_cast<GHit*>(hits1), v.pol, ctx->d_err, began);
        g_launches++;
        return cudaGetLastError();
    }
    uint32_t* queue = ctx->d_scratch + 4;
    cudaError_t e = cudaMemsetAsync(queue, 0, sizeof(uint32_t), s);
    if (e != cudaSuccess) return e;
    LaunchScope scope(ctx, BVHGPU_K_SCENE_BOUNCE, s);
    e = with_variant(v.shape, v.stack, [&](auto sh, auto tg) {
        using SH = decltype(sh);
        using STK = typename decltype(tg)::type;
        auto* k = k_scene_persistent_bounce<SH::block, SH::minb, STK>;
        const size_t smem = stack_smem_bytes<STK>(SH::block);
        int per_sm = 0;
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k, SH::block, smem);
        k<<<std::max(1, per_sm) * ctx->num_sms, SH::block, smem, s>>>(sd, rays, n, seed, static_cast<GHit*>(hits0),
                                                                     static_cast<GHit*>(hits1), queue, v.pol,
                                                                     v.refill, ctx->d_err);
        return cudaGetLastError();
    });
    g_launches++;
    return e;
}

cudaError_t launch_scene_bounce_rays(bvhgpu_ctx* ctx, DeviceScene& sc, const float4* rays, const void* hits0,
                                     uint32_t n, uint32_t seed, float4* out, uint8_t* valid, cudaStream_t s) {
    if (n == 0) return cudaSuccess;
    uint32_t depth = 1;
    SceneData sd = scene_data(ctx, sc, &depth);
    LaunchScope scope(ctx, BVHGPU_K_OTHER, s);
    k_scene_bounce_rays<<<grid_for(n, kBlock), kBlock, 0, s>>>(sd, rays, static_cast<const GHit*>(hits0), n, seed,
                                                               out, valid);
    g_launches++;
    return cudaGetLastError();
}

cudaError_t launch_wobble(bvhgpu_ctx* ctx, float* verts, const float* dirs, const float* r0, const float* phase,
                          uint32_t nv, float amp, float freq, const float* time, cudaStream_t s) {
    LaunchScope scope(ctx, BVHGPU_K_OTHER, s);
    k_wobble<<<grid_for(nv, 256), 256, 0, s>>>(verts, dirs, r0, phase, nv, amp, freq, time);
    g_launches++;
    return cudaGetLastError();
}

cudaError_t launch_animate_instances(bvhgpu_ctx* ctx, DeviceScene& sc, const float* rot0, const float* axis,
                                     const float* omega, const float* scale, const float* trans, const float* time,
                                     cudaStream_t s) {
    LaunchScope scope(ctx, BVHGPU_K_OTHER, s);
    k_animate_instances<<<grid_for(sc.nobjects, 128), 128, 0, s>>>(sc.xf, sc.inv, rot0, axis, omega, scale, trans,
                                                                   sc.nobjects, time);
    g_launches++;
    return cudaGetLastError();
}

cudaError_t launch_advance_time(bvhgpu_ctx* ctx, float* time, float dt, cudaStream_t s) {
    LaunchScope scope(ctx, BVHGPU_K_OTHER, s);
    k_advance_time<<<1, 1, 0, s>>>(time, dt);
    g_launches++;
    return cudaGetLastError();
}

}  // namespace bvhgpu
