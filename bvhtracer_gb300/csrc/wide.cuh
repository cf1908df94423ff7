// Traversal with one warp per ray.
//
// For launches of few rays (wide_rays): one thread per ray leaves most of the GPU idle and its time
// is one lane's walk, so here a warp takes one ray.  Every lane follows the same reference nodes in
// the reference's order; a leaf is tested by all lanes at once, small leaves (or leaves whose margins
// are too wide) in order as in coop_leaf, large ones through their hidden tree: up to 8 nodes' children
// are tested per iteration, one box per lane, and the live leaves' pairs one per lane.  Any order
// of testing inside a leaf is exact (smallest t, ties to the lowest index; a hit from an earlier leaf
// keeps equal t out).  What bounds it: the latency of the dependent node loads of one ray.
#pragma once

#include <cuda_runtime.h>

#include <algorithm>

#include "common.cuh"
#include "internal.hpp"

namespace bvhgpu {

constexpr unsigned kWarp = 0xFFFFFFFFu;
constexpr uint32_t kWideStack = 256;    // pending reference nodes, as the largest stack variant
constexpr uint32_t kWideTlas = 64;      // pending TLAS nodes, as the one-thread kernels
constexpr uint32_t kWideNodes = 224;    // pending hidden nodes; fuller: the leaf is tested in order
constexpr uint32_t kWideLeaves = 96;    // live hidden leaves waiting to be tested
constexpr uint32_t kLeafPairs = kHiddenLeafTris / 2u;    // pairs of a hidden leaf, at most
constexpr uint32_t kLeavesPerRound = 32u / kLeafPairs;  // hidden leaves tested at once, one pair per lane
constexpr int kWideWarps = 2;           // warps (rays) per block
// Leaves of at most this many triangles are tested in order (8 rounds of 64).  4,000 camera rays
// against a 4,096-triangle soup / a 20,480-triangle sphere: 13 / 15 us at 256, 512 and 1,024, 19 / 15
// at 32, 13 / 27 at 1,500.
constexpr uint32_t kWideInOrder = 512;

struct WideSmem {  // one per warp
    uint2 stack[kWideStack];
    uint2 nodes[kWideNodes];
    uint2 leaves[kWideLeaves];
};

// The warp's best hit of the leaf in every lane (smallest t, ties to the lowest index).
__device__ __forceinline__ void wide_reduce(Best& b) {
    // accepted t are positive, so their bits order as the values do; a lane without a hit holds the
    // incoming t with index ~0
    const uint32_t t = __reduce_min_sync(kWarp, b.k == kMiss ? 0x7F800000u : __float_as_uint(b.t));
    if (t == 0x7F800000u) return;
    b.k = __reduce_min_sync(kWarp, (b.k != kMiss && __float_as_uint(b.t) == t) ? b.k : kMiss);
    b.t = __uint_as_float(t);
}

// Tests the leaf [first, first + cnt) in index order, pairs dealt over the lanes.
__device__ __forceinline__ void wide_in_order(const GBlas& g, uint32_t first, uint32_t cnt, const LaneRay& r, Best& b) {
    const unsigned lane = threadIdx.x & 31u;
    const f2 OX = f2_pack(r.o.x, r.o.x), OY = f2_pack(r.o.y, r.o.y), OZ = f2_pack(r.o.z, r.o.z);
    const f2 DX = f2_pack(r.d.x, r.d.x), DY = f2_pack(r.d.y, r.d.y), DZ = f2_pack(r.d.z, r.d.z);
    const f2 Z = f2_neg_zero();
    const uint32_t end = first + cnt;
    for (uint32_t p = (first >> 1) + lane; p < (end + 1u) >> 1; p += 32u) {
        const uint32_t kA = 2u * p;
        const PairData pd = load_pair(g.pairs + 5ull * p);
        b.take(ray_terms(pd, origin_terms(pd, OX, OY, OZ, Z), DX, DY, DZ, Z, kA >= first, kA + 1u < end), kA);
    }
}

// Walks the hidden tree `root` under margins lc.  False: the node list overflowed (test in order).
__device__ __forceinline__ bool wide_hidden(const GBlas& g, uint2 root, LeafCull& lc, const LaneRay& r, Best& b,
                                            WideSmem& sm) {
    const unsigned lane = threadIdx.x & 31u;
    const unsigned below = (1u << lane) - 1u;
    const f2 OX = f2_pack(r.o.x, r.o.x), OY = f2_pack(r.o.y, r.o.y), OZ = f2_pack(r.o.z, r.o.z);
    const f2 DX = f2_pack(r.d.x, r.d.x), DY = f2_pack(r.d.y, r.d.y), DZ = f2_pack(r.d.z, r.d.z);
    const f2 Z = f2_neg_zero();
    uint32_t nn = 1u, nl = 0u;
    if (lane == 0u) sm.nodes[0] = make_uint2(root.y, root.x);  // (count, first)
    __syncwarp();
    while (nn | nl) {
        if (nn && nl + 32u <= kWideLeaves) {
            // the children of the newest up to 8 nodes, one box per lane
            const uint32_t take = min(nn, 8u);
            nn -= take;
            const uint32_t slot = lane >> 2, c = lane & 3u;
            bool live = false;
            uint2 e = make_uint2(0u, 0u);
            if (slot < take) {
                const uint2 nd = sm.nodes[nn + slot];
                if (c <= ((nd.x >> kWideShift) & 3u)) {
                    const float4* N = g.nodes + 2ull * (nd.y + c);
                    const float4 lo = __ldg(N), hi = __ldg(N + 1);
                    float te;
                    live = hidden_box(lo, hi, r.rd, lc, te);
                    e = make_uint2(ubits(hi.w), ubits(lo.w));
                }
            }
            const bool leaf = (e.x & kHiddenLeaf) != 0u;
            const unsigned ml = __ballot_sync(kWarp, live && leaf), mn = __ballot_sync(kWarp, live && !leaf);
            if (nn + (uint32_t)__popc(mn) > kWideNodes) return false;
            __syncwarp();  // the entries taken above have been read
            if (live && leaf) sm.leaves[nl + __popc(ml & below)] = e;
            if (live && !leaf) sm.nodes[nn + __popc(mn & below)] = e;
            nl += (uint32_t)__popc(ml);
            nn += (uint32_t)__popc(mn);
            __syncwarp();
            if (nn && nl < kLeavesPerRound) continue;
        }
        // the newest live leaves, one pair per lane
        const uint32_t take = min(nl, kLeavesPerRound);
        if (take == 0u) continue;
        nl -= take;
        const uint32_t slot = lane / kLeafPairs, q = lane % kLeafPairs;
        if (slot < take) {
            const uint2 e = sm.leaves[nl + slot];
            if (q < (e.x & ~kHiddenLeaf)) {
                const uint32_t p = e.y + q;
                uint2 idx;
                const PairData pd = load_hidden_pair(g.pairs + 5ull * p, idx);
                const PairHit h = ray_terms(pd, origin_terms(pd, OX, OY, OZ, Z), DX, DY, DZ, Z, idx.x != kMiss, idx.y != kMiss);
                if (h.okA && (h.tA < b.t || (h.tA == b.t && b.k != kMiss && idx.x < b.k))) {
                    b.t = h.tA;
                    b.k = idx.x;
                }
                if (h.okB && (h.tB < b.t || (h.tB == b.t && b.k != kMiss && idx.y < b.k))) {
                    b.t = h.tB;
                    b.k = idx.y;
                }
            }
        }
        __syncwarp();
        wide_reduce(b);
        lc.thi = leaf_thi(lc, b.t);
    }
    return true;
}

// The closest hit of one ray in BLAS g by the whole warp: every lane holds the same r and ends with the
// same.  False: stopped (an error flag or the deadline), r incomplete.
__device__ __forceinline__ bool wide_blas(const GBlas& g, LaneRay& r, LeafPolicy pol, WideSmem& sm, const Deadline& deadline,
                                          uint32_t* err) {
    const unsigned lane = threadIdx.x & 31u;
    uint32_t cnt = g.root_count, first = g.root_first, sp = 0u, steps = 0u;
    const uint32_t max_steps = 2u * (g.nodes_used + g.ntris) + 16u;
    for (;;) {
        if (++steps > max_steps) {
            if (lane == 0u) atomicOr(err, kErrSteps);
            return false;
        }
        if (deadline.expired(err)) return false;
        bool pop = true;
        if (cnt == 0u) {
            const float4* N = g.nodes + 2ull * first;
            const float4 l0 = __ldg(N), l1 = __ldg(N + 1), r0 = __ldg(N + 2), r1 = __ldg(N + 3);
            float dl, dr;
            const bool hl = slab(l0, l1, r.o, r.rd, r.ct, dl), hr = slab(r0, r1, r.o, r.rd, r.ct, dr);
            const bool left_near = (hl ? dl : FLT_MAX) < (hr ? dr : FLT_MAX);
            if (left_near ? hl : hr) {
                if (left_near ? hr : hl) {
                    if (sp >= kWideStack) {
                        if (lane == 0u) atomicOr(err, kErrStack);
                        return false;
                    }
                    if (lane == 0u)
                        sm.stack[sp] = left_near ? make_uint2(ubits(r1.w), ubits(r0.w)) : make_uint2(ubits(l1.w), ubits(l0.w));
                    ++sp;
                    __syncwarp();
                }
                cnt = left_near ? ubits(l1.w) : ubits(r1.w);
                first = left_near ? ubits(l0.w) : ubits(r0.w);
                pop = false;
            }
        } else {
            Best b{r.ct, kMiss};
            bool done = false;
            if (cnt > kWideInOrder && g.hx != nullptr && pol.max_duv > 0.0f) {
                const uint2 e = __ldg(g.hx + first);
                if (e.x != 0u) {
                    const float4 a = __ldg(g.cones + 2ull * (e.y & kConeMask)), q = __ldg(g.cones + 2ull * (e.y & kConeMask) + 1);
                    const LeafCone cone = {a.x, a.y, a.z, a.w, q.x, q.y};
                    LeafCull lc = leaf_cull(cull_ray_rd(r.o.x, r.o.y, r.o.z, r.d.x, r.d.y, r.d.z, r.rd.x, r.rd.y, r.rd.z),
                                            q.z, q.w, r.ct, pol.max_duv, cone);
                    if (lc.on) {
                        done = wide_hidden(g, e, lc, r, b, sm);
                        if (!done) b = Best{r.ct, kMiss};
                        __syncwarp();
                    }
                }
            }
            if (!done) wide_in_order(g, first, cnt, r, b);
            wide_reduce(b);
            if (b.k != kMiss) {
                const float4* T = g.tris + 3ull * b.k;
                float t, u, v;
                tri_test(__ldg(T), __ldg(T + 1), __ldg(T + 2), r.o, r.d, t, u, v);  // the winner's u, v
                r.ct = b.t;
                r.hu = u;
                r.hv = v;
                r.hp = b.k;
                r.hit = true;
                r.inst = r.inst_cur;
            }
        }
        if (pop) {
            if (sp == 0u) return true;
            const uint2 e = sm.stack[--sp];
            cnt = e.x;
            first = e.y;
            __syncwarp();
        }
    }
}

// Launches of at most this many rays run one warp per ray (under the kernel's default launch config
// only: a config set by the caller or the tuner names the one-thread kernels' variants).  A one-thread
// kernel's time hardly grows until the GPU is full and starts from the scene's longest walk; the
// warp's grows with the rays.  One thread -> one warp per ray, in us, at 8,000 / 16,000 / 32,000 / 64,000 rays:
//  closest hit, sphere of 320 triangles   23 | 23 | 27 | 29 -> 16 | 25 | 50 | 86
//               soup of 300               24 | 24 | 43 | 43 -> 23 | 37 | 85 | 143
//               sphere of 5,120           58 | 72 | 72 | 74 -> 21 | 35 | 62 | 114
//               sphere of 81,920          194 | 203 | 203 | 248 -> 30 | 43 | 78 | 140
//               soup of 4,096             123 | 199 | 260 | 293 -> 24 | 39 | 81 | 134
//  bounce, 320 / 5,120 / 81,920           67 | 59 | 64 | 66 -> 27 | 42 | 75 | 134;  120 | 119 | 122 | 120 ->
//                                         35 | 56 | 100 | 181;  266 | 280 | 282 | 300 -> 49 | 75 | 134 | 237
//  margins too wide to cull, all leaves in order: 20,000-triangle soup in units of 3 edges
//                                         214 | 217 | 262 | 294 -> 44 | 69 | 122; sphere of 81,920, radius 100, 597 | 690 | 743 |
//                                         952 -> 107 | 168 | 294 | 532
//  Lambertian forward, 1,280 / 327,680    90 | 88 | 96 | 87 -> 19 | 30 | 53 | 96;  197 | 210 | 215 | 224 -> 30 | 46 | 82 | 144
//  scene of 3 small objects               25 | 23 | 23 | 23 -> 15 | 19 | 27 | 44
//  scene of 1,000 objects                 236 | 257 | 277 | 312 -> 47 | 72 | 126 | 226
//  scene bounce, 1,000 objects            541 | 548 | 574 | 636 -> 86 | 125 | 217 | 399
//  scene of 1,000 objects of 80 triangles 104 | 104 | 109 | 123 -> 52 | 87 | 142 | 259
//  its bounce                             282 | 295 | 303 | 314 -> 87 | 140 | 242 | 444
// `small`: the line for fewer than 4,096 triangles (all objects' together); 8,192 where a ray's work is
// one closest hit in one small mesh.
inline uint32_t wide_rays(const bvhgpu_ctx* ctx, int kernel, uint64_t ntris, uint32_t small = 16384u) {
    if (!default_tune(ctx->tune[kernel], kernel)) return 0u;
    return ntris < 4096u ? small : ntris < 65536u ? 32768u : 65536u;
}

// The word in which a warp-per-ray launch keeps its start (Deadline::start), zeroed on the stream, or null where
// no deadline can apply: none set, and no capture whose replays may come under one.
inline cudaError_t launch_start(bvhgpu_ctx* ctx, cudaStream_t s, unsigned long long** first) {
    *first = nullptr;
    cudaStreamCaptureStatus capture = cudaStreamCaptureStatusNone;
    cudaError_t e = cudaStreamIsCapturing(s, &capture);
    if (e != cudaSuccess || (ctx->deadline_ns == 0u && capture == cudaStreamCaptureStatusNone)) return e;
    *first = reinterpret_cast<unsigned long long*>(ctx->d_scratch + 12);
    return cudaMemsetAsync(*first, 0, sizeof(**first), s);
}

// The line of a scene.  Where many objects are tiny a ray's walk is mostly TLAS, which the warp follows no
// faster than a thread: the line stays at 16,384, with a bounce at 32,768.
inline uint32_t wide_rays(const bvhgpu_ctx* ctx, int kernel, const DeviceScene& sc) {
    const uint32_t n = wide_rays(ctx, kernel, sc.instanced_tris);
    if (sc.nobjects < 128u || sc.instanced_tris >= 200ull * sc.nobjects) return n;
    return std::min(n, kernel == BVHGPU_K_SCENE_BOUNCE ? 32768u : 16384u);
}

}  // namespace bvhgpu
