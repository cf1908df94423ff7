// Plans the hidden trees of a BLAS on the device (no reference counterpart).
//
// Every reference leaf with at least kHiddenMinLeaf triangles gets a tree over its triangles: a range
// of triangles is split by binned SAH (16 bins of the centroids along the widest centroid axis, cost =
// area x count of each side), in halves by order when the centroids coincide or below 32 binary
// levels, down to at most kHiddenLeafTris triangles; two levels of splits make one 4-wide node.
//
// The trees grow level by level, one block per 4-wide node: k_plan_split splits its range and both
// halves (centroid bounds, bins and a stable partition, each a pass of the block over the range),
// k_plan_scan numbers the children and writes them, or in a level of many nodes k_plan_emit, and queues
// those to be split.  Node order and tree shape depend on the triangles only.  The leaves' packed pairs
// are numbered at the end by a prefix sum over the triangle positions.  Boxes and cones come from the refresh (k_hidden_refresh).
//
// What bounds it: one block's passes over the largest range, then the launches of the levels (about
// log4(largest leaf / 8)).  The same planning on one host core made a model of 81,920 triangles take
// 28.1 ms to upload, now 0.96 ms; 20,480 triangles 7.0 -> 0.73 ms; 1,280 triangles 0.49 -> 0.18 ms.
#include <cuda_runtime.h>

#include <algorithm>
#include <cfloat>
#include <vector>

#include "common.cuh"
#include "internal.hpp"

namespace bvhgpu {
namespace {

constexpr int kBins = 16;
constexpr int kPlanThreads = 512;
constexpr uint32_t kSahLevels = 16;  // 4-wide levels split by SAH; deeper ones in halves
constexpr uint32_t kPlanSmall = 2048;  // triangles of a model whose levels are queued ahead

struct PlanNode {
    uint32_t a, b;  // range of triangle positions
    uint32_t me;    // hidden node (counted from the first), kNoRefresh for a root
    uint32_t cone;
};

struct PlanCounters {
    uint32_t nhid, nnext, ncones, largest;  // hidden nodes so far, next level's nodes, cones, its largest range
    uint32_t nhp;                           // hidden pairs
    uint32_t decide;                        // the first refresh's word (launch_hidden_refresh)
    uint32_t levels;                        // levels split so far
};

__device__ __forceinline__ uint32_t rank_of(float f) {  // order-preserving
    const uint32_t b = __float_as_uint(f);
    return (b & 0x80000000u) ? ~b : (b | 0x80000000u);
}
__device__ __forceinline__ float unrank(uint32_t r) {
    return __uint_as_float((r & 0x80000000u) ? (r & 0x7FFFFFFFu) : ~r);
}
__device__ __forceinline__ float half_area(const float* lo, const float* hi) {
    const float e0 = hi[0] - lo[0], e1 = hi[1] - lo[1], e2 = hi[2] - lo[2];
    return e0 * e1 + e1 * e2 + e2 * e0;
}
__device__ __forceinline__ int bin_of(float c, float lo, float ext) {
    const float x = (c - lo) / ext * (float)kBins;
    return x >= 0.0f ? min(kBins - 1, (int)x) : 0;  // NaN -> 0
}

__global__ void k_plan_info(const float* __restrict__ tris, uint32_t n, float4* __restrict__ cen, float4* __restrict__ lo,
                            float4* __restrict__ hi, uint32_t* __restrict__ ids, uint32_t* __restrict__ np_at) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float* v = tris + 9ull * i;
    float c[3], l[3], h[3];
    for (int k = 0; k < 3; ++k) {
        c[k] = (v[k] + v[3 + k] + v[6 + k]) / 3.0f;
        l[k] = fminf(v[k], fminf(v[3 + k], v[6 + k]));
        h[k] = fmaxf(v[k], fmaxf(v[3 + k], v[6 + k]));
    }
    cen[i] = make_float4(c[0], c[1], c[2], 0.0f);
    lo[i] = make_float4(l[0], l[1], l[2], 0.0f);
    hi[i] = make_float4(h[0], h[1], h[2], 0.0f);
    ids[i] = i;
    np_at[i] = 0u;
}

struct PlanSmem {
    uint32_t cl[3], ch[3];               // centroid bounds (ranks)
    uint32_t cnt[kBins];
    uint32_t blo[kBins][3], bhi[kBins][3];  // bin boxes (ranks)
    uint32_t warp_left[kPlanThreads / 32];
    int axis, best;
    float lo, ext;
    uint32_t nl;
};

// Splits in[x, y) into out[x, y), both parts non-empty; returns the split position (every thread).
// (in and out swap roles within the kernel: no read-only loads.)
__device__ uint32_t block_split(const uint32_t* in, uint32_t* out, uint32_t x, uint32_t y,
                                bool sah, const float4* __restrict__ cen, const float4* __restrict__ lo,
                                const float4* __restrict__ hi, PlanSmem& sm) {
    const uint32_t tid = threadIdx.x, nt = blockDim.x;
    const uint32_t mid = x + (y - x) / 2u;
    __syncthreads();  // the shared state of an earlier split has been read
    if (tid < 3) {
        sm.cl[tid] = 0xFFFFFFFFu;
        sm.ch[tid] = 0u;
    }
    for (uint32_t k = tid; k < kBins * 3; k += nt) {
        (&sm.blo[0][0])[k] = rank_of(FLT_MAX);
        (&sm.bhi[0][0])[k] = rank_of(-FLT_MAX);
    }
    if (tid < kBins) sm.cnt[tid] = 0u;
    if (tid == 0) sm.best = -1;
    __syncthreads();
    if (sah) {
        float l[3] = {FLT_MAX, FLT_MAX, FLT_MAX}, h[3] = {-FLT_MAX, -FLT_MAX, -FLT_MAX};
        for (uint32_t j = x + tid; j < y; j += nt) {
            const float4 c = cen[in[j]];
            l[0] = fminf(l[0], c.x);
            l[1] = fminf(l[1], c.y);
            l[2] = fminf(l[2], c.z);
            h[0] = fmaxf(h[0], c.x);
            h[1] = fmaxf(h[1], c.y);
            h[2] = fmaxf(h[2], c.z);
        }
        for (int k = 0; k < 3; ++k) {
            const uint32_t a = __reduce_min_sync(0xFFFFFFFFu, rank_of(l[k])), b = __reduce_max_sync(0xFFFFFFFFu, rank_of(h[k]));
            if ((tid & 31u) == 0u) {
                atomicMin(&sm.cl[k], a);
                atomicMax(&sm.ch[k], b);
            }
        }
        __syncthreads();
        if (tid == 0) {
            float ext[3];
            for (int k = 0; k < 3; ++k) ext[k] = unrank(sm.ch[k]) - unrank(sm.cl[k]);
            int ax = 0;
            for (int k = 1; k < 3; ++k)
                if (ext[k] > ext[ax]) ax = k;
            sm.axis = ax;
            sm.lo = unrank(sm.cl[ax]);
            sm.ext = ext[ax];
        }
        __syncthreads();
    }
    const int ax = sah ? sm.axis : 0;
    const float clo = sah ? sm.lo : 0.0f, ext = sah ? sm.ext : 0.0f;
    if (sah && ext > 0.0f && ext < FLT_MAX) {
        for (uint32_t j = x + tid; j < y; j += nt) {
            const uint32_t id = in[j];
            const float4 c = cen[id], l = lo[id], h = hi[id];
            const int b = bin_of(ax == 0 ? c.x : ax == 1 ? c.y : c.z, clo, ext);
            atomicAdd(&sm.cnt[b], 1u);
            atomicMin(&sm.blo[b][0], rank_of(l.x));
            atomicMin(&sm.blo[b][1], rank_of(l.y));
            atomicMin(&sm.blo[b][2], rank_of(l.z));
            atomicMax(&sm.bhi[b][0], rank_of(h.x));
            atomicMax(&sm.bhi[b][1], rank_of(h.y));
            atomicMax(&sm.bhi[b][2], rank_of(h.z));
        }
        __syncthreads();
        if (tid < 32) {
            // lane i: the plane after bin i (left = bins 0..i, right = the rest)
            const int i = (int)tid;
            float cost = FLT_MAX;
            uint32_t ln = 0;
            if (i < kBins - 1) {
                float llo[3] = {FLT_MAX, FLT_MAX, FLT_MAX}, lhi[3] = {-FLT_MAX, -FLT_MAX, -FLT_MAX};
                float rlo[3] = {FLT_MAX, FLT_MAX, FLT_MAX}, rhi[3] = {-FLT_MAX, -FLT_MAX, -FLT_MAX};
                uint32_t rn = 0;
                for (int q = 0; q < kBins; ++q) {
                    const bool left = q <= i;
                    if (left) ln += sm.cnt[q]; else rn += sm.cnt[q];
                    for (int k = 0; k < 3; ++k) {
                        const float a = unrank(sm.blo[q][k]), b = unrank(sm.bhi[q][k]);
                        if (left) {
                            llo[k] = fminf(llo[k], a);
                            lhi[k] = fmaxf(lhi[k], b);
                        } else {
                            rlo[k] = fminf(rlo[k], a);
                            rhi[k] = fmaxf(rhi[k], b);
                        }
                    }
                }
                if (ln != 0u && rn != 0u) cost = half_area(llo, lhi) * (float)ln + half_area(rlo, rhi) * (float)rn;
                if (!(cost < FLT_MAX)) cost = FLT_MAX;
            }
            // the first plane of the smallest cost
            float best = cost;
            int bi = i;
            for (int off = 16; off > 0; off >>= 1) {
                const float oc = __shfl_xor_sync(0xFFFFFFFFu, best, off);
                const int oi = __shfl_xor_sync(0xFFFFFFFFu, bi, off);
                if (oc < best || (oc == best && oi < bi)) {
                    best = oc;
                    bi = oi;
                }
            }
            if (i == bi && best < FLT_MAX) {
                sm.best = bi;
                sm.nl = ln;
            }
        }
        __syncthreads();
    }
    const int best = sm.best;
    if (best < 0) {
        for (uint32_t j = x + tid; j < y; j += nt) out[j] = in[j];
        __syncthreads();
        return mid;
    }
    // stable partition, blockDim triangles at a time
    const uint32_t nl = sm.nl, warps = nt / 32u, w = tid >> 5, lane = tid & 31u;
    uint32_t left_base = x, right_base = x + nl;
    for (uint32_t j0 = x; j0 < y; j0 += nt) {
        const uint32_t j = j0 + tid;
        const bool in_range = j < y;
        uint32_t id = 0u;
        bool left = false;
        if (in_range) {
            id = in[j];
            const float4 c = cen[id];
            left = bin_of(ax == 0 ? c.x : ax == 1 ? c.y : c.z, clo, ext) <= best;
        }
        const unsigned ml = __ballot_sync(0xFFFFFFFFu, left);
        __syncthreads();  // warp_left of the previous chunk has been read
        if (lane == 0u) sm.warp_left[w] = (uint32_t)__popc(ml);
        __syncthreads();
        uint32_t before = 0u, total = 0u;
        for (uint32_t q = 0; q < warps; ++q) {
            const uint32_t v = sm.warp_left[q];
            if (q < w) before += v;
            total += v;
        }
        const uint32_t lrank = before + (uint32_t)__popc(ml & ((1u << lane) - 1u));
        if (in_range) out[left ? left_base + lrank : right_base + (tid - lrank)] = id;
        left_base += total;
        right_base += min(nt, y - j0) - total;
    }
    __syncthreads();
    return x + nl;
}

// One block per node: its 2 to 4 ranges, res = {end of range 0, of range 1, of range 2, ranges}.
__global__ void k_plan_split(const PlanNode* __restrict__ cur, uint32_t* ids, uint32_t* tmp, const float4* __restrict__ cen,
                             const float4* __restrict__ lo, const float4* __restrict__ hi, int sah, uint4* __restrict__ res,
                             const PlanCounters* __restrict__ ctr) {
    __shared__ PlanSmem sm;
    if (blockIdx.x >= ctr->nnext) return;
    const PlanNode nd = cur[blockIdx.x];
    const uint32_t m = block_split(ids, tmp, nd.a, nd.b, sah != 0, cen, lo, hi, sm);
    uint32_t r[4], k = 0u;
    auto half = [&](uint32_t x, uint32_t y) {
        if (y - x > kHiddenLeafTris) {
            r[k++] = block_split(tmp, ids, x, y, sah != 0, cen, lo, hi, sm);
        } else {
            for (uint32_t j = x + threadIdx.x; j < y; j += blockDim.x) ids[j] = tmp[j];
        }
        r[k++] = y;
    };
    half(nd.a, m);
    half(m, nd.b);
    if (threadIdx.x == 0) res[blockIdx.x] = make_uint4(r[0], k > 2 ? r[1] : nd.b, k > 3 ? r[2] : nd.b, k);
}

__device__ __forceinline__ void plan_ranges(const PlanNode& nd, uint4 s, uint32_t* r) {
    r[0] = nd.a;
    r[1] = s.x;
    r[2] = s.y;
    r[3] = s.z;
    r[s.w] = nd.b;
}

struct PlanOut {  // where a level's nodes go
    uint32_t nodes_used;
    PlanNode* next;
    uint2 *meta, *range;
    uint4* up;
    uint32_t* np_at;
    uint2* table;
};

// Node nd of a level that has nhid0 hidden nodes and ncones0 cones before it, o = {children, children to be
// split} of the level's nodes before nd: its own record (or table entry), its children's links, the next
// level's queue.
__device__ __forceinline__ void plan_emit(const PlanNode& nd, uint4 s, uint2 o, uint32_t nhid0, uint32_t ncones0, const PlanOut& out) {
    uint32_t r[5];
    plan_ranges(nd, s, r);
    const uint32_t li = nhid0 + o.x, k = s.w;
    const uint2 own = make_uint2(out.nodes_used + li, kHiddenInterior | ((k - 1u) << kWideShift) | nd.cone);
    if (nd.me == kNoRefresh)
        out.table[nd.a] = own;
    else
        out.meta[nd.me] = own;
    uint32_t q = o.y;
    for (uint32_t c = 0; c < k; ++c) {
        const uint32_t x = r[c], y = r[c + 1];
        out.up[li + c] = make_uint4(li, k, nd.me, nd.cone);
        if (y - x > kHiddenLeafTris) {
            out.next[q] = PlanNode{x, y, li + c, ncones0 + q};
            out.range[li + c] = make_uint2(0u, 0u);
            ++q;
        } else {
            out.range[li + c] = make_uint2(x, y);
            out.np_at[x] = (y - x + 1u) / 2u;
        }
    }
}

// One block numbers a level's children and moves the counters on.  EMIT: and writes its nodes; else
// off[i] = {children, children to be split} before node i.
template <bool EMIT>
__global__ void __launch_bounds__(1024) k_plan_scan(const PlanNode* __restrict__ cur, const uint4* __restrict__ res,
                                                    uint2* __restrict__ off, PlanOut out, PlanCounters* ctr) {
    __shared__ uint32_t wk[32], wi[32];
    const uint32_t n = ctr->nnext, nhid0 = ctr->nhid, ncones0 = ctr->ncones;
    if (n == 0u) return;
    const uint32_t tid = threadIdx.x, lane = tid & 31u, w = tid >> 5;
    uint32_t base_k = 0u, base_i = 0u, largest = 0u;
    for (uint32_t j0 = 0; j0 < n; j0 += 1024u) {
        const uint32_t j = j0 + tid;
        uint32_t k = 0u, in = 0u;
        PlanNode nd;
        uint4 s;
        if (j < n) {
            nd = cur[j];
            s = res[j];
            uint32_t r[5];
            plan_ranges(nd, s, r);
            k = s.w;
            for (uint32_t c = 0; c < k; ++c) {
                const uint32_t len = r[c + 1] - r[c];
                if (len > kHiddenLeafTris) {
                    ++in;
                    largest = max(largest, len);
                }
            }
        }
        uint32_t sk = k, si = in;  // inclusive prefix in the warp
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t a = __shfl_up_sync(0xFFFFFFFFu, sk, o), b = __shfl_up_sync(0xFFFFFFFFu, si, o);
            if (lane >= (uint32_t)o) {
                sk += a;
                si += b;
            }
        }
        __syncthreads();
        if (lane == 31u) {
            wk[w] = sk;
            wi[w] = si;
        }
        __syncthreads();
        uint32_t bk = 0u, bi = 0u, tk = 0u, ti = 0u;
        for (uint32_t q = 0; q < 32u; ++q) {
            if (q < w) {
                bk += wk[q];
                bi += wi[q];
            }
            tk += wk[q];
            ti += wi[q];
        }
        if (j < n) {
            const uint2 o = make_uint2(base_k + bk + sk - k, base_i + bi + si - in);
            if (EMIT)
                plan_emit(nd, s, o, nhid0, ncones0, out);
            else
                off[j] = o;
        }
        base_k += tk;
        base_i += ti;
    }
    largest = __reduce_max_sync(0xFFFFFFFFu, largest);
    __syncthreads();
    if (lane == 0u) wk[w] = largest;
    __syncthreads();
    if (tid == 0) {
        for (int q = 1; q < 32; ++q) wk[0] = max(wk[0], wk[q]);
        ctr->largest = wk[0];
        ctr->nnext = base_i;
        ctr->nhid = nhid0 + base_k;
        ctr->ncones = ncones0 + base_i;
        ctr->levels += 1u;
    }
}

// One thread per node of a level of n, after its scan.
__global__ void k_plan_emit(const PlanNode* __restrict__ cur, const uint4* __restrict__ res, uint32_t n,
                            const uint2* __restrict__ off, uint32_t nhid0, uint32_t ncones0, PlanOut out) {
    const uint32_t j = blockIdx.x * blockDim.x + threadIdx.x;
    if (j < n) plan_emit(cur[j], res[j], off[j], nhid0, ncones0, out);
}

// Exclusive prefix sum of v[0, n) into out: tiles of 1,024, then the tiles' sums.
__global__ void __launch_bounds__(1024) k_scan_tiles(const uint32_t* __restrict__ v, uint32_t n, uint32_t* __restrict__ out,
                                                     uint32_t* __restrict__ sums) {
    __shared__ uint32_t ws[32];
    const uint32_t i = blockIdx.x * 1024u + threadIdx.x, lane = threadIdx.x & 31u, w = threadIdx.x >> 5;
    const uint32_t x = i < n ? v[i] : 0u;
    uint32_t s = x;
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t a = __shfl_up_sync(0xFFFFFFFFu, s, o);
        if (lane >= (uint32_t)o) s += a;
    }
    if (lane == 31u) ws[w] = s;
    __syncthreads();
    uint32_t before = 0u;
    for (uint32_t q = 0; q < w; ++q) before += ws[q];
    if (i < n) out[i] = before + s - x;
    if (threadIdx.x == 1023u) sums[blockIdx.x] = before + s;
}
__global__ void __launch_bounds__(1024) k_scan_sums(uint32_t* __restrict__ sums, uint32_t n, PlanCounters* ctr) {
    __shared__ uint32_t ws[32];
    const uint32_t lane = threadIdx.x & 31u, w = threadIdx.x >> 5;
    uint32_t base = 0u;
    for (uint32_t j0 = 0; j0 < n; j0 += 1024u) {
        const uint32_t i = j0 + threadIdx.x;
        const uint32_t x = i < n ? sums[i] : 0u;
        uint32_t s = x;
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t a = __shfl_up_sync(0xFFFFFFFFu, s, o);
            if (lane >= (uint32_t)o) s += a;
        }
        __syncthreads();
        if (lane == 31u) ws[w] = s;
        __syncthreads();
        uint32_t before = 0u, total = 0u;
        for (uint32_t q = 0; q < 32u; ++q) {
            if (q < w) before += ws[q];
            total += ws[q];
        }
        if (i < n) sums[i] = base + before + s - x;
        base += total;
    }
    if (threadIdx.x == 0) ctr->nhp = base;
}

// One thread per table entry; per hidden node: its record (box zero until the refresh), its links and a leaf's
// pair slots; per reference leaf: its link for the roots' cones (fold_root_cones, kernels_scene.cu).
__global__ void k_plan_finish(const uint2* __restrict__ meta, const uint2* __restrict__ range, const uint4* __restrict__ up,
                              uint32_t nhid, const uint32_t* __restrict__ ids, const uint32_t* __restrict__ pair_at,
                              const uint32_t* __restrict__ sums, uint32_t p0, float4* __restrict__ nodes,
                              uint4* __restrict__ hup, uint2* __restrict__ slots, const float4* __restrict__ ref_nodes,
                              uint32_t nodes_used, const uint32_t* __restrict__ leaves, uint32_t nleaves,
                              const uint2* __restrict__ table, uint32_t table_u2, uint2* __restrict__ hx) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < table_u2) hx[i] = table[i];
    uint4* links = hup + nhid;
    if (i < nleaves) {
        const float4* N = ref_nodes + 2ull * leaves[i];
        const uint2 e = table[__float_as_uint(N[0].w)];
        links[i] = e.x ? make_uint4(e.x - nodes_used, e.y & kConeMask, __float_as_uint(N[1].w), 0u)
                       : make_uint4(kNoRefresh, 0u, 0u, 0u);
    }
    if (i >= nhid) return;
    hup[i] = up[i];
    const uint2 r = range[i];
    uint2 m = meta[i];
    if (r.x != r.y) {
        const uint32_t p = pair_at[r.x] + sums[r.x >> 10], np = (r.y - r.x + 1u) / 2u;
        m = make_uint2(p0 + p, kHiddenLeaf | np);
        for (uint32_t q = 0; q < np; ++q) {
            const uint32_t x = r.x + 2u * q;
            slots[p + q] = make_uint2(ids[x], x + 1u < r.y ? ids[x + 1u] : kMiss);
        }
    }
    nodes[2ull * i] = make_float4(0.0f, 0.0f, 0.0f, __uint_as_float(m.x));
    nodes[2ull * i + 1] = make_float4(0.0f, 0.0f, 0.0f, __uint_as_float(m.y));
}

inline unsigned grid_for(uint32_t n, int block) { return (unsigned)((n + block - 1) / block); }

}  // namespace

cudaError_t plan_hidden(bvhgpu_ctx* ctx, const bvhgpu_node* nodes, uint32_t nodes_used, const std::vector<uint32_t>& leaves,
                        const float* d_tris9, uint32_t ntris, HiddenPlan& plan, cudaStream_t s) {
    std::vector<PlanNode> roots;
    uint32_t largest = 0;
    for (uint32_t li : leaves) {
        const bvhgpu_node& n = nodes[li];
        if (n.primitive_count < kHiddenMinLeaf) continue;
        roots.push_back(PlanNode{n.left_first, n.left_first + n.primitive_count, kNoRefresh, (uint32_t)roots.size()});
        largest = std::max(largest, n.primitive_count);
    }
    plan = HiddenPlan();
    if (roots.empty()) return cudaSuccess;
    // one work area: a node has at least two children and a leaf one triangle, so there are fewer than
    // 2 ntris hidden nodes, and a level's nodes hold more than kHiddenLeafTris triangles each
    const uint32_t max_nodes = 2u * ntris, max_level = ntris / kHiddenLeafTris + 1u, tiles = grid_for(ntris, 1024);
    size_t bytes = 0;
    auto part = [&](size_t b) {
        const size_t at = bytes;
        bytes += (b + 255u) & ~(size_t)255u;
        return at;
    };
    const size_t o_cen = part(16ull * ntris), o_lo = part(16ull * ntris), o_hi = part(16ull * ntris), o_ids = part(4ull * ntris),
                 o_tmp = part(4ull * ntris), o_np = part(4ull * ntris), o_at = part(4ull * ntris), o_sums = part(4ull * tiles),
                 o_q0 = part(sizeof(PlanNode) * max_level), o_q1 = part(sizeof(PlanNode) * max_level),
                 o_res = part(16ull * max_level), o_off = part(8ull * max_level), o_meta = part(8ull * max_nodes),
                 o_range = part(8ull * max_nodes), o_ctr = part(sizeof(PlanCounters));
    plan.table_u2 = hidden_table_u2(ntris);
    const size_t o_up = part(16ull * max_nodes), o_table = part(8ull * plan.table_u2);
    cudaError_t e = cudaSuccess;
    char* W;
    if (bytes <= ctx->stage_out_bytes) {
        W = static_cast<char*>(ctx->stage_out);  // the context's own staging memory, free between calls
    } else {
        if ((e = cudaMalloc(&plan.work, bytes)) != cudaSuccess) return e;
        W = static_cast<char*>(plan.work);
    }
    auto* cen = reinterpret_cast<float4*>(W + o_cen);
    auto* lo = reinterpret_cast<float4*>(W + o_lo);
    auto* hi = reinterpret_cast<float4*>(W + o_hi);
    plan.ids = reinterpret_cast<uint32_t*>(W + o_ids);
    auto* tmp = reinterpret_cast<uint32_t*>(W + o_tmp);
    auto* np_at = reinterpret_cast<uint32_t*>(W + o_np);
    plan.pair_at = reinterpret_cast<uint32_t*>(W + o_at);
    plan.sums = reinterpret_cast<uint32_t*>(W + o_sums);
    PlanNode* q[2] = {reinterpret_cast<PlanNode*>(W + o_q0), reinterpret_cast<PlanNode*>(W + o_q1)};
    auto* res = reinterpret_cast<uint4*>(W + o_res);
    auto* off = reinterpret_cast<uint2*>(W + o_off);
    plan.meta = reinterpret_cast<uint2*>(W + o_meta);
    plan.range = reinterpret_cast<uint2*>(W + o_range);
    plan.up = reinterpret_cast<uint4*>(W + o_up);
    plan.table = reinterpret_cast<uint2*>(W + o_table);
    auto* ctr = reinterpret_cast<PlanCounters*>(W + o_ctr);
    PlanCounters h = {0u, (uint32_t)roots.size(), (uint32_t)roots.size(), largest, 0u, 0u, 0u};
    plan.decide = &ctr->decide;
    if ((e = cudaMemcpyAsync(q[0], roots.data(), sizeof(PlanNode) * roots.size(), cudaMemcpyHostToDevice, s)) != cudaSuccess ||
        (e = cudaMemcpyAsync(ctr, &h, sizeof(h), cudaMemcpyHostToDevice, s)) != cudaSuccess ||
        (e = cudaMemsetAsync(plan.table, 0, 8ull * plan.table_u2, s)) != cudaSuccess)
        return e;
    LaunchScope scope(ctx, BVHGPU_K_OTHER, s);
    k_plan_info<<<grid_for(ntris, 256), 256, 0, s>>>(d_tris9, ntris, cen, lo, hi, plan.ids, np_at);
    g_launches++;
    // Small models: the levels that a balanced tree has, and one more, are queued at once, their launches
    // sized by what a level can hold, and the pairs numbered behind them, with one wait for it all: upload of
    // one leaf of 100 triangles 230 -> 177 us (planned on the host 182), of 1,280 triangles 325 -> 230.
    const bool small = ntris <= kPlanSmall;
    uint32_t level = 0, most = h.nnext, ahead = 1;
    if (small)
        for (uint32_t reach = kHiddenLeafTris; reach < largest; reach *= 4u) ++ahead;
    while (h.nnext != 0u) {
        for (; ahead != 0u; --ahead) {
            PlanNode* cur = q[level & 1u];
            const PlanOut out = {nodes_used, q[(level & 1u) ^ 1u], plan.meta, plan.range, plan.up, np_at, plan.table};
            // small ranges: one triangle or two a thread
            const int threads = h.largest > 512u ? kPlanThreads : h.largest > 128u ? 128 : 64;
            k_plan_split<<<most, threads, 0, s>>>(cur, plan.ids, tmp, cen, lo, hi, level < kSahLevels ? 1 : 0, res, ctr);
            if (most <= 1024u) {
                k_plan_scan<true><<<1, 1024, 0, s>>>(cur, res, off, out, ctr);
                g_launches += 2;
            } else {  // most is the level's own count: only small models queue ahead
                k_plan_scan<false><<<1, 1024, 0, s>>>(cur, res, off, out, ctr);
                k_plan_emit<<<grid_for(most, 128), 128, 0, s>>>(cur, res, most, off, h.nhid, h.ncones, out);
                g_launches += 3;
            }
            most = std::min(4u * most, max_level);
            ++level;
        }
        if (small) {
            k_scan_tiles<<<tiles, 1024, 0, s>>>(np_at, ntris, plan.pair_at, plan.sums);
            k_scan_sums<<<1, 1024, 0, s>>>(plan.sums, tiles, ctr);
            g_launches += 2;
        }
        if ((e = cudaMemcpyAsync(ctx->host_word, ctr, sizeof(h), cudaMemcpyDeviceToHost, s)) != cudaSuccess ||
            (e = cudaStreamSynchronize(s)) != cudaSuccess)
            return e;
        h = *static_cast<const PlanCounters*>(ctx->host_word);
        most = h.nnext;
        ahead = 1;
    }
    if (!small) {
        k_scan_tiles<<<tiles, 1024, 0, s>>>(np_at, ntris, plan.pair_at, plan.sums);
        k_scan_sums<<<1, 1024, 0, s>>>(plan.sums, tiles, ctr);
        g_launches += 2;
        if ((e = cudaMemcpyAsync(ctx->host_word, ctr, sizeof(h), cudaMemcpyDeviceToHost, s)) != cudaSuccess ||
            (e = cudaStreamSynchronize(s)) != cudaSuccess)
            return e;
        h = *static_cast<const PlanCounters*>(ctx->host_word);
    }
    plan.nhid = h.nhid;
    plan.nhp = h.nhp;
    plan.ncones = h.ncones;
    plan.depth = h.levels;
    return cudaGetLastError();
}

cudaError_t finish_hidden(bvhgpu_ctx* ctx, const HiddenPlan& plan, DeviceBlas& b, cudaStream_t s) {
    if (plan.nhid == 0u) return cudaSuccess;
    LaunchScope scope(ctx, BVHGPU_K_OTHER, s);
    k_plan_finish<<<grid_for(std::max({plan.nhid, b.nleaves, plan.table_u2}), 128), 128, 0, s>>>(
        plan.meta, plan.range, plan.up, plan.nhid, plan.ids, plan.pair_at, plan.sums, pairs_in_order(b.ntris),
        b.nodes + 2ull * b.nodes_used, b.hup, b.hx + plan.table_u2, b.nodes, b.nodes_used, b.leaves, b.nleaves, plan.table,
        plan.table_u2, b.hx);
    g_launches++;
    return cudaGetLastError();
}

}  // namespace bvhgpu
