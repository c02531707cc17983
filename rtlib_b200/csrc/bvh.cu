// BVH build over triangles (the binary linear hierarchy, then the eight-wide one rays walk) and
// batched hit queries (rtpg_scene_*).
//
// This is the hit-query boundary of the integrator: RTLib answers closest-hit and occlusion
// queries with OptiX (optixTrace in TraceRadiance / TraceOccluded, SimpleKernel.h:347-366,
// over a GAS built in RTLibExtOPX7TestApplication.cpp:170-198).  No OptiX SDK exists on this
// machine, so queries go to this CUDA BVH instead.
#include <cub/cub.cuh>
#include <new>
#include <type_traits>
#include <vector>

#include "common.cuh"
#include "bvh_dev.cuh"
#include "hashgrid_dev.cuh"  // morton3_63

namespace rtpg {

__device__ __forceinline__ unsigned fbits_ord(float f) {
    const unsigned u = __float_as_uint(f);
    return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
__device__ __forceinline__ float ord_fbits(unsigned u) {
    return __uint_as_float((u & 0x80000000u) ? (u & 0x7fffffffu) : ~u);
}

__global__ void k_scene_bounds(const float* __restrict__ v, const uint32_t* __restrict__ idx, uint32_t nt,
                               unsigned* __restrict__ bounds) {
    float lo[3] = {INFINITY, INFINITY, INFINITY}, hi[3] = {-INFINITY, -INFINITY, -INFINITY};
    for (uint32_t t = blockIdx.x * blockDim.x + threadIdx.x; t < nt; t += gridDim.x * blockDim.x) {
        for (int k = 0; k < 3; ++k) {
            const uint32_t vi = idx[3 * t + k];
            for (int a = 0; a < 3; ++a) {
                // bounds of the centroids are enough for the Morton grid
                const float c = v[3 * vi + a];
                lo[a] = fminf(lo[a], c);
                hi[a] = fmaxf(hi[a], c);
            }
        }
    }
    for (int a = 0; a < 3; ++a) {
        float l = lo[a], h = hi[a];
        for (int o = 16; o > 0; o >>= 1) {
            l = fminf(l, __shfl_xor_sync(0xffffffffu, l, o));
            h = fmaxf(h, __shfl_xor_sync(0xffffffffu, h, o));
        }
        if ((threadIdx.x & 31) == 0) {
            atomicMin(bounds + a, fbits_ord(l));
            atomicMax(bounds + 3 + a, fbits_ord(h));
        }
    }
}

__global__ void k_scene_morton(const float* __restrict__ v, const uint32_t* __restrict__ idx, uint32_t nt,
                               const unsigned* __restrict__ bounds, unsigned long long* __restrict__ keys,
                               uint32_t* __restrict__ vals) {
    float lo[3], ext[3];
    for (int a = 0; a < 3; ++a) {
        lo[a] = ord_fbits(bounds[a]);
        ext[a] = fmaxf(ord_fbits(bounds[3 + a]) - lo[a], 1e-30f);
    }
    for (uint32_t t = blockIdx.x * blockDim.x + threadIdx.x; t < nt; t += gridDim.x * blockDim.x) {
        uint32_t q[3];
        for (int a = 0; a < 3; ++a) {
            const float c = (v[3 * idx[3 * t] + a] + v[3 * idx[3 * t + 1] + a] + v[3 * idx[3 * t + 2] + a]) / 3.0f;
            const float f = fminf(fmaxf((c - lo[a]) / ext[a], 0.0f), 1.0f);
            q[a] = min((uint32_t)(f * 2097152.0f), 2097151u);
        }
        keys[t] = morton3_63(q[0], q[1], q[2]);
        vals[t] = t;
    }
}

__device__ __forceinline__ int bvh_delta(const unsigned long long* __restrict__ k, int n, int i, int j) {
    if (j < 0 || j >= n) return -1;
    const unsigned long long a = k[i], b = k[j];
    if (a == b) return 64 + __clz((uint32_t)i ^ (uint32_t)j);
    return __clzll(a ^ b);
}

// Karras 2012: node i covers a key range whose split is found by binary search
__global__ void k_scene_hierarchy(const unsigned long long* __restrict__ keys, int n, BvhNode* __restrict__ nodes,
                                  uint32_t* __restrict__ parent_i, uint32_t* __restrict__ parent_l) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n - 1; i += gridDim.x * blockDim.x) {
        const int d = (bvh_delta(keys, n, i, i + 1) - bvh_delta(keys, n, i, i - 1)) >= 0 ? 1 : -1;
        const int dmin = bvh_delta(keys, n, i, i - d);
        int lmax = 2;
        while (bvh_delta(keys, n, i, i + lmax * d) > dmin) lmax <<= 1;
        int l = 0;
        for (int t = lmax >> 1; t >= 1; t >>= 1)
            if (bvh_delta(keys, n, i, i + (l + t) * d) > dmin) l += t;
        const int j = i + l * d;
        const int dnode = bvh_delta(keys, n, i, j);
        int s = 0;
        for (int t = (l + 1) >> 1;; t = (t + 1) >> 1) {
            if (bvh_delta(keys, n, i, i + (s + t) * d) > dnode) s += t;
            if (t == 1) break;
        }
        const int gamma = i + s * d + min(d, 0);
        const int lo = min(i, j), hi = max(i, j);
        uint32_t c0, c1;
        if (lo == gamma) { c0 = kBvhLeafBit | (uint32_t)gamma; parent_l[gamma] = i; }
        else { c0 = (uint32_t)gamma; parent_i[gamma] = i; }
        if (hi == gamma + 1) { c1 = kBvhLeafBit | (uint32_t)(gamma + 1); parent_l[gamma + 1] = i; }
        else { c1 = (uint32_t)(gamma + 1); parent_i[gamma + 1] = i; }
        nodes[i].child[0] = c0;
        nodes[i].child[1] = c1;
        nodes[i].pad[0] = nodes[i].pad[1] = 0;
    }
}

__global__ void k_scene_leaves(const float* __restrict__ v, const uint32_t* __restrict__ idx, uint32_t nt,
                               const uint32_t* __restrict__ order, BvhTri* __restrict__ tris, uint32_t* __restrict__ prim) {
    for (uint32_t k = blockIdx.x * blockDim.x + threadIdx.x; k < nt; k += gridDim.x * blockDim.x) {
        const uint32_t p = order[k];
        const uint32_t a = idx[3 * p], b = idx[3 * p + 1], c = idx[3 * p + 2];
        float4 r[3];
        tri_transform(v[3 * a], v[3 * a + 1], v[3 * a + 2], v[3 * b], v[3 * b + 1], v[3 * b + 2], v[3 * c], v[3 * c + 1],
                      v[3 * c + 2], r);
        tris[k] = BvhTri{r[0], r[1], r[2]};
        prim[k] = p;
    }
}

// the leaves back in scene order, as pairs, for small scenes
__global__ void k_scene_flat(const BvhTri* __restrict__ tris, const uint32_t* __restrict__ prim, uint32_t nt,
                             FlatPair* __restrict__ flat) {
    auto put = [&](uint32_t i, const BvhTri& t) {
        float* const w = reinterpret_cast<float*>(flat + i / 2) + (i & 1u);
        const float4 r[3] = {t.r0, t.r1, t.r2};
        for (int a = 0; a < 3; ++a) {
            w[8 * a] = r[a].x;
            w[8 * a + 2] = r[a].y;
            w[8 * a + 4] = r[a].z;
            w[8 * a + 6] = r[a].w;
        }
    };
    for (uint32_t k = blockIdx.x * blockDim.x + threadIdx.x; k < nt; k += gridDim.x * blockDim.x) put(prim[k], tris[k]);
    // u = -1 everywhere
    if ((nt & 1u) && blockIdx.x == 0 && threadIdx.x == 0)
        put(nt, BvhTri{make_float4(0.f, 0.f, 0.f, -1.f), make_float4(0.f, 0.f, 0.f, 0.f), make_float4(1.f, 0.f, 0.f, 0.f)});
}

// the box of scene triangle p, widened by a relative margin so that it contains the triangle
// as the hit test sees it
__device__ __forceinline__ void tri_box(const float* __restrict__ v, const uint32_t* __restrict__ idx, uint32_t p,
                                        float* lo, float* hi) {
    const uint32_t a = idx[3 * p], b = idx[3 * p + 1], c = idx[3 * p + 2];
    for (int k = 0; k < 3; ++k) {
        const float x0 = v[3 * a + k], x1 = v[3 * b + k], x2 = v[3 * c + k];
        lo[k] = fminf(x0, fminf(x1, x2));
        hi[k] = fmaxf(x0, fmaxf(x1, x2));
        const float m = 1e-6f * fmaxf(fabsf(lo[k]), fabsf(hi[k])) + 1e-12f;
        lo[k] -= m;
        hi[k] += m;
    }
}

// the leaves' boxes for the walk, and their largest finite absolute coordinate (as ordered bits: a
// nonnegative float's bits order as it does)
__global__ void k_scene_leaf_boxes(const float* __restrict__ v, const uint32_t* __restrict__ idx,
                                   const uint32_t* __restrict__ prim, uint32_t nt, float4* __restrict__ box,
                                   unsigned* __restrict__ max_abs) {
    float m = 0.0f;
    for (uint32_t k = blockIdx.x * blockDim.x + threadIdx.x; k < nt; k += gridDim.x * blockDim.x) {
        float lo[3], hi[3];
        tri_box(v, idx, prim[k], lo, hi);
        box[2 * size_t(k)] = make_float4(lo[0], lo[1], lo[2], hi[0]);
        box[2 * size_t(k) + 1] = make_float4(hi[1], hi[2], 0.0f, 0.0f);
        for (int a = 0; a < 3; ++a) {
            if (isfinite(lo[a])) m = fmaxf(m, fabsf(lo[a]));
            if (isfinite(hi[a])) m = fmaxf(m, fabsf(hi[a]));
        }
    }
    for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
    if ((threadIdx.x & 31) == 0) atomicMax(max_abs, __float_as_uint(m));
}

// bottom-up boxes: the second thread to reach an interior node merges its children
__global__ void k_scene_boxes(const float* __restrict__ v, const uint32_t* __restrict__ idx,
                              const uint32_t* __restrict__ prim, uint32_t nt, BvhNode* nodes, const uint32_t* parent_i,
                              const uint32_t* parent_l, float4* ibox, unsigned* flags) {
    for (uint32_t k = blockIdx.x * blockDim.x + threadIdx.x; k < nt; k += gridDim.x * blockDim.x) {
        uint32_t node = parent_l[k];
        for (;;) {
            __threadfence();
            if (atomicAdd(flags + node, 1u) == 0) break;
            __threadfence();
            float lo[2][3], hi[2][3];
            for (int c = 0; c < 2; ++c) {
                const uint32_t ch = nodes[node].child[c];
                if (ch & kBvhLeafBit) {
                    tri_box(v, idx, prim[ch & ~kBvhLeafBit], lo[c], hi[c]);
                } else {
                    const float4 a = __ldcg(ibox + 2 * ch), b = __ldcg(ibox + 2 * ch + 1);
                    lo[c][0] = a.x; lo[c][1] = a.y; lo[c][2] = a.z;
                    hi[c][0] = b.x; hi[c][1] = b.y; hi[c][2] = b.z;
                }
            }
            nodes[node].a = make_float4(lo[0][0], lo[0][1], lo[0][2], hi[0][0]);
            nodes[node].b = make_float4(hi[0][1], hi[0][2], lo[1][0], lo[1][1]);
            nodes[node].c = make_float4(lo[1][2], hi[1][0], hi[1][1], hi[1][2]);
            __stcg(ibox + 2 * node, make_float4(fminf(lo[0][0], lo[1][0]), fminf(lo[0][1], lo[1][1]),
                                                fminf(lo[0][2], lo[1][2]), 0.0f));
            __stcg(ibox + 2 * node + 1, make_float4(fmaxf(hi[0][0], hi[1][0]), fmaxf(hi[0][1], hi[1][1]),
                                                    fmaxf(hi[0][2], hi[1][2]), 0.0f));
            if (node == 0) break;
            node = parent_i[node];
        }
    }
}

// ------------------------------------------------------------------ walked hierarchy, binary stage
// A second binary hierarchy over the same leaves by parallel locally-ordered clustering (Meister
// and Bittner, IEEE TVCG 24(3), 2018): clusters stay in Morton order, each looks kPlocRadius
// neighbours to either side for the one whose common box has the least surface area, and pairs that
// chose each other merge.  The linear hierarchy puts a large triangle (a wall) among the small ones
// around its centroid and so inflates every box above it; here it waits until large clusters are
// left and ends up near the root.  Equal areas are told apart by the smaller i ^ j, which is symmetric
// and distinct for a cluster's candidates, so the least pair always merges.
// Boxes that contain one another in order merge one pair a round: each one's best partner is a
// smaller one.  Clusters that are left after kPlocRounds rounds pair with their neighbour in order
// (i with i ^ 1, which halves them each round).  The 1.05 M-triangle rooms take 74 rounds, soups of random
// triangles 49 for 200,000.
constexpr int kPlocRadius = 16;
constexpr int kPlocBlock = 256;
constexpr uint32_t kPlocRounds = 88;  // a round adds at most one level (see k_wide_level)

__device__ __forceinline__ float box_area(float4 alo, float4 ahi, float4 blo, float4 bhi) {
    const float x = fmaxf(ahi.x, bhi.x) - fminf(alo.x, blo.x), y = fmaxf(ahi.y, bhi.y) - fminf(alo.y, blo.y),
                z = fmaxf(ahi.z, bhi.z) - fminf(alo.z, blo.z);
    return x * y + y * z + z * x;
}
// a cluster: lo.xyz and its reference (kBvhLeafBit | leaf or node), hi.xyz
__global__ void k_ploc_init(const float4* __restrict__ leaf_box, uint32_t n, float4* __restrict__ lo, float4* __restrict__ hi) {
    for (uint32_t k = blockIdx.x * blockDim.x + threadIdx.x; k < n; k += gridDim.x * blockDim.x) {
        const float4 a = leaf_box[2 * size_t(k)], b = leaf_box[2 * size_t(k) + 1];
        lo[k] = make_float4(a.x, a.y, a.z, __uint_as_float(kBvhLeafBit | k));
        hi[k] = make_float4(a.w, b.x, b.y, 0.0f);
    }
}
// The partner of cluster i of n: lo, hi point at it among its neighbours.
__device__ __forceinline__ uint32_t ploc_partner(const float4* lo, const float4* hi, uint32_t i, uint32_t n, int radius) {
    const float4 mlo = *lo, mhi = *hi;
    float best = INFINITY;
    uint32_t arg = i ^ 1u;
    if (arg >= n) arg = i - 1;
    for (int d = -radius; d <= radius; ++d) {
        const int j = (int)i + d;
        if (d == 0 || j < 0 || j >= (int)n) continue;
        const float a = box_area(mlo, mhi, lo[d], hi[d]);
        if (a < best || (a == best && ((uint32_t)j ^ i) < (arg ^ i))) {
            best = a;
            arg = (uint32_t)j;
        }
    }
    return arg;
}
// clusters a and b become a node (a: the merged cluster)
__device__ __forceinline__ void ploc_merge(float4& alo, float4& ahi, float4 blo, float4 bhi, BvhNode* nodes, uint32_t* count,
                                           uint32_t* next) {
    const uint32_t ra = __float_as_uint(alo.w), rb = __float_as_uint(blo.w), id = atomicAdd(next, 1u);
    BvhNode nd;
    nd.a = make_float4(alo.x, alo.y, alo.z, ahi.x);
    nd.b = make_float4(ahi.y, ahi.z, blo.x, blo.y);
    nd.c = make_float4(blo.z, bhi.x, bhi.y, bhi.z);
    nd.child[0] = ra;
    nd.child[1] = rb;
    nd.pad[0] = nd.pad[1] = 0;
    nodes[id] = nd;
    count[id] = ((ra & kBvhLeafBit) ? 1u : count[ra]) + ((rb & kBvhLeafBit) ? 1u : count[rb]);
    alo = make_float4(fminf(alo.x, blo.x), fminf(alo.y, blo.y), fminf(alo.z, blo.z), __uint_as_float(id));
    ahi = make_float4(fmaxf(ahi.x, bhi.x), fmaxf(ahi.y, bhi.y), fmaxf(ahi.z, bhi.z), 0.0f);
}
// A round over many clusters, three kernels and a scan; their number is on the device (the host only
// knows a bound, the grids' size).
__global__ void __launch_bounds__(kPlocBlock) k_ploc_nearest(const float4* __restrict__ lo, const float4* __restrict__ hi,
                                                             const uint32_t* __restrict__ clusters, int radius,
                                                             uint32_t* __restrict__ nearest) {
    __shared__ float4 s_lo[kPlocBlock + 2 * kPlocRadius], s_hi[kPlocBlock + 2 * kPlocRadius];
    const uint32_t n = *clusters;
    if (blockIdx.x * kPlocBlock >= n) return;
    const int base = (int)(blockIdx.x * kPlocBlock) - kPlocRadius;
    for (int k = threadIdx.x; k < kPlocBlock + 2 * kPlocRadius; k += kPlocBlock) {
        const int g = min(max(base + k, 0), (int)n - 1);
        s_lo[k] = lo[g];
        s_hi[k] = hi[g];
    }
    __syncthreads();
    const uint32_t i = blockIdx.x * kPlocBlock + threadIdx.x, me = threadIdx.x + kPlocRadius;
    if (i < n) nearest[i] = ploc_partner(s_lo + me, s_hi + me, i, n, radius);
}
__global__ void k_ploc_merge(float4* lo, float4* hi, const uint32_t* __restrict__ clusters, uint32_t bound,
                             const uint32_t* __restrict__ nearest, BvhNode* nodes, uint32_t* count, uint32_t* next,
                             uint32_t* __restrict__ keep) {
    const uint32_t n = *clusters;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < bound; i += gridDim.x * blockDim.x) {
        const uint32_t j = i < n ? nearest[i] : 0u;
        const bool pair = i < n && nearest[j] == i;
        keep[i] = i < n && (!pair || i < j);
        if (!pair || i > j) continue;
        float4 alo = lo[i], ahi = hi[i];
        ploc_merge(alo, ahi, lo[j], hi[j], nodes, count, next);
        lo[i] = alo;
        hi[i] = ahi;
    }
}
__global__ void k_ploc_compact(const float4* __restrict__ lo, const float4* __restrict__ hi,
                               const uint32_t* __restrict__ clusters, const uint32_t* __restrict__ keep,
                               const uint32_t* __restrict__ at, float4* __restrict__ lo2, float4* __restrict__ hi2,
                               uint32_t* __restrict__ left) {
    const uint32_t n = *clusters;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        if (i == n - 1) *left = at[i] + keep[i];
        if (!keep[i]) continue;
        lo2[at[i]] = lo[i];
        hi2[at[i]] = hi[i];
    }
}
// All rounds from kPlocFinish clusters or fewer on, by one CTA in shared memory.  Launches and the look at
// the number of clusters are most of a round's time there (45 us): creating a scene of 66 / 3000 /
// 20,000 / 200,000 triangles took 1.12 / 1.89 / 3.42 / 4.66 ms with a look per round and five allocations,
// 0.60 / 0.98 / 1.88 / 2.48 now.
constexpr uint32_t kPlocFinish = 2048;
constexpr int kPlocFinishBlock = 1024;
constexpr size_t kPlocFinishSmem = kPlocFinish * (2 * sizeof(float4) + sizeof(uint32_t));
__global__ void __launch_bounds__(kPlocFinishBlock) k_ploc_finish(const float4* __restrict__ lo, const float4* __restrict__ hi,
                                                                  const uint32_t* __restrict__ clusters, uint32_t rounds,
                                                                  BvhNode* nodes, uint32_t* count, uint32_t* next) {
    extern __shared__ float4 s_box[];
    float4 *const s_lo = s_box, *const s_hi = s_box + kPlocFinish;
    uint32_t* const s_near = reinterpret_cast<uint32_t*>(s_box + 2 * kPlocFinish);
    __shared__ uint32_t s_warp[kPlocFinishBlock / 32];
    uint32_t n = *clusters;
    for (uint32_t k = threadIdx.x; k < n; k += kPlocFinishBlock) {
        s_lo[k] = lo[k];
        s_hi[k] = hi[k];
    }
    __syncthreads();
    for (; n > 1; ++rounds) {
        const int radius = rounds < kPlocRounds ? kPlocRadius : 0;
        const uint32_t per = n > kPlocFinishBlock ? 2 : 1, i0 = threadIdx.x * per;
        for (uint32_t k = 0; k < per; ++k)
            if (i0 + k < n) s_near[i0 + k] = ploc_partner(s_lo + i0 + k, s_hi + i0 + k, i0 + k, n, radius);
        __syncthreads();
        float4 vlo[2], vhi[2];
        bool keep[2] = {false, false};
#pragma unroll
        for (uint32_t k = 0; k < 2; ++k) {
            const uint32_t i = i0 + k;
            if (k >= per || i >= n) continue;
            const uint32_t j = s_near[i];
            const bool pair = s_near[j] == i;
            keep[k] = !pair || i < j;
            if (!keep[k]) continue;
            vlo[k] = s_lo[i];
            vhi[k] = s_hi[i];
            if (pair) ploc_merge(vlo[k], vhi[k], s_lo[j], s_hi[j], nodes, count, next);
        }
        uint32_t left, at = block_exclusive_scan<kPlocFinishBlock>(uint32_t(keep[0]) + uint32_t(keep[1]), s_warp, left);
#pragma unroll
        for (uint32_t k = 0; k < 2; ++k)
            if (keep[k]) {
                s_lo[at] = vlo[k];
                s_hi[at++] = vhi[k];
            }
        n = left;
        __syncthreads();
    }
}

// ------------------------------------------------------------------ eight-wide hierarchy
// One level of the collapse, one thread per node of it: starting from the two children of its
// binary node, the child of largest surface area is replaced by its own two children until
// there are eight; single triangles become leaves.  From level kCountLevel on
// the child with most triangles is opened instead, which bounds the depth: on the way to any
// triangle a level then either descends seven binary levels or at least halves the triangles
// (at most 31 times), so a binary hierarchy of D levels takes at most kCountLevel + 31 + (D - 31) / 7
// levels: 60 for a clustered hierarchy (kPlocRounds rounds and at most 31 that halve the clusters).
// Nodes with fewer than eight children have leaves only, at least two, so there are at most 5/8 as
// many nodes as triangles.
constexpr uint32_t kCountLevel = 16;
struct WideChild {
    uint32_t ref;    // binary node or kBvhLeafBit | leaf
    uint32_t count;  // its leaves
    float lo[3], hi[3];
    __device__ __forceinline__ float area() const {
        const float x = hi[0] - lo[0], y = hi[1] - lo[1], z = hi[2] - lo[2];
        return x * y + y * z + z * x;
    }
};
__device__ __forceinline__ WideChild wide_child(const BvhNode& nd, const uint32_t* __restrict__ count, float max_abs,
                                                int k) {
    WideChild c;
    c.ref = nd.child[k];
    const float b0[6] = {nd.a.x, nd.a.y, nd.a.z, nd.a.w, nd.b.x, nd.b.y}, b1[6] = {nd.b.z, nd.b.w, nd.c.x, nd.c.y, nd.c.z, nd.c.w};
    // a triangle with a vertex that is not finite is never hit, but its box must not spoil its
    // neighbours' planes
    for (int a = 0; a < 3; ++a) {
        c.lo[a] = fminf(fmaxf(k ? b1[a] : b0[a], -max_abs), max_abs);
        c.hi[a] = fmaxf(fminf(k ? b1[3 + a] : b0[3 + a], max_abs), -max_abs);
    }
    c.count = (c.ref & kBvhLeafBit) ? 1u : count[c.ref];
    return c;
}
// The build's numbers on the device: nodes allocated, triangles placed, bits of the largest coordinate,
// clustered nodes, clusters of even and odd rounds; first node of every level of the collapse
// (first[level + 1] ends it), CTAs of a level's launch that are done.
struct BuildCounts {
    uint32_t nodes, tris, max_abs, merged, clusters[2];
    uint32_t first[kWideStack + 2], done[kWideStack];
};
// root: the binary node of every wide node
__device__ __forceinline__ void wide_node(const BvhNode* __restrict__ nodes, const uint32_t* __restrict__ count,
                                          const BvhTri* __restrict__ tris, const uint32_t* __restrict__ prim, uint32_t w,
                                          uint32_t level, uint32_t* root, uint32_t cap, WideNode* __restrict__ wide,
                                          WideTri* __restrict__ wtris, BuildCounts* counts) {
    const float max_abs = __uint_as_float(counts->max_abs);
    WideChild c[8];
    int n = 2;
    {
        const BvhNode nd = nodes[root[w]];
        c[0] = wide_child(nd, count, max_abs, 0);
        c[1] = wide_child(nd, count, max_abs, 1);
    }
    while (n < 8) {
        int best = -1;
        float key = -1.0f;
        for (int k = 0; k < n; ++k) {
            if (c[k].count == 1) continue;
            const float a = level >= kCountLevel ? (float)c[k].count : c[k].area();
            if (best < 0 || a > key) {
                best = k;
                key = a;
            }
        }
        if (best < 0) break;
        const BvhNode nd = nodes[c[best].ref];
        c[best] = wide_child(nd, count, max_abs, 0);
        c[n++] = wide_child(nd, count, max_abs, 1);
    }
    float lo[3], hi[3];
    for (int a = 0; a < 3; ++a) {
        lo[a] = c[0].lo[a];
        hi[a] = c[0].hi[a];
        for (int k = 1; k < n; ++k) {
            lo[a] = fminf(lo[a], c[k].lo[a]);
            hi[a] = fmaxf(hi[a], c[k].hi[a]);
        }
    }
    // slots: the pair of a free slot and an unplaced child whose centre lies furthest towards the
    // slot's octant, until all are placed
    int slot_of[8];
    {
        uint32_t placed = 0, taken = 0;
        for (int j = 0; j < n; ++j) {
            int bk = -1, bs = 0;
            float bv = 0.0f;
            for (int k = 0; k < n; ++k) {
                if (placed >> k & 1u) continue;
                float d[3];
                for (int a = 0; a < 3; ++a) d[a] = (c[k].lo[a] + c[k].hi[a]) - (lo[a] + hi[a]);
                for (int q = 0; q < 8; ++q) {
                    if (taken >> q & 1u) continue;
                    const float val = ((q & 1) ? d[0] : -d[0]) + ((q & 2) ? d[1] : -d[1]) + ((q & 4) ? d[2] : -d[2]);
                    if (bk < 0 || val > bv) {
                        bk = k;
                        bs = q;
                        bv = val;
                    }
                }
            }
            slot_of[bk] = bs;
            placed |= 1u << bk;
            taken |= 1u << bs;
        }
    }
    int in_slot[8];
    for (int q = 0; q < 8; ++q) in_slot[q] = -1;
    uint32_t imask = 0, lmask = 0;
    for (int k = 0; k < n; ++k) {
        in_slot[slot_of[k]] = k;
        (c[k].count > 1 ? imask : lmask) |= 1u << slot_of[k];
    }
    WideNode nd;
    // planes: q = 0 and q = 255 on the box, a step of at least 2 ulp of the coordinates
    double step[3];
    nd.imask = imask;
    for (int a = 0; a < 3; ++a) {
        int m = 0;
        frexp(fmax(fabs((double)lo[a]), fabs((double)hi[a])), &m);
        const float least = fmaxf((float)ldexp(1.0, m - 22), 0x1p-100f);
        nd.step[a] = fmaxf(__double2float_ru(((double)hi[a] - (double)lo[a]) / 255.0), least);
        step[a] = nd.step[a];
        nd.org[a] = lo[a];
    }
    nd.lmask = lmask;
    nd.pad0 = 0;
    nd.pad1 = 0;
    nd.child_base = imask ? atomicAdd(&counts->nodes, (uint32_t)__popc(imask)) : 0u;
    nd.tri_base = lmask ? atomicAdd(&counts->tris, (uint32_t)__popc(lmask)) : 0u;
    uint32_t child = nd.child_base, tri = nd.tri_base;
    for (int q = 0; q < 8; ++q) {
        const int k = in_slot[q];
        for (int a = 0; a < 3; ++a) {
            nd.qlo[a][q] = 0;
            nd.qhi[a][q] = 0;
        }
        if (k < 0) continue;
        for (int a = 0; a < 3; ++a) {
            const double x0 = ((double)c[k].lo[a] - (double)nd.org[a]) / step[a], x1 = ((double)c[k].hi[a] - (double)nd.org[a]) / step[a];
            nd.qlo[a][q] = (uint8_t)fmin(fmax(floor(x0), 0.0), 255.0);
            nd.qhi[a][q] = (uint8_t)fmin(fmax(ceil(x1), 0.0), 255.0);
        }
        if (imask >> q & 1u) {
            if (child < cap) root[child] = c[k].ref;
            ++child;
        } else {
            const uint32_t leaf = c[k].ref & ~kBvhLeafBit;
            WideTri t;
            t.tr = tris[leaf];
            t.leaf = leaf;
            t.prim = prim[leaf];
            t.pad[0] = t.pad[1] = 0;
            wtris[tri++] = t;
        }
    }
    wide[w] = nd;
}
__global__ void __launch_bounds__(128) k_wide_level(const BvhNode* __restrict__ nodes, const uint32_t* __restrict__ count,
                                                    const BvhTri* __restrict__ tris, const uint32_t* __restrict__ prim,
                                                    uint32_t level, uint32_t* root, uint32_t cap,
                                                    WideNode* __restrict__ wide, WideTri* __restrict__ wtris,
                                                    BuildCounts* counts) {
    const uint32_t end = min(counts->first[level + 1], cap);
    for (uint32_t w = counts->first[level] + blockIdx.x * blockDim.x + threadIdx.x; w < end; w += gridDim.x * blockDim.x)
        wide_node(nodes, count, tris, prim, w, level, root, cap, wide, wtris, counts);
    // the last CTA to finish tells where the level after the next begins
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0 && atomicAdd(counts->done + level, 1u) == gridDim.x - 1)
        counts->first[level + 2] = atomicAdd(&counts->nodes, 0u);
}

// rounds of clustering, or levels of the collapse, between two looks of the host at how far they are
constexpr int kBuildLook = 4;
static_assert(kWideStack % kBuildLook == 0 && (kPlocFinish >> kBuildLook) > 1, "looks end at the bounds");

struct HitOut {
    float* t;
    uint32_t* prim;
    float* uv;
    __device__ __forceinline__ void put(int64_t i, const Hit& h) const {
        if (t) t[i] = h.prim == 0xffffffffu ? -1.0f : h.t;
        if (prim) prim[i] = h.prim;
        if (uv) reinterpret_cast<float2*>(uv)[i] = make_float2(h.u, h.v);
    }
};
template <bool ANY>
__global__ void __launch_bounds__(128) k_scene_intersect_flat(SceneDev s, int64_t n, const float* __restrict__ org,
                                                              const float* __restrict__ dir, const float* __restrict__ tmin,
                                                              const float* __restrict__ tmax, HitOut o) {
    for (int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; i < n; i += int64_t(gridDim.x) * blockDim.x) {
        Hit h;
        h.prim = 0xffffffffu;
        h.t = h.u = h.v = 0.0f;
        if (s.ntris)
            h = flat_trace<ANY>(s.flat, flat_pairs(s.ntris), org[3 * i], org[3 * i + 1], org[3 * i + 2], dir[3 * i], dir[3 * i + 1],
                                dir[3 * i + 2], tmin ? tmin[i] : 0.0f, tmax ? tmax[i] : 1e20f);
        o.put(i, h);
    }
}
// Each warp owns `share` consecutive rays.  Walks end at very different steps, so whenever fewer
// than kRefill lanes are still walking the others take the warp's next rays.
constexpr int kRefill = 28;
constexpr int kWalkCtas = 8;
template <bool ANY>
__global__ void __launch_bounds__(128, 8) k_scene_intersect(SceneDev s, int64_t n, int64_t share, const float* __restrict__ org,
                                                         const float* __restrict__ dir, const float* __restrict__ tmin,
                                                         const float* __restrict__ tmax, HitOut o) {
    const uint32_t lane = threadIdx.x & 31u;
    int64_t next = (int64_t(blockIdx.x) * (blockDim.x >> 5) + (threadIdx.x >> 5)) * share;
    const int64_t end = min(next + share, n);
    if (next >= end) return;
    int64_t i = -1;
    WideWalk<ANY> w(s, 0.f, 0.f, 0.f, 1.f, 1.f, 1.f, 0.f, 0.f);
    w.g.y = 0u;
    uint2 stack[kWideStack];
    for (;;) {
        const unsigned idle = __ballot_sync(0xffffffffu, !w.alive());
        if (idle && (next < end ? __popc(idle) > 32 - kRefill : idle == 0xffffffffu)) {
            if (!w.alive()) {
                if (i >= 0) o.put(i, w.h);
                i = next + __popc(idle & ((1u << lane) - 1u));
                if (i < end)
                    w = WideWalk<ANY>(s, org[3 * i], org[3 * i + 1], org[3 * i + 2], dir[3 * i], dir[3 * i + 1], dir[3 * i + 2],
                                      tmin ? tmin[i] : 0.0f, tmax ? tmax[i] : 1e20f);
                else
                    i = -1;
            }
            if (next >= end) break;
            next += __popc(idle);
        }
        w.step(s, stack);
    }
}

}  // namespace rtpg

using namespace rtpg;

struct rtpg_scene {
    SceneDev dev{};
    BvhNode* nodes = nullptr;
    float4* leaf_box = nullptr;
    WideNode* wide = nullptr;
    WideTri* wtris = nullptr;
    FlatPair* flat = nullptr;
    std::vector<void*> allocs;
    size_t bytes = 0;
    template <class T>
    int alloc(T** p, size_t count) {
        void* q = nullptr;
        cudaError_t e = cudaMalloc(&q, std::max<size_t>(count, 1) * sizeof(T));
        if (e != cudaSuccess) {
            cudaGetLastError();
            return fail(RTPG_ENOMEM, "cudaMalloc(%zu bytes) failed: %s", count * sizeof(T), cudaGetErrorString(e));
        }
        allocs.push_back(q);
        bytes += count * sizeof(T);
        *p = static_cast<T*>(q);
        return RTPG_OK;
    }
    ~rtpg_scene() {
        for (void* p : allocs) cudaFree(p);
    }
};

namespace rtpg {
SceneDev scene_device_view(const rtpg_scene* s) { return s->dev; }
}

extern "C" {

int rtpg_scene_create(const float* vertices, uint32_t num_vertices, const uint32_t* indices, uint32_t num_triangles,
                      void* stream, rtpg_scene** out) {
    if (!out || (num_triangles && (!vertices || !indices))) return fail(RTPG_EINVAL, "rtpg_scene_create: bad arguments");
    if (num_triangles >= kBvhLeafBit) return fail(RTPG_EINVAL, "rtpg_scene_create: too many triangles");
    (void)num_vertices;
    cudaStream_t st = as_stream(stream);
    auto* s = new (std::nothrow) rtpg_scene();
    if (!s) return fail(RTPG_ENOMEM, "rtpg_scene_create: out of host memory");
    const uint32_t n = num_triangles;
    int r;
    unsigned* bounds = nullptr;
    unsigned long long *k0 = nullptr, *k1 = nullptr;
    uint32_t *v0 = nullptr, *v1 = nullptr, *pi = nullptr, *pl = nullptr;
    float4* ibox = nullptr;
    unsigned* flags = nullptr;
    BvhTri* tris = nullptr;  // the triangles in leaf order, and their scene indices
    uint32_t *prim = nullptr, *root = nullptr;
    BuildCounts* counts = nullptr;
    uint32_t *pcount = nullptr, *nearest = nullptr, *keep = nullptr, *at = nullptr;
    BvhNode* pnodes = nullptr;
    float4 *clo[2] = {nullptr, nullptr}, *chi[2] = {nullptr, nullptr};
    uint8_t *sort_temp = nullptr, *scan_temp = nullptr;
    cub::DoubleBuffer<unsigned long long> dk(nullptr, nullptr);
    cub::DoubleBuffer<uint32_t> dv(nullptr, nullptr);
    // small scenes are a flat list; the others get both hierarchies
    const bool flat = n <= kFlatTris;
    const uint32_t wide_cap = n / 8 * 5 + 8;
    if (n > 0 && flat && (r = s->alloc(&s->flat, flat_pairs(n)))) {
        delete s;
        return r;
    }
    // one allocation holds what rays read: each of more than 1 MB costs 0.3 ms
    char* arrays = nullptr;
    for (int pass = 0; pass < 2 && n > 0 && !flat; ++pass) {  // sizes, then places
        size_t at_byte = 0;
        auto take = [&](auto** p, size_t count) {
            if (pass) *p = reinterpret_cast<std::remove_reference_t<decltype(*p)>>(arrays + at_byte);
            at_byte += (count * sizeof(**p) + 255) & ~size_t(255);
        };
        take(&s->nodes, n - 1);
        take(&s->leaf_box, 2 * size_t(n));
        take(&s->wide, wide_cap);
        take(&s->wtris, n);
        if (!pass && (r = s->alloc(&arrays, at_byte))) {
            delete s;
            return r;
        }
    }
    s->dev.nodes = s->nodes;
    s->dev.leaf_box = s->leaf_box;
    s->dev.wide = s->wide;
    s->dev.wtris = s->wtris;
    s->dev.flat = s->flat;
    s->dev.ntris = n;
    if (n == 0) {
        *out = s;
        return RTPG_OK;
    }
    // all scratch in one allocation, freed at the end
    size_t sort_bytes = 0, scan_bytes = 0;
    cudaError_t e = cub::DeviceRadixSort::SortPairs(nullptr, sort_bytes, dk, dv, (int)n, 0, 63, st);
    if (!e && !flat) e = cub::DeviceScan::ExclusiveSum(nullptr, scan_bytes, keep, at, (int)n, st);
    if (e) {
        delete s;
        return fail(RTPG_ECUDA, "rtpg_scene_create: %s", cudaGetErrorString(e));
    }
    void* scratch = nullptr;
    for (int pass = 0; pass < 2; ++pass) {  // sizes, then places
        size_t at_byte = 0;
        auto take = [&](auto** p, size_t count) {
            if (pass) *p = reinterpret_cast<std::remove_reference_t<decltype(*p)>>(static_cast<char*>(scratch) + at_byte);
            at_byte += (count * sizeof(**p) + 255) & ~size_t(255);
        };
        take(&bounds, 6);
        take(&k0, n);
        take(&k1, n);
        take(&v0, n);
        take(&v1, n);
        take(&tris, n);
        take(&prim, n);
        take(&sort_temp, sort_bytes);
        if (!flat) {
            take(&pi, n);
            take(&pl, n);
            take(&ibox, 2 * size_t(n));
            take(&flags, n);
            take(&root, wide_cap);
            take(&counts, 1);
            take(&pcount, n);
            take(&nearest, n);
            take(&keep, n);
            take(&at, n);
            take(&pnodes, n);
            for (int k = 0; k < 2; ++k) {
                take(&clo[k], n);
                take(&chi[k], n);
            }
            take(&scan_temp, scan_bytes);
        }
        if (!pass && (e = cudaMalloc(&scratch, at_byte))) {
            cudaGetLastError();
            delete s;
            return fail(RTPG_ENOMEM, "rtpg_scene_create: scratch allocation failed");
        }
    }
    const unsigned init[6] = {0xffffffffu, 0xffffffffu, 0xffffffffu, 0u, 0u, 0u};
    const int g = grid_for(n, 256, 8);
    int rc = RTPG_OK;
    do {
        if ((e = cudaMemcpyAsync(bounds, init, sizeof(init), cudaMemcpyHostToDevice, st))) break;
        k_scene_bounds<<<g, 256, 0, st>>>(vertices, indices, n, bounds);
        k_scene_morton<<<g, 256, 0, st>>>(vertices, indices, n, bounds, k0, v0);
        dk = cub::DoubleBuffer<unsigned long long>(k0, k1);
        dv = cub::DoubleBuffer<uint32_t>(v0, v1);
        if ((e = cub::DeviceRadixSort::SortPairs(sort_temp, sort_bytes, dk, dv, (int)n, 0, 63, st))) break;
        k_scene_leaves<<<g, 256, 0, st>>>(vertices, indices, n, dv.Current(), tris, prim);
        if (flat) {
            k_scene_flat<<<1, 64, 0, st>>>(tris, prim, n, s->flat);
        } else {
            k_scene_hierarchy<<<g, 256, 0, st>>>(dk.Current(), (int)n, s->nodes, pi, pl);
            if ((e = cudaMemsetAsync(flags, 0, 4ull * n, st))) break;
            k_scene_boxes<<<g, 256, 0, st>>>(vertices, indices, prim, n, s->nodes, pi, pl, ibox, flags);
            BuildCounts now{};
            now.nodes = now.first[1] = 1;
            now.clusters[0] = n;
            if ((e = cudaMemcpyAsync(counts, &now, sizeof(now), cudaMemcpyHostToDevice, st))) break;
            k_scene_leaf_boxes<<<g, 256, 0, st>>>(vertices, indices, prim, n, s->leaf_box, &counts->max_abs);
            k_ploc_init<<<g, 256, 0, st>>>(s->leaf_box, n, clo[0], chi[0]);
            // a round at most halves the clusters, so kBuildLook of them leave more than one
            uint32_t bound = n, rounds = 0;
            while (bound > kPlocFinish && !e) {
                const int gn = (int)((bound + kPlocBlock - 1) / kPlocBlock), gc = grid_for(bound, 256, 8);
                for (int k = 0; k < kBuildLook && !e; ++k, ++rounds) {
                    const int a = rounds & 1, b = a ^ 1, radius = rounds < kPlocRounds ? kPlocRadius : 0;
                    k_ploc_nearest<<<gn, kPlocBlock, 0, st>>>(clo[a], chi[a], counts->clusters + a, radius, nearest);
                    k_ploc_merge<<<gc, 256, 0, st>>>(clo[a], chi[a], counts->clusters + a, bound, nearest, pnodes, pcount,
                                                     &counts->merged, keep);
                    if ((e = cub::DeviceScan::ExclusiveSum(scan_temp, scan_bytes, keep, at, (int)bound, st))) break;
                    k_ploc_compact<<<gc, 256, 0, st>>>(clo[a], chi[a], counts->clusters + a, keep, at, clo[b], chi[b],
                                                       counts->clusters + b);
                }
                if (e || (e = cudaMemcpyAsync(&bound, counts->clusters + (rounds & 1), 4, cudaMemcpyDeviceToHost, st))) break;
                e = cudaStreamSynchronize(st);
            }
            if (e || (e = cudaFuncSetAttribute(k_ploc_finish, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kPlocFinishSmem))) break;
            k_ploc_finish<<<1, kPlocFinishBlock, kPlocFinishSmem, st>>>(clo[rounds & 1], chi[rounds & 1],
                                                                      counts->clusters + (rounds & 1), rounds, pnodes, pcount,
                                                                      &counts->merged);
            const uint32_t bin_root = n - 2;  // made last
            if ((e = cudaMemcpyAsync(root, &bin_root, 4, cudaMemcpyHostToDevice, st))) break;
            const int gw = (int)std::min<uint32_t>((wide_cap + 127) / 128, kSMs * 16);
            uint32_t level = 0;
            do {
                for (int k = 0; k < kBuildLook; ++k, ++level)
                    k_wide_level<<<gw, 128, 0, st>>>(pnodes, pcount, tris, prim, level, root, wide_cap, s->wide, s->wtris, counts);
                if ((e = cudaMemcpyAsync(&now, counts, sizeof(now), cudaMemcpyDeviceToHost, st))) break;
                if ((e = cudaStreamSynchronize(st))) break;
            } while (now.first[level + 1] > now.first[level] && now.nodes <= wide_cap && level < (uint32_t)kWideStack);
            if (e) break;
            if (now.first[level + 1] > now.first[level] || now.nodes > wide_cap) {
                rc = fail(RTPG_ECAPACITY, "rtpg_scene_create: hierarchy of %u nodes in %u levels exceeds its bounds", now.nodes, level);
                break;
            }
            memcpy(&s->dev.max_abs, &now.max_abs, 4);
        }
        if ((e = cudaGetLastError())) break;
        if ((e = cudaStreamSynchronize(st))) break;
    } while (0);
    cudaFree(scratch);
    if (e != cudaSuccess) {
        delete s;
        return fail(RTPG_ECUDA, "rtpg_scene_create: %s", cudaGetErrorString(e));
    }
    if (rc) {
        delete s;
        return rc;
    }
    *out = s;
    return RTPG_OK;
}

int rtpg_scene_destroy(rtpg_scene* s) {
    if (!s) return fail(RTPG_EINVAL, "rtpg_scene_destroy: null handle");
    delete s;
    return RTPG_OK;
}

// Batched TraceRadiance (any_hit = 0, closest hit) / TraceOccluded (any_hit = 1).
int rtpg_scene_intersect(rtpg_scene* s, int64_t n, const float* org, const float* dir, const float* tmin,
                         const float* tmax, int any_hit, float* out_t, uint32_t* out_prim, float* out_uv, void* stream) {
    if (!s) return fail(RTPG_EINVAL, "rtpg_scene_intersect: null handle");
    if (n < 0 || (n > 0 && (!org || !dir))) return fail(RTPG_EINVAL, "rtpg_scene_intersect: bad arguments");
    if (n == 0) return RTPG_OK;
    cudaStream_t st = as_stream(stream);
    const HitOut o{out_t, out_prim, out_uv};
    if (s->dev.flat || s->dev.ntris == 0) {
        const int g = grid_for(n, 128, 16);
        if (any_hit) k_scene_intersect_flat<true><<<g, 128, 0, st>>>(s->dev, n, org, dir, tmin, tmax, o);
        else k_scene_intersect_flat<false><<<g, 128, 0, st>>>(s->dev, n, org, dir, tmin, tmax, o);
    } else {
        // a share of at least a warp's rays on at most kWalkCtas CTAs per SM
        const int64_t warps = int64_t(kSMs) * kWalkCtas * 4;
        const int64_t share = std::max<int64_t>(32, (n + warps - 1) / warps);
        const int g = (int)((n + 4 * share - 1) / (4 * share));
        if (any_hit) k_scene_intersect<true><<<g, 128, 0, st>>>(s->dev, n, share, org, dir, tmin, tmax, o);
        else k_scene_intersect<false><<<g, 128, 0, st>>>(s->dev, n, share, org, dir, tmin, tmax, o);
    }
    RTPG_LAUNCH_CHECK();
    return RTPG_OK;
}

}  // extern "C"
