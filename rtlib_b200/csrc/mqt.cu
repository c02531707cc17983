// Morton-indexed directional quadtrees, one complete tree per hash-grid cell (RTLib's "HashTree"
// guide: MortonQuadTreeT / MortonQuadTreeWrapperT, OPX7UtilsMorton.h:253-531, host wrapper
// RTMortonQuadTreeWrapperT :590-764, pyramid build mortonBuildKernel,
// OPX7UtilsMortonBuild.cu:2-16).
//
// Layout in HBM: building leaves, int64 fixed point, cell-major: leaves[cell * 4^L + code]
// (the reference records only the leaf level too, OPX7UtilsMorton.h:282-283); sampling
// pyramid, float, per cell (4^(L+1)-1)/3 entries, level l at offset (4^l-1)/3 (+ mqt_dev.cuh's
// alignment shift), Morton order inside a level (code = part1by1(y) << 1 | part1by1(x)).
//
// Update (RTMortonQuadTreeWrapperT::Update + LaunchBuildKernel, :640-651, :916-941) is one
// kernel: the leaves of every cell in use are reduced with exact integer sums, written as a float
// pyramid to the sampling buffer and zeroed (RTLib launches 1024x more blocks than cells and
// loops serially per cell).
#include <algorithm>
#include <new>
#include <vector>

#include "common.cuh"
#include "limits.cuh"
#include "mqt_dev.cuh"

namespace rtpg {


// what one record adds: leaf (UINT64_MAX: nothing) and fixed-point value
__device__ __forceinline__ unsigned long long mqt_record_key(const MqtDev& t, int64_t i, const uint32_t* __restrict__ cell,
                                                             const float* __restrict__ dir, int canonical,
                                                             const float* __restrict__ value, unsigned long long& v) {
    const uint32_t c = cell[i];
    const float x = value[i];
    if (c == 0xffffffffu || c >= t.ncells || !isfinite(x) || !(x > 0.0f)) return ~0ull;
    float2 uv;
    if (canonical) uv = reinterpret_cast<const float2*>(dir)[i];
    else uv = dir_to_canonical_mqt(dir[3 * i], dir[3 * i + 1], dir[3 * i + 2]);
    v = to_fx(x, t.fx, t.status);
    return ((unsigned long long)c << (2 * t.level)) + mqt_leaf_code(t.level, uv.x, uv.y);
}

// One record per thread, one plain 64-bit atomic each: a frame's records spread over the leaves
// of many cells, where aggregating equal keys within the warp only adds its 64-bit match.
// The cell is marked as touched by a byte store.  Popular cells would get thousands of those, which
// queue up in L2 behind one another (and a look at the byte first finds the L1 line of the first
// look), so each CTA remembers the cells it marked in a direct-mapped table in shared memory; large
// CTAs share one table among many records.  2^22 records into 377 k / 1474 cells of 4^4 leaves:
// 258 / 255 us aggregated and without marks, 150 / 97 us here with the cells' flags side by side (139 / 75 us
// without marks); mqt_touched_shift spreads them since.
constexpr int kRecThreads = 1024;
constexpr uint32_t kRecTags = 8192;  // 32 KB, two CTAs per SM
__global__ void __launch_bounds__(kRecThreads) k_mqt_record(MqtDev t, int64_t n, const uint32_t* __restrict__ cell,
                                                            const float* __restrict__ dir, int canonical,
                                                            const float* __restrict__ value) {
    __shared__ uint32_t s_tag[kRecTags];
    for (uint32_t k = threadIdx.x; k < kRecTags; k += kRecThreads) s_tag[k] = 0xffffffffu;
    __syncthreads();
    const int64_t stride = int64_t(gridDim.x) * blockDim.x;
    for (int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; i < n; i += stride) {
        unsigned long long v;
        const unsigned long long key = mqt_record_key(t, i, cell, dir, canonical, value, v);
        if (key == ~0ull) continue;
        atomicAdd(t.leaves + key, v);
        const uint32_t c = uint32_t(key >> (2 * t.level));
        mqt_mark(t, c, s_tag + c % kRecTags);
    }
}

// The same for trees of few leaves in all (`nleaf`), where records queue up on the leaves
// themselves: every CTA sums all leaves in shared memory and adds the nonzero ones once.  A sum is
// two 32-bit words, the low word's carry added to the high one (64-bit shared adds are
// compare-and-swap loops).  2^22 records into 10 cells of 16 leaves: 798 us with one atomic per
// record, 40 us here.
constexpr uint32_t kRecPrivLeaves = 16384;  // 128 KB
__global__ void __launch_bounds__(kRecThreads) k_mqt_record_private(MqtDev t, int64_t n, const uint32_t* __restrict__ cell,
                                                                    const float* __restrict__ dir, int canonical,
                                                                    const float* __restrict__ value, uint32_t nleaf) {
    extern __shared__ uint32_t s_sum[];
    uint32_t *lo = s_sum, *hi = s_sum + nleaf;
    for (uint32_t k = threadIdx.x; k < 2 * nleaf; k += kRecThreads) s_sum[k] = 0u;
    __syncthreads();
    const int64_t stride = int64_t(gridDim.x) * blockDim.x;
    for (int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; i < n; i += stride) {
        unsigned long long v;
        const unsigned long long key = mqt_record_key(t, i, cell, dir, canonical, value, v);
        if (key == ~0ull) continue;
        const uint32_t low = (uint32_t)v, old = atomicAdd(lo + key, low);
        const uint32_t up = (uint32_t)(v >> 32) + (old + low < low ? 1u : 0u);
        if (up) atomicAdd(hi + key, up);
    }
    __syncthreads();
    // each CTA starts at another leaf, so that they do not all add to the same one at once
    for (uint32_t j = threadIdx.x; j < nleaf; j += kRecThreads) {
        const uint32_t k = (j + blockIdx.x * 97u) % nleaf;
        const unsigned long long v = ((unsigned long long)hi[k] << 32) | lo[k];
        if (!v) continue;
        atomicAdd(t.leaves + k, v);
        t.touched[size_t(k >> (2 * t.level)) << t.touched_shift] = 1;
    }
}

// ------------------------------------------------------------------ build
// Bound by HBM: a cell's leaves are read (8 B each), its pyramid written (4 B a node).  The
// building leaves of a cell are nonzero only if it was recorded into since the last build
// (`touched`), its pyramid only if the last build wrote sums there (`live`): a cell with neither
// is skipped, leaves are read only where touched, and a 32-byte sector of leaves is zeroed only if
// it holds something.  At level 4 with 36 % of 2^20 cells in use and 4 M records: 1206 us when every cell
// was read, zeroed and rewritten (level 4: 5.7 GB), 277 us now (1.4 GB, 77 % of the copy rate).
//
// A lane takes four leaves (one 32-byte load and, as floats, one 16-byte store) and sums them to
// their parent; four and sixteen lanes' parents come from butterfly shuffles, wider nodes from
// sums over the lane's further leaves 128 apart.  Lanes are consecutive in memory at every step and
// no shared memory is used.  Sums are exact integers, in any order the same.
constexpr int kMqtWarps = 8;

__device__ __forceinline__ void ld_leaves(const unsigned long long* p, unsigned long long* v) {
    asm volatile("ld.global.v4.u64 {%0,%1,%2,%3}, [%4];" : "=l"(v[0]), "=l"(v[1]), "=l"(v[2]), "=l"(v[3]) : "l"(p) : "memory");
}
__device__ __forceinline__ void zero_leaves(unsigned long long* p) {
    asm volatile("st.global.v4.u64 [%0], {%1,%1,%1,%1};" ::"l"(p), "l"(0ull) : "memory");
}
__device__ __forceinline__ unsigned long long xor_add(unsigned long long s, int o) {
    return s + __shfl_xor_sync(0xffffffffu, s, o);
}

// The subtree of S levels (4 or 5) whose root is node `sub` of level `top` of a cell: its leaves
// (lf: its first one) are summed and zeroed, its nodes written to the cell's pyramid w; returns
// the subtree's sum.  The whole warp calls it.  read = false: the leaves are zero.
template <int S>
__device__ __forceinline__ unsigned long long mqt_build_subtree(unsigned long long* lf, float* w, uint32_t top,
                                                                uint32_t sub, bool read, FixedPoint fx) {
    static_assert(S == 4 || S == 5, "a warp's share is 256 or 1024 leaves");
    constexpr int NC = (1 << (2 * (S - 1))) / 32;  // four-leaf groups per lane
    const uint32_t lane = threadIdx.x & 31u;
    unsigned long long v[NC][4];
#pragma unroll
    for (int c = 0; c < NC; ++c) {
        if (read) ld_leaves(lf + 4 * (c * 32 + lane), v[c]);
        else v[c][0] = v[c][1] = v[c][2] = v[c][3] = 0ull;
    }
    unsigned long long run = 0, all = 0;
    float* const w0 = w + mqt_base(top + S) + (size_t(sub) << (2 * S));
    float* const w1 = w + mqt_base(top + S - 1) + (size_t(sub) << (2 * (S - 1)));
    float* const w2 = w + mqt_base(top + S - 2) + (size_t(sub) << (2 * (S - 2)));
    float* const w3 = w + mqt_base(top + S - 3) + (size_t(sub) << (2 * (S - 3)));
#pragma unroll
    for (int c = 0; c < NC; ++c) {
        const uint32_t g = c * 32 + lane;
        if (v[c][0] | v[c][1] | v[c][2] | v[c][3]) zero_leaves(lf + 4 * g);
        *reinterpret_cast<float4*>(w0 + 4 * g) = make_float4(fx_to_float(v[c][0], fx), fx_to_float(v[c][1], fx),
                                                             fx_to_float(v[c][2], fx), fx_to_float(v[c][3], fx));
        unsigned long long s = v[c][0] + v[c][1] + v[c][2] + v[c][3];
        w1[g] = fx_to_float(s, fx);
        s = xor_add(xor_add(s, 1), 2);
        if ((lane & 3u) == 0) w2[g >> 2] = fx_to_float(s, fx);
        s = xor_add(xor_add(s, 4), 8);
        if ((lane & 15u) == 0) w3[g >> 4] = fx_to_float(s, fx);
        run += xor_add(s, 16);
        if (S == 5 && (c & 1)) {  // the level between: two groups of 32
            if (lane == 0) w[mqt_base(top + 1) + (size_t(sub) << 2) + (c >> 1)] = fx_to_float(run, fx);
        }
        if (S == 4 || (c & 1)) {
            all += run;
            run = 0;
        }
    }
    if (lane == 0) w[mqt_base(top) + sub] = fx_to_float(all, fx);
    return all;
}

// Levels 1 to 3: 32, 8 or 2 cells per warp, a lane per four leaves.
template <int L>
__global__ void __launch_bounds__(32 * kMqtWarps) k_mqt_build_small(MqtDev t) {
    static_assert(L >= 1 && L <= 3, "levels 1..3");
    constexpr uint32_t G = 1u << (2 * (L - 1));  // lanes of a cell
    constexpr uint32_t NLEAF = 4 * G;
    const uint32_t lane = threadIdx.x & 31u, g = lane % G;
    const uint32_t nw = gridDim.x * kMqtWarps, per = 32 / G;
    for (uint32_t base = (blockIdx.x * kMqtWarps + (threadIdx.x >> 5)) * per; base < t.ncells; base += nw * per) {
        const uint32_t c = base + lane / G;
        const bool touched = c < t.ncells && t.touched[size_t(c) << t.touched_shift], live = c < t.ncells && t.live[c];
        if (!__any_sync(0xffffffffu, touched || live)) continue;
        unsigned long long v[4] = {0ull, 0ull, 0ull, 0ull};
        unsigned long long* lf = t.leaves + size_t(c) * NLEAF + 4 * g;
        if (touched) ld_leaves(lf, v);
        if (v[0] | v[1] | v[2] | v[3]) zero_leaves(lf);
        const bool out = touched || live;
        float* w = t.pyramid + size_t(c) * mqt_stride(L);
        if (out)
            *reinterpret_cast<float4*>(w + mqt_base(L) + 4 * g) =
                make_float4(fx_to_float(v[0], t.fx), fx_to_float(v[1], t.fx), fx_to_float(v[2], t.fx), fx_to_float(v[3], t.fx));
        unsigned long long s = v[0] + v[1] + v[2] + v[3];
        if (out) w[mqt_base(L - 1) + g] = fx_to_float(s, t.fx);
        if (L >= 2) {
            s = xor_add(xor_add(s, 1), 2);
            if (out && (lane & 3u) == 0) w[mqt_base(L >= 2 ? L - 2 : 0) + (g >> 2)] = fx_to_float(s, t.fx);
        }
        if (L >= 3) {
            s = xor_add(xor_add(s, 4), 8);
            if (out && (lane & 15u) == 0) w[mqt_base(0)] = fx_to_float(s, t.fx);
        }
        __syncwarp();
        if (out && g == 0) {
            t.touched[size_t(c) << t.touched_shift] = 0;
            t.live[c] = touched ? 1 : 0;
        }
    }
}

// Levels 4 and 5: a warp per cell.  A warp looks at eight cells' flags at a time.
template <int L>
__global__ void __launch_bounds__(32 * kMqtWarps) k_mqt_build_warp(MqtDev t) {
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t nw = gridDim.x * kMqtWarps;
    for (uint32_t base = (blockIdx.x * kMqtWarps + (threadIdx.x >> 5)) * 8; base < t.ncells; base += nw * 8) {
        const uint32_t c0 = base + lane;
        const bool mine = lane < 8 && c0 < t.ncells;
        const bool touched = mine && t.touched[size_t(c0) << t.touched_shift], live = mine && t.live[c0];
        const unsigned read = __ballot_sync(0xffffffffu, touched);
        for (unsigned todo = __ballot_sync(0xffffffffu, touched || live); todo; todo &= todo - 1) {
            const uint32_t k = __ffs(todo) - 1;
            mqt_build_subtree<L>(t.leaves + (size_t(base + k) << (2 * L)), t.pyramid + size_t(base + k) * mqt_stride(L), 0, 0,
                                 (read >> k) & 1u, t.fx);
        }
        if (touched || live) {
            t.touched[size_t(c0) << t.touched_shift] = 0;
            t.live[c0] = touched ? 1 : 0;
        }
    }
}

// Levels 6 and 7: a CTA of 4 or 16 warps per cell, each warp a subtree of five levels; the one or
// two levels above come from the warps' sums in shared memory.
template <int L>
__global__ void __launch_bounds__(L == 6 ? 128 : 512) k_mqt_build_block(MqtDev t) {
    static_assert(L == 6 || L == 7, "levels 6, 7");
    constexpr uint32_t W = L == 6 ? 4 : 16, TOP = L - 5;
    __shared__ unsigned long long s_sum[W];
    const uint32_t warp = threadIdx.x >> 5;
    for (uint32_t c = blockIdx.x; c < t.ncells; c += gridDim.x) {
        const bool touched = t.touched[size_t(c) << t.touched_shift], live = t.live[c];
        if (!touched && !live) continue;
        float* w = t.pyramid + size_t(c) * mqt_stride(L);
        const unsigned long long s = mqt_build_subtree<5>(t.leaves + (size_t(c) << (2 * L)) + size_t(warp) * 1024, w, TOP, warp,
                                                          touched, t.fx);
        if ((threadIdx.x & 31u) == 0) s_sum[warp] = s;
        __syncthreads();
        if (L == 7 && threadIdx.x < 4) {
            const unsigned long long* p = s_sum + 4 * threadIdx.x;
            w[mqt_base(1) + threadIdx.x] = fx_to_float(p[0] + p[1] + p[2] + p[3], t.fx);
        }
        if (threadIdx.x == 0) {
            unsigned long long r = 0;
            for (uint32_t k = 0; k < W; ++k) r += s_sum[k];
            w[mqt_base(0)] = fx_to_float(r, t.fx);
            t.touched[size_t(c) << t.touched_shift] = 0;
            t.live[c] = touched ? 1 : 0;
        }
        __syncthreads();
    }
}

// ------------------------------------------------------------------ sample / pdf
struct MqtSampleOut {
    float *uv, *pdf, *dir, *pdf_tree;
};
__device__ __forceinline__ void mqt_sample_one(const MqtDev& t, int64_t i, const uint32_t* __restrict__ cell,
                                               const uint32_t* __restrict__ seeds, uint32_t seed_base, const MqtSampleOut& o) {
    const uint32_t c = cell[i];
    uint32_t rng = seeds ? seeds[i] : (pcg1d(seed_base + (uint32_t)i) | 1u);
    float pdf;
    const float2 uv = mqt_sample_and_pdf(t, c, rng, pdf);
    if (o.uv) reinterpret_cast<float2*>(o.uv)[i] = uv;
    if (o.pdf_tree) o.pdf_tree[i] = pdf;
    // MortonQuadTreeWrapperT::SampleAndPdf (OPX7UtilsMorton.h:486-500):
    // pdf *= (0.25f * RTLIB_M_INV_PI), evaluated in double as written
    if (o.pdf) o.pdf[i] = (float)((double)pdf * (0.25 * kInvPiD));
    if (o.dir) {
        const float3 d = canonical_to_dir_mqt(uv.x, uv.y);
        o.dir[3 * i] = d.x;
        o.dir[3 * i + 1] = d.y;
        o.dir[3 * i + 2] = d.z;
    }
}
__global__ void __launch_bounds__(256) k_mqt_sample(MqtDev t, int64_t n, const uint32_t* __restrict__ cell,
                                                    const uint32_t* __restrict__ seeds, uint32_t seed_base, MqtSampleOut o) {
    const int64_t stride = int64_t(gridDim.x) * blockDim.x;
    for (int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; i < n; i += stride)
        mqt_sample_one(t, i, cell, seeds, seed_base, o);
}

__global__ void __launch_bounds__(256) k_mqt_pdf(MqtDev t, int64_t n, const uint32_t* __restrict__ cell,
                                                 const float* __restrict__ dir, int canonical, float* __restrict__ out,
                                                 int tree_level) {
    const int64_t stride = int64_t(gridDim.x) * blockDim.x;
    for (int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; i < n; i += stride) {
        float2 uv;
        if (canonical) uv = reinterpret_cast<const float2*>(dir)[i];
        else uv = dir_to_canonical_mqt(dir[3 * i], dir[3 * i + 1], dir[3 * i + 2]);
        const float p = mqt_pdf(t, cell[i], uv.x, uv.y);
        // MortonQuadTreeWrapperT::Pdf (:515-524): tree.Pdf(dir2) * 0.25f * RTLIB_M_INV_PI
        out[i] = tree_level ? p : (float)((double)(p * 0.25f) * kInvPiD);
    }
}

// ------------------------------------------------------------------ export
// Floats [at, at + m) of the pyramids without their rows' shift.  Rows copied to host memory one by one
// (a strided copy) take twice to seven times as long as one run of bytes, so a chunk is packed first:
// 2^20 trees of level 3 with their leaves 348 -> 188 ms, 2^18 of level 2 60.7 -> 8.7 ms (178 and 7.9 as
// one run).
constexpr size_t kExportFloats = 1u << 18;  // 1 MB: allocations past that cost 0.3 ms
__global__ void __launch_bounds__(256) k_mqt_pack(MqtDev t, uint64_t at, uint32_t m, float* __restrict__ out) {
    const uint32_t per = mqt_level_offset(t.level + 1);
    for (uint32_t k = blockIdx.x * blockDim.x + threadIdx.x; k < m; k += gridDim.x * blockDim.x) {
        const uint64_t c = (at + k) / per;
        out[k] = t.pyramid[c * mqt_stride(t.level) + kMqtShift + ((at + k) - c * per)];
    }
}

}  // namespace rtpg

using namespace rtpg;

struct rtpg_mqt {
    MqtDev dev{};
    float* staging = nullptr;  // of exports: kExportFloats, or all there are
    std::vector<void*> allocs;
    size_t bytes = 0;
    template <class T>
    int alloc(T** p, size_t count) {
        void* q = nullptr;
        cudaError_t e = cudaMalloc(&q, count * sizeof(T));
        if (e != cudaSuccess) {
            cudaGetLastError();
            return fail(RTPG_ENOMEM, "cudaMalloc(%zu bytes) failed: %s", count * sizeof(T), cudaGetErrorString(e));
        }
        allocs.push_back(q);
        bytes += count * sizeof(T);
        *p = static_cast<T*>(q);
        return RTPG_OK;
    }
    ~rtpg_mqt() {
        for (void* p : allocs) cudaFree(p);
    }
};

extern "C" {

// RTMortonQuadTreeWrapperT(ctx, maxHashSize, maxTreeLevel, fraction) + Allocate (MO.h:597-638)
int rtpg_mqt_create(uint32_t num_cells, uint32_t level, float fraction, int32_t fixed_point_bits, rtpg_mqt** out) {
    if (!out || num_cells == 0) return fail(RTPG_EINVAL, "rtpg_mqt_create: bad arguments");
    if (level < 1 || level > kMqtMaxLevel) return fail(RTPG_EINVAL, "rtpg_mqt_create: level must be in [1, %u]", kMqtMaxLevel);
    if (fixed_point_bits == 0) fixed_point_bits = 24;
    if (fixed_point_bits < 0 || fixed_point_bits > 40) return fail(RTPG_EINVAL, "rtpg_mqt_create: fixed_point_bits in [0,40]");
    auto* h = new (std::nothrow) rtpg_mqt();
    if (!h) return fail(RTPG_ENOMEM, "rtpg_mqt_create: out of host memory");
    MqtDev& t = h->dev;
    t.ncells = num_cells;
    t.level = level;
    t.fraction = fraction;
    t.touched_shift = mqt_touched_shift(num_cells);
    t.fx.scale = ldexpf(1.0f, fixed_point_bits);
    t.fx.inv_scale = ldexpf(1.0f, -fixed_point_bits);
    const size_t nleaf = (size_t)num_cells << (2 * level), npyr = (size_t)num_cells * mqt_stride(level);
    int r;
    if ((r = h->alloc(&t.leaves, nleaf)) || (r = h->alloc(&t.pyramid, npyr)) || (r = h->alloc(&t.status, 1)) ||
        (r = h->alloc(&t.touched, (size_t)num_cells << t.touched_shift)) || (r = h->alloc(&t.live, num_cells)) ||
        (r = h->alloc(&h->staging, std::min<size_t>(kExportFloats, (size_t)num_cells * mqt_level_offset(level + 1))))) {
        delete h;
        return r;
    }
    if (cudaMemset(t.leaves, 0, nleaf * 8) != cudaSuccess || cudaMemset(t.pyramid, 0, npyr * 4) != cudaSuccess ||
        cudaMemset(t.status, 0, 4) != cudaSuccess || cudaMemset(t.touched, 0, (size_t)num_cells << t.touched_shift) != cudaSuccess ||
        cudaMemset(t.live, 0, num_cells) != cudaSuccess) {
        delete h;
        return fail(RTPG_ECUDA, "rtpg_mqt_create: memset failed");
    }
    const cudaError_t e = cudaFuncSetAttribute(k_mqt_record_private, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                               int(kRecPrivLeaves * 8));
    if (e != cudaSuccess) {
        delete h;
        return fail(RTPG_ECUDA, "cudaFuncSetAttribute: %s", cudaGetErrorString(e));
    }
    *out = h;
    return RTPG_OK;
}

int rtpg_mqt_destroy(rtpg_mqt* h) {
    if (!h) return fail(RTPG_EINVAL, "rtpg_mqt_destroy: null handle");
    delete h;
    return RTPG_OK;
}

// RTMortonQuadTreeWrapperT::Allocate on an existing wrapper: zero both buffers (MO.h:618-637)
int rtpg_mqt_clear(rtpg_mqt* h, void* stream) {
    if (!h) return fail(RTPG_EINVAL, "rtpg_mqt_clear: null handle");
    cudaStream_t st = as_stream(stream);
    const MqtDev& t = h->dev;
    RTPG_CUDA(cudaMemsetAsync(t.leaves, 0, ((size_t)t.ncells << (2 * t.level)) * 8, st));
    RTPG_CUDA(cudaMemsetAsync(t.pyramid, 0, (size_t)t.ncells * mqt_stride(t.level) * 4, st));
    RTPG_CUDA(cudaMemsetAsync(t.touched, 0, (size_t)t.ncells << t.touched_shift, st));
    RTPG_CUDA(cudaMemsetAsync(t.live, 0, t.ncells, st));
    RTPG_CUDA(cudaMemsetAsync(t.status, 0, 4, st));
    return RTPG_OK;
}

// MortonQuadTreeWrapperT::Record (MO.h:477-484): cell UINT32_MAX is skipped.
int rtpg_mqt_record(rtpg_mqt* h, int64_t n, const uint32_t* cell, const float* dir, int dir_is_canonical,
                    const float* value, void* stream) {
    if (!h) return fail(RTPG_EINVAL, "rtpg_mqt_record: null handle");
    if (n < 0 || (n > 0 && (!cell || !dir || !value))) return fail(RTPG_EINVAL, "rtpg_mqt_record: bad arguments");
    if (dir_is_canonical && !aligned8(dir)) return fail(RTPG_EINVAL, "rtpg_mqt_record: misaligned float2 array");
    if (n == 0) return RTPG_OK;
    const MqtDev& t = h->dev;
    cudaStream_t st = as_stream(stream);
    // private sums on so many CTAs that flushing them takes at most half as many adds as there
    // are records; below sixteen records per leaf there is little to gather
    const uint64_t nleaf = (uint64_t)t.ncells << (2 * t.level);
    if (nleaf <= kRecPrivLeaves && (int64_t)(16 * nleaf) <= n)
        k_mqt_record_private<<<(int)std::min<int64_t>(kSMs, n / (int64_t)(2 * nleaf)), kRecThreads, nleaf * 8, st>>>(
            t, n, cell, dir, dir_is_canonical, value, (uint32_t)nleaf);
    else
        k_mqt_record<<<grid_for(n, kRecThreads, 2), kRecThreads, 0, st>>>(t, n, cell, dir, dir_is_canonical, value);
    RTPG_LAUNCH_CHECK();
    return RTPG_OK;
}

// Update + mortonBuildKernel: building leaves -> sampling pyramid, building cleared.
int rtpg_mqt_update(rtpg_mqt* h, void* stream) {
    if (!h) return fail(RTPG_EINVAL, "rtpg_mqt_update: null handle");
    const MqtDev& t = h->dev;
    cudaStream_t st = as_stream(stream);
    // warps of `cells` cells each, at most one resident wave of 8 CTAs per SM
    auto grid = [&](uint32_t cells) {
        const uint32_t per = cells * kMqtWarps;
        return (int)std::min<uint32_t>(t.ncells / per + (t.ncells % per != 0), kSMs * 8);
    };
    const int block = 32 * kMqtWarps, gb = (int)std::min<uint32_t>(t.ncells, kSMs * 8);
    switch (t.level) {
        case 1: k_mqt_build_small<1><<<grid(32), block, 0, st>>>(t); break;
        case 2: k_mqt_build_small<2><<<grid(8), block, 0, st>>>(t); break;
        case 3: k_mqt_build_small<3><<<grid(2), block, 0, st>>>(t); break;
        case 4: k_mqt_build_warp<4><<<grid(8), block, 0, st>>>(t); break;
        case 5: k_mqt_build_warp<5><<<grid(8), block, 0, st>>>(t); break;
        case 6: k_mqt_build_block<6><<<gb, 128, 0, st>>>(t); break;
        default: k_mqt_build_block<7><<<gb, 512, 0, st>>>(t); break;
    }
    RTPG_LAUNCH_CHECK();
    return RTPG_OK;
}

// MortonQuadTreeWrapperT::SampleAndPdf (MO.h:486-500); out_pdf includes the 1/(4 pi) factor,
// out_pdf_tree is MortonQuadTreeT::SampleAndPdf's pdf (MO.h:286-344).
int rtpg_mqt_sample_pdf(rtpg_mqt* h, int64_t n, const uint32_t* cell, const uint32_t* seeds, uint32_t seed_base,
                        float* out_uv, float* out_pdf, float* out_dir, float* out_pdf_tree, void* stream) {
    if (!h) return fail(RTPG_EINVAL, "rtpg_mqt_sample_pdf: null handle");
    if (n < 0 || (n > 0 && !cell)) return fail(RTPG_EINVAL, "rtpg_mqt_sample_pdf: bad arguments");
    if (!aligned8(out_uv)) return fail(RTPG_EINVAL, "rtpg_mqt_sample_pdf: misaligned float2 array");
    if (n == 0) return RTPG_OK;
    const MqtSampleOut o{out_uv, out_pdf, out_dir, out_pdf_tree};
    k_mqt_sample<<<grid_for(n, 256, 8), 256, 0, as_stream(stream)>>>(h->dev, n, cell, seeds, seed_base, o);
    RTPG_LAUNCH_CHECK();
    return RTPG_OK;
}

// MortonQuadTreeWrapperT::Pdf (MO.h:515-524) or, tree_level = 1, MortonQuadTreeT::Pdf (:401-414).
int rtpg_mqt_pdf(rtpg_mqt* h, int64_t n, const uint32_t* cell, const float* dir, int dir_is_canonical, float* out,
                 int tree_level, void* stream) {
    if (!h) return fail(RTPG_EINVAL, "rtpg_mqt_pdf: null handle");
    if (n < 0 || (n > 0 && (!cell || !dir || !out))) return fail(RTPG_EINVAL, "rtpg_mqt_pdf: bad arguments");
    if (dir_is_canonical && !aligned8(dir)) return fail(RTPG_EINVAL, "rtpg_mqt_pdf: misaligned float2 array");
    if (n == 0) return RTPG_OK;
    k_mqt_pdf<<<grid_for(n, 256, 8), 256, 0, as_stream(stream)>>>(h->dev, n, cell, dir, dir_is_canonical, out, tree_level);
    RTPG_LAUNCH_CHECK();
    return RTPG_OK;
}

int rtpg_mqt_export(rtpg_mqt* h, int64_t* host_leaves, float* host_pyramid, void* stream) {
    if (!h) return fail(RTPG_EINVAL, "rtpg_mqt_export: null handle");
    cudaStream_t st = as_stream(stream);
    const MqtDev& t = h->dev;
    if (host_leaves)
        RTPG_CUDA(cudaMemcpyAsync(host_leaves, t.leaves, ((size_t)t.ncells << (2 * t.level)) * 8, cudaMemcpyDeviceToHost, st));
    if (host_pyramid) {
        const uint64_t n = (uint64_t)t.ncells * mqt_level_offset(t.level + 1);
        for (uint64_t at = 0; at < n; at += kExportFloats) {
            const uint32_t m = (uint32_t)std::min<uint64_t>(kExportFloats, n - at);
            k_mqt_pack<<<grid_for(m, 256, 8), 256, 0, st>>>(t, at, m, h->staging);
            RTPG_LAUNCH_CHECK();
            RTPG_CUDA(cudaMemcpyAsync(host_pyramid + at, h->staging, (size_t)m * 4, cudaMemcpyDeviceToHost, st));
        }
    }
    RTPG_CUDA(cudaStreamSynchronize(st));
    return RTPG_OK;
}

int rtpg_mqt_status(rtpg_mqt* h, uint32_t* host_status, int clear, void* stream) {
    if (!h || !host_status) return fail(RTPG_EINVAL, "rtpg_mqt_status: null argument");
    cudaStream_t st = as_stream(stream);
    RTPG_CUDA(cudaMemcpyAsync(host_status, h->dev.status, 4, cudaMemcpyDeviceToHost, st));
    if (clear) RTPG_CUDA(cudaMemsetAsync(h->dev.status, 0, 4, st));
    RTPG_CUDA(cudaStreamSynchronize(st));
    return RTPG_OK;
}

}  // extern "C"

namespace rtpg {
MqtDev mqt_device_view(const rtpg_mqt* h) { return h->dev; }
}

// ================================================================== pass controller
// RTMortonQuadTreeControllerT (OPX7UtilsMorton.h:766-993): the doubling pass schedule of the
// hash-grid guide with a LOCATE phase.  BegTrace at Start clears both quadtree buffers
// (RTMortonQuadTreeWrapperT::Allocate); EndTrace after a finished pass beyond
// iteration_for_built runs Update + mortonBuildKernel (rtpg_mqt_update here).
struct rtpg_mqt_controller {
    rtpg_mqt* tree;
    uint32_t sample_for_budget, samples_per_launch, iteration_for_built, iteration_for_locate;
    float ratio_for_budget;
    bool start = false, executing = false;
    uint32_t per_all = 0, per_tmp = 0, remain = 0, pass = 0, iteration = 0;
    int32_t state = RTPG_MQT_TRACE_RECORD;
};

extern "C" {

int rtpg_mqt_controller_create(rtpg_mqt* tree, uint32_t sample_for_budget, uint32_t iteration_for_built,
                               uint32_t iteration_for_locate, float ratio_for_budget, uint32_t samples_per_launch,
                               rtpg_mqt_controller** out) {
    if (!tree || !out || samples_per_launch == 0) return fail(RTPG_EINVAL, "rtpg_mqt_controller_create: bad arguments");
    auto* c = new (std::nothrow) rtpg_mqt_controller();
    if (!c) return fail(RTPG_ENOMEM, "rtpg_mqt_controller_create: out of host memory");
    c->tree = tree;
    c->sample_for_budget = sample_for_budget;
    c->samples_per_launch = samples_per_launch;
    c->iteration_for_built = iteration_for_built;
    c->iteration_for_locate = iteration_for_locate;
    c->ratio_for_budget = ratio_for_budget;
    *out = c;
    return RTPG_OK;
}
int rtpg_mqt_controller_destroy(rtpg_mqt_controller* c) {
    if (!c) return fail(RTPG_EINVAL, "rtpg_mqt_controller_destroy: null handle");
    delete c;
    return RTPG_OK;
}
int rtpg_mqt_controller_start(rtpg_mqt_controller* c) {
    if (!c) return fail(RTPG_EINVAL, "rtpg_mqt_controller_start: null handle");
    c->start = true;
    return RTPG_OK;
}
// BegTrace (OPX7UtilsMorton.h:818-889)
int rtpg_mqt_controller_begin(rtpg_mqt_controller* c, void* stream) {
    if (!c) return fail(RTPG_EINVAL, "rtpg_mqt_controller_begin: null handle");
    if (c->start) {
        c->per_all = 0;
        c->per_tmp = 0;
        c->iteration = 0;
        c->start = false;
        c->executing = true;
        c->remain = ((c->sample_for_budget - 1 + c->samples_per_launch) / c->samples_per_launch) * c->samples_per_launch;
        c->pass = 0;
        c->state = RTPG_MQT_TRACE_RECORD;
        int r = rtpg_mqt_clear(c->tree, stream);
        if (r) return r;
    }
    if (!c->executing) return RTPG_OK;
    if (c->per_tmp == 0) {
        c->remain -= c->pass;
        c->pass = std::min<uint32_t>(c->remain, (1u << c->iteration) * c->samples_per_launch);
        if ((c->remain - c->pass < 2 * c->pass) ||
            (c->per_all >= c->ratio_for_budget * static_cast<float>(c->sample_for_budget)))
            c->pass = c->remain;
    }
    if (c->iteration > c->iteration_for_built)
        c->state = c->remain > c->pass ? RTPG_MQT_TRACE_RECORD_AND_SAMPLE : RTPG_MQT_TRACE_SAMPLE;
    else if (c->iteration > c->iteration_for_locate)
        c->state = RTPG_MQT_TRACE_RECORD;
    else
        c->state = RTPG_MQT_TRACE_LOCATE;
    return RTPG_OK;
}
// EndTrace (OPX7UtilsMorton.h:891-922)
int rtpg_mqt_controller_end(rtpg_mqt_controller* c, void* stream) {
    if (!c) return fail(RTPG_EINVAL, "rtpg_mqt_controller_end: null handle");
    if (!c->executing) return RTPG_OK;
    c->per_all += c->samples_per_launch;
    c->per_tmp += c->samples_per_launch;
    if (c->per_tmp >= c->pass) {
        c->iteration++;
        if (c->iteration > c->iteration_for_built) {
            int r = rtpg_mqt_update(c->tree, stream);
            if (r) return r;
        }
        c->per_tmp = 0;
    }
    if (c->per_all > c->sample_for_budget) {
        c->executing = false;
        c->per_all = 0;
    }
    return RTPG_OK;
}
int rtpg_mqt_controller_get(rtpg_mqt_controller* c, int32_t* state, uint32_t* iteration, uint32_t* samples_in_pass,
                            int32_t* executing) {
    if (!c) return fail(RTPG_EINVAL, "rtpg_mqt_controller_get: null handle");
    if (state) *state = c->state;
    if (iteration) *iteration = c->iteration;
    if (samples_in_pass) *samples_in_pass = c->per_tmp;
    if (executing) *executing = c->executing ? 1 : 0;
    return RTPG_OK;
}

}  // extern "C"
