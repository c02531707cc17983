// Device-side Morton quadtree routines (MortonQuadTreeT, OPX7UtilsMorton.h:253-449).
#pragma once
#include "common.cuh"
#include "canonical.cuh"

namespace rtpg {

// Deepest supported level (the build gives a cell of level 7 sixteen warps).  RTLib's configured
// maximum is 6 (OPX7/CMakeLists.txt:103).
constexpr uint32_t kMqtMaxLevel = 7;
constexpr double kInvPiD = 0.318309886183790691216444201927515678107738494873046875;

struct MqtDev {
    uint32_t ncells, level;
    float fraction;
    FixedPoint fx;
    unsigned long long* leaves;  // ncells * 4^L, building
    float* pyramid;              // ncells * mqt_stride(level), sampling
    // per cell: recorded into since the last build (its leaves may be nonzero); its pyramid may
    // be nonzero.  The build reads and writes only the cells that need it.  Cell c's first flag is
    // touched[c << touched_shift] (see mqt_touched_shift).
    uint8_t *touched, *live;
    uint32_t touched_shift;
    unsigned* status;
};

__host__ __device__ __forceinline__ uint32_t mqt_level_offset(uint32_t l) { return ((1u << (2 * l)) - 1u) / 3u; }
// Device layout of a cell's pyramid: the levels one after the other, shifted by three floats, so
// that the four children of a node are one aligned 16-byte vector ((4^l - 1) / 3 = 1 mod 4) and
// a cell starts on a 32-byte sector; root and first children share the first sector.
constexpr uint32_t kMqtShift = 3;
__host__ __device__ __forceinline__ uint32_t mqt_base(uint32_t l) { return mqt_level_offset(l) + kMqtShift; }
__host__ __device__ __forceinline__ uint32_t mqt_stride(uint32_t level) { return mqt_level_offset(level + 1) + kMqtShift; }

// MortonUtils::Part1By1_16 / Comp1By1_16 (OPX7UtilsMorton.h:41-89)
__device__ __forceinline__ uint32_t part1by1(uint32_t x) {
    x &= 0x0000FFFF;
    x = (x ^ (x << 8)) & 0x00FF00FF;
    x = (x ^ (x << 4)) & 0x0F0F0F0F;
    x = (x ^ (x << 2)) & 0x33333333;
    x = (x ^ (x << 1)) & 0x55555555;
    return x;
}
__device__ __forceinline__ uint32_t compact1by1(uint32_t x) {
    x &= 0x55555555;
    x = (x ^ (x >> 1)) & 0x33333333;
    x = (x ^ (x >> 2)) & 0x0F0F0F0F;
    x = (x ^ (x >> 4)) & 0x00FF00FF;
    x = (x ^ (x >> 8)) & 0x0000FFFF;
    return x;
}

// leaf Morton code of MortonQuadTreeT::Record (:267-270): uint(uv * 2^L) per axis, clamped
// to 2^L - 1 (uv == 1 would otherwise address past the level)
__device__ __forceinline__ uint32_t mqt_leaf_code(uint32_t level, float u, float v) {
    const float nn = (float)(1u << level);
    const uint32_t maxi = (1u << level) - 1u;
    uint32_t px = __float2uint_rz(__fmul_rn(u, nn)), py = __float2uint_rz(__fmul_rn(v, nn));
    px = px > maxi ? maxi : px;
    py = py > maxi ? maxi : py;
    return (part1by1(py) << 1) + part1by1(px);
}

__device__ __forceinline__ float2 dir_to_canonical_mqt(float x, float y, float z) { return dir_to_canonical(x, y, z); }
__device__ __forceinline__ float3 canonical_to_dir_mqt(float u, float v) { return canonical_to_dir(u, v); }

// One level of MortonQuadTreeT::SampleAndPdf (:286-344), float order as written: the quadrant a
// draw selects among the sums q of a node with sum `total`.
__device__ __forceinline__ uint32_t mqt_choose_exact(float4 q, float total, float draw) {
    const float partial_l = __fadd_rn(q.x, q.z);
    const float boundary = __fdiv_rn(partial_l, total);
    const bool right = !(draw < boundary);
    const float partial = right ? __fadd_rn(q.y, q.w) : partial_l;
    const float sample = __fdiv_rn(right ? __fsub_rn(draw, boundary) : draw,
                                   right ? __fsub_rn(1.0f, boundary) : boundary);
    return (right ? 1u : 0u) | (sample >= __fdiv_rn(right ? q.y : q.x, partial) ? 2u : 0u);
}
// The same choice without its three divisions wherever they cannot matter: the boundary is
// approximated (2 ulp of at most 1: 2.4e-7) and the second comparison num / den >= c / partial is
// taken as num * partial >= c * den.  num and den are then off by at most 4e-7 each, c <= partial
// up to rounding, and the rounded quotients by 2^-24 relative each, so the products differ by at
// most 1.1e-6 * partial from what decides.  Closer calls (about two draws in a million), and every
// comparison that a zero or non-finite sum makes unordered, take the divisions.
__device__ __forceinline__ uint32_t mqt_choose(float4 q, float total, float draw) {
    const float partial_l = __fadd_rn(q.x, q.z);
    const float b = __fdividef(partial_l, total);
    const float off = __fsub_rn(draw, b);
    const bool right = off >= 0.0f;
    const float partial = right ? __fadd_rn(q.y, q.w) : partial_l;
    const float num = right ? off : draw, den = right ? __fsub_rn(1.0f, b) : b;
    const float d = __fsub_rn(__fmul_rn(num, partial), __fmul_rn(right ? q.y : q.x, den));
    if (fabsf(off) > 1e-6f && fabsf(d) > __fmul_rn(2e-6f, partial)) return (right ? 1u : 0u) | (d >= 0.0f ? 2u : 0u);
    return mqt_choose_exact(q, total, draw);
}

// MortonQuadTreeT::SampleAndPdf (:286-344)
// A cell outside [0, ncells) (UINT32_MAX marks a hash-grid miss) samples like an empty
// tree: uniform with pdf 1 (RTLib reads out of bounds there).
__device__ __forceinline__ float2 mqt_sample_and_pdf(const MqtDev& t, uint32_t cell, uint32_t& rng, float& pdf) {
    const float* w = t.pyramid + (size_t)(cell < t.ncells ? cell : 0u) * mqt_stride(t.level);
    const float root = cell < t.ncells ? w[mqt_base(0)] : 0.0f;
    if (root <= 0.0f) {
        const float a = rnd1(rng);
        const float b = rnd1(rng);
        pdf = 1.0f;
        return make_float2(a, b);
    }
    float total = root;
    uint32_t size = 4, offset = mqt_base(1), code = 0;
    for (uint32_t l = 0; l < t.level; ++l) {
        const float4 q = *reinterpret_cast<const float4*>(w + offset + (code << 2));
        const uint32_t cl = mqt_choose(q, total, rnd1(rng));
        total = cl == 0 ? q.x : (cl == 1 ? q.y : (cl == 2 ? q.z : q.w));
        code = (code << 2) + cl;
        offset += size;
        size *= 4;
    }
    // division by 2^L as the exact product with its reciprocal
    const float inv = __uint_as_float((127u - t.level) << 23);
    const uint32_t xi = compact1by1(code), yi = compact1by1(code >> 1);
    const float rx = rnd1(rng);
    const float px = __fmul_rn(__fadd_rn((float)xi, rx), inv);
    const float ry = rnd1(rng);
    const float py = __fmul_rn(__fadd_rn((float)yi, ry), inv);
    pdf = __fmul_rn(__fdiv_rn(total, root), (float)(1u << (2 * t.level)));
    return make_float2(px, py);
}

// Marks cell c as touched unless `tag`, its entry of a direct-mapped table of cells the CTA has
// marked (shared memory, UINT32_MAX: none), says that was done.  Any lane's entry will do.
__device__ __forceinline__ void mqt_mark(const MqtDev& t, uint32_t c, volatile uint32_t* tag) {
    if (*tag == c) return;
    *tag = c;
    t.touched[size_t(c) << t.touched_shift] = 1;
}
// Flags that many CTAs mark lie apart, up to a sector each, while they fit 1 MB: stores to one line queue up
// in L2.  2 x 10^5 / 10^6 / 4 x 10^6 records into 4096 cells of 4^4 leaves: 23.1 / 84 / 171 us with the flags side
// by side (17.1 / 64 / 243 when records were aggregated by warps and not marked), 8.8 / 23.1 / 49.7 now.
inline uint32_t mqt_touched_shift(uint32_t ncells) {
    uint32_t s = 0;
    while (s < 5 && (uint64_t)ncells << (s + 1) <= 1u << 20) ++s;
    return s;
}

// MortonQuadTreeT::Pdf (:401-414)
__device__ __forceinline__ float mqt_pdf(const MqtDev& t, uint32_t cell, float u, float v) {
    if (cell >= t.ncells) return 1.0f;
    const float* w = t.pyramid + (size_t)cell * mqt_stride(t.level);
    const float root = w[mqt_base(0)];
    if (root <= 0.0f) return 1.0f;
    const float nn = (float)(1u << t.level);
    const uint32_t idx = mqt_base(t.level) + mqt_leaf_code(t.level, u, v);
    return __fmul_rn(__fmul_rn(__fdiv_rn(w[idx], root), nn), nn);
}

}  // namespace rtpg
