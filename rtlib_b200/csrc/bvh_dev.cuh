// Triangle BVH for closest-hit / any-hit queries (the part RTLib delegates to OptiX:
// TraceRadiance / TraceOccluded, SimpleKernel.h:347-366).  Two hierarchies over the same
// triangles:
//   - a binary linear BVH: 63-bit Morton codes of the triangle centroids, radix-sorted, hierarchy
//     by Karras' split search, boxes by a bottom-up pass.  It defines which triangle a query
//     reports: a leaf's box must pass box_hit, and of triangles at exactly the same distance
//     the one a near-first walk of this hierarchy meets first wins;
//   - the hierarchy that rays walk: eight children per node, their boxes quantised to eight bits
//     per plane (see WideNode), collapsed from a binary hierarchy that clustering builds (k_ploc_*).
#pragma once
#include "common.cuh"

namespace rtpg {

constexpr uint32_t kBvhLeafBit = 0x80000000u;

struct __align__(16) BvhNode {
    float4 a;  // c0.lo.xyz, c0.hi.x
    float4 b;  // c0.hi.yz, c1.lo.xy
    float4 c;  // c1.lo.z, c1.hi.xyz
    uint32_t child[2];  // kBvhLeafBit | leaf index, or interior node index
    uint32_t pad[2];
};

// A triangle as the affine map of world space onto its own frame (Baldwin and Weber, "Fast
// Ray-Triangle Intersections by Coordinate Transformation", JCGT 5(3), 2016): a point x has
// barycentric coordinates u = dot(r0.xyz, x) + r0.w and v = dot(r1.xyz, x) + r1.w, and
// dot(r2.xyz, x) + r2.w is its offset along the face normal in units of the normal's length.
// tri_transform forms the rows in double precision from the vertices, once per scene.
struct __align__(16) BvhTri {
    float4 r0, r1, r2;
};

// The rows of triangle (a, b, c): with e1 = b - a, e2 = c - a, n = e1 x e2, the inverse of the
// matrix [e1 e2 n] is [e2 x n; n x e1; n] / |n|^2, translated by -a.  Every operation is a
// double operation rounded as written (the file is built without contraction), then the rows
// are rounded to float: the CPU restatement forms them the same way, bit for bit.
__host__ __device__ inline void tri_transform(float ax_, float ay_, float az_, float bx_, float by_, float bz_, float cx_,
                                              float cy_, float cz_, float4* r) {
    const double ax = ax_, ay = ay_, az = az_;
    const double e1x = (double)bx_ - ax, e1y = (double)by_ - ay, e1z = (double)bz_ - az;
    const double e2x = (double)cx_ - ax, e2y = (double)cy_ - ay, e2z = (double)cz_ - az;
    const double nx = e1y * e2z - e1z * e2y, ny = e1z * e2x - e1x * e2z, nz = e1x * e2y - e1y * e2x;
    const double nn = nx * nx + ny * ny + nz * nz;
    const double m[3][3] = {{e2y * nz - e2z * ny, e2z * nx - e2x * nz, e2x * ny - e2y * nx},
                            {ny * e1z - nz * e1y, nz * e1x - nx * e1z, nx * e1y - ny * e1x},
                            {nx, ny, nz}};
    for (int k = 0; k < 3; ++k) {
        const double w = -(m[k][0] * ax + m[k][1] * ay + m[k][2] * az);
        r[k] = make_float4((float)(m[k][0] / nn), (float)(m[k][1] / nn), (float)(m[k][2] / nn), (float)(w / nn));
    }
}

// Scenes of at most kFlatTris triangles are also kept as a flat list in their own order and
// traced by testing every triangle: all lanes of a warp then run the same loop over the same
// triangle (one broadcast load per triangle), where the BVH walk leaves most lanes idle, and the
// lowest index wins a tie of equal distances, as in a brute-force test.  The list holds pairs:
// triangle 2k in the low and 2k + 1 in the high word of every row element, the operands of packed
// fused multiply-adds.  An odd list ends with a triangle that is never hit.
constexpr uint32_t kFlatTris = 64;
struct __align__(16) FlatPair {
    unsigned long long r0[4], r1[4], r2[4];
};
__host__ __device__ constexpr uint32_t flat_pairs(uint32_t n) { return (n + 1) / 2; }

// A node of the walked hierarchy, after Ylitie, Karras and Laine, "Efficient Incoherent Ray
// Traversal on GPUs Through Compressed Wide BVHs" (HPG 2017): up to eight children in slots that
// follow the octants of the node, so that visiting slot (k xor octant) for descending k is about
// front to back for every ray octant, without sorting.  96 bytes = three 32-byte loads.
//   org, step  planes of axis a: a lower one at org[a] + (q - kPlaneMargin) * step[a], an upper one at
//              org[a] + (q + kPlaneMargin) * step[a]; q = 0 and 255 lie on the node's own box, so that walls
//              there stay thin
//   imask      slots that hold interior children, stored one after the other from child_base in
//              slot order
//   lmask      slots that hold a triangle, stored one after the other from tri_base in slot order
//   qlo, qhi   per axis and slot, rounded outwards
// A leaf is one triangle: more of them per leaf cost more tests than they save nodes (closest hits
// of 2^20 rays in 1.05 M triangles: 1493 us with one, 1492 with two, 1596 with three).
// With steps that are powers of two and planes rounded outwards by up to a step, a wall of a node's box was
// a slab as thick as two steps, entered by every ray that starts or ends on it: next event estimation in Cornell
// boxes whose light is 32 / 512 / 2048 triangles took 1-6 % longer than with two exact boxes a node (1280 x 720,
// 8 samples: 8.63 / 9.31 / 10.40 ms): 8.81 / 9.61 / 11.04 then, 8.46 / 9.11 / 10.53 now.
constexpr float kPlaneMargin = 0.03125f;
struct __align__(32) WideNode {
    float org[3];
    uint32_t imask, child_base, tri_base, lmask, pad0;
    uint8_t qlo[3][8], qhi[3][8];
    float step[3];
    uint32_t pad1;
};
static_assert(sizeof(WideNode) == 96, "three 32-byte sectors");
// A leaf triangle of the walked hierarchy: its rows, its leaf in the binary hierarchy and its scene
// index.  64 bytes = two 32-byte loads.
struct __align__(32) WideTri {
    BvhTri tr;
    uint32_t leaf, prim, pad[2];
};
static_assert(sizeof(WideTri) == 64, "two 32-byte sectors");
constexpr int kWideStack = 64;  // the build keeps the hierarchy shallower (k_wide_level)

struct SceneDev {
    const BvhNode* nodes;   // n - 1 interior nodes of the binary hierarchy (root 0)
    const float4* leaf_box; // per leaf of it: (lo.xyz, hi.x), (hi.yz, -, -)
    const WideNode* wide;   // null for scenes traced as a flat list
    const WideTri* wtris;
    const FlatPair* flat;   // n <= kFlatTris: the triangles in scene order, else null
    uint32_t ntris;
    float max_abs;          // largest absolute coordinate of the leaf boxes
};

struct Hit {
    float t, u, v;
    uint32_t prim;  // 0xffffffff: miss
};

// Slab test with the ray's origin pre-scaled (oix = ox * ix, ...): each slab distance is one
// fused multiply-add, lo * ix - ox * ix with a single rounding.  The test of a leaf's box is part of
// what a query reports (see the top of the file); rounding is monotonic, so whatever box
// contains a box that passes passes too.
__device__ __forceinline__ bool box_hit(float lox, float loy, float loz, float hix, float hiy, float hiz, float oix,
                                        float oiy, float oiz, float ix, float iy, float iz, float tmin, float tmax,
                                        float& tnear) {
    const float tx0 = __fmaf_rn(lox, ix, -oix), tx1 = __fmaf_rn(hix, ix, -oix);
    const float ty0 = __fmaf_rn(loy, iy, -oiy), ty1 = __fmaf_rn(hiy, iy, -oiy);
    const float tz0 = __fmaf_rn(loz, iz, -oiz), tz1 = __fmaf_rn(hiz, iz, -oiz);
    const float t0 = fmaxf(fmaxf(fminf(tx0, tx1), fminf(ty0, ty1)), fmaxf(fminf(tz0, tz1), tmin));
    const float t1 = fminf(fminf(fmaxf(tx0, tx1), fmaxf(ty0, ty1)), fminf(fmaxf(tz0, tz1), tmax));
    tnear = t0;
    return t0 <= t1;
}

// The hit of ray o + t d on triangle tr: the ray meets the triangle's plane at
// t = -(dot(r2.xyz, o) + r2.w) / dot(r2.xyz, d), where u and v follow as o's coordinates plus
// t times d's.  Each dot product is a chain of fused multiply-adds and 1 / den the correctly
// rounded reciprocal, so the CPU restatement (fmaf, 1.0f / den) reproduces every value; the
// test runs without a branch, as every lane of a warp tests the same triangle.  Returns t in
// (tmin, tmax) or a negative value (also for a ray parallel to the plane: t is then infinite
// or NaN).
__device__ __forceinline__ float tri_hit(const BvhTri& tr, float ox, float oy, float oz, float dx, float dy, float dz,
                                         float tmin, float tmax, float& u, float& v) {
    const float den = __fmaf_rn(tr.r2.x, dx, __fmaf_rn(tr.r2.y, dy, __fmul_rn(tr.r2.z, dz)));
    const float num = __fmaf_rn(tr.r2.x, ox, __fmaf_rn(tr.r2.y, oy, __fmaf_rn(tr.r2.z, oz, tr.r2.w)));
    const float t = __fmul_rn(-num, __frcp_rn(den));
    const float ud = __fmaf_rn(tr.r0.x, dx, __fmaf_rn(tr.r0.y, dy, __fmul_rn(tr.r0.z, dz)));
    const float uo = __fmaf_rn(tr.r0.x, ox, __fmaf_rn(tr.r0.y, oy, __fmaf_rn(tr.r0.z, oz, tr.r0.w)));
    const float vd = __fmaf_rn(tr.r1.x, dx, __fmaf_rn(tr.r1.y, dy, __fmul_rn(tr.r1.z, dz)));
    const float vo = __fmaf_rn(tr.r1.x, ox, __fmaf_rn(tr.r1.y, oy, __fmaf_rn(tr.r1.z, oz, tr.r1.w)));
    u = __fmaf_rn(t, ud, uo);
    v = __fmaf_rn(t, vd, vo);
    const bool hit = (t > tmin) & (t < tmax) & (u >= 0.0f) & (v >= 0.0f) & (__fadd_rn(u, v) <= 1.0f);
    return hit ? t : -1.0f;
}

// two floats as one operand of the packed instructions: each word rounds as the scalar operation
__device__ __forceinline__ unsigned long long pack2(float a, float b) {
    unsigned long long r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ float2 unpack2(unsigned long long v) {
    float2 r;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
    return r;
}
__device__ __forceinline__ unsigned long long fma2(unsigned long long a, unsigned long long b, unsigned long long c) {
    unsigned long long r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
__device__ __forceinline__ unsigned long long mul2(unsigned long long a, unsigned long long b) {
    unsigned long long r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ unsigned long long add2(unsigned long long a, unsigned long long b) {
    unsigned long long r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ float min3_nan(float a, float b, float c) {  // NaN if any is
    float r;
    asm("min.NaN.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
    return r;
}

// closest hit (ANY = false) or any hit (ANY = true) in (tmin, tmax) by testing every triangle
// of a small scene (npairs pairs in scene order).  tri_hit's operations, two triangles at a time: the
// same roundings, half the multiply-adds to issue.  u >= 0, v >= 0 and u + v <= 1 are one comparison
// of the least of u, v and 1 - (u + v), whose sign is exact.  k_bounce of the guided Cornell render
// (36 triangles, 512 launches at 512 x 512): 25.0 -> 22.1 ms; unrolled by 1, 3, 4: 24.9, 22.4, 22.6.
// LANES > 1: that many neighbouring lanes hold the same ray and test every LANES-th pair each; all of
// them return the hit.  The pairs come from memory then (the constant bank serves one address at a
// time).
template <bool ANY, int LANES = 1>
__device__ __forceinline__ Hit flat_trace(const FlatPair* pairs, uint32_t npairs, float ox, float oy, float oz, float dx,
                                          float dy, float dz, float tmin, float tmax) {
    Hit h;
    h.t = tmax;
    h.prim = 0xffffffffu;
    h.u = h.v = 0.0f;
    const unsigned long long px = pack2(ox, ox), py = pack2(oy, oy), pz = pack2(oz, oz);
    const unsigned long long qx = pack2(dx, dx), qy = pack2(dy, dy), qz = pack2(dz, dz);
    const unsigned long long one = pack2(1.0f, 1.0f), minus = pack2(-1.0f, -1.0f);
#pragma unroll 2
    for (uint32_t k = LANES > 1 ? threadIdx.x % LANES : 0; k < npairs; k += LANES) {
        const FlatPair& p = pairs[k];
        const float2 den = unpack2(fma2(p.r2[0], qx, fma2(p.r2[1], qy, mul2(p.r2[2], qz))));
        const float2 num = unpack2(fma2(p.r2[0], px, fma2(p.r2[1], py, fma2(p.r2[2], pz, p.r2[3]))));
        const unsigned long long ud = fma2(p.r0[0], qx, fma2(p.r0[1], qy, mul2(p.r0[2], qz)));
        const unsigned long long uo = fma2(p.r0[0], px, fma2(p.r0[1], py, fma2(p.r0[2], pz, p.r0[3])));
        const unsigned long long vd = fma2(p.r1[0], qx, fma2(p.r1[1], qy, mul2(p.r1[2], qz)));
        const unsigned long long vo = fma2(p.r1[0], px, fma2(p.r1[1], py, fma2(p.r1[2], pz, p.r1[3])));
        const float ta = __fmul_rn(-num.x, __frcp_rn(den.x)), tb = __fmul_rn(-num.y, __frcp_rn(den.y));
        const unsigned long long t2 = pack2(ta, tb);
        const unsigned long long u2 = fma2(t2, ud, uo), v2 = fma2(t2, vd, vo);
        const float2 w = unpack2(fma2(add2(u2, v2), minus, one));
        const float2 u = unpack2(u2), v = unpack2(v2);
        const bool ina = min3_nan(u.x, v.x, w.x) >= 0.0f, inb = min3_nan(u.y, v.y, w.y) >= 0.0f;
        if (ina & (ta > tmin) & (ta < h.t) & (ta > 0.0f)) {
            h.t = ta;
            h.u = u.x;
            h.v = v.x;
            h.prim = 2 * k;
            if (ANY) break;
        }
        if (inb & (tb > tmin) & (tb < h.t) & (tb > 0.0f)) {
            h.t = tb;
            h.u = u.y;
            h.v = v.y;
            h.prim = 2 * k + 1;
            if (ANY) break;
        }
    }
    const uint32_t group = ((1u << (LANES % 32)) - 1u) << (threadIdx.x % 32 / LANES * LANES);
#pragma unroll
    for (int o = 1; o < LANES; o *= 2) {  // the nearest, of equal distances the lowest index
        const float t = __shfl_xor_sync(group, h.t, o), u = __shfl_xor_sync(group, h.u, o), v = __shfl_xor_sync(group, h.v, o);
        const uint32_t prim = __shfl_xor_sync(group, h.prim, o);
        if (t < h.t || (t == h.t && prim < h.prim)) h = Hit{t, u, v, prim};
    }
    return h;
}

// whether the box test of the binary hierarchy lets the ray reach leaf `leaf`
struct RayInv {
    float ix, iy, iz;
    __device__ __forceinline__ RayInv(float dx, float dy, float dz)
        : ix(1.0f / (fabsf(dx) > 1e-30f ? dx : copysignf(1e-30f, dx))),
          iy(1.0f / (fabsf(dy) > 1e-30f ? dy : copysignf(1e-30f, dy))),
          iz(1.0f / (fabsf(dz) > 1e-30f ? dz : copysignf(1e-30f, dz))) {}
};
__device__ __forceinline__ bool leaf_reached(const SceneDev& s, uint32_t leaf, float ox, float oy, float oz,
                                             const RayInv& r, float tmin, float tmax) {
    const float4 a = s.leaf_box[2 * size_t(leaf)], b = s.leaf_box[2 * size_t(leaf) + 1];
    float t0;
    return box_hit(a.x, a.y, a.z, a.w, b.x, b.y, ox * r.ix, oy * r.iy, oz * r.iz, r.ix, r.iy, r.iz, tmin, tmax, t0);
}
// Whether a near-first walk of the binary hierarchy meets leaf a before leaf b: decided at the
// node where their ways part.  A node's left child ends at the leaf its index names.
static __device__ __noinline__ bool meets_first(const BvhNode* nodes, uint32_t a, uint32_t b, float ox, float oy, float oz,
                                                RayInv r, float tmin, float tmax) {
    const uint32_t lo = min(a, b), hi = max(a, b);
    uint32_t cur = 0;
    for (;;) {
        const BvhNode nd = nodes[cur];
        const uint32_t split = nd.child[0] & ~kBvhLeafBit;
        if (hi <= split) {
            cur = nd.child[0];
        } else if (lo > split) {
            cur = nd.child[1];
        } else {
            const float oix = ox * r.ix, oiy = oy * r.iy, oiz = oz * r.iz;
            float t0, t1;
            box_hit(nd.a.x, nd.a.y, nd.a.z, nd.a.w, nd.b.x, nd.b.y, oix, oiy, oiz, r.ix, r.iy, r.iz, tmin, tmax, t0);
            box_hit(nd.b.z, nd.b.w, nd.c.x, nd.c.y, nd.c.z, nd.c.w, oix, oiy, oiz, r.ix, r.iy, r.iz, tmin, tmax, t1);
            return (t0 <= t1) == (a <= split);
        }
    }
}

__device__ __forceinline__ void ld32(const void* p, uint32_t* v) {
    asm("ld.global.nc.v8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
        : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7])
        : "l"(p));
}
// byte j of w as the float 32768 + byte, in one instruction (a conversion would go to the
// quarter-rate unit, 48 times a node)
template <int J>
__device__ __forceinline__ float plane(uint32_t w) {
    return __uint_as_float(__byte_perm(w, 0x47000000u, 0x7604u | (J << 4)));
}

// What a walk needs of its ray: reciprocal directions, and the origin's products with them widened
// by what rounding can do.  Whatever leaf box passes box_hit must not be lost to a quantised box
// around it: box_hit's slab distances are off by at most 2^-23 (|o| + |plane|) |1/d|, the ones
// here by as much again, so planes are moved apart by 2^-21 (|o| + max_abs), (a ten-thousandth
// of a millimetre per metre of scene).  Forming 32768 + q and the products with the step adds less than
// 2^-7 of a quantisation step, which kPlaneMargin covers.
struct WideRay {
    RayInv inv;
    float px, py, pz, ex, ey, ez;  // origin product, widening
    uint32_t octinv;               // 7 - octant: bit a set where the direction is positive
    __device__ __forceinline__ WideRay(const SceneDev& s, float ox, float oy, float oz, float dx, float dy, float dz)
        : inv(dx, dy, dz) {
        ex = 0x1p-21f * (fabsf(ox) + s.max_abs) * fabsf(inv.ix);
        ey = 0x1p-21f * (fabsf(oy) + s.max_abs) * fabsf(inv.iy);
        ez = 0x1p-21f * (fabsf(oz) + s.max_abs) * fabsf(inv.iz);
        px = ox * inv.ix; py = oy * inv.iy; pz = oz * inv.iz;
        octinv = (inv.ix < 0.0f ? 0u : 1u) | (inv.iy < 0.0f ? 0u : 2u) | (inv.iz < 0.0f ? 0u : 4u);
    }
};

__device__ __forceinline__ float max3(float a, float b, float c) {
    float r;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
    return r;
}
__device__ __forceinline__ float min3(float a, float b, float c) {
    float r;
    asm("min.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
    return r;
}
// Slots of the node's children whose box the ray may hit in [tmin, tmax]; v: the node.  The mask is summed in the mantissa of a float, off the integer pipe that the byte
// permutes and the min / max keep busy.
__device__ __forceinline__ uint32_t wide_hits(const WideRay& r, const uint32_t* v, float tmin, float tmax) {
    const float px = __uint_as_float(v[0]), py = __uint_as_float(v[1]), pz = __uint_as_float(v[2]);
    const float sx = __uint_as_float(v[20]) * r.inv.ix, sy = __uint_as_float(v[21]) * r.inv.iy, sz = __uint_as_float(v[22]) * r.inv.iz;
    const float mx = kPlaneMargin * fabsf(sx), my = kPlaneMargin * fabsf(sy), mz = kPlaneMargin * fabsf(sz);
    const float ox = __fmaf_rn(-32768.0f, sx, __fmaf_rn(px, r.inv.ix, -r.px)), oy = __fmaf_rn(-32768.0f, sy, __fmaf_rn(py, r.inv.iy, -r.py)),
                oz = __fmaf_rn(-32768.0f, sz, __fmaf_rn(pz, r.inv.iz, -r.pz));
    const float nx = ox - (mx + r.ex), fx = ox + (mx + r.ex), ny = oy - (my + r.ey), fy = oy + (my + r.ey), nz = oz - (mz + r.ez), fz = oz + (mz + r.ez);
    const bool bx = r.inv.ix < 0.0f, by = r.inv.iy < 0.0f, bz = r.inv.iz < 0.0f;
    float hits = 8388608.0f;  // 2^23: its last eight bits are the mask
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        const uint32_t lx = v[8 + h], ly = v[10 + h], lz = v[12 + h], hx = v[14 + h], hy = v[16 + h], hz = v[18 + h];
        const uint32_t ax = bx ? hx : lx, ay = by ? hy : ly, az = bz ? hz : lz;
        const uint32_t cx = bx ? lx : hx, cy = by ? ly : hy, cz = bz ? lz : hz;
        auto child = [&](float x0, float y0, float z0, float x1, float y1, float z1, float bit) {
            const float t0 = max3(fmaxf(__fmaf_rn(x0, sx, nx), tmin), __fmaf_rn(y0, sy, ny), __fmaf_rn(z0, sz, nz));
            const float t1 = min3(fminf(__fmaf_rn(x1, sx, fx), tmax), __fmaf_rn(y1, sy, fy), __fmaf_rn(z1, sz, fz));
            if (t0 <= t1) hits += bit;
        };
        const float b = h ? 16.0f : 1.0f;
        child(plane<0>(ax), plane<0>(ay), plane<0>(az), plane<0>(cx), plane<0>(cy), plane<0>(cz), b);
        child(plane<1>(ax), plane<1>(ay), plane<1>(az), plane<1>(cx), plane<1>(cy), plane<1>(cz), 2.0f * b);
        child(plane<2>(ax), plane<2>(ay), plane<2>(az), plane<2>(cx), plane<2>(cy), plane<2>(cz), 4.0f * b);
        child(plane<3>(ax), plane<3>(ay), plane<3>(az), plane<3>(cx), plane<3>(cy), plane<3>(cz), 8.0f * b);
    }
    return __float_as_uint(hits) & 0xffu;
}
// bit k of the result is bit k ^ octinv of m
__device__ __forceinline__ uint32_t octant_order(uint32_t m, uint32_t octinv) {
    if (octinv & 1u) m = (m & 0x55u) << 1 | (m >> 1 & 0x55u);
    if (octinv & 2u) m = (m & 0x33u) << 2 | (m >> 2 & 0x33u);
    if (octinv & 4u) m = (m & 0x0fu) << 4 | m >> 4;
    return m;
}

// One ray's walk, a step at a time: a step visits a node, or tests one triangle of the last node
// visited while there are any.  The stack is the caller's (an array indexed at run time, which would
// keep the whole struct out of registers).
template <bool ANY>
struct WideWalk {
    float ox, oy, oz, dx, dy, dz, tmin, tmax;
    WideRay r;
    Hit h;
    uint32_t leaf, todo, tri_base, lmask;
    uint2 g;  // node group: first child, pending children in bits 24..31 (octant order) | imask
    int sp;

    __device__ __forceinline__ WideWalk(const SceneDev& s, float ox_, float oy_, float oz_, float dx_, float dy_, float dz_,
                                        float tmin_, float tmax_)
        : ox(ox_), oy(oy_), oz(oz_), dx(dx_), dy(dy_), dz(dz_), tmin(tmin_), tmax(tmax_), r(s, ox, oy, oz, dx, dy, dz) {
        h.t = tmax;
        h.prim = 0xffffffffu;
        h.u = h.v = 0.0f;
        leaf = todo = tri_base = lmask = 0;
        g = make_uint2(0u, 0x80000000u);  // the root: slot 7 ^ octinv of no node
        sp = 0;
    }
    __device__ __forceinline__ bool alive() const { return g.y > 0x00ffffffu || todo; }
    __device__ __forceinline__ void step(const SceneDev& s, uint2* stack) {
        if (alive() && !todo) {
            const uint32_t k = 31u - __clz(g.y);
            const uint32_t slot = (k - 24u) ^ r.octinv;
            const uint32_t node = g.x + __popc(g.y & 0xffu & ~(0xffffffffu << slot));
            g.y &= ~(1u << k);
            if (g.y > 0x00ffffffu) stack[sp++] = g;
            uint32_t v[24];
            const char* const p = reinterpret_cast<const char*>(s.wide + node);
            ld32(p, v);
            ld32(p + 32, v + 8);
            ld32(p + 64, v + 16);
            const uint32_t hits = wide_hits(r, v, tmin, h.t), imask = v[3];
            g = make_uint2(v[4], octant_order(hits & imask, r.octinv) << 24 | imask);
            tri_base = v[5];
            lmask = v[6];
            todo = hits & lmask;
            if (g.y <= 0x00ffffffu) {
                if (sp == 0) g.y = 0u;  // no node left
                else g = stack[--sp];
            }
        }
        if (todo) {
            const uint32_t j = __ffs(todo) - 1;
            todo &= todo - 1;
            uint32_t w[16];
            const char* const q = reinterpret_cast<const char*>(s.wtris + tri_base + __popc(lmask & ~(0xffffffffu << j)));
            ld32(q, w);
            ld32(q + 32, w + 8);
            BvhTri tr;
            tr.r0 = make_float4(__uint_as_float(w[0]), __uint_as_float(w[1]), __uint_as_float(w[2]), __uint_as_float(w[3]));
            tr.r1 = make_float4(__uint_as_float(w[4]), __uint_as_float(w[5]), __uint_as_float(w[6]), __uint_as_float(w[7]));
            tr.r2 = make_float4(__uint_as_float(w[8]), __uint_as_float(w[9]), __uint_as_float(w[10]), __uint_as_float(w[11]));
            float u, v;
            // equal distances pass, to be told apart below
            const bool any = h.prim != 0xffffffffu;
            const float t = tri_hit(tr, ox, oy, oz, dx, dy, dz, tmin, any ? __uint_as_float(__float_as_uint(h.t) + 1u) : h.t, u, v);
            if (t > 0.0f && leaf_reached(s, w[12], ox, oy, oz, r.inv, tmin, tmax) &&
                (ANY || t < h.t || meets_first(s.nodes, w[12], leaf, ox, oy, oz, r.inv, tmin, tmax))) {
                h.t = t;
                h.u = u;
                h.v = v;
                h.prim = w[13];
                leaf = w[12];
                if (ANY) g.y = todo = 0u;
            }
        }
    }
};

// closest hit (ANY = false) or any hit (ANY = true) in (tmin, tmax) through the hierarchy.  The warp's rays step together:
// without the vote that ends each step its lanes drift apart for good and a node is visited by a
// few of them (closest hits of 2^20 rays in 1.05 M triangles: 1490 us without, 946 us with it).
// Bound by the integer pipe (byte permutes, min / max) at 12 of 32 lanes.  Per-ray loops of the
// binary hierarchy took 1787 us for the same rays (8.8 lanes, L1 82 % busy with 64-byte nodes).
template <bool ANY>
__device__ __forceinline__ Hit bvh_trace(const SceneDev& s, float ox, float oy, float oz, float dx, float dy, float dz,
                                         float tmin, float tmax) {
    WideWalk<ANY> w(s, ox, oy, oz, dx, dy, dz, tmin, tmax);
    uint2 stack[kWideStack];
    const unsigned mask = __activemask();
    do w.step(s, stack);
    while (__any_sync(mask, w.alive()));
    return w.h;
}

}  // namespace rtpg
