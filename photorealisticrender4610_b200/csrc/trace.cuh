// Device ray traversal: the reference's closest-hit and any-hit BVH walks
// (BVH.cpp:311-473) with Möller-Trumbore (Triangle.hpp:46-92) and the
// analytic sphere (Sphere.hpp:22-44), over the 64-byte child-pair nodes of
// device_types.h.
//
// Bit-exactness. Everything here is compiled with --fmad=false and IEEE
// division/sqrt, and every expression keeps the reference's operation order,
// so each slab distance, determinant and t is the float the reference's
// IEEE build computes. The traversal order (near child first on
// tLeft <= tRight, cull on tBox < closestT at push and at pop) is the
// reference's, so ties resolve to the same triangle.
//
// Stacks live in shared memory, one column per thread ([depth][block]
// layout), so a warp's pushes and pops hit distinct banks.
//
// Checked build (-DPRR_CHECKED): every node and triangle fetch is tested
// against the array's length and every stack push against the column's
// depth. A failed test records an error code (first one wins), the offending
// value and a count in the scene's status words and keeps the access in
// bounds (an out-of-range node reads as two empty boxes, a triangle as a
// degenerate one that never hits, an overflowing push is dropped), so the
// kernel runs to its end and the host reads the status (prr_check_status).
// Nothing traps and nothing waits. In the normal build the tests compile to
// nothing.
#pragma once
#include <cuda_runtime.h>

#include "device_types.h"

namespace prr {

#define kInf (__int_as_float(0x7f800000))

// Error codes of the checked build's status words.
enum : uint32_t { kCheckNode = 1, kCheckTri = 2, kCheckStack = 3, kCheckQueue = 4 };

// status[0] = first error code, status[1] = its value, status[2] = errors seen
__device__ __forceinline__ void check_fail(uint32_t *status, uint32_t code, uint32_t value) {
    if (!status)
        return;
    if (atomicCAS(status, 0u, code) == 0u)
        atomicExch(status + 1, value);
    atomicAdd(status + 2, 1u);
}

// What a checked fetch tests against.
struct TraceBounds {
    uint32_t n_nodes, n_qnodes, n_tris;
    uint32_t *check;
};

__device__ __forceinline__ TraceBounds bounds_of(const DevScene &S) {
    return TraceBounds{S.n_nodes, S.n_qnodes, S.n_tris, S.check};
}

struct RayD {
    float ox, oy, oz;
    float dx, dy, dz;
};

// BVHAccel::precompute (BVH.cpp:290-299)
struct RayPre {
    float ox, oy, oz;
    float ix, iy, iz;
    bool nx, ny, nz; // octant: direction negative on that axis
};

__device__ __forceinline__ RayPre precompute(const RayD &r) {
    RayPre p;
    p.ox = r.ox;
    p.oy = r.oy;
    p.oz = r.oz;
    p.ix = (r.dx != 0.f) ? (1.f / r.dx) : kInf;
    p.iy = (r.dy != 0.f) ? (1.f / r.dy) : kInf;
    p.iz = (r.dz != 0.f) ? (1.f / r.dz) : kInf;
    p.nx = r.dx < 0.f;
    p.ny = r.dy < 0.f;
    p.nz = r.dz < 0.f;
    return p;
}

// Three-input max and min (sm_100's max.f32 / min.f32 with three sources).
// Like fmaxf/fminf they ignore a NaN input (the result is the max or min of
// the others), so fmax3(a, b, c) == fmaxf(fmaxf(a, b), c) and likewise for
// fmin3, in one instruction instead of two.
__device__ __forceinline__ float fmax3(float a, float b, float c) {
    float d;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
    return d;
}

__device__ __forceinline__ float fmin3(float a, float b, float c) {
    float d;
    asm("min.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
    return d;
}

// BVHAccel::nodeIntersect (BVH.hpp:115-124) on bounds
// [minX,maxX,minY,maxY,minZ,maxZ]. The reference folds the three axes into
// tMin = 0 and tMax = +inf one at a time with std::max(tMin, t0) and
// std::min(tMax, t1); fmaxf/fminf agree with those for every input, NaN
// included (the running bound is never NaN, and both return it when the new
// term is NaN), and so do the three-input forms over the same terms.
__device__ __forceinline__ float slab(float x0, float x1, float y0, float y1, float z0, float z1,
                                      const RayPre &p) {
    const float t0x = ((p.nx ? x1 : x0) - p.ox) * p.ix;
    const float t1x = ((p.nx ? x0 : x1) - p.ox) * p.ix;
    const float t0y = ((p.ny ? y1 : y0) - p.oy) * p.iy;
    const float t1y = ((p.ny ? y0 : y1) - p.oy) * p.iy;
    const float t0z = ((p.nz ? z1 : z0) - p.oz) * p.iz;
    const float t1z = ((p.nz ? z0 : z1) - p.oz) * p.iz;
    const float tmin = fmax3(fmaxf(0.f, t0x), t0y, t0z);
    const float tmax = fmin3(fminf(kInf, t1x), t1y, t1z);
    return tmin <= tmax ? tmin : kInf;
}

// The same precomputation with the origin and the reciprocal direction held
// twice per axis, as the register pairs of sm_100's packed float2 arithmetic:
// one packed subtract and one packed multiply give an axis's distances to both
// of its planes. Used by the query-set kernels and by the any-hit walk of the
// wavefront's shadow stage, which have the registers for the pairs (in the
// closest-hit walk of the extend stage the six extra registers cost a
// resident block per SM, more than the packed arithmetic saves).
struct RayPair {
    float2 o2x, o2y, o2z; // (o, o) per axis
    float2 i2x, i2y, i2z; // (1/d, 1/d) per axis
    bool nx, ny, nz;      // octant: direction negative on that axis
};

__device__ __forceinline__ RayPair precompute_pair(const RayD &r) {
    const RayPre q = precompute(r);
    RayPair p;
    p.o2x = make_float2(q.ox, q.ox);
    p.o2y = make_float2(q.oy, q.oy);
    p.o2z = make_float2(q.oz, q.oz);
    p.i2x = make_float2(q.ix, q.ix);
    p.i2y = make_float2(q.iy, q.iy);
    p.i2z = make_float2(q.iz, q.iz);
    p.nx = q.nx;
    p.ny = q.ny;
    p.nz = q.nz;
    return p;
}

// (a.x - b.x, a.y - b.y), each rounded to nearest like the scalar subtract.
__device__ __forceinline__ float2 fsub2(float2 a, float2 b) {
    float2 d;
    asm("{\n\t.reg .b64 a2, b2, d2;\n\t"
        "mov.b64 a2, {%2, %3};\n\t"
        "mov.b64 b2, {%4, %5};\n\t"
        "sub.rn.f32x2 d2, a2, b2;\n\t"
        "mov.b64 {%0, %1}, d2;\n\t}"
        : "=f"(d.x), "=f"(d.y)
        : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
    return d;
}

// slab() on the packed form: per axis (t at the min plane, t at the max
// plane) as (plane - o) * inv, each lane the float the scalar form computes;
// the octant then picks which of the two enters, as the reference picks the
// plane before subtracting.
__device__ __forceinline__ float slab(float x0, float x1, float y0, float y1, float z0, float z1,
                                      const RayPair &p) {
    const float2 tx = __fmul2_rn(fsub2(make_float2(x0, x1), p.o2x), p.i2x);
    const float2 ty = __fmul2_rn(fsub2(make_float2(y0, y1), p.o2y), p.i2y);
    const float2 tz = __fmul2_rn(fsub2(make_float2(z0, z1), p.o2z), p.i2z);
    const float t0x = p.nx ? tx.y : tx.x, t1x = p.nx ? tx.x : tx.y;
    const float t0y = p.ny ? ty.y : ty.x, t1y = p.ny ? ty.x : ty.y;
    const float t0z = p.nz ? tz.y : tz.x, t1z = p.nz ? tz.x : tz.y;
    const float tmin = fmax3(fmaxf(0.f, t0x), t0y, t0z);
    const float tmax = fmin3(fminf(kInf, t1x), t1y, t1z);
    return tmin <= tmax ? tmin : kInf;
}

__device__ __forceinline__ float slab6(const float *b, const RayPre &p) {
    return slab(b[0], b[1], b[2], b[3], b[4], b[5], p);
}

__device__ __forceinline__ float slab6(const float *b, const RayPair &p) {
    return slab(b[0], b[1], b[2], b[3], b[4], b[5], p);
}

struct NodeV {
    float4 a, b, c;
    uint4 link;
};

// 32 bytes from 32-byte aligned read-only global memory in one load
// instruction (sm_100's 256-bit vector load): half a node, or a whole Tri
// record. Builds with -DPRR_LDG128 use two 128-bit loads instead.
__device__ __forceinline__ void ldg256(const void *p, float4 &lo, float4 &hi) {
#ifdef PRR_LDG128
    lo = __ldg(reinterpret_cast<const float4 *>(p));
    hi = __ldg(reinterpret_cast<const float4 *>(p) + 1);
#else
    asm("ld.global.nc.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
        : "=f"(lo.x), "=f"(lo.y), "=f"(lo.z), "=f"(lo.w), "=f"(hi.x), "=f"(hi.y), "=f"(hi.z),
          "=f"(hi.w)
        : "l"(p));
#endif
}

__device__ __forceinline__ NodeV load_node(const WNode *nodes, uint32_t idx) {
    const WNode *q = nodes + idx;
    NodeV n;
    float4 l;
    ldg256(q, n.a, n.b);
    ldg256(reinterpret_cast<const float4 *>(q) + 2, n.c, l);
    n.link = make_uint4(__float_as_uint(l.x), __float_as_uint(l.y), __float_as_uint(l.z),
                        __float_as_uint(l.w));
    return n;
}

// ---- four-wide nodes

struct QuadV {
    float4 mn[3], mx[3]; // per axis: the four children's minima, maxima
    uint4 ref;
};

__device__ __forceinline__ QuadV load_quad(const QNode *nodes, uint32_t idx,
                                           const TraceBounds &B) {
    QuadV n;
#ifdef PRR_CHECKED
    if (idx >= B.n_qnodes) {
        check_fail(B.check, kCheckNode, idx);
        for (int a = 0; a < 3; a++) { // four empty boxes: no slab test enters them
            n.mn[a] = make_float4(kInf, kInf, kInf, kInf);
            n.mx[a] = make_float4(-kInf, -kInf, -kInf, -kInf);
        }
        n.ref = make_uint4(kLeafBit, kLeafBit, kLeafBit, kLeafBit);
        return n;
    }
#endif
    (void) B;
    const float4 *q = reinterpret_cast<const float4 *>(nodes + idx);
    ldg256(q, n.mn[0], n.mx[0]);
    ldg256(q + 2, n.mn[1], n.mx[1]);
    ldg256(q + 4, n.mn[2], n.mx[2]);
    n.ref = __ldg(reinterpret_cast<const uint4 *>(q + 6));
    return n;
}

// min that returns NaN when either operand is NaN
__device__ __forceinline__ float fmin_nan(float a, float b) {
    float d;
    asm("min.NaN.f32 %0, %1, %2;" : "=f"(d) : "f"(a), "f"(b));
    return d;
}

// Distances to one axis's near and far planes of the four children, each the
// float the binary slab() computes for that child.
__device__ __forceinline__ void quad_axis(const float4 &mn, const float4 &mx, bool neg, float o,
                                          float inv, float (&t0)[4], float (&t1)[4]) {
    t0[0] = ((neg ? mx.x : mn.x) - o) * inv;
    t0[1] = ((neg ? mx.y : mn.y) - o) * inv;
    t0[2] = ((neg ? mx.z : mn.z) - o) * inv;
    t0[3] = ((neg ? mx.w : mn.w) - o) * inv;
    t1[0] = ((neg ? mn.x : mx.x) - o) * inv;
    t1[1] = ((neg ? mn.y : mx.y) - o) * inv;
    t1[2] = ((neg ? mn.z : mx.z) - o) * inv;
    t1[3] = ((neg ? mn.w : mx.w) - o) * inv;
}

__device__ __forceinline__ void quad_axis(const float4 &mn, const float4 &mx, bool neg, float2 o,
                                          float2 inv, float (&t0)[4], float (&t1)[4]) {
    const float2 a = __fmul2_rn(fsub2(make_float2(neg ? mx.x : mn.x, neg ? mx.y : mn.y), o), inv);
    const float2 b = __fmul2_rn(fsub2(make_float2(neg ? mx.z : mn.z, neg ? mx.w : mn.w), o), inv);
    const float2 c = __fmul2_rn(fsub2(make_float2(neg ? mn.x : mx.x, neg ? mn.y : mx.y), o), inv);
    const float2 d = __fmul2_rn(fsub2(make_float2(neg ? mn.z : mx.z, neg ? mn.w : mx.w), o), inv);
    t0[0] = a.x;
    t0[1] = a.y;
    t0[2] = b.x;
    t0[3] = b.y;
    t1[0] = c.x;
    t1[1] = c.y;
    t1[2] = d.x;
    t1[3] = d.y;
}

// Entry distances of the four children (slab() of each), and of the two
// binary nodes between them and this one (e01 over children 0 and 1, e23 over
// 2 and 3), which only decide the order the sides are walked in.
//
// Why a walk over these nodes equals the binary walk: a node's box is the
// union of its children's, and rounding is monotone, so a child's entry
// distance is never below its parent's and a child is entered only when its
// parent is; whether a leaf's triangles are tested therefore depends on the
// leaf's own distance and on the order of the leaves alone. The order comes
// from comparing siblings' entry distances at each binary node: between the
// grandchildren of a side those computed here, between the two sides e01 and
// e23, the near distances of the union boxes -- per axis the smaller of the
// children's near distances, or NaN (an axis without a bound) when one of
// them is, since then the union's near plane is either at the ray's origin
// too or behind it. Where a side's own box is missed its entry distance is
// not the binary walk's +inf, but then none of its children is entered.
__device__ __forceinline__ void quad_fold(const float (&x0)[4], const float (&x1)[4],
                                          const float (&y0)[4], const float (&y1)[4],
                                          const float (&z0)[4], const float (&z1)[4],
                                          float (&t)[4], float &e01, float &e23) {
#pragma unroll
    for (int k = 0; k < 4; k++) {
        const float tmin = fmax3(fmaxf(0.f, x0[k]), y0[k], z0[k]);
        // NaN when no axis bounds the exit: not tmin > tmax, as tmin <= +inf
        const float tmax = fmin3(x1[k], y1[k], z1[k]);
        t[k] = tmin > tmax ? kInf : tmin;
    }
    e01 = fmax3(fmaxf(0.f, fmin_nan(x0[0], x0[1])), fmin_nan(y0[0], y0[1]),
                fmin_nan(z0[0], z0[1]));
    e23 = fmax3(fmaxf(0.f, fmin_nan(x0[2], x0[3])), fmin_nan(y0[2], y0[3]),
                fmin_nan(z0[2], z0[3]));
}

__device__ __forceinline__ void quad_test(const QuadV &n, const RayPre &p, float (&t)[4],
                                          float &e01, float &e23) {
    float x0[4], x1[4], y0[4], y1[4], z0[4], z1[4];
    quad_axis(n.mn[0], n.mx[0], p.nx, p.ox, p.ix, x0, x1);
    quad_axis(n.mn[1], n.mx[1], p.ny, p.oy, p.iy, y0, y1);
    quad_axis(n.mn[2], n.mx[2], p.nz, p.oz, p.iz, z0, z1);
    quad_fold(x0, x1, y0, y1, z0, z1, t, e01, e23);
}

__device__ __forceinline__ void quad_test(const QuadV &n, const RayPair &p, float (&t)[4],
                                          float &e01, float &e23) {
    float x0[4], x1[4], y0[4], y1[4], z0[4], z1[4];
    quad_axis(n.mn[0], n.mx[0], p.nx, p.o2x, p.i2x, x0, x1);
    quad_axis(n.mn[1], n.mx[1], p.ny, p.o2y, p.i2y, y0, y1);
    quad_axis(n.mn[2], n.mx[2], p.nz, p.o2z, p.i2z, z0, z1);
    quad_fold(x0, x1, y0, y1, z0, z1, t, e01, e23);
}

// The children of a four-wide node in walk order, with their entry distances
// (t0 <= t1 and t2 <= t3).
struct QuadOrder {
    float t0, t1, t2, t3;
    uint32_t r0, r1, r2, r3;
    // whether some child is entered (its box nearer than best), and the first
    __device__ __forceinline__ bool any(float best) const { return t0 < best || t2 < best; }
    __device__ __forceinline__ uint32_t next(float best) const { return t0 < best ? r0 : r2; }
    __device__ __forceinline__ float next_t(float best) const { return t0 < best ? t0 : t2; }
    // push(ref, t) for the entered children but the first, last in walk order first
    template <class Push> __device__ __forceinline__ void rest(float best, Push &&push) const {
        if (t3 < best)
            push(r3, t3);
        if (t0 < best && t2 < best)
            push(r2, t2);
        if (t1 < best)
            push(r1, t1);
    }
};

template <class P>
__device__ __forceinline__ QuadOrder quad_order(const QuadV &n, const P &p) {
    float t[4], e01, e23;
    quad_test(n, p, t, e01, e23);
    const bool s0 = !(t[0] <= t[1]), s1 = !(t[2] <= t[3]), sw = !(e01 <= e23);
    const float an = s0 ? t[1] : t[0], af = s0 ? t[0] : t[1];
    const float bn = s1 ? t[3] : t[2], bf = s1 ? t[2] : t[3];
    const uint32_t ar = s0 ? n.ref.y : n.ref.x, aq = s0 ? n.ref.x : n.ref.y;
    const uint32_t br = s1 ? n.ref.w : n.ref.z, bq = s1 ? n.ref.z : n.ref.w;
    QuadOrder q;
    q.t0 = sw ? bn : an;
    q.t1 = sw ? bf : af;
    q.t2 = sw ? an : bn;
    q.t3 = sw ? af : bf;
    q.r0 = sw ? br : ar;
    q.r1 = sw ? bq : aq;
    q.r2 = sw ? ar : br;
    q.r3 = sw ? aq : bq;
    return q;
}

// True for a ray that an inverted box (+inf..-inf, an empty slot) does not
// stop: on every axis its origin is NaN or its direction NaN or infinite. Such
// a ray hits no triangle (its Möller-Trumbore t is NaN or 0), so mesh walks
// are skipped for it, and empty slots are never entered.
template <class P> __device__ __forceinline__ bool no_slab(const P &p) {
    return slab(kInf, -kInf, kInf, -kInf, kInf, -kInf, p) < kInf;
}

struct TriV {
    float4 p, q, r;
};

__device__ __forceinline__ TriV load_tri(const Tri *tris, const float *e2z, uint32_t idx) {
    TriV v;
    ldg256(tris + idx, v.p, v.q);
    v.r = make_float4(__ldg(e2z + idx), 0.f, 0.f, 0.f);
    return v;
}

// Checked forms: the plain fetch unless the build is checked and the index is
// out of range.
__device__ __forceinline__ NodeV load_node(const WNode *nodes, uint32_t idx,
                                           const TraceBounds &B) {
#ifdef PRR_CHECKED
    if (idx >= B.n_nodes) {
        check_fail(B.check, kCheckNode, idx);
        NodeV n; // two empty boxes: no slab test enters them
        n.a = make_float4(kInf, -kInf, kInf, -kInf);
        n.b = make_float4(kInf, -kInf, kInf, -kInf);
        n.c = make_float4(kInf, -kInf, kInf, -kInf);
        n.link = make_uint4(0u, 0u, 0u, 0u);
        return n;
    }
#endif
    return load_node(nodes, idx);
}

__device__ __forceinline__ TriV load_tri(const Tri *tris, const float *e2z, uint32_t idx,
                                         const TraceBounds &B) {
#ifdef PRR_CHECKED
    if (idx >= B.n_tris) {
        check_fail(B.check, kCheckTri, idx);
        TriV v; // all zero: det = 0 fails the parallel test
        v.p = v.q = v.r = make_float4(0.f, 0.f, 0.f, 0.f);
        return v;
    }
#endif
    return load_tri(tris, e2z, idx);
}

__device__ __forceinline__ NodeV load_node(const DevScene &S, uint32_t idx) {
    return load_node(S.nodes, idx, bounds_of(S));
}

__device__ __forceinline__ QuadV load_quad(const DevScene &S, uint32_t idx) {
    return load_quad(S.qnodes, idx, bounds_of(S));
}

__device__ __forceinline__ TriV load_tri(const DevScene &S, uint32_t idx) {
    return load_tri(S.tris, S.tri_e2z, idx, bounds_of(S));
}

// Triangle::hitTest (Triangle.hpp:46-64), evaluated without early exits. The
// miss tests are kept in their negated form so NaNs fall through exactly as
// the reference's `if (cond) return miss` chain lets them.
__device__ __forceinline__ bool tri_hit(const TriV &T, const RayD &r, float &t, float &u,
                                        float &v) {
    const float v0x = T.p.x, v0y = T.p.y, v0z = T.p.z;
    const float e1x = T.p.w, e1y = T.q.x, e1z = T.q.y;
    const float e2x = T.q.z, e2y = T.q.w, e2z = T.r.x;
    // P = d x e2
    const float px = r.dy * e2z - r.dz * e2y;
    const float py = r.dz * e2x - r.dx * e2z;
    const float pz = r.dx * e2y - r.dy * e2x;
    const float det = px * e1x + py * e1y + pz * e1z;
    const float inv = 1.f / det;
    const float tx = r.ox - v0x, ty = r.oy - v0y, tz = r.oz - v0z;
    u = (px * tx + py * ty + pz * tz) * inv;
    // Q = T x e1
    const float qx = ty * e1z - tz * e1y;
    const float qy = tz * e1x - tx * e1z;
    const float qz = tx * e1y - ty * e1x;
    v = (qx * r.dx + qy * r.dy + qz * r.dz) * inv;
    t = (qx * e2x + qy * e2y + qz * e2z) * inv;
    return !(fabsf(det) < 1e-6f) && !(u < 0.f) && !(v < 0.f || u + v > 1.f) && !(t <= 1e-3f);
}

// Triangle::intersectT (Triangle.hpp:75-92) followed by the caller's
// `t >= 0 && t < tMax` check (BVH.cpp:395-398).
__device__ __forceinline__ bool tri_occludes(const TriV &T, const RayD &r, float tmax) {
    const float v0x = T.p.x, v0y = T.p.y, v0z = T.p.z;
    const float e1x = T.p.w, e1y = T.q.x, e1z = T.q.y;
    const float e2x = T.q.z, e2y = T.q.w, e2z = T.r.x;
    const float px = r.dy * e2z - r.dz * e2y;
    const float py = r.dz * e2x - r.dx * e2z;
    const float pz = r.dx * e2y - r.dy * e2x;
    const float det = px * e1x + py * e1y + pz * e1z;
    const float inv = 1.f / det;
    const float tx = r.ox - v0x, ty = r.oy - v0y, tz = r.oz - v0z;
    const float u = (px * tx + py * ty + pz * tz) * inv;
    const float qx = ty * e1z - tz * e1y;
    const float qy = tz * e1x - tx * e1z;
    const float qz = tx * e1y - ty * e1x;
    const float v = (qx * r.dx + qy * r.dy + qz * r.dz) * inv;
    const float t = (qx * e2x + qy * e2y + qz * e2z) * inv;
    return !(fabsf(det) < 1e-6f) && !(u < 0.f || u > 1.f) && !(v < 0.f || u + v > 1.f) &&
           (t > 1e-3f && t < tmax);
}

// Shared-memory accesses by 32-bit shared address (a pointer that may also
// name global memory compiles to generic accesses, which cost the LSU more).
__device__ __forceinline__ void sts(uint32_t a, uint2 v) {
    asm volatile("st.shared.v2.u32 [%0], {%1, %2};" ::"r"(a), "r"(v.x), "r"(v.y));
}
__device__ __forceinline__ void sts(uint32_t a, uint32_t v) {
    asm volatile("st.shared.u32 [%0], %1;" ::"r"(a), "r"(v));
}
__device__ __forceinline__ void lds(uint32_t a, uint2 &v) {
    asm volatile("ld.shared.v2.u32 {%0, %1}, [%2];" : "=r"(v.x), "=r"(v.y) : "r"(a));
}
__device__ __forceinline__ void lds(uint32_t a, uint32_t &v) {
    asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(a));
}

// Per-thread stack with a bounded shared-memory part. A position is the byte
// address `top` of the next free entry of the thread's shared-memory column
// (step bytes apart, [entry][thread], so a warp's pushes hit distinct banks);
// positions at `limit` and beyond stand for entries of a buffer that lies
// outside: LOCAL entries of the thread's local memory, or, where those are too
// few (or none, LOCAL = 0), a global buffer laid out [entry - cap][grid thread].
// A warp's spills are coalesced in both. The bound
// on a walk's entries is found when its tree is packed; the outer part is
// only reached deep in unbalanced subtrees and stays in L1/L2, and the code
// for it sits behind one comparison per step. Fewer shared entries leave more
// of the SM's L1 for node and triangle fetches and let more blocks be
// resident.
template <class E, int LOCAL = 0> struct StackCol {
    uint32_t base, step, limit;
    E *gl;                   // global part (LOCAL > 0: nullptr where `local` serves)
    E *local = nullptr;      // LOCAL entries of the thread's own
    int total = 1 << 30;     // entries in both parts (tested by the checked build)
    uint32_t *check = nullptr;
    __device__ __forceinline__ StackCol(E *sm, E *global, E *own, int cap, int total_,
                                        uint32_t *check_)
        : base((uint32_t) __cvta_generic_to_shared(sm) + threadIdx.x * (uint32_t) sizeof(E)),
          step(blockDim.x * (uint32_t) sizeof(E)), gl(global), local(own), total(total_),
          check(check_) {
        limit = base + (uint32_t) cap * step;
    }
    __device__ __forceinline__ E *spill_at(uint32_t top) const {
        const size_t k = (top - limit) / step;
        if (LOCAL > 0 && !gl)
            return local + k;
        return gl + k * (gridDim.x * blockDim.x) + blockIdx.x * blockDim.x + threadIdx.x;
    }
    __device__ __forceinline__ bool ok(uint32_t top) const {
#ifdef PRR_CHECKED
        if (top < base || (top - base) / step >= (uint32_t) total) {
            check_fail(check, kCheckStack, (top - base) / step);
            return false;
        }
#endif
        (void) top;
        return true;
    }
    // three more entries fit in the shared part
    __device__ __forceinline__ bool room3(uint32_t top) const { return top + 2 * step < limit; }
    // an entry known to lie in the shared part
    __device__ __forceinline__ void put_sm(uint32_t &top, E v) const {
        if (!ok(top))
            return;
        sts(top, v);
        top += step;
    }
    __device__ __forceinline__ void put(uint32_t &top, E v) const {
        if (!ok(top))
            return;
        if (top < limit)
            sts(top, v);
        else
            *spill_at(top) = v;
        top += step;
    }
    __device__ __forceinline__ E pop(uint32_t &top) const {
        top -= step;
        E v{};
        if (!ok(top))
            return v;
        if (top < limit)
            lds(top, v);
        else
            v = *spill_at(top);
        return v;
    }
    __device__ __forceinline__ bool empty(uint32_t top) const { return top == base; }
};

// Push a node's entered children but the first (closest hit: with their entry
// distances; any hit: references alone).
template <int LOCAL>
__device__ __forceinline__ void push_rest(const StackCol<uint2, LOCAL> &st, uint32_t &top,
                                          const QuadOrder &q, float best) {
    if (st.room3(top))
        q.rest(best, [&](uint32_t c, float t) {
            st.put_sm(top, make_uint2(c, __float_as_uint(t)));
        });
    else
        q.rest(best, [&](uint32_t c, float t) {
            st.put(top, make_uint2(c, __float_as_uint(t)));
        });
}
template <int LOCAL>
__device__ __forceinline__ void push_rest(const StackCol<uint32_t, LOCAL> &st, uint32_t &top,
                                          const QuadOrder &q, float tmax) {
    if (st.room3(top))
        q.rest(tmax, [&](uint32_t c, float) { st.put_sm(top, c); });
    else
        q.rest(tmax, [&](uint32_t c, float) { st.put(top, c); });
}

// Asks for a child's first bytes in L1: for batches so small that memory is idle
// and a walk waits on one fetch after another (a child waiting on the stack is
// then at hand when it is popped).
__device__ __forceinline__ void fetch_child(const QNode *nodes, const Tri *tris, uint32_t ref) {
    const void *g = (ref & kLeafBit) ? (const void *) (tris + leaf_first(ref))
                                     : (const void *) (nodes + ref);
    asm volatile("prefetch.global.L1 [%0];" ::"l"(g));
}

// Per-thread stack column in shared memory.
struct SmemStack {
    uint2 *base; // &smem[tid]; entry k at base[k * stride]
    int stride;
    int sp;
    int cap = 1 << 30;         // entries in the column (tested by the checked build)
    uint32_t *check = nullptr; // where the checked build reports
    __device__ __forceinline__ void push(uint32_t ref, float t) {
#ifdef PRR_CHECKED
        if (sp >= cap) {
            check_fail(check, kCheckStack, (uint32_t) sp);
            return;
        }
#endif
        base[sp * stride] = make_uint2(ref, __float_as_uint(t));
        sp++;
    }
    __device__ __forceinline__ uint2 pop() {
        --sp;
        return base[sp * stride];
    }
};

// Work of a binary walk: interior nodes of either level, triangle tests, object
// leaves (mesh entries and sphere tests).
struct WalkCounts {
    unsigned nodes = 0, tris = 0, objects = 0;
};

// BVHAccel::Intersect, triangle fast path (BVH.cpp:311-415) on one mesh's
// four-wide nodes. best_t enters as +inf (every mesh-level search starts
// fresh, BVH.cpp:331). Returns the winning triangle's global leaf-order index,
// or -1.
template <int LOCAL>
__device__ __forceinline__ int blas_closest_quad(const QNode *__restrict__ nodes,
                                                 const Tri *__restrict__ tris,
                                                 const float *__restrict__ e2z, uint32_t root,
                                                 const RayD &r, const RayPre &p,
                                                 const StackCol<uint2, LOCAL> &st, float &best_t,
                                                 float &best_u, float &best_v,
                                                 const TraceBounds &B) {
    if (!(root & kLeafBit) && no_slab(p))
        return -1;
    uint32_t top = st.base;
    uint32_t ref = root;
    int hit = -1;
    for (;;) {
        if (!(ref & kLeafBit)) {
            const QuadOrder q = quad_order(load_quad(nodes, ref, B), p);
            push_rest(st, top, q, best_t);
            if (q.any(best_t)) {
                ref = q.next(best_t);
                continue;
            }
        } else {
            const uint32_t first = leaf_first(ref);
            const uint32_t cnt = leaf_count(ref);
            for (uint32_t i = 0; i < cnt; i++) {
                const TriV T = load_tri(tris, e2z, first + i, B);
                float t, u, v;
                if (tri_hit(T, r, t, u, v) && t < best_t) {
                    best_t = t;
                    best_u = u;
                    best_v = v;
                    hit = (int) (first + i);
                }
            }
        }
        // pop the next entry whose box is still nearer than the closest hit
        for (;;) {
            if (st.empty(top))
                return hit;
            const uint2 e = st.pop(top);
            if (__uint_as_float(e.y) < best_t) {
                ref = e.x;
                break;
            }
        }
    }
}

// The same search on the binary nodes, for the kernels that run a whole path
// per thread (plain renderer, photons, caustic samples): the four-wide step's
// registers cost those more than its shorter walk saves (museum-like scene of
// 122,880 triangles at 480x270, 16 spp: 12.4 ms, 14.4 four-wide; Cornell box
// 2.2 against 2.7).
template <bool COUNT = false>
__device__ __forceinline__ int blas_closest(const WNode *__restrict__ nodes,
                                            const Tri *__restrict__ tris,
                                            const float *__restrict__ e2z, uint32_t root,
                                            const RayD &r, const RayPre &p, SmemStack &st,
                                            float &best_t, float &best_u, float &best_v,
                                            const TraceBounds &B, WalkCounts *wc = nullptr) {
    const int sp0 = st.sp;
    uint32_t ref = root;
    int hit = -1;
    for (;;) {
        if (!(ref & kLeafBit)) {
            if constexpr (COUNT)
                wc->nodes++;
            const NodeV n = load_node(nodes, ref, B);
            const float tl = slab(n.a.x, n.a.y, n.a.z, n.a.w, n.b.x, n.b.y, p);
            const float tr = slab(n.b.z, n.b.w, n.c.x, n.c.y, n.c.z, n.c.w, p);
            if (tl <= tr) {
                if (tl < best_t) {
                    if (tr < best_t)
                        st.push(n.link.y, tr);
                    ref = n.link.x;
                    continue;
                }
            } else {
                if (tr < best_t) {
                    if (tl < best_t)
                        st.push(n.link.x, tl);
                    ref = n.link.y;
                    continue;
                }
            }
        } else {
            const uint32_t first = leaf_first(ref);
            const uint32_t cnt = leaf_count(ref);
            for (uint32_t i = 0; i < cnt; i++) {
                if constexpr (COUNT)
                    wc->tris++;
                const TriV T = load_tri(tris, e2z, first + i, B);
                float t, u, v;
                if (tri_hit(T, r, t, u, v) && t < best_t) {
                    best_t = t;
                    best_u = u;
                    best_v = v;
                    hit = (int) (first + i);
                }
            }
        }
        // pop the next entry whose box is still nearer than the closest hit
        for (;;) {
            if (st.sp == sp0)
                return hit;
            const uint2 e = st.pop();
            if (__uint_as_float(e.y) < best_t) {
                ref = e.x;
                break;
            }
        }
    }
}

template <bool COUNT = false>
__device__ __forceinline__ bool blas_occluded(const WNode *__restrict__ nodes,
                                              const Tri *__restrict__ tris,
                                              const float *__restrict__ e2z, uint32_t root,
                                              const float *root_box, const RayD &r,
                                              const RayPre &p, SmemStack &st, float tmax,
                                              const TraceBounds &B, WalkCounts *wc = nullptr) {
    if (!(slab6(root_box, p) < tmax))
        return false;
    const int sp0 = st.sp;
    uint32_t ref = root;
    for (;;) {
        if (!(ref & kLeafBit)) {
            if constexpr (COUNT)
                wc->nodes++;
            const NodeV n = load_node(nodes, ref, B);
            const float tl = slab(n.a.x, n.a.y, n.a.z, n.a.w, n.b.x, n.b.y, p);
            const float tr = slab(n.b.z, n.b.w, n.c.x, n.c.y, n.c.z, n.c.w, p);
            const uint32_t axis = n.link.z;
            const bool neg = axis == 0 ? p.nx : (axis == 1 ? p.ny : p.nz);
            // octant 0 -> near = left
            const uint32_t near_ref = neg ? n.link.y : n.link.x;
            const uint32_t far_ref = neg ? n.link.x : n.link.y;
            const float tnear = neg ? tr : tl;
            const float tfar = neg ? tl : tr;
            if (tfar < tmax)
                st.push(far_ref, 0.f);
            if (tnear < tmax) {
                ref = near_ref;
                continue;
            }
        } else {
            const uint32_t first = leaf_first(ref);
            const uint32_t cnt = leaf_count(ref);
            for (uint32_t i = 0; i < cnt; i++) {
                if constexpr (COUNT)
                    wc->tris++;
                const TriV T = load_tri(tris, e2z, first + i, B);
                if (tri_occludes(T, r, tmax)) {
                    st.sp = sp0;
                    return true;
                }
            }
        }
        if (st.sp == sp0)
            return false;
        ref = st.pop().x;
    }
}

// Sphere::getIntersection (Sphere.hpp:22-44) with solveQuadratic
// (global.hpp:19-33). The reference calls the double sqrt there and mixes
// -0.5 (a double) into both roots, so those steps run in double and round to
// float exactly where the reference's assignments do.
__device__ __forceinline__ bool sphere_hit(const DevObject &s, const RayD &r, float &t_out) {
    const float Lx = r.ox - s.cx, Ly = r.oy - s.cy, Lz = r.oz - s.cz;
    const float a = r.dx * r.dx + r.dy * r.dy + r.dz * r.dz;
    const float b = 2 * (r.dx * Lx + r.dy * Ly + r.dz * Lz);
    const float c = (Lx * Lx + Ly * Ly + Lz * Lz) - s.radius2;
    const float discr = b * b - 4 * a * c;
    float x0, x1;
    if (discr < 0)
        return false;
    else if (discr == 0) {
        x0 = x1 = (float) (-0.5 * (double) b / (double) a);
    } else {
        const double sq = sqrt((double) discr);
        const float q = (b > 0) ? (float) (-0.5 * ((double) b + sq))
                                : (float) (-0.5 * ((double) b - sq));
        x0 = q / a;
        x1 = c / q;
    }
    if (x0 > x1) {
        float tmp = x0;
        x0 = x1;
        x1 = tmp;
    }
    float t0 = x0;
    if (t0 < 0)
        t0 = x1;
    if (t0 < 0)
        return false;
    t_out = t0;
    return true;
}

// sphere_hit called out of line, for walks inlined in a kernel that waits on
// instruction fetch: its double-precision steps are long and rarely run.
static __device__ __noinline__ bool sphere_hit_ool(const DevObject &s, const RayD &r, float &t) {
    return sphere_hit(s, r, t);
}

struct SceneHit {
    int obj;      // object index, -1 on a miss
    int tri;      // global leaf-order triangle index (meshes), -1 for spheres
    float t, u, v;
};

// Scene::intersect -> BVHAccel::Intersect, general path (BVH.cpp:359-369):
// every scene-BVH leaf object is intersected on its own (meshes start their
// own search at +inf) and replaces the winner when tnear < closestT.
template <bool COUNT = false, bool OOL = false>
__device__ __forceinline__ SceneHit scene_closest(const DevScene &S, const RayD &r,
                                                  const RayPre &p, SmemStack &tst,
                                                  SmemStack &bst, WalkCounts *wc = nullptr) {
    SceneHit h;
    h.obj = -1;
    h.tri = -1;
    h.t = kInf;
    h.u = h.v = 0.f;
    if (S.n_objects == 0)
        return h;
    float closest = kInf;
    const int sp0 = tst.sp;
    uint32_t ref = S.tlas_root;
    for (;;) {
        if (!(ref & kLeafBit)) {
            if constexpr (COUNT)
                wc->nodes++;
            const NodeV n = load_node(S, ref);
            const float tl = slab(n.a.x, n.a.y, n.a.z, n.a.w, n.b.x, n.b.y, p);
            const float tr = slab(n.b.z, n.b.w, n.c.x, n.c.y, n.c.z, n.c.w, p);
            if (tl <= tr) {
                if (tl < closest) {
                    if (tr < closest)
                        tst.push(n.link.y, tr);
                    ref = n.link.x;
                    continue;
                }
            } else {
                if (tr < closest) {
                    if (tl < closest)
                        tst.push(n.link.x, tl);
                    ref = n.link.y;
                    continue;
                }
            }
        } else {
            const int k = (int) (ref & ~kLeafBit);
            const DevObject &o = S.objects[k];
            if constexpr (COUNT)
                wc->objects++;
            if (o.kind == kObjMesh) {
                float t = kInf, u = 0.f, v = 0.f;
                const int tri = blas_closest<COUNT>(S.nodes, S.tris, S.tri_e2z, o.root, r, p, bst, t, u, v,
                                             bounds_of(S), wc);
                if (tri >= 0 && t < closest) {
                    closest = t;
                    h.obj = k;
                    h.tri = tri;
                    h.t = t;
                    h.u = u;
                    h.v = v;
                }
            } else {
                float t;
                if ((OOL ? sphere_hit_ool(o, r, t) : sphere_hit(o, r, t)) && t < closest) {
                    closest = t;
                    h.obj = k;
                    h.tri = -1;
                    h.t = t;
                }
            }
        }
        for (;;) {
            if (tst.sp == sp0)
                return h;
            const uint2 e = tst.pop();
            if (__uint_as_float(e.y) < closest) {
                ref = e.x;
                break;
            }
        }
    }
}

// Scene::intersectP -> BVHAccel::IntersectP over objects (BVH.cpp:421-473):
// MeshTriangle::intersectT answers 1e-3 when its own IntersectP finds an
// occluder (Triangle.hpp:141-147) and Sphere falls back to
// Object::intersectT (Object.hpp:24-29); the caller then requires
// t >= 0 && t < tMax.
template <bool COUNT = false, bool OOL = false>
__device__ __forceinline__ bool scene_occluded(const DevScene &S, const RayD &r,
                                               const RayPre &p, SmemStack &tst, SmemStack &bst,
                                               float tmax, WalkCounts *wc = nullptr) {
    if (S.n_objects == 0)
        return false;
    if (!(slab6(S.tlas_box, p) < tmax))
        return false;
    const int sp0 = tst.sp;
    uint32_t ref = S.tlas_root;
    for (;;) {
        if (!(ref & kLeafBit)) {
            if constexpr (COUNT)
                wc->nodes++;
            const NodeV n = load_node(S, ref);
            const float tl = slab(n.a.x, n.a.y, n.a.z, n.a.w, n.b.x, n.b.y, p);
            const float tr = slab(n.b.z, n.b.w, n.c.x, n.c.y, n.c.z, n.c.w, p);
            const uint32_t axis = n.link.z;
            const bool neg = axis == 0 ? p.nx : (axis == 1 ? p.ny : p.nz);
            const uint32_t near_ref = neg ? n.link.y : n.link.x;
            const uint32_t far_ref = neg ? n.link.x : n.link.y;
            const float tnear = neg ? tr : tl;
            const float tfar = neg ? tl : tr;
            if (tfar < tmax)
                tst.push(far_ref, 0.f);
            if (tnear < tmax) {
                ref = near_ref;
                continue;
            }
        } else {
            const DevObject &o = S.objects[ref & ~kLeafBit];
            bool occ;
            if constexpr (COUNT)
                wc->objects++;
            if (o.kind == kObjMesh) {
                occ = blas_occluded<COUNT>(S.nodes, S.tris, S.tri_e2z, o.root, o.root_box, r, p, bst, tmax,
                                    bounds_of(S), wc) &&
                      (1e-3f < tmax);
            } else {
                float t;
                occ = (OOL ? sphere_hit_ool(o, r, t) : sphere_hit(o, r, t)) && t < tmax && t >= 0.f;
            }
            if (occ) {
                tst.sp = sp0;
                return true;
            }
        }
        if (tst.sp == sp0)
            return false;
        ref = tst.pop().x;
    }
}

} // namespace prr
