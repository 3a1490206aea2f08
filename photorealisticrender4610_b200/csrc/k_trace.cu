// Batch ray-query kernels: mesh closest hit / any hit (the BVHAccel::Intersect
// and IntersectP micro-path, BVH.cpp:311-473) and scene-level closest hit /
// any hit (Scene::intersect / intersectP, Scene.cpp:29-35).
//
// One lane traces one ray at a time over the four-wide mesh nodes. A persistent
// grid hands rays to lanes one by one (trace_rays); how many rays a warp holds
// at once follows from the batch size.
#include "prr_internal.h"
#include "trace_step.cuh"

#include <algorithm>

namespace prr {

namespace {

__device__ __forceinline__ RayD load_ray(const float *__restrict__ O, const float *__restrict__ D,
                                         int64_t i) {
    RayD r;
    r.ox = __ldg(O + i * 3 + 0);
    r.oy = __ldg(O + i * 3 + 1);
    r.oz = __ldg(O + i * 3 + 2);
    r.dx = __ldg(D + i * 3 + 0);
    r.dy = __ldg(D + i * 3 + 1);
    r.dz = __ldg(D + i * 3 + 2);
    return r;
}

// Möller-Trumbore in fp64 on the input vertices: the winner's t re-solved for
// the 1e-6-relative check, once per ray.
__device__ double tri_t64(const float *__restrict__ v, const RayD &r) {
    const double v0x = v[0], v0y = v[1], v0z = v[2];
    const double e1x = (double) v[3] - v0x, e1y = (double) v[4] - v0y, e1z = (double) v[5] - v0z;
    const double e2x = (double) v[6] - v0x, e2y = (double) v[7] - v0y, e2z = (double) v[8] - v0z;
    const double ox = r.ox, oy = r.oy, oz = r.oz, dx = r.dx, dy = r.dy, dz = r.dz;
    const double tx = ox - v0x, ty = oy - v0y, tz = oz - v0z;
    const double px = dy * e2z - dz * e2y, py = dz * e2x - dx * e2z, pz = dx * e2y - dy * e2x;
    const double qx = ty * e1z - tz * e1y, qy = tz * e1x - tx * e1z, qz = tx * e1y - ty * e1x;
    const double det = px * e1x + py * e1y + pz * e1z;
    return (qx * e2x + qy * e2y + qz * e2z) / det;
}

// What every query kernel needs besides its rays and outputs.
struct TraceCfg {
    unsigned *counter;           // next ray to hand out (nullptr: fixed shares)
    void *spill;                 // global part of the stacks (nullptr: local_stack serves)
    uint32_t share;              // rays of a warp's share: n over the grid's warps
    int lanes;                   // lanes of a warp that take rays: share, at most 32
    int refill;                  // idle lanes that trigger a refill (at most lanes)
    int stack_sm, stack_cap;     // stack entries: in shared memory, in all
};

// Stack entries of a thread's own local memory, beyond those in shared memory:
// enough for a four-wide walk of any tree whose binary walk's stack (one entry
// per level) fits where kStackSm shared entries do, without a buffer that
// captured calls, whose replays may overlap, would have to share.
constexpr int kLocalStack = 24;
template <class E> using QueryStack = StackCol<E, kLocalStack>;

struct MeshArgs {
    const QNode *nodes;
    const Tri *tris;
    const float *e2z;
    const TriMeta *meta;
    const float *verts;
    uint32_t root;
    const float *O, *D;
    uint32_t n;
    int32_t *out_id;
    float *out_t;
    double *out_t64;
    TraceCfg c;
    TraceBounds B;        // array bounds and status words (checked build)
    const uint32_t *perm; // trace order -> input index (nullptr: input order)
};

// Input index of the ray traced in position i.
__device__ __forceinline__ uint32_t ray_at(const MeshArgs &a, uint32_t i) {
    return a.perm ? __ldg(a.perm + i) : i;
}

__device__ __forceinline__ void write_hit(const MeshArgs &a, int64_t i, const RayD &r, int hit,
                                          float t) {
    a.out_id[i] = hit >= 0 ? __ldg(&a.meta[hit].id) : -1;
    a.out_t[i] = t;
    if (a.out_t64)
        a.out_t64[i] = hit >= 0 ? tri_t64(a.verts + (size_t) hit * 9, r)
                                : __longlong_as_double(0x7ff8000000000000LL);
}

// Hands the rays [0, n) to the lanes of the grid and steps them. Each loop
// iteration performs ONE step of every busy lane's ray; a lane whose ray is
// done stays idle until `refill` lanes of its warp are, then the warp takes
// that many new rays at once: rays finishing at different depths do not hold
// their warp hostage, and every ray still takes its steps in its own order.
//
// A batch smaller than the grid's lanes is spread over all of its warps, each
// holding n / warps rays in its first lanes: a step of a warp runs the node
// and the triangle code one after the other for whichever lanes are at one or
// the other, so a small batch, which is as slow as its longest ray, finishes
// sooner the fewer rays share a warp (4,099 rays on 10,000 triangles: 72 us,
// 174 with 32 rays a warp over the binary nodes; 20,000 rays on 300,000: 320
// against 444).
//
// Rays come from the counter, or, without one (batches of one or two rounds of
// the grid's lanes, and calls under stream capture, which allocate nothing),
// from a contiguous share per warp.
template <class Body>
__device__ __forceinline__ void trace_rays(Body &b, uint32_t n, const TraceCfg &c) {
    const unsigned full = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    const unsigned all = 0xffffffffu >> (32 - c.lanes); // lanes that take rays
    unsigned taken = 0; // rays this warp has taken of its share
    bool more = true;   // warp-uniform: rays are left to take
    bool busy = false;
    for (;;) {
        const unsigned im = __ballot_sync(full, !busy) & all;
        if (!more && im == all)
            break;
        if (more && __popc(im) >= c.refill) {
            const int cnt = __popc(im);
            uint32_t base = 0, end = n;
            if (c.counter) {
                if (lane == 0)
                    base = atomicAdd(c.counter, (unsigned) cnt);
                base = __shfl_sync(full, base, 0);
            } else {
                const uint32_t first =
                    ((blockIdx.x * blockDim.x + threadIdx.x) >> 5) * c.share;
                base = first + taken;
                end = min(n, first + c.share);
                taken += cnt;
            }
            more = base + cnt < end;
            const uint32_t i = base + __popc(im & ((1u << lane) - 1u));
            if ((im >> lane & 1u) && i < end)
                busy = b.start(i);
        }
        if (busy && b.step()) {
            b.finish();
            busy = false;
        }
    }
}

// One ray of a closest-hit query on one mesh. A step is one four-wide node
// (the slab tests of BVH.cpp:368-397 at two levels), or one triangle of the
// current leaf (BVH.cpp:343-357), followed when needed by the pop of
// BVH.cpp:400-407. FEW, here and below: the form for small batches, which
// tests a leaf's triangles in one step, their loads under way together, and
// asks for the children it pushes.
template <bool FEW> struct MeshClosest {
    const MeshArgs &a;
    const QueryStack<uint2> col;
    uint32_t idx = 0;
    RayD r;
    RayPair p;
    float best = 0.f;
    int hit = -1;
    uint32_t ref = 0; // next node, or the leaf triangles left to test (a leaf reference)
    uint32_t top = 0;

    __device__ __forceinline__ MeshClosest(const MeshArgs &args, uint2 *smem, uint2 *own)
        : a(args), col(smem, (uint2 *) args.c.spill, own, args.c.stack_sm, args.c.stack_cap,
                       args.B.check) {}

    __device__ __forceinline__ bool start(uint32_t i) {
        idx = ray_at(a, i);
        r = load_ray(a.O, a.D, idx);
        p = precompute_pair(r);
        best = kInf;
        hit = -1;
        top = col.base;
        if (no_slab(p)) {
            finish();
            return false;
        }
        ref = a.root;
        return true;
    }

    __device__ __forceinline__ bool step() {
        if (ref & kLeafBit) {
            const uint32_t tri = leaf_first(ref);
            if constexpr (FEW) {
                const uint32_t ntri = leaf_count(ref);
                // the whole leaf, its loads under way together
                TriV T[4];
#pragma unroll
                for (uint32_t k = 0; k < 4; k++)
                    if (k < ntri)
                        T[k] = load_tri(a.tris, a.e2z, tri + k, a.B);
#pragma unroll
                for (uint32_t k = 0; k < 4; k++)
                    if (k < ntri) {
                        float t, u, v;
                        if (tri_hit(T[k], r, t, u, v) && t < best) {
                            best = t;
                            hit = (int) (tri + k);
                        }
                    }
            } else {
                const TriV T = load_tri(a.tris, a.e2z, tri, a.B);
                float t, u, v;
                if (tri_hit(T, r, t, u, v) && t < best) {
                    best = t;
                    hit = (int) tri;
                }
                ref = leaf_rest(ref);
                if (ref)
                    return false;
            }
        } else {
            const QuadOrder q = quad_order(load_quad(a.nodes, ref, a.B), p);
            if constexpr (FEW)
                q.rest(best, [&](uint32_t x, float) { fetch_child(a.nodes, a.tris, x); });
            push_rest(col, top, q, best);
            if (q.any(best)) {
                ref = q.next(best);
                return false;
            }
        }
        while (!col.empty(top)) {
            const uint2 e = col.pop(top);
            if (__uint_as_float(e.y) < best) {
                ref = e.x;
                return false;
            }
        }
        return true;
    }

    __device__ __forceinline__ void finish() { write_hit(a, idx, r, hit, best); }
};

// 56 registers, so 9 resident blocks of 128 with 24 stack entries in shared
// memory. 1M triangles, 4,194,304 reordered rays: 3.21 ms against 3.64 over the
// binary nodes (634M against 791M warp instructions for 1M rays: bound by issue
// and the latency of L2; whole stacks in shared memory, 6 blocks, gave 3.70).
// 300,000 triangles, 1,500,007 rays in input order, default call: 1.67 ms
// against 3.09 for one ray per thread over the binary nodes.
__global__ void __maxnreg__(64) k_mesh_closest_refill(const __grid_constant__ MeshArgs a) {
    extern __shared__ uint2 smem[];
    uint2 own[kLocalStack];
    MeshClosest<false> b(a, smem, own);
    trace_rays(b, a.n, a.c);
}

// For batches that give each ray a lane of its own: the walk that keeps more
// loads under way (96 registers, 5 blocks of 128). 10,000 triangles, 4,099 rays
// 76 -> 67 us, 40,000 rays 157 -> 126; 300,000 triangles, 1,000 rays 196 -> 161,
// 40,000 rays 340 -> 285. An SM's registers hold blocks of up to kFewBlock
// threads of it; larger ones take the form above.
constexpr int kFewBlock = 640;
__global__ void __launch_bounds__(kFewBlock)
    k_mesh_closest_few(const __grid_constant__ MeshArgs a) {
    extern __shared__ uint2 smem[];
    uint2 own[kLocalStack];
    MeshClosest<true> b(a, smem, own);
    trace_rays(b, a.n, a.c);
}

// Persistent: each warp takes the next 32 rays from the counter until none
// are left. The counter is zeroed on the stream before the launch. 55 registers
// (61 without the bound), so the 9 blocks of 128 that the stacks leave room for:
// 4,194,304 rays on 10,000, 300,000 and 1,000,000 triangles 4.08, 7.65 and 5.64
// ms; whole stacks in shared memory 3.94, 7.44 and 5.76, but 30 and 34 entries
// are more than blocks of 1,024 have room for.
__global__ void __maxnreg__(56)
    k_mesh_closest_persistent(const __grid_constant__ MeshArgs a) {
    extern __shared__ uint2 smem[];
    uint2 own[kLocalStack];
    const QueryStack<uint2> st(smem, (uint2 *) a.c.spill, own, a.c.stack_sm, a.c.stack_cap,
                               a.B.check);
    const int lane = threadIdx.x & 31;
    for (;;) {
        uint32_t base = 0;
        if (lane == 0)
            base = atomicAdd(a.c.counter, 32u);
        base = __shfl_sync(0xffffffffu, base, 0);
        if (base >= a.n)
            break;
        if (base + lane < a.n) {
            const int64_t i = ray_at(a, base + lane);
            const RayD r = load_ray(a.O, a.D, i);
            const RayPre p = precompute(r);
            float t = kInf, u = 0.f, v = 0.f;
            const int hit =
                blas_closest_quad(a.nodes, a.tris, a.e2z, a.root, r, p, st, t, u, v, a.B);
            write_hit(a, i, r, hit, t);
        }
    }
}

// Persistent closest hit with postponed leaves (phased): a lane that reaches a
// leaf parks it and keeps walking interior nodes until it reaches a second
// leaf; each warp step is then either a node step for every lane that can
// walk or a triangle step for every lane holding a parked leaf (chosen when
// at least `tri_min` lanes hold one), so the two kinds of work no longer
// split a warp. Exactness: leaves are still taken in the reference's DFS
// order, and a parked leaf is re-tested against the closest hit at the time
// its triangles are tested (the box entry < closest test the reference makes
// when it reaches that leaf); the interior nodes walked meanwhile with an
// older closest hit only add leaves that this re-test then drops, since a
// box contains the boxes below it and the slab entry distance is monotone in
// the box.

constexpr uint32_t kNoRef = 0xFFFFFFFFu;

__global__ void __maxnreg__(64)
    k_mesh_closest_phased(const __grid_constant__ MeshArgs a, int refill, int tri_min) {
    extern __shared__ uint2 smem[];
    uint2 own[kLocalStack];
    const QueryStack<uint2> col(smem, (uint2 *) a.c.spill, own, a.c.stack_sm, a.c.stack_cap,
                                a.B.check);
    const int lane = threadIdx.x & 31;
    const unsigned full = 0xffffffffu;
    int64_t idx = -1;
    RayD r{};
    RayPair p{};
    float best = kInf;
    int hit = -1;
    uint32_t ref = kNoRef; // walk position: interior node, leaf waiting for the slot, or none
    float ref_t = 0.f;     // box entry distance of ref
    uint32_t ptri = 0;     // parked leaf: next triangle, triangles left, box entry
    int pcnt = 0;
    float pt = 0.f;
    uint32_t top = col.base;
    bool more = true; // warp-uniform: the ray counter is not exhausted
    for (;;) {
        const bool idle = idx < 0;
        const unsigned im = __ballot_sync(full, idle);
        if (!more && im == full)
            break;
        if (more && __popc(im) >= refill) {
            const int cnt = __popc(im);
            uint32_t base = 0;
            if (lane == 0)
                base = atomicAdd(a.c.counter, (unsigned) cnt);
            base = __shfl_sync(full, base, 0);
            if (base + cnt >= a.n)
                more = false;
            if (idle) {
                const uint32_t ni = base + __popc(im & ((1u << lane) - 1u));
                if (ni < a.n) {
                    idx = ray_at(a, ni);
                    r = load_ray(a.O, a.D, idx);
                    p = precompute_pair(r);
                    best = kInf;
                    hit = -1;
                    top = col.base;
                    ref = no_slab(p) ? kNoRef : a.root;
                    ref_t = -kInf; // the root is entered without a box test
                    pcnt = 0;
                }
            }
        }
        const bool act = idx >= 0;
        const bool leaf_wait = ref != kNoRef && (ref & kLeafBit);
        const bool tw = act && pcnt > 0;
        const bool nw = act && !(leaf_wait && pcnt > 0) && !(ref == kNoRef && col.empty(top));
        const unsigned tm = __ballot_sync(full, tw);
        const unsigned nm = __ballot_sync(full, nw);
        if (tm != 0 && (nm == 0 || __popc(tm) >= tri_min)) {
            if (tw) {
                if (pt < best) {
                    pt = -kInf; // the leaf passed; its other triangles follow unconditionally
                    const TriV T = load_tri(a.tris, a.e2z, ptri, a.B);
                    float t, u, v;
                    if (tri_hit(T, r, t, u, v) && t < best) {
                        best = t;
                        hit = (int) ptri;
                    }
                    ptri++;
                    pcnt--;
                } else {
                    pcnt = 0;
                }
            }
        } else if (nw) {
            if (ref != kNoRef && !(ref & kLeafBit)) {
                const QuadOrder q = quad_order(load_quad(a.nodes, ref, a.B), p);
                push_rest(col, top, q, best);
                ref = q.any(best) ? q.next(best) : kNoRef;
                ref_t = q.next_t(best);
            }
            if (ref != kNoRef && (ref & kLeafBit) && pcnt == 0) {
                ptri = leaf_first(ref);
                pcnt = (int) leaf_count(ref);
                pt = ref_t;
                ref = kNoRef;
            }
            while (ref == kNoRef && !col.empty(top)) {
                const uint2 e = col.pop(top);
                if (__uint_as_float(e.y) < best) {
                    ref = e.x;
                    ref_t = __uint_as_float(e.y);
                }
            }
        }
        if (act && ref == kNoRef && col.empty(top) && pcnt == 0) {
            write_hit(a, idx, r, hit, best);
            idx = -1;
        }
    }
}

// One ray of an any-hit query on one mesh (BVHAccel::IntersectP).
template <bool FEW> struct MeshAny {
    const MeshArgs &a;
    const float *tmaxs;
    uint8_t *out;
    const float *box; // the mesh's root box
    const QueryStack<uint32_t> col;
    uint32_t idx = 0;
    RayD r;
    RayPair p;
    float tmax = 0.f;
    uint32_t ref = 0; // as in MeshClosest
    uint32_t top = 0;
    bool occluded = false;

    __device__ __forceinline__ MeshAny(const MeshArgs &args, const float *root_box,
                                       const float *tmax_, uint8_t *hit, uint32_t *smem,
                                       uint32_t *own)
        : a(args), tmaxs(tmax_), out(hit), box(root_box),
          col(smem, (uint32_t *) args.c.spill, own, args.c.stack_sm, args.c.stack_cap,
              args.B.check) {}

    __device__ __forceinline__ bool start(uint32_t i) {
        idx = i;
        r = load_ray(a.O, a.D, i);
        p = precompute_pair(r);
        tmax = __ldg(tmaxs + i);
        top = col.base;
        occluded = false;
        if (!(slab6(box, p) < tmax) || no_slab(p)) {
            finish();
            return false;
        }
        ref = a.root;
        return true;
    }

    __device__ __forceinline__ bool step() {
        if (ref & kLeafBit) {
            const uint32_t tri = leaf_first(ref);
            if constexpr (FEW) {
                const uint32_t ntri = leaf_count(ref);
                TriV T[4];
#pragma unroll
                for (uint32_t k = 0; k < 4; k++)
                    if (k < ntri)
                        T[k] = load_tri(a.tris, a.e2z, tri + k, a.B);
#pragma unroll
                for (uint32_t k = 0; k < 4; k++)
                    if (k < ntri && tri_occludes(T[k], r, tmax))
                        occluded = true;
                if (occluded)
                    return true;
            } else {
                if (tri_occludes(load_tri(a.tris, a.e2z, tri, a.B), r, tmax)) {
                    occluded = true;
                    return true;
                }
                ref = leaf_rest(ref);
                if (ref)
                    return false;
            }
        } else {
            const QuadOrder q = quad_order(load_quad(a.nodes, ref, a.B), p);
            if constexpr (FEW)
                q.rest(tmax, [&](uint32_t x, float) { fetch_child(a.nodes, a.tris, x); });
            push_rest(col, top, q, tmax);
            if (q.any(tmax)) {
                ref = q.next(tmax);
                return false;
            }
        }
        if (col.empty(top))
            return true;
        ref = col.pop(top);
        return false;
    }

    __device__ __forceinline__ void finish() { out[idx] = occluded ? 1 : 0; }
};

struct MeshBox {
    float b[6];
};

template <bool FEW>
__global__ void __maxnreg__(FEW ? 128 : 64) k_mesh_occluded(const __grid_constant__ MeshArgs a,
                                                const __grid_constant__ MeshBox box,
                                                const float *tmax, uint8_t *out) {
    extern __shared__ uint32_t smem32[];
    uint32_t own[kLocalStack];
    MeshAny<FEW> b(a, box.b, tmax, out, smem32, own);
    trace_rays(b, a.n, a.c);
}

// Scene-level queries: the resumable two-level walks of trace_step.cuh.
struct SceneArgs {
    const float *O, *D;
    uint32_t n;
    TraceCfg c;
};

template <class E>
__device__ __forceinline__ QueryStack<E> scene_col(const DevScene &S, const TraceCfg &c, E *smem,
                                                   E *own) {
    return QueryStack<E>(smem, (E *) c.spill, own, c.stack_sm, c.stack_cap, S.check);
}

// Coordinates and normal of the hit of ray r on object ob at ht (tri: leaf-order
// triangle index, of a mesh).
__device__ __forceinline__ void hit_geometry(const DevScene &S, const RayD &r, const DevObject &o,
                                             int tri, float ht, float *geo) {
    // hit coords (Triangle.cpp:37 / Sphere.hpp:37): origin + direction * t
    const float cx = r.ox + r.dx * ht, cy = r.oy + r.dy * ht, cz = r.oz + r.dz * ht;
    float nx, ny, nz;
    if (o.kind == kObjMesh) {
        nx = S.normals[(size_t) tri * 3 + 0];
        ny = S.normals[(size_t) tri * 3 + 1];
        nz = S.normals[(size_t) tri * 3 + 2];
        if (o.attr & kAttrNormals) {
            // Triangle::finalize (Triangle.cpp:44-47): normalize(n0*w0 + n1*u + n2*v)
            float t, u, v;
            tri_hit(load_tri(S, (uint32_t) tri), r, t, u, v);
            const float w0 = 1.f - u - v;
            const float *R = S.attr + (size_t) (o.attr_base + (tri - o.tri_base)) * kAttrFloats;
            nx = R[0] * w0 + R[3] * u + R[6] * v;
            ny = R[1] * w0 + R[4] * u + R[7] * v;
            nz = R[2] * w0 + R[5] * u + R[8] * v;
            const float m2 = nx * nx + ny * ny + nz * nz;
            if (m2 > 0) {
                const float inv = 1 / sqrtf(m2);
                nx = nx * inv;
                ny = ny * inv;
                nz = nz * inv;
            }
        }
    } else {
        // normalize(coords - center) (Vector.hpp:103-111)
        nx = cx - o.cx;
        ny = cy - o.cy;
        nz = cz - o.cz;
        const float m2 = nx * nx + ny * ny + nz * nz;
        if (m2 > 0) {
            const float inv = 1 / sqrtf(m2);
            nx = nx * inv;
            ny = ny * inv;
            nz = nz * inv;
        }
    }
    geo[0] = cx;
    geo[1] = cy;
    geo[2] = cz;
    geo[3] = nx;
    geo[4] = ny;
    geo[5] = nz;
}

// 2,000,003 rays on 122,880 triangles with geometry, half of them incoherent:
// 0.50 ms against 0.74 for one ray per thread; any hit 0.35 against 0.81.
// Geometry: the FEW form writes it as a ray ends, which saves a launch (1,000 rays
// with geometry in the museum-like scene of 7,680 triangles 61.8 -> 56.9 us, in
// the Cornell box 40.4 -> 36.6). The other leaves it to k_scene_finish, as here a
// few lanes at a time would make its loads and stores while the rest of their
// warp waits.
template <bool FEW> struct SceneClosest {
    const DevScene &S;
    const SceneArgs &a;
    int32_t *out_obj, *out_prim;
    float *out_t, *out_geo;
    const QueryStack<uint2> col;
    uint32_t idx = 0;
    ClosestWalk<FEW> w;

    __device__ __forceinline__ SceneClosest(const DevScene &scene, const SceneArgs &args,
                                            int32_t *obj, int32_t *prim, float *t, float *geo,
                                            uint2 *smem, uint2 *own)
        : S(scene), a(args), out_obj(obj), out_prim(prim), out_t(t), out_geo(geo),
          col(scene_col(scene, args.c, smem, own)) {}

    __device__ __forceinline__ bool start(uint32_t i) {
        idx = i;
        if (w.start(S, load_ray(a.O, a.D, i), col))
            return true;
        finish();
        return false;
    }
    __device__ __forceinline__ bool step() { return w.step(S, col); }
    __device__ __forceinline__ void finish() {
        out_obj[idx] = w.hit_obj;
        out_t[idx] = w.best;
        int prim = w.hit_tri;
        if ((FEW || !out_geo) && w.hit_obj >= 0) {
            prim = prim >= 0 ? __ldg(&S.tri_meta[prim].id) : 0;
            if (FEW && out_geo)
                hit_geometry(S, w.r, S.objects[w.hit_obj], w.hit_tri, w.best,
                             out_geo + (size_t) idx * 6);
        }
        out_prim[idx] = prim;
    }
};

template <bool FEW>
__global__ void __maxnreg__(FEW ? 128 : 64)
    k_scene_closest(const __grid_constant__ DevScene S, const __grid_constant__ SceneArgs a,
                    int32_t *out_obj, int32_t *out_prim, float *out_t, float *geo) {
    extern __shared__ uint2 smem[];
    uint2 own[kLocalStack];
    SceneClosest<FEW> b(S, a, out_obj, out_prim, out_t, geo, smem, own);
    trace_rays(b, a.n, a.c);
}

// Hit geometry of a large scene query, one thread per ray, so its loads and
// stores are coalesced. out_prim holds leaf-order triangle indices (-1 for a
// sphere) and is resolved here.
__global__ void __launch_bounds__(256)
    k_scene_finish(const __grid_constant__ DevScene S, const float *O, const float *D, int64_t n,
                   const int32_t *obj, int32_t *prim, const float *ts, float *geo) {
    const int64_t i = (int64_t) blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n)
        return;
    const int ob = obj[i];
    if (ob < 0)
        return; // a miss: prim is -1, its geometry is left as it was
    const int tri = prim[i];
    prim[i] = tri >= 0 ? __ldg(&S.tri_meta[tri].id) : 0;
    hit_geometry(S, load_ray(O, D, i), S.objects[ob], tri, ts[i], geo + i * 6);
}

template <bool FEW> struct SceneAny {
    const DevScene &S;
    const SceneArgs &a;
    const float *tmaxs;
    uint8_t *out;
    const QueryStack<uint32_t> col;
    uint32_t idx = 0;
    AnyWalk<FEW> w;

    __device__ __forceinline__ SceneAny(const DevScene &scene, const SceneArgs &args,
                                        const float *tmax, uint8_t *hit, uint32_t *smem,
                                        uint32_t *own)
        : S(scene), a(args), tmaxs(tmax), out(hit), col(scene_col(scene, args.c, smem, own)) {}

    __device__ __forceinline__ bool start(uint32_t i) {
        idx = i;
        if (w.start(S, load_ray(a.O, a.D, i), __ldg(tmaxs + i), col))
            return true;
        finish();
        return false;
    }
    __device__ __forceinline__ bool step() { return w.step(S, col); }
    __device__ __forceinline__ void finish() { out[idx] = w.occluded ? 1 : 0; }
};

template <bool FEW>
__global__ void __maxnreg__(FEW ? 128 : 64)
    k_scene_occluded(const __grid_constant__ DevScene S, const __grid_constant__ SceneArgs a,
                     const float *tmax, uint8_t *out) {
    extern __shared__ uint32_t smem32[];
    uint32_t own[kLocalStack];
    SceneAny<FEW> b(S, a, tmax, out, smem32, own);
    trace_rays(b, a.n, a.c);
}

// ---------------------------------------------------------------- ray order
// Coherence reordering before a closest-hit batch. Each ray gets a 30-bit key
// from where it enters the mesh's root box (its origin if it starts inside)
// and its normalised direction, each quantised to 5 bits per axis; the
// buckets are the key's top `bits` bits. A counting pass, an exclusive scan
// and a scatter with one atomic per ray give a permutation grouped by bucket
// (the order inside a bucket is whatever the atomics give: it does not matter,
// because every ray's result is written at its own input index and the walk
// of one ray does not depend on any other). Rays that miss the root box get
// the last bucket.

// bit k of v (k < 5) to bit 6k, for a 6-way interleave
__device__ __forceinline__ uint32_t spread6(uint32_t v) {
    uint32_t r = 0;
#pragma unroll
    for (int b = 0; b < 5; b++)
        r |= ((v >> b) & 1u) << (6 * b);
    return r;
}

// bit k of v (k < 5) to bit 3k, for a 3-way interleave
__device__ __forceinline__ uint32_t spread3(uint32_t v) {
    uint32_t r = 0;
#pragma unroll
    for (int b = 0; b < 5; b++)
        r |= ((v >> b) & 1u) << (3 * b);
    return r;
}

__device__ __forceinline__ uint32_t quant5(float u) {
    const float q = u * 32.f;
    return q <= 0.f ? 0u : (q >= 31.f ? 31u : (uint32_t) q);
}

struct RayKeyArgs {
    const float *O, *D;
    int64_t n;
    float box[6]; // root box [minX,maxX,minY,maxY,minZ,maxZ]
    int mode;     // 1 entry and direction interleaved, 2 direction-major, 3 entry-major,
                  // 4 entry and exit point interleaved, 5 entry-major then exit
    int shift;    // key >> shift = bucket
    uint32_t *bucket;
    uint32_t *count;
};

__global__ void k_ray_buckets(RayKeyArgs a) {
    const int64_t i = (int64_t) blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= a.n)
        return;
    const RayD r = load_ray(a.O, a.D, i);
    const RayPre p = precompute(r);
    const float t = slab(a.box[0], a.box[1], a.box[2], a.box[3], a.box[4], a.box[5], p);
    uint32_t key = (1u << 30) - 1u;
    if (t < kInf) {
        const float ex = (r.ox + r.dx * t - a.box[0]) / (a.box[1] - a.box[0]);
        const float ey = (r.oy + r.dy * t - a.box[2]) / (a.box[3] - a.box[2]);
        const float ez = (r.oz + r.dz * t - a.box[4]) / (a.box[5] - a.box[4]);
        const float inv = rsqrtf(r.dx * r.dx + r.dy * r.dy + r.dz * r.dz);
        const uint32_t qx = quant5(ex), qy = quant5(ey), qz = quant5(ez);
        const uint32_t dx = quant5(0.5f + 0.5f * r.dx * inv);
        const uint32_t dy = quant5(0.5f + 0.5f * r.dy * inv);
        const uint32_t dz = quant5(0.5f + 0.5f * r.dz * inv);
        const uint32_t e3 = spread3(qx) << 2 | spread3(qy) << 1 | spread3(qz);
        const uint32_t d3 = spread3(dx) << 2 | spread3(dy) << 1 | spread3(dz);
        if (a.mode == 2) {
            key = d3 << 15 | e3;
        } else if (a.mode == 3) {
            key = e3 << 15 | d3;
        } else if (a.mode >= 4) {
            // where the ray leaves the box: the nearest far slab
            const float fx = ((p.nx ? a.box[0] : a.box[1]) - p.ox) * p.ix;
            const float fy = ((p.ny ? a.box[2] : a.box[3]) - p.oy) * p.iy;
            const float fz = ((p.nz ? a.box[4] : a.box[5]) - p.oz) * p.iz;
            const float tx = fminf(fx, fminf(fy, fz));
            const uint32_t xx = quant5((r.ox + r.dx * tx - a.box[0]) / (a.box[1] - a.box[0]));
            const uint32_t xy = quant5((r.oy + r.dy * tx - a.box[2]) / (a.box[3] - a.box[2]));
            const uint32_t xz = quant5((r.oz + r.dz * tx - a.box[4]) / (a.box[5] - a.box[4]));
            if (a.mode == 4)
                key = spread6(qx) << 5 | spread6(qy) << 4 | spread6(qz) << 3 | spread6(xx) << 2 |
                      spread6(xy) << 1 | spread6(xz);
            else
                key = e3 << 15 | spread3(xx) << 2 | spread3(xy) << 1 | spread3(xz);
        } else {
            key = spread6(qx) << 5 | spread6(qy) << 4 | spread6(qz) << 3 | spread6(dx) << 2 |
                  spread6(dy) << 1 | spread6(dz);
        }
    }
    const uint32_t b = key >> a.shift;
    a.bucket[i] = b;
    atomicAdd(a.count + b, 1u);
}

// Exclusive scan of count[0, m) in place, in tiles of 4096 (1024 threads x 4):
// tile sums first, then the sums' scan, then the tiles.
constexpr int kScanTile = 4096;

__device__ __forceinline__ uint32_t block_exclusive_scan(uint32_t v, uint32_t *sh,
                                                         uint32_t *total) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint32_t x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o)
            x += y;
    }
    if (lane == 31)
        sh[warp] = x;
    __syncthreads();
    if (warp == 0) {
        const int nw = blockDim.x >> 5;
        uint32_t w = lane < nw ? sh[lane] : 0u;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(0xffffffffu, w, o);
            if (lane >= o)
                w += y;
        }
        if (lane < nw)
            sh[lane] = w;
    }
    __syncthreads();
    const uint32_t before = (warp > 0 ? sh[warp - 1] : 0u) + x - v;
    if (total)
        *total = sh[(blockDim.x >> 5) - 1];
    __syncthreads();
    return before;
}

__global__ void k_scan_tile_sums(const uint32_t *count, int64_t m, uint32_t *sums) {
    __shared__ uint32_t sh[32];
    const int64_t base = (int64_t) blockIdx.x * kScanTile + (int64_t) threadIdx.x * 4;
    uint32_t v = 0;
    for (int k = 0; k < 4; k++)
        if (base + k < m)
            v += count[base + k];
    uint32_t total = 0;
    block_exclusive_scan(v, sh, &total);
    if (threadIdx.x == 0)
        sums[blockIdx.x] = total;
}

// one block: exclusive scan of the tile sums (at most 1024 tiles)
__global__ void k_scan_sums(uint32_t *sums, int tiles) {
    __shared__ uint32_t sh[32];
    const uint32_t v = (int) threadIdx.x < tiles ? sums[threadIdx.x] : 0u;
    const uint32_t e = block_exclusive_scan(v, sh, nullptr);
    if ((int) threadIdx.x < tiles)
        sums[threadIdx.x] = e;
}

__global__ void k_scan_tiles(uint32_t *count, int64_t m, const uint32_t *sums) {
    __shared__ uint32_t sh[32];
    const int64_t base = (int64_t) blockIdx.x * kScanTile + (int64_t) threadIdx.x * 4;
    uint32_t c[4], v = 0;
    for (int k = 0; k < 4; k++) {
        c[k] = base + k < m ? count[base + k] : 0u;
        v += c[k];
    }
    uint32_t run = sums[blockIdx.x] + block_exclusive_scan(v, sh, nullptr);
    for (int k = 0; k < 4; k++)
        if (base + k < m) {
            count[base + k] = run;
            run += c[k];
        }
}

__global__ void k_ray_scatter(const uint32_t *bucket, int64_t n, uint32_t *offset,
                              uint32_t *perm) {
    const int64_t i = (int64_t) blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n)
        return;
    const uint32_t pos = atomicAdd(offset + bucket[i], 1u);
    perm[pos] = (uint32_t) i;
}

// Bucket bits for n rays: about 8 rays per bucket, 2^8 .. 2^22 buckets (the
// scan handles at most 1024 tiles of 4096).
int ray_bucket_bits(int64_t n) {
    int b = 0;
    while (b < 30 && (int64_t(1) << b) < n)
        b++;
    return std::max(8, std::min(22, b - 3));
}

// Device bytes of the reordering scratch for n rays.
size_t ray_order_bytes(int64_t n) {
    const int64_t m = int64_t(1) << ray_bucket_bits(n);
    const int64_t tiles = (m + kScanTile - 1) / kScanTile;
    return (size_t) (2 * n + m + tiles) * sizeof(uint32_t);
}

// Fills perm[0, n) with the coherence order of the rays (scratch from
// ray_order_bytes(n), which starts with perm).
int ray_order(const float *o, const float *d, int64_t n, const float box[6], int mode,
              void *scratch, cudaStream_t st) {
    const int bits = ray_bucket_bits(n);
    const int64_t m = int64_t(1) << bits;
    const int64_t tiles = (m + kScanTile - 1) / kScanTile;
    uint32_t *perm = (uint32_t *) scratch;
    uint32_t *bucket = perm + n;
    uint32_t *count = bucket + n;
    uint32_t *sums = count + m;
    RayKeyArgs a;
    a.O = o;
    a.D = d;
    a.n = n;
    for (int k = 0; k < 6; k++)
        a.box[k] = box[k];
    a.mode = mode;
    a.shift = 30 - bits;
    a.bucket = bucket;
    a.count = count;
    PRR_CUDA_TRY(cudaMemsetAsync(count, 0, (size_t) m * sizeof(uint32_t), st));
    const unsigned g = (unsigned) ((n + 255) / 256);
    k_ray_buckets<<<g, 256, 0, st>>>(a);
    k_scan_tile_sums<<<(unsigned) tiles, 1024, 0, st>>>(count, m, sums);
    k_scan_sums<<<1, 1024, 0, st>>>(sums, (int) tiles);
    k_scan_tiles<<<(unsigned) tiles, 1024, 0, st>>>(count, m, sums);
    k_ray_scatter<<<g, 256, 0, st>>>(bucket, n, count, perm);
    PRR_CUDA_TRY(cudaGetLastError());
    return PRR_OK;
}

TraceBounds host_bounds(const DevScene &S) {
    return TraceBounds{S.n_nodes, S.n_qnodes, S.n_tris, S.check};
}

int stack_cap(int depth) {
    // entries outstanding <= the bound found when the tree was packed; one spare slot
    return std::max(1, depth + 1);
}

int set_smem(const void *fn, size_t bytes) {
    // The stack columns live in shared memory: ask for the largest carveout so
    // the resident-block count the occupancy query reports is what launches.
    cudaFuncSetAttribute(fn, cudaFuncAttributePreferredSharedMemoryCarveout,
                         cudaSharedmemCarveoutMaxShared);
    if (bytes > 48 * 1024) {
        cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                             (int) bytes);
        if (e != cudaSuccess)
            return fail(PRR_ERR_CUDA, std::string("cudaFuncSetAttribute: ") + cudaGetErrorString(e));
    }
    return PRR_OK;
}

} // namespace

int device_sm_count() {
    static int sms = [] {
        int dev = 0, v = 0;
        cudaGetDevice(&dev);
        if (cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || v <= 0)
            v = 148;
        return v;
    }();
    return sms;
}

namespace {

// Stack entries a query kernel keeps in shared memory: 9 blocks of 128
// threads, what its registers allow, fill an SM's shared memory at 24 entries
// of 8 bytes. Deeper entries go to local memory, or, where kLocalStack are too
// few, to a per-call global buffer.
constexpr int kStackSm = 24;
constexpr size_t kMaxSmem = 227 * 1024; // shared memory of a block at most

// Device scratch of one call, from the library's stream-ordered pool and given
// back on the stream: concurrent calls on other streams get their own.
struct CallScratch {
    char *ptr = nullptr;
    cudaStream_t st = nullptr;
    ~CallScratch() {
        if (ptr)
            cudaFreeAsync(ptr, st);
    }
    int alloc(size_t bytes, cudaStream_t stream) {
        cudaMemPool_t pool;
        PRR_CUDA_TRY(library_pool(&pool));
        st = stream;
        PRR_CUDA_TRY(cudaMallocFromPoolAsync((void **) &ptr, bytes, pool, stream));
        return PRR_OK;
    }
};

// True while the stream is being captured into a graph: such calls allocate
// nothing and keep no counter, as a replayed graph may overlap other calls. The
// entries of a stack that local memory does not hold are then all shared.
bool capturing(cudaStream_t st) {
    cudaStreamCaptureStatus s = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(st, &s) != cudaSuccess) {
        cudaGetLastError();
        return true;
    }
    return s != cudaStreamCaptureStatusNone;
}

// Rays of one launch: the kernels index with 32 bits. Larger batches are
// traced launch after launch on their stream.
constexpr int64_t kMaxLaunch = int64_t(1) << 31;

// Batches traced by the FEW form of a kernel: up to 640 rays per SM, what its
// residents (4 or 5 blocks of 128) hold at once or little more. Closest hit on
// one mesh takes it to 740, and on large meshes (walks of 24 stack entries and
// more, from about 50,000 triangles on) to 1,280, their rays being slower apart
// than the larger batch's queueing. Times of the form over the other's, at
// 110,000, 130,000 and 160,000 rays: 1,000 triangles 1.03, 1.10, 1.13; 10,000
// 0.97, 1.05, 1.05; 100,000 0.83, 0.84, 0.90; 1,000,000 0.87, 0.89, 0.88 (250,000
// rays 0.96); scene level, museum-like of 1,920 to 491,520 triangles, 94,000
// rays 0.89 to 0.84, 130,000 1.06 to 0.93.
bool few_rays(int64_t n, int per_sm = 640) { return n <= (int64_t) device_sm_count() * per_sm; }

// Launch shape of a query kernel over n rays: shared memory, grid, and the
// scratch it needs (counter and stack spill). The grid is what the device
// holds at once, less for batches that give its warps less than one ray each.
struct TraceLaunch {
    size_t smem = 0;
    unsigned grid = 1;
    CallScratch scratch;
};

//
// A counter costs a call an allocation, a clear and the atomics, so rays are
// counted out only when a warp's share is more than a few rounds of its lanes
// (count_from). Closest hit on one mesh: one round, 32 (10,000 triangles,
// 200,000 rays 260 us, 275 with fixed shares of two). The other queries, whose
// rays differ less: two, 64 (94,000 rays, counted / fixed: any hit on 10,000
// triangles 40.9 / 35.5 us, closest hit in the Cornell box 18.4 / 15.0, in the
// museum-like scene of 30,720 triangles 78.9 / 74.5, of 491,520 105 / 107).
int plan_trace(TraceLaunch &L, TraceCfg &c, const void *fn, int block, int cap, size_t entry,
               int64_t n, int blocks_per_sm, int refill, int count_from, bool counter_always,
               unsigned *counter, bool in_capture, cudaStream_t st) {
    c.stack_cap = cap;
    c.stack_sm = std::min(cap, kStackSm);
    if (in_capture)
        c.stack_sm = std::max(c.stack_sm, cap - kLocalStack);
    const bool local = cap - c.stack_sm <= kLocalStack;
    c.counter = nullptr;
    c.spill = nullptr;
    L.smem = (size_t) c.stack_sm * block * entry;
    if (L.smem > kMaxSmem)
        return fail(PRR_ERR_UNSUPPORTED, "BVH too deep for the shared-memory stack");
    if (int rc = set_smem(fn, L.smem))
        return rc;
    int bps = 0; // blocks resident per SM
    PRR_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&bps, fn, block, L.smem));
    if (bps == 0)
        return fail(PRR_ERR_INTERNAL, "no block of the query kernel fits an SM");
    if (blocks_per_sm > 0)
        bps = blocks_per_sm;
    const int64_t resident = (int64_t) device_sm_count() * bps;
    const int64_t warps = resident * (block / 32);
    c.share = (uint32_t) ((n + warps - 1) / warps);
    c.lanes = (int) std::min(32u, c.share);
    c.refill = std::min(refill, c.lanes);
    const int64_t per_block = (int64_t) c.lanes * (block / 32);
    L.grid = (unsigned) std::min<int64_t>(resident, (n + per_block - 1) / per_block);
    const bool count = counter_always || (n > warps * count_from && !in_capture);
    size_t bytes = count && !counter ? 256 : 0;
    const size_t spill_at = bytes;
    if (!local)
        bytes += (size_t) (cap - c.stack_sm) * L.grid * block * entry;
    if (bytes)
        if (int rc = L.scratch.alloc(bytes, st))
            return rc;
    if (!local)
        c.spill = L.scratch.ptr + spill_at;
    if (count) {
        c.counter = counter ? counter : (unsigned *) L.scratch.ptr;
        PRR_CUDA_TRY(cudaMemsetAsync(c.counter, 0, sizeof(unsigned), st));
    }
    return PRR_OK;
}

} // namespace

int launch_mesh_closest(const Scene &s, int object, const float *o, const float *d, int64_t n,
                        int32_t *id, float *t, double *t64, unsigned *counter,
                        const prr_trace_config *cfg, cudaStream_t st) {
    if (n == 0)
        return PRR_OK;
    for (; n > kMaxLaunch; n -= kMaxLaunch, o += kMaxLaunch * 3, d += kMaxLaunch * 3,
                           id += kMaxLaunch, t += kMaxLaunch, t64 += t64 ? kMaxLaunch : 0)
        if (int rc = launch_mesh_closest(s, object, o, d, kMaxLaunch, id, t, t64, counter, cfg,
                                         st))
            return rc;
    const HostObject &obj = s.objects[object];
    MeshArgs a;
    a.nodes = s.dev.qnodes;
    a.tris = s.dev.tris;
    a.e2z = s.dev.tri_e2z;
    a.meta = s.dev.tri_meta;
    a.verts = s.dev.verts;
    a.root = obj.qroot;
    a.O = o;
    a.D = d;
    a.n = (uint32_t) n;
    a.out_id = id;
    a.out_t = t;
    a.out_t64 = t64;
    a.perm = nullptr;
    a.B = host_bounds(s.dev);
    const int block = (cfg && cfg->block_size > 0) ? cfg->block_size : 128;
    if (block % 32 != 0 || block > 1024)
        return fail(PRR_ERR_INVALID_ARGUMENT, "block_size must be a multiple of 32 <= 1024");
    const int mode = cfg ? cfg->persistent : 0;
    if (mode < 0 || mode > 3)
        return fail(PRR_ERR_INVALID_ARGUMENT, "persistent must be 0, 1, 2 or 3");
    const int sort = cfg ? cfg->sort_rays : 0;
    if (sort < 0 || sort > 5)
        return fail(PRR_ERR_INVALID_ARGUMENT, "sort_rays must be 0 to 5");
    const bool in_capture = capturing(st);
    // a counter of the scene serves captured persistent launches, which
    // allocate nothing; every other call gets its own
    if (in_capture && mode > 0 && !counter)
        counter = (unsigned *) s.d_counter.ptr;
    const bool few =
        mode == 0 && block <= kFewBlock && few_rays(n, obj.qstack >= 24 ? 1280 : 740);
    const int cap = stack_cap(obj.qstack);
    const void *fn = mode == 1   ? (const void *) k_mesh_closest_persistent
                     : mode == 3 ? (const void *) k_mesh_closest_phased
                     : few       ? (const void *) k_mesh_closest_few
                                 : (const void *) k_mesh_closest_refill;
    const int refill = mode >= 2 && cfg->batch > 0 ? std::min(cfg->batch, 32) : 8;
    TraceLaunch L;
    if (int rc = plan_trace(L, a.c, fn, block, cap, sizeof(uint2), n,
                            mode > 0 ? cfg->blocks_per_sm : 0, refill, 32, mode > 0, counter,
                            in_capture, st))
        return rc;
    CallScratch order;
    if (sort > 0 && n < (int64_t(1) << 31)) {
        if (int rc = order.alloc(ray_order_bytes(n), st))
            return rc;
        float box[6];
        for (int k = 0; k < 6; k++)
            box[k] = obj.bvh.bounds[k];
        if (int rc = ray_order(o, d, n, box, sort, order.ptr, st))
            return rc;
        a.perm = (const uint32_t *) order.ptr;
    }
    if (mode == 1)
        k_mesh_closest_persistent<<<L.grid, block, L.smem, st>>>(a);
    else if (mode == 3)
        k_mesh_closest_phased<<<L.grid, block, L.smem, st>>>(
            a, refill, cfg->leaf_batch > 0 ? std::min(cfg->leaf_batch, 32) : 16);
    else if (few)
        k_mesh_closest_few<<<L.grid, block, L.smem, st>>>(a);
    else
        k_mesh_closest_refill<<<L.grid, block, L.smem, st>>>(a);
    PRR_CUDA_TRY(cudaGetLastError());
    return PRR_OK;
}

int launch_mesh_occluded(const Scene &s, int object, const float *o, const float *d,
                         const float *tmax, int64_t n, uint8_t *hit, cudaStream_t st) {
    if (n == 0)
        return PRR_OK;
    for (; n > kMaxLaunch; n -= kMaxLaunch, o += kMaxLaunch * 3, d += kMaxLaunch * 3,
                           tmax += kMaxLaunch, hit += kMaxLaunch)
        if (int rc = launch_mesh_occluded(s, object, o, d, tmax, kMaxLaunch, hit, st))
            return rc;
    const HostObject &obj = s.objects[object];
    MeshArgs a{};
    a.nodes = s.dev.qnodes;
    a.tris = s.dev.tris;
    a.e2z = s.dev.tri_e2z;
    a.root = obj.qroot;
    a.O = o;
    a.D = d;
    a.n = (uint32_t) n;
    a.B = host_bounds(s.dev);
    MeshBox box;
    for (int k = 0; k < 6; k++)
        box.b[k] = obj.bvh.bounds[k];
    const int block = 128;
    TraceLaunch L;
    auto kern = few_rays(n) ? k_mesh_occluded<true> : k_mesh_occluded<false>;
    if (int rc = plan_trace(L, a.c, (const void *) kern, block, stack_cap(obj.qstack),
                            sizeof(uint32_t), n, 0, 8, 64, false, nullptr, capturing(st), st))
        return rc;
    kern<<<L.grid, block, L.smem, st>>>(a, box, tmax, hit);
    PRR_CUDA_TRY(cudaGetLastError());
    return PRR_OK;
}

int launch_scene_closest(const Scene &s, const float *o, const float *d, int64_t n,
                         int32_t *obj, int32_t *prim, float *t, float *geo, cudaStream_t st) {
    if (n == 0)
        return PRR_OK;
    for (; n > kMaxLaunch; n -= kMaxLaunch, o += kMaxLaunch * 3, d += kMaxLaunch * 3,
                           obj += kMaxLaunch, prim += kMaxLaunch, t += kMaxLaunch,
                           geo += geo ? kMaxLaunch * 6 : 0)
        if (int rc = launch_scene_closest(s, o, d, kMaxLaunch, obj, prim, t, geo, st))
            return rc;
    const int block = 128;
    SceneArgs a{o, d, (uint32_t) n, {}};
    TraceLaunch L;
    const bool few = few_rays(n);
    auto kern = few ? k_scene_closest<true> : k_scene_closest<false>;
    if (int rc = plan_trace(L, a.c, (const void *) kern, block,
                            stack_cap(s.dev.blas_stack + s.dev.tlas_stack),
                            sizeof(uint2), n, 0, 8, 64, false, nullptr, capturing(st), st))
        return rc;
    kern<<<L.grid, block, L.smem, st>>>(s.dev, a, obj, prim, t, geo);
    if (geo && !few)
        k_scene_finish<<<(unsigned) ((n + 255) / 256), 256, 0, st>>>(s.dev, o, d, n, obj, prim, t,
                                                                     geo);
    PRR_CUDA_TRY(cudaGetLastError());
    return PRR_OK;
}

int launch_scene_occluded(const Scene &s, const float *o, const float *d, const float *tmax,
                          int64_t n, uint8_t *hit, cudaStream_t st) {
    if (n == 0)
        return PRR_OK;
    for (; n > kMaxLaunch; n -= kMaxLaunch, o += kMaxLaunch * 3, d += kMaxLaunch * 3,
                           tmax += kMaxLaunch, hit += kMaxLaunch)
        if (int rc = launch_scene_occluded(s, o, d, tmax, kMaxLaunch, hit, st))
            return rc;
    const int block = 128;
    SceneArgs a{o, d, (uint32_t) n, {}};
    TraceLaunch L;
    auto kern = few_rays(n) ? k_scene_occluded<true> : k_scene_occluded<false>;
    if (int rc = plan_trace(L, a.c, (const void *) kern, block,
                            stack_cap(s.dev.blas_stack + s.dev.tlas_stack),
                            sizeof(uint32_t), n, 0, 8, 64, false, nullptr, capturing(st), st))
        return rc;
    kern<<<L.grid, block, L.smem, st>>>(s.dev, a, tmax, hit);
    PRR_CUDA_TRY(cudaGetLastError());
    return PRR_OK;
}

} // namespace prr
