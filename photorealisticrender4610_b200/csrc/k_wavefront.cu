// Wavefront integrator: Integrator::castRay (Integrator.cpp:104-263) cut into
// stages that run over queues of paths instead of one path per thread.
//
// A pass traces samples [base, base + k) of every pixel of the window at once
// (P = k * pixels paths). Per bounce:
//   extend   closest hit of every queued ray; the path is appended to the
//            miss, delta (mirror/glass) or surface (diffuse/emissive) queue of
//            its hit -- the sort by material, made with warp-aggregated appends
//   miss     background / env contributions, path ends
//   delta    specular chain step (Integrator.cpp:143-169)
//   surface  NEE towards emitters and the environment (shadow rays queued with
//            their would-be contributions), BSDF sample, next ray queued
//   shadow   any-hit of the queued shadow rays; visible contributions added
// The pending part of a non-delta bounce -- the MIS terms for an env miss or
// an emitter hit, beta *= f/pdf, Russian roulette (Integrator.cpp:205-256) --
// runs at the start of the stage that sees the next hit, so every path makes
// the same random draws and the same additions to L in the same order as
// castRay. At the end of a pass each pixel adds its k results in sample order,
// so the film is the plain renderer's, bit for bit.
//
// Every kernel reads its queue length from device memory, so a pass is one
// fixed launch sequence; it is captured once in a CUDA graph and replayed.
#include "integrator.cuh"
#include "prr_internal.h"
#include "trace_step.cuh"

#include <algorithm>
#include <cstring>

namespace prr {
namespace {

enum : int { kFlagSpecular = 1, kFlagPending = 2, kFlagEndAfterShadow = 4 };
enum : int {
    kCntRay0 = 0, kCntRay1 = 1, kCntMiss = 2, kCntDelta = 3, kCntSurf = 4, kCntShadow = 5,
    kCntExtend = 6, kCntShadowJobs = 7, kCntRays = 8, kCntShadowRays = 10, kCntShadowFetch = 12,
    kCntActive = 13, kCntSlots = 16
};

// One request of a multi-request step (the render server): its scene, camera
// and window, the samples this step traces, and where its paths and pixels
// start in the step's arrays.
struct WfReq {
    const DevScene *scene;
    DevCamera camera;
    int W, x0, y0, ww, wh, npix; // image width, window, window pixels
    int s0, nspp;                // samples [s0, s0 + nspp) of every window pixel
    int max_depth;
    float clamp;
    uint64_t seed;
    int64_t path_base, pix_base; // first path / first pixel of this request in the step
    float3 *film;                // running per-pixel sums, window order
    unsigned long long rays[2];  // closest, shadow rays traced (added by the kernels)
};

struct Wf {
    int P, npix, spp_pass;
    int W, x0, y0, ww, wh;
    int max_depth;
    float clamp;
    uint64_t seed;
    int tlas_cap, blas_cap; // stack entries a walk may need at the scene and mesh level
    int stack_sm;           // entries of the two kept in shared memory
    int count_stack;        // binary-walk entries of the counting variants, both levels
    void *spill;            // global part of the stacks ([entry][grid thread])
    // path state
    uint64_t *rng;
    float4 *ro, *rd;     // current ray
    float4 *beta;        // xyz
    float4 *L;           // xyz
    int *bounce, *flags;
    float4 *pend;        // pending BSDF: f/pdf xyz, pdf
    float4 *prev;        // pending BSDF: hit point it left from
    int4 *hit;           // obj, tri, t bits
    float4 *slo, *sld, *slc; // light shadow ray: origin+tmax, dir+valid, contribution
    float4 *seo, *sed, *sec; // env shadow ray
    float4 *result;      // final L per path
    float3 *film;        // per pixel running sum, in path order (tile_pixel)
    // queues
    int *qray[2], *qmiss, *qdelta, *qsurf, *qshadow, *qjob;
    uint8_t *vis;        // per shadow job (2 per path): 1 when nothing occludes
    unsigned *cnt;       // kCntSlots counters (64-bit ray totals at kCntRays, kCntShadowRays)
    int *pass_base;      // first sample of the current pass (advanced by the film kernel)
    int sample_offset;
    // ordered queues: stages tag paths instead of appending them, and a stable
    // partition builds the next queues in path (= pixel) order
    int ordered;
    uint8_t *tag;        // per path: bucket of the pending partition, 0xFF none
    unsigned *tile;      // per partition tile: 8 bucket counts, then offsets
    // adaptive sampling (min_spp < max_spp): each pass traces the next
    // spp_pass samples of the pixels still active; the film stage replays the
    // reference's per-sample Welford stop (Renderer.cpp:74-95) on them
    int adaptive, min_spp, max_spp;
    float threshold;
    int *act, *act_next; // active pixels (window-local indices), in pixel order
    uint8_t *ptag;       // per active slot: 0 = stays active, 0xFF = done
    float4 *wel0, *wel1; // per pixel: (n, mean r, g, b), (M2 r, g, b, -)
    // multi-request steps: the request table and each path's request
    WfReq *reqs;
    int n_reqs;
    int *req;
    // traversal counts (kStat* slots), filled only by the counting variants of
    // the extend and shadow stages
    unsigned long long *stats;
    uint32_t *check; // status words of the checked build (nullptr: not reported)
};

// The stages of a bounce are launched with programmatic dependence
// (launch_stage): the blocks of a stage are set up while the stage before it
// drains, and wait here, before they touch memory, until that stage has ended
// and its writes are visible. Every block of every stage waits, also one with
// nothing to do, so a stage that has ended implies all before it. The next
// stage is let in only after the wait: let in before it, the blocks of two
// later stages would hold slots that the draining stage's last blocks free.
// Launches with full ordering / let in before the wait / after it: museum-like
// scene at 960x540 x 16, depth 8, 12.33 / 12.15 / 12.12 ms; adaptive at 320x180
// up to 64 spp, depth 12, 6.63 / 6.38 / 6.34; 97x61 x 4 1.50 / 1.26 / 1.24; a
// box of 256x256 x 16 at depth 5 1.54 / 1.43 / 1.38.
__device__ __forceinline__ void stage_begin() {
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;");
}

// q[slot] = v for an appended queue entry; the checked build tests the slot
// against the queue's capacity (and drops and reports an entry beyond it).
__device__ __forceinline__ void queue_put(const Wf &w, int *q, int slot, int64_t cap, int v) {
#ifdef PRR_CHECKED
    if (slot < 0 || (int64_t) slot >= cap) {
        check_fail(w.check, kCheckQueue, (uint32_t) slot);
        return;
    }
#endif
    (void) w;
    (void) cap;
    q[slot] = v;
}

// A queue's length as a stage reads it. The checked build tests it against
// the queue's capacity (and reports and clamps a longer one).
__device__ __forceinline__ int queue_len(const Wf &w, unsigned n, int64_t cap) {
#ifdef PRR_CHECKED
    if ((int64_t) n > cap) {
        if (blockIdx.x == 0 && threadIdx.x == 0)
            check_fail(w.check, kCheckQueue, n);
        return (int) cap;
    }
#endif
    (void) w;
    (void) cap;
    return (int) n;
}

// Slots of Wf::stats: traversal work of closest-hit (extend) and shadow rays
// (interior nodes of either BVH level, triangle tests, object leaves: mesh
// entries and sphere tests) and the extend results by class.
enum : int {
    kStatClosestNodes = 0, kStatClosestTris = 1, kStatClosestObjects = 2,
    kStatShadowNodes = 3, kStatShadowTris = 4, kStatShadowObjects = 5,
    kStatMiss = 6, kStatDelta = 7, kStatSurface = 8, kStatSlots = 9
};
static_assert(kStatSlots == kWfStatSlots, "counter slots of prr_render_counts");

// Adds a lane's counts to the stats slots [slot, slot + n), one atomic per
// slot per warp.
template <int N>
__device__ __forceinline__ void flush_stats(unsigned long long *stats, int slot,
                                            const unsigned (&c)[N]) {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int k = 0; k < N; k++) {
        unsigned long long v = c[k];
        for (int off = 16; off > 0; off >>= 1)
            v += __shfl_down_sync(0xffffffffu, v, off);
        if (lane == 0 && v)
            atomicAdd(stats + slot + k, v);
    }
}

// Per-path scene, clamp and depth: the kernel's own for a render, the path's
// request's for a server step.
template <bool MULTI>
__device__ __forceinline__ const DevScene &scene_of(const DevScene &S0, const Wf &w, int p) {
    if constexpr (MULTI)
        return *w.reqs[w.req[p]].scene;
    else
        return S0;
}
template <bool MULTI> __device__ __forceinline__ float clamp_of(const Wf &w, int p) {
    if constexpr (MULTI)
        return w.reqs[w.req[p]].clamp;
    else
        return w.clamp;
}
template <bool MULTI> __device__ __forceinline__ int depth_of(const Wf &w, int p) {
    if constexpr (MULTI)
        return w.reqs[w.req[p]].max_depth;
    else
        return w.max_depth;
}
// the request whose [base, base + count) range holds index x (bases ascending)
__device__ __forceinline__ int find_req(const WfReq *reqs, int n, int64_t x, bool pixels) {
    int lo = 0, hi = n - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        const int64_t b = pixels ? reqs[mid].pix_base : reqs[mid].path_base;
        if (b <= x)
            lo = mid;
        else
            hi = mid - 1;
    }
    return lo;
}
// Adds one to a per-request ray counter for every lane of `mask` whose
// predicate holds, one atomic per request present in the warp.
__device__ __forceinline__ void count_req_rays(const Wf &w, unsigned mask, bool pred, int r,
                                               int which) {
    const unsigned m = __ballot_sync(mask, pred);
    if (!pred)
        return;
    const unsigned same = __match_any_sync(m, r);
    if ((threadIdx.x & 31) == __ffs(same) - 1)
        atomicAdd(&w.reqs[r].rays[which], (unsigned long long) __popc(same));
}

__device__ __forceinline__ uint8_t dir_octant(V3 d) {
    return (uint8_t) ((d.x < 0.f) | ((d.y < 0.f) << 1) | ((d.z < 0.f) << 2));
}

__device__ __forceinline__ int warp_append(unsigned *counter, bool pred) {
    const unsigned active = __activemask();
    const unsigned mask = __ballot_sync(active, pred);
    if (!mask)
        return -1;
    const int lane = threadIdx.x & 31;
    const int leader = __ffs(mask) - 1;
    unsigned base = 0;
    if (lane == leader)
        base = atomicAdd(counter, (unsigned) __popc(mask));
    base = __shfl_sync(active, base, leader);
    return pred ? (int) (base + __popc(mask & ((1u << lane) - 1u))) : -1;
}

__device__ __forceinline__ V3 ld3(const float4 *a, int i) {
    const float4 v = a[i];
    return v3(v.x, v.y, v.z);
}
__device__ __forceinline__ void st3(float4 *a, int i, V3 v, float w = 0.f) {
    a[i] = make_float4(v.x, v.y, v.z, w);
}

__device__ __forceinline__ void finish(const Wf &w, int p, V3 L) {
    if (!finite3(L))
        L = v3(0.f);
    w.result[p] = make_float4(L.x, L.y, L.z, 0.f);
}

// The paths of a pass: a pixel's samples in a row, pixel after pixel, so the 32
// paths a warp starts share one or two pixels, and after a bounce, sorted by
// octant, they still leave from the same surfaces: fewer nodes, triangles and
// texels per warp than with one sample of 32 pixels (museum-like 960x540, 16
// spp 12.12 -> 11.66 ms; adaptive 320x180, up to 64 spp, 6.30 -> 5.95; eight
// served frames 9.77 -> 9.29). The film stages then read a pixel's samples
// from a row each: 0.3% of the frame, 0.2% before.
//
// Window pixel q in path order: tiles of 8x4 pixels (narrower at the right
// edge, lower at the bottom), row by row of tiles, so a warp's 32 paths start
// in a small square instead of a long row and stay closer together (1% on
// every frame tried: museum-like 480x270, adaptive up to 256 spp, 44.0 -> 43.5
// ms).
__device__ __forceinline__ void tile_pixel(int q, int ww, int wh, int &x, int &y) {
    const int strip = q / (4 * ww);
    int r = q - strip * 4 * ww;
    const int h = min(4, wh - strip * 4);
    const int tx = r / (8 * h);
    r -= tx * 8 * h;
    const int tw = min(8, ww - tx * 8);
    y = strip * 4 + r / tw;
    x = tx * 8 + r % tw;
}

// ---- generate: camera rays for every (pixel, sample) of the pass
template <bool MULTI> __global__ void k_wf_generate(DevScene S, Wf w) {
    const int base = MULTI ? 0 : *w.pass_base;
    const int stride = gridDim.x * blockDim.x;
    // fixed spp: every pixel; adaptive: the active ones (their count is on
    // the device, set by the previous pass); server step: every request's
    // window times its samples of this step, request after request
    const int nq = w.adaptive ? (int) w.cnt[kCntActive] : w.npix;
    const int P = (w.adaptive && !MULTI) ? nq * w.spp_pass : w.P;
    for (int p = blockIdx.x * blockDim.x + threadIdx.x; p < P; p += stride) {
        int i, j;
        uint32_t m, sample;
        uint64_t seed;
        const DevCamera *cam;
        if constexpr (MULTI) {
            const int r = find_req(w.reqs, w.n_reqs, p, false);
            const WfReq &R = w.reqs[r];
            const int o = (int) (p - R.path_base);
            const int q = o / R.nspp;
            tile_pixel(q, R.ww, R.wh, i, j);
            i += R.x0;
            j += R.y0;
            m = (uint32_t) i + (uint32_t) j * (uint32_t) R.W;
            sample = (uint32_t) (R.s0 + (o - q * R.nspp));
            seed = R.seed;
            cam = &R.camera;
            w.req[p] = r;
        } else {
            const int a = p / w.spp_pass;
            const int q = w.adaptive ? w.act[a] : a;
            tile_pixel(q, w.ww, w.wh, i, j);
            i += w.x0;
            j += w.y0;
            m = (uint32_t) i + (uint32_t) j * (uint32_t) w.W;
            sample = (uint32_t) (w.sample_offset + base + (p - a * w.spp_pass));
            seed = w.seed;
            cam = &S.camera;
        }
        Rng rng{path_state(seed, m, sample)};
        const float xo = rng.next();
        const float yo = rng.next();
        const Ray3 r = generate_ray(*cam, i, j, xo, yo, rng);
        w.rng[p] = rng.s;
        st3(w.ro, p, r.o);
        st3(w.rd, p, r.d);
        st3(w.beta, p, v3(1.f));
        st3(w.L, p, v3(0.f));
        w.bounce[p] = 0;
        w.flags[p] = 0;
        w.qray[0][p] = p;
        w.tag[p] = 0xFF;
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        w.cnt[kCntRay0] = (unsigned) P;
        w.cnt[kCntRay1] = 0;
    }
}

// ---- per bounce: rotate the ray queues, clear the stage queues
__global__ void k_wf_begin(Wf w, int it) {
    stage_begin();
    // bounce `it` reads ray queue it&1 (filled by the previous bounce, or by
    // generate) and its shading stages append to queue (it+1)&1
    const int in = it & 1;
    if (threadIdx.x == 0) {
        w.cnt[kCntRay0 + (in ^ 1)] = 0;
        w.cnt[kCntMiss] = w.cnt[kCntDelta] = w.cnt[kCntSurf] = w.cnt[kCntShadow] = 0;
        w.cnt[kCntExtend] = w.cnt[kCntShadowJobs] = w.cnt[kCntShadowFetch] = 0;
        unsigned long long *tot = reinterpret_cast<unsigned long long *>(w.cnt + kCntRays);
        *tot += w.cnt[kCntRay0 + in];
    }
}

// The lanes of a warp that take rays of a queue of n: all 32, or as many as
// spread a short queue (a small frame, the last bounces) over every warp of
// the grid. A short queue takes as long as its longest ray, and a warp steps
// faster the fewer rays it holds.
__device__ __forceinline__ int lanes_used(int n) {
    const int warps = gridDim.x * (blockDim.x >> 5);
    return max(1, min(32, n / warps + 1));
}

// ---- extend: closest hit of the queued rays, then sort by material class.
// Persistent: a lane whose ray is finished takes the next queued ray once
// `refill` lanes of its warp are idle (one atomic per refill).
// This thread's stack: stack_sm entries in shared memory, the rest in the spill
// buffer.
template <class E> __device__ __forceinline__ StackCol<E> path_stack(const Wf &w, E *smem) {
    return StackCol<E>(smem, (E *) w.spill, nullptr, w.stack_sm, w.tlas_cap + w.blas_cap,
                       w.check);
}

template <bool MULTI>
__device__ __forceinline__ const DevScene &lane_scene(const DevScene &S0, const DevScene *ls) {
    if constexpr (MULTI)
        return *ls;
    else
        return S0;
}

// A traced path's hit record and its place among the next stages: its class
// as a tag (ordered queues) or an entry of its class's queue. All lanes of the
// warp call it; cls < 0: nothing to write.
__device__ __forceinline__ int hit_class(const DevScene &S, int obj) {
    if (obj < 0)
        return 0;
    const int kind = S.materials[S.objects[obj].material].kind;
    return (kind == kMatMirror || kind == kMatGlass) ? 1 : 2;
}
__device__ __forceinline__ void route_path(const Wf &w, int p, int cls) {
    if (w.ordered) {
        if (cls >= 0)
            w.tag[p] = (uint8_t) cls;
        return;
    }
    const int a = warp_append(w.cnt + kCntMiss, cls == 0);
    const int b = warp_append(w.cnt + kCntDelta, cls == 1);
    const int c = warp_append(w.cnt + kCntSurf, cls == 2);
    if (cls == 0)
        queue_put(w, w.qmiss, a, w.P, p);
    else if (cls == 1)
        queue_put(w, w.qdelta, b, w.P, p);
    else if (cls == 2)
        queue_put(w, w.qsurf, c, w.P, p);
}

template <bool MULTI>
__device__ __forceinline__ void wf_extend(const DevScene &S0, const Wf &w, int it, int refill) {
    extern __shared__ uint2 smem[];
    const StackCol<uint2> st = path_stack(w, smem);
    const int *qin = w.qray[it & 1];
    const int n = queue_len(w, w.cnt[kCntRay0 + (it & 1)], w.P);
    const unsigned full = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    // a lane without a ray has p = -1, or -2 when it takes none
    int p = -1;
    // this lane's ray's scene (server steps; a valid scene before the first ray)
    const DevScene *ls = MULTI ? w.reqs[0].scene : nullptr;
    ClosestWalk<> cw;
    bool more = n > 0;
    if (!more)
        return;
    refill = min(refill, lanes_used(n));
    if (lane >= lanes_used(n))
        p = -2;
    for (;;) {
        const bool idle = p == -1;
        const unsigned im = __ballot_sync(full, idle);
        if (!more && __all_sync(full, p < 0))
            break;
        bool done = false;
        if (more && __popc(im) >= refill) {
            const int cnt = __popc(im);
            unsigned base = 0;
            if (lane == 0)
                base = atomicAdd(w.cnt + kCntExtend, (unsigned) cnt);
            base = __shfl_sync(full, base, 0);
            if ((int) (base + cnt) >= n)
                more = false;
            const int k = (int) base + __popc(im & ((1u << lane) - 1u));
            const bool take = idle && k < n;
            int r = 0;
            if (take) {
                p = qin[k];
                if constexpr (MULTI) {
                    r = w.req[p];
                    ls = w.reqs[r].scene;
                }
                const float4 o = w.ro[p], d = w.rd[p];
                done = !cw.start(lane_scene<MULTI>(S0, ls), RayD{o.x, o.y, o.z, d.x, d.y, d.z},
                                 st);
            }
            if constexpr (MULTI)
                count_req_rays(w, full, take, r, 0);
        }
        const DevScene &S = lane_scene<MULTI>(S0, ls);
        if (p >= 0 && !done)
            done = cw.step(S, st);
        int cls = -1;
        if (done) {
            w.hit[p] = make_int4(cw.hit_obj, cw.hit_tri, __float_as_int(cw.best), 0);
            cls = hit_class(S, cw.hit_obj);
        }
        route_path(w, p, cls);
        if (done)
            p = -1;
    }
}

// The counting form of the extend stage (prr_render_counts): the binary walk,
// which visits the nodes the reference visits, one ray per thread.
__global__ void k_wf_extend_count(DevScene S, Wf w, int it, int) {
    stage_begin();
    extern __shared__ uint2 smem[];
    SmemStack tst{smem + threadIdx.x, (int) blockDim.x, 0, S.tlas_depth + 1, w.check};
    SmemStack bst{smem + (size_t) (S.tlas_depth + 1) * blockDim.x + threadIdx.x, (int) blockDim.x,
                  0, S.blas_depth + 1, w.check};
    const int n = queue_len(w, w.cnt[kCntRay0 + (it & 1)], w.P);
    unsigned cls_n[3] = {0, 0, 0};
    WalkCounts c;
    for (int base = blockIdx.x * blockDim.x; base < n; base += gridDim.x * blockDim.x) {
        const int k = base + threadIdx.x;
        int p = 0, cls = -1;
        if (k < n) {
            p = w.qray[it & 1][k];
            const float4 o = w.ro[p], d = w.rd[p];
            const RayD r{o.x, o.y, o.z, d.x, d.y, d.z};
            const SceneHit h = scene_closest<true>(S, r, precompute(r), tst, bst, &c);
            w.hit[p] = make_int4(h.obj, h.tri, __float_as_int(h.t), 0);
            cls = hit_class(S, h.obj);
            cls_n[cls]++;
        }
        route_path(w, p, cls);
    }
    const unsigned work[3] = {c.nodes, c.tris, c.objects};
    flush_stats(w.stats, kStatClosestNodes, work);
    flush_stats(w.stats, kStatMiss, cls_n);
}

// Hit record -> Inter (Triangle::finalize / Sphere::getIntersection fields).
__device__ __forceinline__ Inter load_inter(const DevScene &S, const Wf &w, int p) {
    const int4 h = w.hit[p];
    Inter in;
    in.hit = h.x >= 0;
    in.a = no_attr();
    if (!in.hit) {
        in.mat = -1;
        in.p = in.n = v3(0.f);
        return in;
    }
    const float t = __int_as_float(h.z);
    const V3 o = ld3(w.ro, p), d = ld3(w.rd, p);
    const DevObject &ob = S.objects[h.x];
    in.mat = ob.material;
    if (ob.kind == kObjMesh) {
        in.p = o + t * d;
        in.n = v3(S.normals[(size_t) h.y * 3], S.normals[(size_t) h.y * 3 + 1],
                  S.normals[(size_t) h.y * 3 + 2]);
        finalize_attr(S, ob, h.y, RayD{o.x, o.y, o.z, d.x, d.y, d.z}, in.n, in.a);
    } else {
        in.p = o + d * t;
        in.n = normalize(in.p - v3(ob.cx, ob.cy, ob.cz));
    }
    return in;
}

// The tail of a non-delta bounce (Integrator.cpp:205-256) for the hit of the
// ray it spawned, then the head of the next loop iteration. Returns false
// when the path has ended (its result is written). `it` and `specular` are
// the loop variables of the iteration that now processes `in`.
__device__ __forceinline__ bool enter_iteration(const DevScene &S, const Wf &w, int p,
                                                const Inter &in, Rng &rng, V3 &beta, V3 &L,
                                                int &it, bool &specular, float clamp,
                                                int max_depth) {
    const int k = w.bounce[p];
    const int fl = w.flags[p];
    const V3 bg = v3(S.background[0], S.background[1], S.background[2]);
    if (fl & kFlagPending) {
        const float4 pe = w.pend[p];
        const V3 scale = v3(pe.x, pe.y, pe.z);
        const float bpdf = pe.w;
        const V3 wi = ld3(w.rd, p);
        const bool indirect = k > 0;
        if (!in.hit) {
            V3 c;
            if (S.env.loaded) {
                const V3 el = env_lookup(S.env, wi);
                const float ep = env_pdf(S.env, wi);
                c = beta * scale * mis(bpdf, ep) * el;
            } else {
                c = beta * scale * bg;
            }
            L = L + (indirect ? clamp_indirect(c, clamp) : c);
            return false;
        }
        const DevMaterial &hm = S.materials[in.mat];
        if (hm.kind == kMatEmissive) {
            const V3 hp = ld3(w.prev, p);
            const float cos_l = smax(0.f, dot(-wi, normalized(in.n)));
            const V3 dd = in.p - hp;
            const float hd2 = dot(dd, dd);
            const float pdf_area = S.total_emit_area > 0.f ? 1.f / S.total_emit_area : 0.f;
            const float pdf_sa = pdf_area * hd2 / smax(cos_l, 1e-4f);
            const V3 c = beta * scale * mis(bpdf, pdf_sa) *
                         v3(hm.emission[0], hm.emission[1], hm.emission[2]);
            L = L + (indirect ? clamp_indirect(c, clamp) : c);
            return false;
        }
        beta = beta * scale;
        if (!finite3(beta))
            return false;
        if (k >= 3) {
            const float mc = max3(beta);
            const float q = smax(0.05f, 1.f - mc);
            if (rng.next() < q)
                return false;
            beta = beta * (1.f / (1.f - q));
        }
        it = k + 1;
        specular = false;
    } else if (fl & kFlagSpecular) {
        it = k + 1;
        specular = true;
    } else {
        it = 0;
        specular = false;
    }
    if (it >= max_depth)
        return false;
    if (it == 0 || specular) {
        const V3 d = ld3(w.rd, p);
        if (!in.hit) {
            const V3 b = S.env.loaded ? env_lookup(S.env, d) : bg;
            const V3 c = beta * b;
            L = L + ((it > 0) ? clamp_indirect(c, clamp) : c);
        } else if (S.materials[in.mat].kind == kMatEmissive) {
            const DevMaterial &hm = S.materials[in.mat];
            const V3 c = beta * v3(hm.emission[0], hm.emission[1], hm.emission[2]);
            L = L + ((it > 0) ? clamp_indirect(c, clamp) : c);
        }
    }
    return in.hit;
}

// ---- miss: the path leaves the scene
template <bool MULTI> __global__ void k_wf_miss(DevScene S0, Wf w) {
    stage_begin();
    const int n = queue_len(w, w.cnt[kCntMiss], w.P);
    const int stride = gridDim.x * blockDim.x;
    for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < n; k += stride) {
        const int p = w.qmiss[k];
        const DevScene &S = scene_of<MULTI>(S0, w, p);
        Rng rng{w.rng[p]};
        V3 beta = ld3(w.beta, p), L = ld3(w.L, p);
        Inter in;
        in.hit = false;
        in.mat = -1;
        in.a = no_attr();
        int it;
        bool spec;
        enter_iteration(S, w, p, in, rng, beta, L, it, spec, clamp_of<MULTI>(w, p),
                        depth_of<MULTI>(w, p));
        finish(w, p, L);
    }
}

// ---- delta: one step of the specular chain
template <bool MULTI> __global__ void k_wf_delta(DevScene S0, Wf w, int it_next) {
    stage_begin();
    const int n = queue_len(w, w.cnt[kCntDelta], w.P);
    int *qout = w.qray[it_next & 1];
    const int stride = gridDim.x * blockDim.x;
    for (int base = blockIdx.x * blockDim.x; base < n; base += stride) {
        const int k = base + threadIdx.x;
        bool cont = false;
        int p = 0;
        if (k < n) {
            p = w.qdelta[k];
            const DevScene &S = scene_of<MULTI>(S0, w, p);
            const int max_depth = depth_of<MULTI>(w, p);
            Rng rng{w.rng[p]};
            V3 beta = ld3(w.beta, p), L = ld3(w.L, p);
            const Inter in = load_inter(S, w, p);
            int it;
            bool spec;
            if (!enter_iteration(S, w, p, in, rng, beta, L, it, spec, clamp_of<MULTI>(w, p),
                                 max_depth)) {
                finish(w, p, L);
            } else {
                const DevMaterial &m = S.materials[in.mat];
                const V3 cd = ld3(w.rd, p);
                const Shading sd = build_shading(S, m, in.n, in.a);
                const BSDFSample bs = delta_sample(m, sd, -cd, rng);
                if (bs.pdf < 1e-6f) {
                    finish(w, p, L);
                } else {
                    beta = beta * bs.f / bs.pdf;
                    const bool trans = dot(bs.wi, in.n) < 0.f;
                    const V3 off = trans ? -in.n : in.n;
                    if (trans)
                        beta = beta * sd.base;
                    // the next ray is only looked at if the loop runs again
                    if (it + 1 >= max_depth) {
                        finish(w, p, L);
                    } else {
                        st3(w.ro, p, in.p + off * PRR_EPS);
                        st3(w.rd, p, bs.wi);
                        st3(w.beta, p, beta);
                        st3(w.L, p, L);
                        w.bounce[p] = it;
                        w.flags[p] = kFlagSpecular;
                        w.rng[p] = rng.s;
                        cont = true;
                    }
                }
            }
        }
        if (w.ordered) {
            if (cont)
                w.tag[p] = dir_octant(ld3(w.rd, p));
        } else {
            const int slot = warp_append(w.cnt + kCntRay0 + (it_next & 1), cont);
            if (cont)
                queue_put(w, qout, slot, w.P, p);
        }
    }
}

// ---- surface: NEE + BSDF sampling of a non-delta bounce
// 64 registers (1,024 threads per SM): this stage waits on scattered path state
// and scene data, so resident warps matter more than a few spills. In blocks of
// 512 whose warps start each path together, so that they read its long code at
// about the same time (museum-like 960x540, 16 spp: 12.34 ms, 12.45 in blocks of
// 128; barriers between the three directions cost more than they gain, 12.46).
constexpr int kSurfaceBlock = 512;
template <bool MULTI>
__global__ void __launch_bounds__(kSurfaceBlock, 2)
    k_wf_surface(DevScene S0, Wf w, int it_next) {
    stage_begin();
    const int n = queue_len(w, w.cnt[kCntSurf], w.P);
    int *qout = w.qray[it_next & 1];
    const int stride = gridDim.x * blockDim.x;
    for (int base = blockIdx.x * blockDim.x; base < n; base += stride) {
        __syncthreads();
        const int k = base + threadIdx.x;
        bool cont = false, shadow = false, jl = false, je = false;
        uint8_t oct = 0;
        int p = 0;
        if (k < n) {
            p = w.qsurf[k];
            const DevScene &S = scene_of<MULTI>(S0, w, p);
            Rng rng{w.rng[p]};
            V3 beta = ld3(w.beta, p), L = ld3(w.L, p);
            const Inter in = load_inter(S, w, p);
            int it;
            bool spec;
            if (!enter_iteration(S, w, p, in, rng, beta, L, it, spec, clamp_of<MULTI>(w, p),
                                 depth_of<MULTI>(w, p))) {
                finish(w, p, L);
            } else {
                const DevMaterial &m = S.materials[in.mat];
                const V3 cd = ld3(w.rd, p);
                const V3 hp = in.p;
                const V3 sn = dot(cd, in.n) < 0.f ? in.n : -in.n;
                const Shading sd = build_shading<true>(S, m, sn, in.a);
                const V3 wo = -cd;
                const float indirect = it > 0 ? 1.f : 0.f;
                // The three directions that leave the hit: towards an emitter,
                // towards the environment, and the BSDF sample. One loop, so the
                // BSDF evaluation stands once in the code. The first two
                // contributions are formed now and added by the shadow stage if
                // their light is visible.
                V3 wi = v3(0.f), f = v3(0.f);
                float bp = 0.f;
#pragma unroll 1
                for (int d = 0; d < 3; d++) {
                    float pdf = 0.f, tmax = kInf;
                    V3 em = v3(0.f);
                    bool ok = false;
                    if (d == 0) {
                        if (S.total_emit_area > 0.f) {
                            const LightPoint lp = sample_light(S, rng);
                            const float pdf_area = 1.0f / S.total_emit_area;
                            const V3 to = lp.p - hp;
                            const float dist2 = dot(to, to);
                            const float dist = sqrtf(dist2);
                            wi = to / dist;
                            const float cos_l = smax(0.f, dot(-wi, normalized(lp.n)));
                            ok = cos_l > 0.f;
                            if (ok) {
                                pdf = pdf_area * dist2 / cos_l;
                                tmax = dist - 2.f * PRR_EPS;
                                const DevMaterial &lm = S.materials[lp.material];
                                em = v3(lm.emission[0], lm.emission[1], lm.emission[2]);
                            }
                        }
                    } else if (d == 1) {
                        if (S.env.loaded) {
                            wi = env_importance(S.env, rng, pdf);
                            ok = !(pdf < 1e-6f);
                            if (ok)
                                em = env_lookup(S.env, wi);
                        }
                    } else {
                        ok = m.kind == kMatDiffuse && diffuse_direction(m, sd, wo, rng, wi);
                    }
                    f = v3(0.f);
                    bp = 0.f;
                    if (ok)
                        mat_eval_pdf(m, sd, wi, wo, &f, &bp);
                    if (d < 2 && ok) {
                        V3 c = mis(pdf, bp) * em * f / (d == 0 ? pdf : pdf + 1e-6f);
                        c = beta * c;
                        if (!(c.x == 0.f && c.y == 0.f && c.z == 0.f)) {
                            const V3 o = hp + wi * PRR_EPS;
                            (d == 0 ? w.slo : w.seo)[p] = make_float4(o.x, o.y, o.z, tmax);
                            (d == 0 ? w.sld : w.sed)[p] = make_float4(wi.x, wi.y, wi.z, 1.f);
                            (d == 0 ? w.slc : w.sec)[p] = make_float4(c.x, c.y, c.z, indirect);
                            if (d == 0)
                                jl = true;
                            else
                                je = true;
                        }
                    }
                }
                // a ray's direction carries its flag (w = 0: none); its origin and
                // contribution are read only when set
                shadow = jl || je;
                if (shadow && !jl)
                    w.sld[p] = make_float4(0.f, 0.f, 0.f, 0.f);
                if (shadow && !je)
                    w.sed[p] = make_float4(0.f, 0.f, 0.f, 0.f);
                BSDFSample bs;
                bs.wi = wi;
                bs.pdf = bp;
                bs.f = bp > 1e-6f ? f : v3(0.f); // DiffuseMaterial::sample
                if (bs.pdf < 1e-6f) {
                    if (shadow) {
                        st3(w.L, p, L);
                        w.flags[p] = kFlagEndAfterShadow;
                    } else {
                        finish(w, p, L);
                    }
                } else {
                    const V3 scale = bs.f / bs.pdf;
                    const V3 off = dot(bs.wi, sd.f.N) >= 0.f ? sd.f.N : -sd.f.N;
                    st3(w.ro, p, hp + off * PRR_EPS);
                    st3(w.rd, p, bs.wi);
                    oct = dir_octant(bs.wi);
                    st3(w.pend, p, scale, bs.pdf);
                    if (S.has_emissive_kind) // read only on an emissive hit
                        st3(w.prev, p, hp);
                    st3(w.beta, p, beta);
                    // L is as loaded: a hit adds to it only on an emissive
                    // material, which has no BSDF sample
                    w.bounce[p] = it;
                    w.flags[p] = kFlagPending;
                    cont = true;
                }
                w.rng[p] = rng.s;
            }
        }
        if (w.ordered) {
            if (cont)
                w.tag[p] = oct;
        } else {
            const int slot = warp_append(w.cnt + kCntRay0 + (it_next & 1), cont);
            if (cont)
                queue_put(w, qout, slot, w.P, p);
        }
        const int sslot = warp_append(w.cnt + kCntShadow, shadow);
        if (shadow)
            queue_put(w, w.qshadow, sslot, w.P, p);
        const int j0 = warp_append(w.cnt + kCntShadowJobs, jl);
        if (jl)
            queue_put(w, w.qjob, j0, 2 * (int64_t) w.P, p * 2);
        const int j1 = warp_append(w.cnt + kCntShadowJobs, je);
        if (je)
            queue_put(w, w.qjob, j1, 2 * (int64_t) w.P, p * 2 + 1);
    }
}

// ---- shadow: visibility of every queued NEE ray (persistent, per-lane refill)
// Adds up the rays each lane traced.
__device__ __forceinline__ void count_shadow_rays(const Wf &w, unsigned rays) {
    for (int off = 16; off > 0; off >>= 1)
        rays += __shfl_down_sync(0xffffffffu, rays, off);
    if ((threadIdx.x & 31) == 0 && rays)
        atomicAdd(reinterpret_cast<unsigned long long *>(w.cnt + kCntShadowRays),
                  (unsigned long long) rays);
}

template <bool MULTI>
__device__ __forceinline__ void wf_shadow(const DevScene &S0, const Wf &w, int refill) {
    extern __shared__ uint32_t smem32[];
    const StackCol<uint32_t> st = path_stack(w, smem32);
    const int n = queue_len(w, w.cnt[kCntShadowJobs], 2 * (int64_t) w.P);
    const unsigned full = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    int job = -1; // -2: a lane that takes no rays
    // this lane's ray's scene (server steps; a valid scene before the first ray)
    const DevScene *ls = MULTI ? w.reqs[0].scene : nullptr;
    AnyWalk<> aw;
    bool more = n > 0;
    if (!more)
        return;
    unsigned rays = 0;
    refill = min(refill, lanes_used(n));
    if (lane >= lanes_used(n))
        job = -2;
    for (;;) {
        const bool idle = job == -1;
        const unsigned im = __ballot_sync(full, idle);
        if (!more && __all_sync(full, job < 0))
            break;
        if (more && __popc(im) >= refill) {
            const int cnt = __popc(im);
            unsigned base = 0;
            if (lane == 0)
                base = atomicAdd(w.cnt + kCntShadowFetch, (unsigned) cnt);
            base = __shfl_sync(full, base, 0);
            if ((int) (base + cnt) >= n)
                more = false;
            const int k = (int) base + __popc(im & ((1u << lane) - 1u));
            const bool take = idle && k < n;
            int r = 0;
            if (take) {
                job = w.qjob[k];
                const int p = job >> 1;
                if constexpr (MULTI) {
                    r = w.req[p];
                    ls = w.reqs[r].scene;
                }
                const float4 o = (job & 1) ? w.seo[p] : w.slo[p];
                const float4 d = (job & 1) ? w.sed[p] : w.sld[p];
                rays++;
                if (!aw.start(lane_scene<MULTI>(S0, ls), RayD{o.x, o.y, o.z, d.x, d.y, d.z}, o.w,
                              st)) {
                    w.vis[job] = aw.occluded ? 0 : 1;
                    job = -1;
                }
            }
            if constexpr (MULTI)
                count_req_rays(w, full, take, r, 1);
        }
        if (job >= 0 && aw.step(lane_scene<MULTI>(S0, ls), st)) {
            w.vis[job] = aw.occluded ? 0 : 1;
            job = -1;
        }
    }
    count_shadow_rays(w, rays);
}

// The counting form, as k_wf_extend_count.
__global__ void k_wf_shadow_count(DevScene S, Wf w, int) {
    stage_begin();
    extern __shared__ uint2 smem[];
    SmemStack tst{smem + threadIdx.x, (int) blockDim.x, 0, S.tlas_depth + 1, w.check};
    SmemStack bst{smem + (size_t) (S.tlas_depth + 1) * blockDim.x + threadIdx.x, (int) blockDim.x,
                  0, S.blas_depth + 1, w.check};
    const int n = queue_len(w, w.cnt[kCntShadowJobs], 2 * (int64_t) w.P);
    unsigned rays = 0;
    WalkCounts c;
    for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < n; k += gridDim.x * blockDim.x) {
        const int job = w.qjob[k], p = job >> 1;
        const float4 o = (job & 1) ? w.seo[p] : w.slo[p];
        const float4 d = (job & 1) ? w.sed[p] : w.sld[p];
        const RayD r{o.x, o.y, o.z, d.x, d.y, d.z};
        rays++;
        w.vis[job] = scene_occluded<true>(S, r, precompute(r), tst, bst, o.w, &c) ? 0 : 1;
    }
    const unsigned work[3] = {c.nodes, c.tris, c.objects};
    flush_stats(w.stats, kStatShadowNodes, work);
    count_shadow_rays(w, rays);
}

// The traversal stages on the four-wide nodes, 64 registers at most (8 resident
// blocks of 128). Tighter caps gain blocks but spill the four boxes' distances:
// museum-like scene of 491,520 triangles at 960x540, 16 spp, append-order
// queues: 16.9 ms, 17.6 at 56 registers, 19.0 at 48; 18.5 on the binary nodes
// (at their best cap, 48). 13.2 ms with the default queues and one walk for
// both levels.
template <bool MULTI>
__global__ void __maxnreg__(64) k_wf_extend(DevScene S, Wf w, int it, int refill) {
    stage_begin();
    wf_extend<MULTI>(S, w, it, refill);
}
template <bool MULTI>
__global__ void __maxnreg__(64) k_wf_shadow(DevScene S, Wf w, int refill) {
    stage_begin();
    wf_shadow<MULTI>(S, w, refill);
}

// ---- add the visible NEE contributions, light first, then env, as castRay
template <bool MULTI> __global__ void k_wf_shadow_resolve(Wf w) {
    stage_begin();
    const int n = queue_len(w, w.cnt[kCntShadow], w.P);
    const int stride = gridDim.x * blockDim.x;
    for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < n; k += stride) {
        const int p = w.qshadow[k];
        V3 L = ld3(w.L, p);
        for (int r = 0; r < 2; r++) {
            const float4 d = r == 0 ? w.sld[p] : w.sed[p];
            if (d.w == 0.f || !w.vis[p * 2 + r])
                continue;
            const float4 c = r == 0 ? w.slc[p] : w.sec[p];
            const V3 cv = v3(c.x, c.y, c.z);
            L = L + (c.w != 0.f ? clamp_indirect(cv, clamp_of<MULTI>(w, p)) : cv);
        }
        if (w.flags[p] & kFlagEndAfterShadow)
            finish(w, p, L);
        else
            st3(w.L, p, L);
    }
}

// ---- film: add the pass's samples per pixel in sample order
// ---- ordered queues: a stable partition of the per-path tags into bucket
// queues, in path order within each bucket. A tile is 4096 paths: 256
// threads x 16 tags read as one 16-byte vector. Tiles are counted, the tile
// counts scanned per bucket, then each tile writes its paths to their buckets
// in order and clears their tags for the next partition. The tag array is
// padded with 0xFF to whole tiles.
constexpr int kPartThreads = 256;
constexpr int kPartTile = kPartThreads * 16;

struct PartSpec {
    uint8_t *tag;       // the tags, padded with 0xFF to whole tiles
    const int *map;     // item k is written as map[k] (nullptr: k itself)
    int *q[8];          // bucket b's queue; concatenated: all in q[0], bucket order
    int nb;             // buckets (<= 8)
    int concat;
    int count_slot[8];  // counter slot receiving bucket b's size (-1: none)
    int total_slot;     // counter slot receiving the total (-1: none)
    int from[2];        // counters of the items that may carry a tag (-1: not looked at)
};
constexpr int kSkipTiles = 128; // tiles from which on an empty partition is looked for

// No item carries a tag: a bounce without paths (the passes after an adaptive
// frame's last pixel has stopped, the last bounces of most passes), whose
// partitions then leave the P tags unread. 960x540, up to 256 spp, every pixel
// stopped in the first of 16 passes: 26.0 -> 17.3 ms. The kernels ask for their
// first data before they look (ld_now): waiting for the counters first made
// short launches longer (a render of 0.88 ms by 4%). Few tiles are read in no
// time, so small passes do not look.
__device__ __forceinline__ bool part_empty(const Wf &w, const PartSpec &ps) {
    return ps.from[0] >= 0 && (w.cnt[ps.from[0]] | w.cnt[ps.from[1]]) == 0;
}

// A load issued where it stands in the code, whatever is known of its use.
__device__ __forceinline__ uint4 ld_now(const uint4 *p) {
    uint4 v;
    asm volatile("ld.global.v4.u32 {%0, %1, %2, %3}, [%4];"
                 : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
                 : "l"(p));
    return v;
}

// How many of the 16 tag bytes in v equal b.
__device__ __forceinline__ unsigned count_tag(const uint4 &v, unsigned b) {
    const unsigned bb = b * 0x01010101u;
    return (__popc(__vcmpeq4(v.x, bb)) + __popc(__vcmpeq4(v.y, bb)) +
            __popc(__vcmpeq4(v.z, bb)) + __popc(__vcmpeq4(v.w, bb))) >> 3;
}

__global__ void __launch_bounds__(kPartThreads) k_part_count(Wf w, PartSpec ps) {
    stage_begin();
    const uint4 v = ld_now(reinterpret_cast<const uint4 *>(ps.tag) + blockIdx.x * kPartThreads +
                           threadIdx.x);
    if (part_empty(w, ps))
        return;
    const int nb = ps.nb;
    __shared__ unsigned c[8];
    if (threadIdx.x < 8)
        c[threadIdx.x] = 0;
    __syncthreads();
#pragma unroll
    for (int b = 0; b < 8; b++)
        if (b < nb) {
            const unsigned r = __reduce_add_sync(0xffffffffu, count_tag(v, b));
            if ((threadIdx.x & 31) == 0 && r)
                atomicAdd(&c[b], r);
        }
    __syncthreads();
    if (threadIdx.x < 8)
        w.tile[blockIdx.x * 8 + threadIdx.x] = c[threadIdx.x];
}

// Exclusive scan over the tiles, all buckets at once: one block, one tile per
// thread per round. Tile counts become the tiles' first output slots.
__global__ void __launch_bounds__(1024) k_part_scan(Wf w, int ntiles, PartSpec ps) {
    stage_begin();
    // this thread's tile of the first round
    uint4 a = make_uint4(0u, 0u, 0u, 0u), b = a;
    if ((int) threadIdx.x < ntiles) {
        a = ld_now(reinterpret_cast<const uint4 *>(w.tile) + threadIdx.x * 2);
        b = ld_now(reinterpret_cast<const uint4 *>(w.tile) + threadIdx.x * 2 + 1);
    }
    if (part_empty(w, ps)) {
        if (threadIdx.x < 8 && ps.count_slot[threadIdx.x] >= 0)
            w.cnt[ps.count_slot[threadIdx.x]] = 0;
        if (threadIdx.x == 8 && ps.total_slot >= 0)
            w.cnt[ps.total_slot] = 0;
        return;
    }
    __shared__ unsigned wsum[32][8];
    __shared__ unsigned carry[8];
    __shared__ unsigned total[8];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    if (threadIdx.x < 8)
        carry[threadIdx.x] = 0;
    __syncthreads();
    for (int r0 = 0; r0 < ntiles; r0 += 1024) {
        const int t = r0 + threadIdx.x;
        if (r0 > 0) {
            a = b = make_uint4(0u, 0u, 0u, 0u);
            if (t < ntiles) {
                a = reinterpret_cast<const uint4 *>(w.tile)[t * 2];
                b = reinterpret_cast<const uint4 *>(w.tile)[t * 2 + 1];
            }
        }
        const unsigned v[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
        unsigned x[8];
#pragma unroll
        for (int k = 0; k < 8; k++) {
            x[k] = v[k];
            for (int o = 1; o < 32; o <<= 1) {
                const unsigned y = __shfl_up_sync(0xffffffffu, x[k], o);
                if (lane >= o)
                    x[k] += y;
            }
            if (lane == 31)
                wsum[wid][k] = x[k];
        }
        __syncthreads();
        // warp 0 scans the 32 warp sums of each bucket
        if (wid == 0) {
#pragma unroll
            for (int k = 0; k < 8; k++) {
                const unsigned s0 = wsum[lane][k];
                unsigned z = s0;
                for (int o = 1; o < 32; o <<= 1) {
                    const unsigned y = __shfl_up_sync(0xffffffffu, z, o);
                    if (lane >= o)
                        z += y;
                }
                wsum[lane][k] = z - s0; // exclusive
                if (lane == 31) {
                    // round total folded into the running carry after use
                    total[k] = z;
                }
            }
        }
        __syncthreads();
        if (t < ntiles) {
            unsigned o[8];
#pragma unroll
            for (int k = 0; k < 8; k++)
                o[k] = carry[k] + wsum[wid][k] + x[k] - v[k];
            reinterpret_cast<uint4 *>(w.tile)[t * 2] = make_uint4(o[0], o[1], o[2], o[3]);
            reinterpret_cast<uint4 *>(w.tile)[t * 2 + 1] = make_uint4(o[4], o[5], o[6], o[7]);
        }
        __syncthreads();
        if (threadIdx.x < 8)
            carry[threadIdx.x] += total[threadIdx.x];
        __syncthreads();
    }
    // bucket bases (concatenated queues) and counts
    if (threadIdx.x == 0) {
        unsigned base = 0;
#pragma unroll
        for (int k = 0; k < 8; k++)
            if (k < ps.nb) {
                total[k] = base; // reuse: first slot of bucket k
                if (ps.count_slot[k] >= 0)
                    w.cnt[ps.count_slot[k]] = carry[k];
                base += carry[k];
            }
        if (ps.total_slot >= 0)
            w.cnt[ps.total_slot] = base;
    }
    __syncthreads();
    if (ps.concat)
        for (int i = threadIdx.x; i < ntiles * 8; i += 1024) {
            const int k = i & 7;
            if (k < ps.nb)
                w.tile[i] += total[k];
        }
}

__global__ void __launch_bounds__(kPartThreads) k_part_scatter(Wf w, PartSpec ps) {
    stage_begin();
    uint4 *tv = reinterpret_cast<uint4 *>(ps.tag) + blockIdx.x * kPartThreads + threadIdx.x;
    const uint4 v = ld_now(tv);
    if (part_empty(w, ps))
        return;
    __shared__ unsigned wsum[kPartThreads / 32][8];
    __shared__ unsigned base[8][kPartThreads];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    unsigned c[8], x[8];
#pragma unroll
    for (int k = 0; k < 8; k++) {
        c[k] = k < ps.nb ? count_tag(v, k) : 0u;
        x[k] = c[k];
        for (int o = 1; o < 32; o <<= 1) {
            const unsigned y = __shfl_up_sync(0xffffffffu, x[k], o);
            if (lane >= o)
                x[k] += y;
        }
        if (lane == 31)
            wsum[wid][k] = x[k];
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < 8; k++) {
        unsigned before = 0;
        for (int u = 0; u < wid; u++)
            before += wsum[u][k];
        base[k][threadIdx.x] = (k < ps.nb ? w.tile[blockIdx.x * 8 + k] : 0u) + before + x[k] - c[k];
    }
    const uint32_t words[4] = {v.x, v.y, v.z, v.w};
    const int first = (blockIdx.x * kPartThreads + threadIdx.x) * 16;
#pragma unroll
    for (int i = 0; i < 16; i++) {
        const unsigned t = (words[i >> 2] >> ((i & 3) * 8)) & 0xFFu;
        if (t < (unsigned) ps.nb) {
            int *q = ps.q[0];
            if (!ps.concat) {
#pragma unroll
                for (int k = 1; k < 8; k++)
                    if (t == (unsigned) k)
                        q = ps.q[k];
            }
            q[base[t][threadIdx.x]++] = ps.map ? ps.map[first + i] : first + i;
        }
    }
    *tv = make_uint4(0xFFFFFFFFu, 0xFFFFFFFFu, 0xFFFFFFFFu, 0xFFFFFFFFu);
}

// ---- adaptive film: each active pixel takes this pass's samples in sample
// order -- running sum, per-channel Welford update, and the stop test after
// every sample once min_spp samples are in (Renderer.cpp:74-95). Samples
// traced past a pixel's stop are dropped, as the reference never draws them.
__global__ void k_wf_film_adaptive(Wf w) {
    const int na = (int) w.cnt[kCntActive];
    const int stride = gridDim.x * blockDim.x;
    for (int a = blockIdx.x * blockDim.x + threadIdx.x; a < na; a += stride) {
        const int q = w.act[a];
        const float4 s0 = w.wel0[q], s1 = w.wel1[q];
        Welford wr{(int) s0.x, s0.y, s1.x}, wg{(int) s0.x, s0.z, s1.y}, wb{(int) s0.x, s0.w, s1.z};
        float3 f = w.film[q];
        bool done = false;
        for (int k = 0; k < w.spp_pass && !done; k++) {
            float4 r = w.result[(size_t) a * w.spp_pass + k];
            if (isnan(r.x) || isnan(r.y) || isnan(r.z))
                r = make_float4(0.f, 0.f, 0.f, 0.f);
            f.x += r.x;
            f.y += r.y;
            f.z += r.z;
            wr.update(r.x);
            wg.update(r.y);
            wb.update(r.z);
            done = wr.n >= w.min_spp && wr.ci() < w.threshold && wg.ci() < w.threshold &&
                   wb.ci() < w.threshold;
        }
        w.film[q] = f;
        w.wel0[q] = make_float4((float) wr.n, wr.mean, wg.mean, wb.mean);
        w.wel1[q] = make_float4(wr.M2, wg.M2, wb.M2, 0.f);
        w.ptag[a] = (done || wr.n >= w.max_spp) ? 0xFF : 0;
    }
    if (blockIdx.x == 0 && threadIdx.x == 0)
        *w.pass_base += w.spp_pass;
}

__global__ void k_wf_copy_active(Wf w) {
    const int na = (int) w.cnt[kCntActive];
    const int stride = gridDim.x * blockDim.x;
    for (int a = blockIdx.x * blockDim.x + threadIdx.x; a < na; a += stride)
        w.act[a] = w.act_next[a];
}

__global__ void k_wf_adaptive_init(Wf w) {
    const int stride = gridDim.x * blockDim.x;
    for (int q = blockIdx.x * blockDim.x + threadIdx.x; q < w.npix; q += stride) {
        w.act[q] = q;
        w.wel0[q] = make_float4(0.f, 0.f, 0.f, 0.f);
        w.wel1[q] = make_float4(0.f, 0.f, 0.f, 0.f);
    }
    if (blockIdx.x == 0 && threadIdx.x == 0)
        w.cnt[kCntActive] = (unsigned) w.npix;
}

// mean = sum / n per pixel (Renderer.cpp:98-99)
__global__ void k_wf_resolve_adaptive(const float3 *film, const float4 *wel0, int npix, int ww,
                                      int wh, float *out, int32_t *spp) {
    const int q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= npix)
        return;
    const float3 f = film[q];
    const int n = (int) wel0[q].x;
    int x, y;
    tile_pixel(q, ww, wh, x, y);
    const size_t o = (size_t) y * ww + x;
    out[o * 3 + 0] = f.x / (float) n;
    out[o * 3 + 1] = f.y / (float) n;
    out[o * 3 + 2] = f.z / (float) n;
    if (spp)
        spp[o] = n;
}

// ---- server step film: every request's window pixels take this step's
// samples in sample order (the same sums as a render of the request alone)
__global__ void k_wf_film_multi(Wf w, int64_t total_pixels) {
    const int64_t stride = (int64_t) gridDim.x * blockDim.x;
    for (int64_t t = (int64_t) blockIdx.x * blockDim.x + threadIdx.x; t < total_pixels;
         t += stride) {
        const int r = find_req(w.reqs, w.n_reqs, t, true);
        const WfReq &R = w.reqs[r];
        const int q = (int) (t - R.pix_base);
        int x, y;
        tile_pixel(q, R.ww, R.wh, x, y);
        float3 &film = R.film[(size_t) y * R.ww + x]; // row order
        float3 f = film;
        for (int s = 0; s < R.nspp; s++) {
            const float4 v = w.result[R.path_base + (int64_t) q * R.nspp + s];
            if (!(isnan(v.x) || isnan(v.y) || isnan(v.z))) {
                f.x += v.x;
                f.y += v.y;
                f.z += v.z;
            }
        }
        film = f;
    }
}

__global__ void k_wf_film(Wf w) {
    const int q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q < w.npix) {
        float3 f = w.film[q];
        for (int s = 0; s < w.spp_pass; s++) {
            const float4 r = w.result[(size_t) q * w.spp_pass + s];
            // a NaN sample is zeroed before accumulation (Renderer.cpp:78-83)
            if (!(isnan(r.x) || isnan(r.y) || isnan(r.z))) {
                f.x += r.x;
                f.y += r.y;
                f.z += r.z;
            }
        }
        w.film[q] = f;
    }
    if (blockIdx.x == 0 && threadIdx.x == 0)
        *w.pass_base += w.spp_pass;
}

__global__ void k_wf_resolve(const float3 *film, int npix, int ww, int wh, int n, float *out,
                             int32_t *spp) {
    const int q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= npix)
        return;
    const float3 f = film[q];
    int x, y;
    tile_pixel(q, ww, wh, x, y);
    const size_t o = (size_t) y * ww + x;
    out[o * 3 + 0] = f.x / (float) n;
    out[o * 3 + 1] = f.y / (float) n;
    out[o * 3 + 2] = f.z / (float) n;
    if (spp)
        spp[o] = n;
}

__global__ void k_wf_rays_out(const unsigned *cnt, unsigned long long *out) {
    out[0] = *reinterpret_cast<const unsigned long long *>(cnt + kCntRays);
    out[1] = *reinterpret_cast<const unsigned long long *>(cnt + kCntShadowRays);
}

template <class T> T *carve(char *&p, size_t n) {
    T *r = reinterpret_cast<T *>(p);
    p += (n * sizeof(T) + 255) & ~size_t(255);
    return r;
}

} // namespace

// One captured pass and everything it was captured with: the kernels' arguments
// and launch shapes, byte for byte.
struct WavefrontPlan {
    cudaGraph_t graph = nullptr;
    cudaGraphExec_t exec = nullptr;
    std::vector<unsigned char> inputs;
    void release() {
        if (exec)
            cudaGraphExecDestroy(exec);
        if (graph)
            cudaGraphDestroy(graph);
        exec = nullptr;
        graph = nullptr;
    }
    ~WavefrontPlan() { release(); }
};

namespace {

// Bytes of the path-state layout for P paths, npix film pixels and the stacks'
// spilled entries.
size_t wf_bytes(size_t P, int npix, size_t spill) {
    const int ntiles = (int) ((P + kPartTile - 1) / kPartTile);
    const int ptiles = (npix + kPartTile - 1) / kPartTile;
    return 256 * 48 + P * (8 + 16 * 16 + 4 * 2 + 4 * 9 + 2 + 4) + (size_t) ntiles * kPartTile +
           (size_t) npix * (16 + 8 + 32) + (size_t) ptiles * kPartTile +
           (size_t) std::max(ntiles, ptiles) * 32 + 4096 + spill;
}

// Carves the per-path arrays, queues, counters and partition buffers of P
// paths and npix pixels out of `buf` (grown as needed).
int wf_layout(DevBuf &buf, Wf &w, size_t P, int npix, size_t spill) {
    const int ntiles = (int) ((P + kPartTile - 1) / kPartTile);
    const int ptiles = (npix + kPartTile - 1) / kPartTile;
    const size_t bytes = wf_bytes(P, npix, spill);
    PRR_CUDA_TRY(buf.ensure(bytes));
    char *cur = (char *) buf.ptr;
    w.rng = carve<uint64_t>(cur, P);
    w.ro = carve<float4>(cur, P);
    w.rd = carve<float4>(cur, P);
    w.beta = carve<float4>(cur, P);
    w.L = carve<float4>(cur, P);
    w.pend = carve<float4>(cur, P);
    w.prev = carve<float4>(cur, P);
    w.hit = carve<int4>(cur, P);
    w.slo = carve<float4>(cur, P);
    w.sld = carve<float4>(cur, P);
    w.slc = carve<float4>(cur, P);
    w.seo = carve<float4>(cur, P);
    w.sed = carve<float4>(cur, P);
    w.sec = carve<float4>(cur, P);
    w.result = carve<float4>(cur, P);
    w.bounce = carve<int>(cur, P);
    w.flags = carve<int>(cur, P);
    w.req = carve<int>(cur, P);
    w.qray[0] = carve<int>(cur, P);
    w.qray[1] = carve<int>(cur, P);
    w.qmiss = carve<int>(cur, P);
    w.qdelta = carve<int>(cur, P);
    w.qsurf = carve<int>(cur, P);
    w.qshadow = carve<int>(cur, P);
    w.qjob = carve<int>(cur, 2 * P);
    w.vis = carve<uint8_t>(cur, 2 * P);
    w.film = carve<float3>(cur, (size_t) npix);
    w.cnt = carve<unsigned>(cur, kCntSlots);
    w.pass_base = carve<int>(cur, 4);
    w.tag = carve<uint8_t>(cur, (size_t) ntiles * kPartTile);
    w.tile = carve<unsigned>(cur, (size_t) std::max(ntiles, ptiles) * 8);
    w.act = carve<int>(cur, (size_t) npix);
    w.act_next = carve<int>(cur, (size_t) npix);
    w.ptag = carve<uint8_t>(cur, (size_t) ptiles * kPartTile);
    w.wel0 = carve<float4>(cur, (size_t) npix);
    w.wel1 = carve<float4>(cur, (size_t) npix);
    w.spill = carve<char>(cur, spill);
    if ((size_t) (cur - (char *) buf.ptr) > bytes)
        return fail(PRR_ERR_INTERNAL, "wavefront buffer layout overflow");
    return PRR_OK;
}

// Launch shape of one bounce: traversal grids, stack split, spill size.
struct WfShape {
    int block, refill, g_ext, g_sh, g_shade, g_gen, ntiles, ptiles;
    size_t smem_ext, smem_sh, spill_bytes;
    void (*ext)(DevScene, Wf, int, int);
    void (*sh)(DevScene, Wf, int);
};

template <bool MULTI>
int wf_shape(Wf &w, int block_req, int stack_req, int refill_req, WfShape &L) {
    const int sms = device_sm_count();
    L.block = block_req > 0 ? block_req : 128;
    // Stacks: the entries of both levels lie in one. The scene's and the mesh's up
    // to stack_req (0: all of them) are kept in shared memory, within 96 KB per
    // block; deeper ones go to the global spill buffer.
    const int max_sm_entries = (96 * 1024) / (L.block * (int) sizeof(uint2));
    const int blas_sm = stack_req > 0 ? std::min(stack_req, w.blas_cap) : w.blas_cap;
    w.stack_sm = std::min(w.tlas_cap + blas_sm, max_sm_entries);
    L.smem_ext = (size_t) w.stack_sm * L.block * sizeof(uint2);
    L.smem_sh = (size_t) w.stack_sm * L.block * sizeof(uint32_t);
    L.ext = k_wf_extend<MULTI>;
    L.sh = k_wf_shadow<MULTI>;
    if constexpr (!MULTI) {
        if (w.stats) {
            // the counting variants (a separate, untimed render): whole binary
            // stacks in shared memory, so one-warp blocks for deep trees
            L.ext = k_wf_extend_count;
            L.sh = k_wf_shadow_count;
            L.block = 32;
            L.smem_ext = L.smem_sh = (size_t) w.count_stack * L.block * sizeof(uint2);
            if (L.smem_ext > 227 * 1024)
                return fail(PRR_ERR_UNSUPPORTED, "BVH too deep for the counting render");
        }
    }
    if (L.smem_ext > 48 * 1024)
        PRR_CUDA_TRY(cudaFuncSetAttribute((const void *) L.ext,
                                          cudaFuncAttributeMaxDynamicSharedMemorySize,
                                          (int) L.smem_ext));
    if (L.smem_sh > 48 * 1024)
        PRR_CUDA_TRY(cudaFuncSetAttribute((const void *) L.sh,
                                          cudaFuncAttributeMaxDynamicSharedMemorySize,
                                          (int) L.smem_sh));
    // Deep stacks want the largest shared-memory split; shallow ones keep the
    // default, since every change of split between consecutive kernels drains
    // the SM (which dominates frames made of many short launches).
    const int carve_pref = L.smem_ext > 16 * 1024 ? (int) cudaSharedmemCarveoutMaxShared
                                                  : (int) cudaSharedmemCarveoutDefault;
    cudaFuncSetAttribute((const void *) L.ext, cudaFuncAttributePreferredSharedMemoryCarveout,
                         carve_pref);
    cudaFuncSetAttribute((const void *) L.sh, cudaFuncAttributePreferredSharedMemoryCarveout,
                         carve_pref);
    L.refill = refill_req > 0 ? std::min(refill_req, 32) : 12;
    int occ_ext = 1, occ_sh = 1;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ_ext, (const void *) L.ext, L.block,
                                                  L.smem_ext);
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ_sh, (const void *) L.sh, L.block,
                                                  L.smem_sh);
    L.g_ext = sms * std::max(1, occ_ext);
    L.g_sh = sms * std::max(1, occ_sh);
    const size_t spill_entries = (size_t) (w.tlas_cap + w.blas_cap - w.stack_sm);
    L.spill_bytes =
        spill_entries * std::max((size_t) L.g_ext * L.block * sizeof(uint2),
                                 (size_t) L.g_sh * L.block * sizeof(uint32_t));
    L.g_shade = sms * 8;
    L.g_gen = (int) std::min<int64_t>(((int64_t) w.P + 255) / 256, (int64_t) sms * 16);
    L.ntiles = (int) (((size_t) w.P + kPartTile - 1) / kPartTile);
    L.ptiles = (w.npix + kPartTile - 1) / kPartTile;
    return PRR_OK;
}

// The stable partitions of the ordered queues.
struct WfParts {
    PartSpec cls[2], ray[2], act; // cls and ray: by the ray queue they read and write
};
WfParts wf_parts(const Wf &w, int ntiles) {
    WfParts P;
    const bool look = ntiles >= kSkipTiles;
    // hit classes -> miss / delta / surface queues
    for (int r = 0; r < 2; r++) {
        PartSpec &c = P.cls[r] = PartSpec{};
        c.tag = w.tag;
        c.q[0] = w.qmiss;
        c.q[1] = w.qdelta;
        c.q[2] = w.qsurf;
        c.nb = 3;
        c.concat = 0;
        std::fill(c.count_slot, c.count_slot + 8, -1);
        c.count_slot[0] = kCntMiss;
        c.count_slot[1] = kCntDelta;
        c.count_slot[2] = kCntSurf;
        c.total_slot = -1;
        c.from[0] = c.from[1] = look ? kCntRay0 + r : -1;
    }
    // next rays -> the ray queue, direction octant major
    for (int r = 0; r < 2; r++) {
        P.ray[r] = PartSpec{};
        P.ray[r].tag = w.tag;
        P.ray[r].q[0] = w.qray[r];
        P.ray[r].nb = 8;
        P.ray[r].concat = 1;
        for (int b = 0; b < 8; b++)
            P.ray[r].count_slot[b] = -1;
        P.ray[r].total_slot = kCntRay0 + r;
        P.ray[r].from[0] = look ? kCntDelta : -1;
        P.ray[r].from[1] = look ? kCntSurf : -1;
    }
    // adaptive: the pixels still active -> the next pass's active list
    P.act = PartSpec{};
    P.act.tag = w.ptag;
    P.act.map = w.act;
    P.act.q[0] = w.act_next;
    P.act.nb = 1;
    P.act.concat = 1;
    std::fill(P.act.count_slot, P.act.count_slot + 8, -1);
    P.act.total_slot = kCntActive;
    P.act.from[0] = P.act.from[1] = -1;
    return P;
}

// Launches a stage behind the one before it (stage_begin).
template <class... P, class... A>
void launch_stage(void (*kern)(P...), unsigned grid, unsigned block, size_t smem, cudaStream_t cs,
                  const A &...args) {
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(block);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = cs;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    cudaLaunchKernelEx(&cfg, kern, static_cast<P>(args)...);
}

void wf_partition(const Wf &w, const PartSpec &ps, int nt, cudaStream_t cs) {
    launch_stage(k_part_count, nt, kPartThreads, 0, cs, w, ps);
    launch_stage(k_part_scan, 1, 1024, 0, cs, w, nt, ps);
    launch_stage(k_part_scatter, nt, kPartThreads, 0, cs, w, ps);
}

// generate + every bounce of one pass (no film stage)
template <bool MULTI>
int wf_enqueue_bounces(const DevScene &S, const Wf &w, const WfShape &L, const WfParts &parts,
                       cudaStream_t cs) {
    k_wf_generate<MULTI><<<L.g_gen, 256, 0, cs>>>(S, w);
    for (int it = 0; it <= w.max_depth; it++) {
        launch_stage(k_wf_begin, 1, 32, 0, cs, w, it);
        launch_stage(L.ext, L.g_ext, L.block, L.smem_ext, cs, S, w, it, L.refill);
        if (w.ordered)
            wf_partition(w, parts.cls[it & 1], L.ntiles, cs);
        launch_stage(k_wf_miss<MULTI>, L.g_shade, 128, 0, cs, S, w);
        launch_stage(k_wf_delta<MULTI>, L.g_shade, 128, 0, cs, S, w, it + 1);
        launch_stage(k_wf_surface<MULTI>, device_sm_count() * 2, kSurfaceBlock, 0, cs, S, w, it + 1);
        launch_stage(L.sh, L.g_sh, L.block, L.smem_sh, cs, S, w, L.refill);
        launch_stage(k_wf_shadow_resolve<MULTI>, L.g_shade, 128, 0, cs, w);
        if (w.ordered)
            wf_partition(w, parts.ray[(it + 1) & 1], L.ntiles, cs);
    }
    PRR_CUDA_TRY(cudaGetLastError());
    return PRR_OK;
}

} // namespace

int render_wavefront(Scene &s, const prr_render_settings &rs, float *out_rgb, int32_t *out_spp,
                     unsigned long long *out_rays, cudaStream_t st) {
    const DevScene &S = s.dev;
    Wf w;
    WfShape L;
    std::memset(&w, 0, sizeof(w)); // padding too: the bytes are compared (WavefrontPlan)
    std::memset(&L, 0, sizeof(L));
    w.W = s.width;
    w.x0 = rs.x0;
    w.y0 = rs.y0;
    w.ww = rs.x1 - rs.x0;
    w.wh = rs.y1 - rs.y0;
    w.npix = w.ww * w.wh;
    w.max_depth = rs.max_depth;
    w.clamp = rs.indirect_clamp;
    w.seed = rs.seed;
    w.sample_offset = rs.sample_offset;
    w.tlas_cap = S.tlas_stack + 1;
    w.blas_cap = S.blas_stack + 1;
    w.count_stack = S.tlas_depth + S.blas_depth + 2;
    w.ordered = s.wf_ordered ? 1 : 0;
    w.adaptive = rs.min_spp < rs.max_spp ? 1 : 0;
    w.min_spp = rs.min_spp;
    w.max_spp = rs.max_spp;
    w.threshold = rs.variance_threshold;
    w.stats = s.wf_stats;
    w.check = S.check;
    // Paths per pass: whole samples of the window, by default at most 32M in
    // flight (10 GB of path state): every bounce of a pass ends in a tail of
    // long rays, so fewer and larger passes pay it less often.
    // Adaptive renders take 8M: all samples of a pass are traced, also those past
    // a pixel's stop. Museum-like scene at 480x270, up to 256 spp, 8M and 32M: all
    // pixels stopped after one sample 17.2 and 34.9 ms, after 3 20.9 and 35.0,
    // but 56.7 and 49.4 where they take nearly all 256.
    const int64_t kDefaultPaths = (int64_t) 1 << 25, kLeastPaths = (int64_t) 1 << 23;
    const bool automatic = s.wf_paths <= 0;
    int64_t target = s.wf_paths;
    if (automatic)
        target = w.adaptive ? kLeastPaths : s.wf_fit > 0 ? s.wf_fit : kDefaultPaths;
    int spp_pass = 1;
    for (;; target >>= 1) {
        spp_pass = (int) std::max<int64_t>(1, target / std::max(1, w.npix));
        spp_pass = std::min(spp_pass, rs.max_spp);
        while (rs.max_spp % spp_pass)
            spp_pass--;
        w.spp_pass = spp_pass;
        w.P = spp_pass * w.npix;
        if (int rc = wf_shape<false>(w, s.wf_block, s.wf_stack, s.wf_refill, L))
            return rc;
        // More than the least is taken only where it leaves other users of the
        // device three quarters of the free memory, looked up when the buffer has
        // to grow; a smaller size that had to do is kept for the next renders.
        const bool shrinks = automatic && target > kLeastPaths;
        const size_t held = s.d_wavefront.bytes;
        const size_t need = wf_bytes((size_t) w.P, w.npix, L.spill_bytes);
        if (shrinks && need > held) {
            size_t free_bytes = 0, total_bytes = 0;
            PRR_CUDA_TRY(cudaMemGetInfo(&free_bytes, &total_bytes));
            if (need > (free_bytes + held) / 4) {
                s.wf_fit = target >> 1;
                continue;
            }
        }
        const int rc = wf_layout(s.d_wavefront, w, (size_t) w.P, w.npix, L.spill_bytes);
        if (rc == PRR_OK)
            break;
        if (rc != PRR_ERR_OUT_OF_MEMORY || !shrinks)
            return rc;
        cudaGetLastError(); // the failed allocation
        s.wf_fit = target >> 1;
    }
    const WfParts parts = wf_parts(w, L.ntiles);

    PRR_CUDA_TRY(cudaMemsetAsync(w.film, 0, (size_t) w.npix * sizeof(float3), st));
    PRR_CUDA_TRY(cudaMemsetAsync(w.tag, 0xFF, (size_t) L.ntiles * kPartTile, st));
    PRR_CUDA_TRY(cudaMemsetAsync(w.cnt, 0, kCntSlots * sizeof(unsigned), st));
    PRR_CUDA_TRY(cudaMemsetAsync(w.pass_base, 0, sizeof(int), st));
    if (w.adaptive) { // after the counters are cleared: it sets the active count
        PRR_CUDA_TRY(cudaMemsetAsync(w.ptag, 0xFF, (size_t) L.ptiles * kPartTile, st));
        k_wf_adaptive_init<<<(w.npix + 255) / 256, 256, 0, st>>>(w);
    }

    // one pass: the bounces, then the film stage
    auto enqueue_pass = [&](cudaStream_t cs) -> int {
        if (int rc = wf_enqueue_bounces<false>(S, w, L, parts, cs))
            return rc;
        if (w.adaptive) {
            k_wf_film_adaptive<<<(w.npix + 255) / 256, 256, 0, cs>>>(w);
            wf_partition(w, parts.act, L.ptiles, cs);
            k_wf_copy_active<<<(w.npix + 255) / 256, 256, 0, cs>>>(w);
        } else {
            k_wf_film<<<(w.npix + 255) / 256, 256, 0, cs>>>(w);
        }
        PRR_CUDA_TRY(cudaGetLastError());
        return PRR_OK;
    };
    const int passes = rs.max_spp / spp_pass;
    if (!s.wf_plan)
        s.wf_plan = std::make_shared<WavefrontPlan>();
    WavefrontPlan &plan = *s.wf_plan;
    if (s.wf_graphs && passes > 1 && !w.stats) {
        // the scene (its background may change after the build), the window, seed
        // and sampling, the buffers, the launch shapes
        std::vector<unsigned char> inputs(sizeof(S) + sizeof(w) + sizeof(L));
        std::memcpy(inputs.data(), &S, sizeof(S));
        std::memcpy(inputs.data() + sizeof(S), &w, sizeof(w));
        std::memcpy(inputs.data() + sizeof(S) + sizeof(w), &L, sizeof(L));
        if (!plan.exec || plan.inputs != inputs) {
            plan.release();
            cudaStream_t cap;
            PRR_CUDA_TRY(cudaStreamCreateWithFlags(&cap, cudaStreamNonBlocking));
            PRR_CUDA_TRY(cudaStreamBeginCapture(cap, cudaStreamCaptureModeThreadLocal));
            int rc = enqueue_pass(cap);
            cudaGraph_t g = nullptr;
            cudaError_t e = cudaStreamEndCapture(cap, &g);
            cudaStreamDestroy(cap);
            if (rc)
                return rc;
            if (e != cudaSuccess)
                return fail(PRR_ERR_CUDA, std::string("graph capture: ") + cudaGetErrorString(e));
            plan.graph = g;
            PRR_CUDA_TRY(cudaGraphInstantiate(&plan.exec, g, 0));
            plan.inputs = std::move(inputs);
        }
        for (int k = 0; k < passes; k++)
            PRR_CUDA_TRY(cudaGraphLaunch(plan.exec, st));
    } else {
        for (int k = 0; k < passes; k++)
            if (int rc = enqueue_pass(st))
                return rc;
    }
    if (w.adaptive)
        k_wf_resolve_adaptive<<<(w.npix + 255) / 256, 256, 0, st>>>(w.film, w.wel0, w.npix, w.ww, w.wh,
                                                                    out_rgb, out_spp);
    else
        k_wf_resolve<<<(w.npix + 255) / 256, 256, 0, st>>>(w.film, w.npix, w.ww, w.wh, rs.max_spp, out_rgb,
                                                            out_spp);
    PRR_CUDA_TRY(cudaGetLastError());
    if (out_rays) {
        k_wf_rays_out<<<1, 1, 0, st>>>(w.cnt, out_rays);
        PRR_CUDA_TRY(cudaGetLastError());
    }
    // generate + per bounce (begin, extend, miss, delta, surface, shadow,
    // shadow_resolve, and two 3-kernel partitions when ordered) + film
    const int64_t per_pass = 2 + (int64_t) (w.max_depth + 1) * (7 + (w.ordered ? 6 : 0)) +
                             (w.adaptive ? 4 : 0);
    s.last_launches = per_pass * passes + 1 + (w.adaptive ? 1 : 0) + (out_rays ? 1 : 0);
    return PRR_OK;
}

int wavefront_step_multi(WfMultiState &ms, const WfStepReq *reqs, int n,
                         int64_t paths_per_launch, int tlas_cap, int blas_cap,
                         unsigned long long *rays_host, cudaStream_t st, int64_t *launches) {
    if (n <= 0)
        return PRR_OK;
    // the request table of the whole step in pinned memory, one copy up
    const size_t table_bytes = (size_t) n * sizeof(WfReq);
    if (table_bytes > ms.h_cap) {
        if (ms.h_table)
            cudaFreeHost(ms.h_table);
        ms.h_table = nullptr;
        ms.h_cap = std::max(table_bytes, 2 * ms.h_cap);
        PRR_CUDA_TRY(cudaMallocHost(&ms.h_table, ms.h_cap));
    }
    PRR_CUDA_TRY(ms.reqs.ensure(ms.h_cap));
    WfReq *table = static_cast<WfReq *>(ms.h_table);
    // launch groups: consecutive requests of at most paths_per_launch paths
    // (a request alone may exceed it); bases count from each group's start
    struct Group {
        int a, b, max_depth;
        int64_t P, npix;
    };
    std::vector<Group> groups;
    Group g{0, 0, 1, 0, 0};
    for (int k = 0; k < n; k++) {
        const WfStepReq &q = reqs[k];
        const int64_t paths = (int64_t) q.ww * q.wh * q.nspp;
        if (k > g.a && g.P + paths > paths_per_launch) {
            groups.push_back(g);
            g = Group{k, k, 1, 0, 0};
        }
        WfReq &t = table[k];
        std::memset(&t, 0, sizeof(t));
        t.scene = q.scene;
        t.camera = q.camera;
        t.W = q.camera.width;
        t.x0 = q.x0;
        t.y0 = q.y0;
        t.ww = q.ww;
        t.wh = q.wh;
        t.npix = q.ww * q.wh;
        t.s0 = q.s0;
        t.nspp = q.nspp;
        t.max_depth = q.max_depth;
        t.clamp = q.clamp;
        t.seed = q.seed;
        t.path_base = g.P;
        t.pix_base = g.npix;
        t.film = q.film;
        g.P += paths;
        g.npix += t.npix;
        g.max_depth = std::max(g.max_depth, q.max_depth);
        g.b = k + 1;
    }
    groups.push_back(g);
    int64_t maxP = 0;
    for (const Group &x : groups)
        maxP = std::max(maxP, x.P);
    if (maxP >= ((int64_t) 1 << 31))
        return fail(PRR_ERR_INVALID_ARGUMENT, "server step too large");
    PRR_CUDA_TRY(cudaMemcpyAsync(ms.reqs.ptr, table, table_bytes, cudaMemcpyHostToDevice, st));
    int64_t nl = 0;
    for (const Group &x : groups) {
        Wf w{};
        w.P = (int) x.P;
        w.npix = 0; // no per-render film or active list in a server step
        w.max_depth = x.max_depth;
        w.ordered = 1;
        w.reqs = ms.reqs.as<WfReq>() + x.a;
        w.n_reqs = x.b - x.a;
        w.tlas_cap = tlas_cap;
        w.blas_cap = blas_cap;
        WfShape L{};
        if (int rc = wf_shape<true>(w, 128, 8, 0, L))
            return rc;
        if (int rc = wf_layout(ms.state, w, (size_t) maxP, 1, L.spill_bytes))
            return rc;
        const WfParts parts = wf_parts(w, L.ntiles);
        PRR_CUDA_TRY(cudaMemsetAsync(w.tag, 0xFF, (size_t) L.ntiles * kPartTile, st));
        PRR_CUDA_TRY(cudaMemsetAsync(w.cnt, 0, kCntSlots * sizeof(unsigned), st));
        if (int rc = wf_enqueue_bounces<true>(DevScene{}, w, L, parts, st))
            return rc;
        k_wf_film_multi<<<(int) std::min<int64_t>((x.npix + 255) / 256,
                                                  (int64_t) device_sm_count() * 16),
                          256, 0, st>>>(w, x.npix);
        PRR_CUDA_TRY(cudaGetLastError());
        // generate + per bounce (begin, extend, 3-kernel partition, miss,
        // delta, surface, shadow, shadow_resolve, 3-kernel partition) + film
        nl += 1 + (int64_t) (w.max_depth + 1) * 13 + 1;
    }
    // the rays each request traced: one strided copy out of the table
    if (rays_host)
        PRR_CUDA_TRY(cudaMemcpy2DAsync(rays_host, 2 * sizeof(unsigned long long),
                                       &ms.reqs.as<WfReq>()[0].rays, sizeof(WfReq),
                                       2 * sizeof(unsigned long long), n,
                                       cudaMemcpyDeviceToHost, st));
    if (launches)
        *launches = nl;
    return PRR_OK;
}

} // namespace prr
