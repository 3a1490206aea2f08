// The path integrator: Integrator::castRay (Integrator.cpp:104-263) with its
// light-sampling helpers (sampleDirectLight :14-34, sampleEnvironmentMap
// :39-66, evalLightSample :78-87, evalEnvironmentSample :93-102, mis
// Integrator.hpp:30-32), restated for one device thread.
#pragma once
#include "shading.cuh"

namespace prr {

// The part of Intersection the integrator reads (Intersection.hpp:12-34).
struct Inter {
    bool hit;
    V3 p, n;
    int mat;
    SurfAttr a;
};

// Triangle::finalize (Triangle.cpp:34-59) for meshes with per-corner data:
// the hit's barycentrics (re-derived by the same Moller-Trumbore test the
// traversal ran), w0 = 1 - u - v, interpolated uv, smooth normal and tangent
// with its handedness.
__device__ __forceinline__ void finalize_attr(const DevScene &S, const DevObject &o, int tri,
                                              const RayD &r, V3 &n, SurfAttr &a) {
    a = no_attr();
    if (!o.attr)
        return;
    float t, u, v;
    tri_hit(load_tri(S, (uint32_t) tri), r, t, u, v);
    const float w0 = 1.f - u - v;
    const float *R = S.attr + (size_t) (o.attr_base + (tri - o.tri_base)) * kAttrFloats;
    if (o.attr & kAttrUV) {
        a.u = R[9] * w0 + R[11] * u + R[13] * v;
        a.v = R[10] * w0 + R[12] * u + R[14] * v;
    }
    if (o.attr & kAttrNormals)
        n = normalize(v3(R[0], R[1], R[2]) * w0 + v3(R[3], R[4], R[5]) * u +
                      v3(R[6], R[7], R[8]) * v);
    if (o.attr & kAttrTangents) {
        a.tan = normalize(v3(R[15], R[16], R[17]) * w0 + v3(R[18], R[19], R[20]) * u +
                          v3(R[21], R[22], R[23]) * v);
        const float w = R[24] * w0 + R[25] * u + R[26] * v;
        a.hand = w >= 0.f ? 1.f : -1.f;
        a.has_tan = 1;
    }
}

// OOL: spheres tested out of line.
template <bool OOL = false>
__device__ __forceinline__ Inter intersect(const DevScene &S, const Ray3 &ray, SmemStack &tst,
                                           SmemStack &bst) {
    RayD r{ray.o.x, ray.o.y, ray.o.z, ray.d.x, ray.d.y, ray.d.z};
    const RayPre p = precompute(r);
    const SceneHit h = scene_closest<false, OOL>(S, r, p, tst, bst);
    Inter in;
    in.hit = h.obj >= 0;
    in.a = no_attr();
    if (!in.hit) {
        in.p = in.n = v3(0.f);
        in.mat = -1;
        return in;
    }
    const DevObject &o = S.objects[h.obj];
    in.mat = o.material;
    if (o.kind == kObjMesh) {
        // Triangle::finalize (Triangle.cpp:34-59): origin + t * direction, face normal
        in.p = ray.o + h.t * ray.d;
        in.n = v3(S.normals[(size_t) h.tri * 3], S.normals[(size_t) h.tri * 3 + 1],
                  S.normals[(size_t) h.tri * 3 + 2]);
        finalize_attr(S, o, h.tri, r, in.n, in.a);
    } else {
        // Sphere::getIntersection (Sphere.hpp:37-39)
        in.p = ray.o + ray.d * h.t;
        in.n = normalize(in.p - v3(o.cx, o.cy, o.cz));
    }
    return in;
}

template <bool OOL = false>
__device__ __forceinline__ bool occluded(const DevScene &S, V3 o, V3 d, float tmax, SmemStack &tst,
                                         SmemStack &bst) {
    RayD r{o.x, o.y, o.z, d.x, d.y, d.z};
    const RayPre p = precompute(r);
    return scene_occluded<false, OOL>(S, r, p, tst, bst, tmax);
}

__device__ __forceinline__ float mis(float a, float b) { return (a * a) / (a * a + b * b + 1e-6f); }

__device__ __forceinline__ V3 clamp_indirect(V3 c, float clamp) {
    if (clamp <= 0.f)
        return c;
    const float lum = (c.x + c.y + c.z) / 3;
    return (lum > clamp) ? c * (clamp / lum) : c;
}

struct PathCounters {
    uint32_t closest, shadow; // rays traced by this path
};

// Integrator::castRay. `rng` must be positioned after the camera draws.
//
// One loop iteration traces the path's ray, finishes the bounce that spawned it
// (its MIS term or its Russian roulette) and shades the hit, so that the
// traversals, the BSDF evaluation and the environment lookup stand once or
// twice in the code instead of two to four times: with them inlined at every
// use the megakernels stalled on instruction fetch (9 warps of every issue
// cycle; Cornell box 256x256, 16 spp, 2.18 ms).
//
// SYNC: every thread of the block calls it together, with run = false for
// those without a path, and the block starts each iteration together. Its
// warps then read the same instructions at about the same time, which pays
// where the rays' walks are short (Cornell box 2.05 -> 1.44 ms in blocks of
// 384) and costs where they are long and uneven (see render_plain).
template <bool SYNC = false>
static __device__ V3 cast_ray(const DevScene &S, Ray3 ray, int max_depth, float clamp, Rng &rng,
                              SmemStack &tst, SmemStack &bst, PathCounters &cnt,
                              bool run = true) {
    enum { kFirst, kSpecular, kPending };
    V3 L = v3(0.f), beta = v3(1.f);
    Ray3 cur = ray;
    const DevEnv &env = S.env;
    const V3 bg = v3(S.background[0], S.background[1], S.background[2]);
// the path has ended: the loop is left, or (SYNC) gone through idle
#define PRR_PATH_END                                                                               \
    if constexpr (SYNC)                                                                            \
        continue;                                                                                  \
    else                                                                                           \
        break
    int bounce = 0;
    int from = kFirst;                     // what spawned the ray
    V3 scale = v3(0.f), prev = v3(0.f);    // pending bounce: f / pdf, the hit it left from
    float bpdf = 0.f;                      // its pdf
    (void) run; // only SYNC reads it
    for (;;) {
        if constexpr (SYNC) {
            if (!__syncthreads_or(run))
                break;
            if (!run)
                continue;
            run = false; // set again where the path goes on
        }
        const Inter in = intersect<SYNC>(S, cur, tst, bst);
        cnt.closest++;
        const bool lit = !in.hit || S.materials[in.mat].kind == kMatEmissive;
        if (from != kFirst && !(from == kPending && lit)) {
            if (from == kPending) {
                beta = beta * scale;
                if (!finite3(beta))
                    PRR_PATH_END;
                // Russian roulette from bounce 3 (Integrator.cpp:250-256)
                if (bounce >= 3) {
                    const float mc = max3(beta);
                    const float q = smax(0.05f, 1.f - mc);
                    if (rng.next() < q)
                        PRR_PATH_END;
                    beta = beta * (1.f / (1.f - q));
                }
            }
            bounce++;
            if (bounce >= max_depth)
                PRR_PATH_END;
        }
        if (lit && (from == kPending || bounce == 0 || from == kSpecular)) {
            // light reached: seen directly (Integrator.cpp:119-139), or by the
            // pending bounce's BSDF sample, weighted (:213-244)
            V3 e;
            if (!in.hit)
                e = env.loaded ? env_lookup(env, cur.d) : bg;
            else {
                const DevMaterial &m = S.materials[in.mat];
                e = v3(m.emission[0], m.emission[1], m.emission[2]);
            }
            V3 c;
            if (from != kPending) {
                c = beta * e;
            } else if (!in.hit) {
                c = env.loaded ? beta * scale * mis(bpdf, env_pdf(env, cur.d)) * e
                               : beta * scale * e;
            } else {
                const float cos_l = smax(0.f, dot(-cur.d, normalized(in.n)));
                const V3 dd = in.p - prev;
                const float hd2 = dot(dd, dd);
                const float pdf_area = S.total_emit_area > 0.f ? 1.f / S.total_emit_area : 0.f;
                const float pdf_sa = pdf_area * hd2 / smax(cos_l, 1e-4f);
                c = beta * scale * mis(bpdf, pdf_sa) * e;
            }
            L = L + ((bounce > 0) ? clamp_indirect(c, clamp) : c);
            if (from == kPending)
                PRR_PATH_END;
        }
        if (!in.hit)
            PRR_PATH_END;
        const DevMaterial &m = S.materials[in.mat];
        const V3 hp = in.p;
        const V3 gn = in.n;
        const bool delta = m.kind == kMatMirror || m.kind == kMatGlass;
        const V3 sn = delta || dot(cur.d, gn) < 0.f ? gn : -gn;
        const Shading sd = build_shading<true>(S, m, sn, in.a);
        const V3 wo = -cur.d;
        if (delta) {
            // delta chain (Integrator.cpp:143-169)
            const BSDFSample bs = delta_sample(m, sd, wo, rng);
            if (bs.pdf < 1e-6f)
                PRR_PATH_END;
            beta = beta * bs.f / bs.pdf;
            const bool trans = dot(bs.wi, gn) < 0.f;
            const V3 off = trans ? -gn : gn;
            cur = Ray3{hp + off * PRR_EPS, bs.wi};
            if (trans)
                beta = beta * sd.base;
            from = kSpecular;
            if constexpr (SYNC)
                run = true;
            continue;
        }
        const bool indirect = bounce > 0;
        // Three directions leave the hit: towards an area emitter
        // (sampleDirectLight + evalLightSample), towards the environment
        // (sampleEnvironmentMap + evalEnvironmentSample), and the BSDF sample
        // (Integrator.cpp:198-244).
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
                if (env.loaded) {
                    wi = env_importance(env, rng, pdf);
                    ok = !(pdf < 1e-6f);
                    if (ok)
                        em = env_lookup(env, wi);
                }
            } else {
                ok = m.kind == kMatDiffuse && diffuse_direction(m, sd, wo, rng, wi);
            }
            f = v3(0.f);
            bp = 0.f;
            if (ok)
                mat_eval_pdf(m, sd, wi, wo, &f, &bp);
            if (d < 2 && ok) {
                // the contribution is formed before the visibility test (it has
                // no side effects); a zero one needs no shadow ray because
                // castRay would add exactly zero either way
                V3 c = beta * (mis(pdf, bp) * em * f / (d == 0 ? pdf : pdf + 1e-6f));
                if (!(c.x == 0.f && c.y == 0.f && c.z == 0.f)) {
                    cnt.shadow++;
                    if (occluded<SYNC>(S, hp + wi * PRR_EPS, wi, tmax, tst, bst))
                        c = v3(0.f);
                }
                L = L + (indirect ? clamp_indirect(c, clamp) : c);
            }
        }
        if (bp < 1e-6f)
            PRR_PATH_END;
        if (!(bp > 1e-6f)) // DiffuseMaterial::sample leaves f at 0 there
            f = v3(0.f);
        scale = f / bp;
        bpdf = bp;
        prev = hp;
        const V3 off = dot(wi, sd.f.N) >= 0.f ? sd.f.N : -sd.f.N;
        cur = Ray3{hp + off * PRR_EPS, wi};
        from = kPending;
        if constexpr (SYNC)
            run = true;
    }
#undef PRR_PATH_END
    if (!finite3(L))
        return v3(0.f);
    return L;
}

// Welford online mean / variance and the 95% confidence stop of the
// adaptive sampler (Renderer.hpp:14-40), with the reference's float steps.
struct Welford {
    int n = 0;
    float mean = 0.f, M2 = 0.f;
    __device__ void update(float x) {
        n++;
        const float delta = x - mean;
        mean += delta / (float) n;
        M2 += delta * (x - mean);
    }
    __device__ float variance() const { return n < 2 ? 0.f : M2 / (float) (n - 1); }
    __device__ float ci() const {
        if (n < 2 || fabsf(mean) < 1e-6f)
            return 1.f;
        return 1.96f * sqrtf(variance() / (float) n) / fabsf(mean);
    }
};

} // namespace prr
