// tracer.cuh -- device code of the path-tracing core (sm_100a).
//
// Restates the reference's hot path in f32 on the GPU:
//   primitive hits   src/sphere.rs:23-62, quad.rs:29-62, triangle.rs:21-64, obj.rs:259-313,
//                    disk.rs:31-58, plane.rs:42-69, constant_medium.rs:25-69, hit.rs:19-43
//   traversal        src/bvh.rs:52-68 + src/scene.rs:816-834 (closest hit: BVH then planes)
//   materials        src/material.rs:59-391, constant_medium.rs:81-89, texture.rs:9-50
//   NEE              src/render.rs:1333-1466
//   integrator       src/render.rs:1472-1537 (iterative form, see path_bounce)
//   camera           src/camera.rs:82-102
// Random numbers come from Philox4x32-10 keyed by (pixel, stratum, bounce, call).
#pragma once

#include <cuda_runtime.h>
#include <math_constants.h>
#include <stdint.h>

#include "device_scene.h"

namespace lum {

// ------------------------------------------------------------------------------- vectors
struct V {
    float x, y, z;
};
__device__ __forceinline__ V mk(float x, float y, float z) { return V{x, y, z}; }
__device__ __forceinline__ V mk(const float* p) { return V{p[0], p[1], p[2]}; }
__device__ __forceinline__ V operator+(V a, V b) { return {a.x + b.x, a.y + b.y, a.z + b.z}; }
__device__ __forceinline__ V operator-(V a, V b) { return {a.x - b.x, a.y - b.y, a.z - b.z}; }
__device__ __forceinline__ V operator-(V a) { return {-a.x, -a.y, -a.z}; }
__device__ __forceinline__ V operator*(V a, float t) { return {a.x * t, a.y * t, a.z * t}; }
__device__ __forceinline__ V operator*(float t, V a) { return a * t; }
__device__ __forceinline__ V mul(V a, V b) { return {a.x * b.x, a.y * b.y, a.z * b.z}; }
__device__ __forceinline__ float dot(V a, V b) { return fmaf(a.x, b.x, fmaf(a.y, b.y, a.z * b.z)); }
__device__ __forceinline__ V cross(V a, V b) {
    return {a.y * b.z - a.z * b.y, a.z * b.x - a.x * b.z, a.x * b.y - a.y * b.x};
}
__device__ __forceinline__ float len2(V a) { return dot(a, a); }
__device__ __forceinline__ V unit(V a) { return a * rsqrtf(len2(a)); }
__device__ __forceinline__ V fma3(V a, float t, V b) { return {fmaf(a.x, t, b.x), fmaf(a.y, t, b.y), fmaf(a.z, t, b.z)}; }
__device__ __forceinline__ V xyz(float4 a) { return {a.x, a.y, a.z}; }
__device__ __forceinline__ bool near_zero(V a) {
    return fabsf(a.x) < 1e-8f && fabsf(a.y) < 1e-8f && fabsf(a.z) < 1e-8f;
}
__device__ __forceinline__ V reflect(V v, V n) { return v - n * (2.0f * dot(v, n)); }
__device__ __forceinline__ bool has_nan(V a) { return isnan(a.x) || isnan(a.y) || isnan(a.z); }

// -------------------------------------------------------------------------------- RNG
// Philox4x32-10 (Salmon et al., SC'11).  U: unroll factor of the ten rounds (philox_unroll).
__device__ __forceinline__ void philox_round(uint4& c, uint32_t k0, uint32_t k1) {
    uint32_t lo0 = 0xD2511F53u * c.x, hi0 = __umulhi(0xD2511F53u, c.x);
    uint32_t lo1 = 0xCD9E8D57u * c.z, hi1 = __umulhi(0xCD9E8D57u, c.z);
    c = make_uint4(hi1 ^ c.y ^ k0, lo1, hi0 ^ c.w ^ k1, lo0);
}
template <int U = 10>
__device__ __forceinline__ uint4 philox(uint4 c, uint32_t k0, uint32_t k1) {
    if constexpr (U >= 10) {
#pragma unroll
        for (int r = 0; r < 10; ++r) {
            if (r > 0) {
                k0 += 0x9E3779B9u;
                k1 += 0xBB67AE85u;
            }
            philox_round(c, k0, k1);
        }
    } else {
#pragma unroll U
        for (int r = 0; r < 10; ++r) {
            if (r > 0) {
                k0 += 0x9E3779B9u;
                k1 += 0xBB67AE85u;
            }
            philox_round(c, k0, k1);
        }
    }
    return c;
}
__device__ __forceinline__ float u24(uint32_t x) { return (float)(x >> 8) * (1.0f / 16777216.0f); }
template <int U = 10>
__device__ __forceinline__ float4 draw4(uint32_t k0, uint32_t k1, uint32_t pixel, uint32_t stratum, uint32_t bounce,
                                        uint32_t call) {
    uint4 o = philox<U>(make_uint4(pixel, stratum, bounce, call), k0, k1);
    return make_float4(u24(o.x), u24(o.y), u24(o.z), u24(o.w));
}
// The rare draws (dispersion, Blend, Subsurface, moving spheres) out of line, as the other code that few
// paths or scenes reach: pixel filters but the box, checkers, backgrounds but sky and solid, the
// panorama camera, media.  Inlined, they made the kernels' loops wait for instructions (2.2 stalled
// warps per issue on mixed scenes and meshes).  On B200 together, same images: twelve mixed scenes
// 160 -> 145 ms, the materials' scene 13.0 -> 11.0, dense mesh (16 spp) 17.2 -> 16.7, quads 7.63 -> 7.60.
// The light sampler, the disk test and the other materials' scatter stay inline: out of line they
// gained nothing or lost 5-8%.
static __device__ __noinline__ float4 draw4_cold(uint32_t k0, uint32_t k1, uint32_t pixel, uint32_t stratum, uint32_t bounce,
                                                 uint32_t call) {
    return draw4<2>(k0, k1, pixel, stratum, bounce, call);
}
enum : uint32_t { CALL_CAMERA = 0, CALL_CAMERA2 = 1, CALL_SCATTER = 2, CALL_NEE = 3, CALL_EXTRA = 4, CALL_BLEND = 5 };

// Direct (rejection-free) samplers; same distributions as src/vec3.rs:96-122.
__device__ __forceinline__ V unit_vector(float a, float b) {
    float z = 1.0f - 2.0f * a;
    float r = sqrtf(fmaxf(0.0f, 1.0f - z * z));
    float s, c;
    sincospif(2.0f * b, &s, &c);
    return {r * c, r * s, z};
}
__device__ __forceinline__ V in_unit_sphere(float a, float b, float c) { return unit_vector(a, b) * cbrtf(c); }

// ------------------------------------------------------------------------------ ray/hit
struct Ray {
    V o, d;
    float time;
};

struct Hit {
    float t;
    int prim;     // index into the reordered primitive array; -1 none; <= -2 : plane (-2 - index)
    float b1, b2; // triangle barycentrics (u, v)
};

// Record k (0-3, a constant at every call site) of primitive i.
__device__ __forceinline__ float4 ldp(const SceneDev& S, int i, int k) {
    return k < 3 ? __ldg(reinterpret_cast<const float4*>(S.prims) + 3 * i + k)
                 : __ldg(reinterpret_cast<const float4*>(S.prims3) + i);
}

// Robust sphere roots (Haines et al., "Precision Improvements for Ray/Sphere Intersection",
// Ray Tracing Gems 2019): discriminant from the ray-to-centre distance, near root from c/q.
// Spheres of radius >= kBigSphere (ground spheres) evaluate o - c and |o - c|^2 - r^2 in
// f64: in f32 that difference loses ~r * 6e-8 absolutely, which near the surface of an
// r = 1000 sphere is a large relative error of the near root.
// a = |d|^2 and ia = 1 / a are the ray's (the caller may compute them once per ray).
// BIG: r >= kBigSphere is known.
template <bool BIG = false>
__device__ __forceinline__ bool sphere_roots(V c, float r, const Ray& ray, float a, float ia, float& t0, float& t1) {
    V oc;
    float cc;
    if (BIG || r >= kBigSphere) {
        double dx = (double)ray.o.x - (double)c.x, dy = (double)ray.o.y - (double)c.y, dz = (double)ray.o.z - (double)c.z;
        oc = mk((float)dx, (float)dy, (float)dz);
        cc = (float)fma(dx, dx, fma(dy, dy, fma(dz, dz, -(double)r * (double)r)));
    } else {
        oc = ray.o - c;
        cc = fmaf(-r, r, len2(oc));
    }
    float b = dot(oc, ray.d);
    V f = fma3(ray.d, -b * ia, oc);
    float disc = a * (r * r - len2(f));
    if (disc < 0.0f) return false;
    float q = -b - copysignf(sqrtf(disc), b);
    float ta = cc / q, tb = q * ia;
    if (q == 0.0f) ta = tb = -b * ia;
    t0 = fminf(ta, tb);
    t1 = fmaxf(ta, tb);
    return true;
}

__device__ __forceinline__ bool sphere_roots(V c, float r, const Ray& ray, float& t0, float& t1) {
    const float a = len2(ray.d);
    return sphere_roots(c, r, ray, a, 1.0f / a, t0, t1);
}

// sphere.rs:24-45: near root if in [tmin, tmax], else far root.  ia: 1 / |d|^2 of the ray, or 0
// to compute it here.
template <bool BIG = false>
__device__ __forceinline__ bool hit_sphere(float4 a, float4 b, const Ray& ray, float tmin, float tmax, float& t,
                                           float ia = 0.0f) {
    V c = xyz(a);
    if (b.w != 0.0f) c = fma3(xyz(b) - c, ray.time, c);   // MovingSphere::center_at
    float t0, t1;
    const float aa = len2(ray.d);
    if (!sphere_roots<BIG>(c, a.w, ray, aa, ia != 0.0f ? ia : 1.0f / aa, t0, t1)) return false;
    if (t0 >= tmin && t0 <= tmax) { t = t0; return true; }
    if (t1 >= tmin && t1 <= tmax) { t = t1; return true; }
    return false;
}

// quad.rs:29-62.  No early returns: a warp's test ends with its last lane anyway (quads 7.59 -> 7.54
// ms, 128x128 box room 0.294 -> 0.290).  The record keeps w = (u x v)/|u x v|^2 and |u x v|, so the plane test,
// the parallel threshold on the unit normal and the planar coordinates are the reference's.
__device__ __forceinline__ bool hit_quad(float4 a, float4 b, float4 c, float4 d, const Ray& ray, float tmin,
                                         float tmax, float& t, float* uv = nullptr) {
    V w = xyz(d);
    const float denom = dot(w, ray.d);
    const float tt = (a.w - dot(w, ray.o)) / denom;
    V p = fma3(ray.d, tt, ray.o);
    V ph = p - xyz(a);
    const float alpha = dot(w, cross(ph, xyz(c)));
    const float beta = dot(w, cross(xyz(b), ph));
    const bool ok = !(fabsf(denom * b.w) < 1e-8f) & (tt >= tmin) & (tt <= tmax) & (alpha >= 0.0f) & (alpha <= 1.0f) &
                    (beta >= 0.0f) & (beta <= 1.0f);
    if (ok) {
        t = tt;
        if (uv) { uv[0] = alpha; uv[1] = beta; }
    }
    return ok;
}

// triangle.rs:21-64 (Moller-Trumbore)
// The barycentric bounds are tested on the numerators against the determinant (u = su / aa in
// [0, 1] <=> su between 0 and aa, and likewise v >= 0, u + v <= 1), so the division is done only
// for the few candidates that pass them; u, v and t are then the reference's f * numerator.
__device__ __forceinline__ bool hit_tri(float4 a, float4 b, float4 c, const Ray& ray, float tmin, float tmax,
                                        float& t, float& bu, float& bv) {
    V e1 = xyz(b), e2 = xyz(c);
    V h = cross(ray.d, e2);
    float aa = dot(e1, h);
    if (fabsf(aa) < 1e-8f) return false;
    V s = ray.o - xyz(a);
    const float su = dot(s, h);
    const float sg = aa > 0.0f ? 1.0f : -1.0f, da = fabsf(aa);   // numerators scaled to aa > 0
    if (!(su * sg >= 0.0f && su * sg <= da)) return false;
    V q = cross(s, e1);
    const float sv = dot(ray.d, q);
    if (sv * sg < 0.0f || (su + sv) * sg > da) return false;
    const float f = 1.0f / aa;
    const float u = f * su, v = f * sv;
    float tt = f * dot(e2, q);
    if (!(tt >= tmin && tt <= tmax)) return false;
    t = tt;
    bu = u;
    bv = v;
    return true;
}

// disk.rs:31-58
__device__ __forceinline__ bool hit_disk(float4 a, float4 b, const Ray& ray, float tmin, float tmax, float& t) {
    V n = xyz(b);
    float denom = dot(n, ray.d);
    if (fabsf(denom) < 1e-8f) return false;
    float tt = dot(xyz(a) - ray.o, n) / denom;
    if (!(tt >= tmin && tt <= tmax)) return false;
    V off = fma3(ray.d, tt, ray.o) - xyz(a);
    if (len2(off) > a.w * a.w) return false;
    t = tt;
    return true;
}

// constant_medium.rs:25-69.  Boundary entry/exit over the whole line (t_min = -inf), the
// second hit at least 1e-4 past the first; the free-flight distance is the reference's
// deterministic hash of the ray, evaluated in f64 without contraction.
__device__ __forceinline__ bool hit_fog(int type, float4 a, float4 b, float4 c, const Ray& ray, float tmin,
                                        float tmax, float& t) {
    float e0, e1;
    if (type == PT_FOG_SPHERE) {
        if (!sphere_roots(xyz(a), a.w, ray, e0, e1)) return false;
    } else {
        float lo = -CUDART_INF_F, hi = CUDART_INF_F;
        float o[3] = {ray.o.x, ray.o.y, ray.o.z}, d[3] = {ray.d.x, ray.d.y, ray.d.z};
        float mn[3] = {a.x, a.y, a.z}, mx[3] = {b.x, b.y, b.z};
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            float inv = 1.0f / d[k];
            float ta = (mn[k] - o[k]) * inv, tb = (mx[k] - o[k]) * inv;
            lo = fmaxf(lo, fminf(ta, tb));
            hi = fminf(hi, fmaxf(ta, tb));
        }
        if (!(lo <= hi)) return false;
        e0 = lo;
        e1 = hi;
    }
    if (!(e1 >= e0 + 0.0001f)) return false;
    float t1 = fmaxf(e0, tmin), t2 = fminf(e1, tmax);
    if (t1 >= t2) return false;
    if (t1 < 0.0f) t1 = 0.0f;
    float rl = sqrtf(len2(ray.d));
    float inside = (t2 - t1) * rl;
    double hv = __dadd_rn(__dadd_rn(__dadd_rn(__dmul_rn((double)ray.o.x, 73856093.0), __dmul_rn((double)ray.o.y, 19349663.0)),
                                    __dmul_rn((double)ray.o.z, 83492791.0)),
                          __dmul_rn((double)ray.d.x, 47392381.0));
    hv = fabs(hv - trunc(hv));
    double hd = (double)c.x * log(fmax(1.0 - hv, 1e-10));
    if (hd > (double)inside) return false;
    t = t1 + (float)hd / rl;
    return true;
}

// hit_fog out of line (see draw4_cold): two box or sphere roots and the f64 free-flight hash, for a
// handful of primitives.
static __device__ __noinline__ bool hit_fog_cold(int type, float4 a, float4 b, float4 c, const Ray& ray, float tmin,
                                                 float tmax, float& t) {
    return hit_fog(type, a, b, c, ray, tmin, tmax, t);
}

// Scene classes of the general megakernel build (CLS): the primitive types and NEE light kinds
// the kernel carries code for.  A scene runs the smallest class that holds all its primitives
// and lights (SceneDev::cls, chosen by lum_scene_create); code a scene cannot reach costs
// instruction-fetch time in the megakernel.
enum : int {
    CLS_ALL = 0,    // every primitive type and light kind
    CLS_QUAD = 1,   // quads (rects, boxes) with rect lights (box room, quad scenes)
    CLS_MESH = 2,   // triangles, disks and media with disk and rect lights (meshes)
    CLS_GROUND = 3, // CLS_ALL, and big spheres apart from the BVH (SceneDev::n_big)
    CLS_MANY = 4,   // CLS_ALL, CLS_MESH and CLS_QUAD for large scenes (many_prims): their warps turn to the
    CLS_MESH_MANY = 5,   // leaves once at most two lanes still look for one (walk_warp)
    CLS_QUAD_MANY = 6
};
// From these sizes a walk is long enough that the last lanes' search for a leaf costs the others more
// than turning to the leaves early does.  Never against always, ms on B200:
//   mixed primitives, 512x512 16 spp: 2,000 4.10 / 4.13, 4,000 4.97 / 4.89 and 4.68 / 4.49, 8,000 5.38 /
//     5.16, 16,000 6.10 / 5.71; 128x128: 2,000 0.58 / 0.60, 4,000 0.70 / 0.68.  But a batch's scenes run side by
//     side, and two builds at once cost more than that: batches of up to 16,000 primitives with the line at
//     16,384 / 4,096 7.67 / 8.16, 16.5 / 17.1, 45.0 / 45.4
//   quads, 512x512 64 spp: 128 2.11 / 2.12, 200 3.01 / 2.98, 300 3.92 / 3.82, 512 5.42 / 5.26, 1,000 7.21 /
//     7.03; 256x256 16 spp, where the longest tasks count: 128 0.240 / 0.256, 300 0.424 / 0.432, 512 0.574 /
//     0.578, 1,000 0.808 / 0.803
//   meshes, 960x540 16 spp: 1,280 triangles 3.17 / 3.25, 20,480 4.03 / 4.04, 81,920 4.57 / 4.45, 327,680 5.25 / 4.90
// Four lanes gave 2% less on the mesh; ratios of waiting to searching lanes (4, 8, 14) no more.
__host__ constexpr int many_prims(int cls) {
    return cls == CLS_MESH ? 65536 : cls == CLS_QUAD ? 512 : 16384;
}
template <int CLS>
__host__ __device__ constexpr bool cls_is_quad() { return CLS == CLS_QUAD || CLS == CLS_QUAD_MANY; }
template <int CLS>
__host__ __device__ constexpr int cls_slack() { return CLS == CLS_MANY || CLS == CLS_MESH_MANY || CLS == CLS_QUAD_MANY ? 2 : 0; }
template <int CLS>
__host__ __device__ constexpr bool cls_is_mesh() { return CLS == CLS_MESH || CLS == CLS_MESH_MANY; }
template <int CLS>
__host__ __device__ constexpr bool cls_has_big() { return CLS == CLS_GROUND; }
template <int CLS>
__host__ __device__ constexpr bool cls_is_all() { return CLS == CLS_ALL || CLS == CLS_GROUND || CLS == CLS_MANY; }

// Unroll factor of the Philox rounds in a build.  The mesh, general and other-materials builds are bound
// by instruction fetch, and each inlined draw site carries the ten rounds: rolled by two the mesh
// ran 186.1 -> 173.3 ms on B200, mixed scenes 150.5 -> 148.8, the materials' scene 11.3 -> 11.2; the
// sphere field, bound by issue, runs 4-6% slower that way and keeps them unrolled, as does the
// quad class (box room 1% slower rolled).
template <int CLS, bool SPH = false>
constexpr int philox_unroll() { return CLS == CLS_QUAD || CLS == CLS_QUAD_MANY || SPH ? 10 : 2; }
template <int CLS>
__host__ __device__ constexpr bool cls_has_prim(int type) {
    return cls_is_all<CLS>() || (cls_is_quad<CLS>() && type == PT_QUAD) ||
           (cls_is_mesh<CLS>() && (type == PT_TRIANGLE || type == PT_DISK || type == PT_FOG_SPHERE || type == PT_FOG_BOX));
}
template <int CLS>
__host__ __device__ constexpr bool cls_has_light(int kind) {   // 1 sphere, 2 rect, 3 disk
    return cls_is_all<CLS>() || (cls_is_quad<CLS>() && kind == 2) || (cls_is_mesh<CLS>() && (kind == 2 || kind == 3));
}

// One primitive test; updates the closest hit when t is within [tmin, hit.t].  The record carries
// its type (record 2's w), so its 48 bytes come in one round trip: with the type in the separate
// meta array, the test waited for it before it fetched records 1 and 2.  The quad class holds
// quads only and reads no type.  On B200: quads 512x512 8.06 -> 7.88 ms, box room 1.73 -> 1.71, the
// materials' scene 14.3 -> 14.2, mixed scenes 179.6 -> 178.3.
// SPH: the scene's primitives are all static spheres (SceneDev::spheres_basic), so the other
// primitive tests are left out of the kernel and a test reads only record 0 (centre, radius).
// ia_ray: 1 / |d|^2 of the ray, computed once per walk by the sphere-class build (0 elsewhere).
template <bool COUNT = false, bool SPH = false, int CLS = CLS_ALL>
__device__ __forceinline__ bool test_prim(const SceneDev& S, int i, const Ray& ray, float tmin, Hit& hit,
                                          TestTally* tl = nullptr, float ia_ray = 0.0f) {
    float4 a = ldp(S, i, 0);
    float t;
    if constexpr (SPH && !COUNT) {
        if (hit_sphere(a, make_float4(0.0f, 0.0f, 0.0f, 0.0f), ray, tmin, hit.t, t, ia_ray)) {
            hit.t = t;
            hit.prim = i;
            return true;
        }
        return false;
    }
    if constexpr (cls_is_quad<CLS>() && !COUNT) {   // every primitive is a quad
        const float4 b = ldp(S, i, 1), c = ldp(S, i, 2), d = ldp(S, i, 3);
        if (hit_quad(a, b, c, d, ray, tmin, hit.t, t)) { hit.t = t; hit.prim = i; return true; }
        return false;
    }
    const float4 b = ldp(S, i, 1), c = ldp(S, i, 2);
    const int type = __float_as_int(c.w) & 15;
    if constexpr (COUNT) tl->prim[type]++;
    switch (type) {
        case PT_SPHERE: {
            if constexpr (!cls_has_prim<CLS>(PT_SPHERE)) return false;
            if (hit_sphere(a, b, ray, tmin, hit.t, t)) { hit.t = t; hit.prim = i; return true; }
            return false;
        }
        case PT_QUAD: {
            if constexpr (!cls_has_prim<CLS>(PT_QUAD)) return false;
            float4 d = ldp(S, i, 3);
            if (hit_quad(a, b, c, d, ray, tmin, hit.t, t)) { hit.t = t; hit.prim = i; return true; }
            return false;
        }
        case PT_TRIANGLE: {
            if constexpr (!cls_has_prim<CLS>(PT_TRIANGLE)) return false;
            float bu, bv;
            if (hit_tri(a, b, c, ray, tmin, hit.t, t, bu, bv)) {
                hit.t = t; hit.prim = i; hit.b1 = bu; hit.b2 = bv;
                return true;
            }
            return false;
        }
        case PT_DISK: {
            if constexpr (!cls_has_prim<CLS>(PT_DISK)) return false;
            if (hit_disk(a, b, ray, tmin, hit.t, t)) { hit.t = t; hit.prim = i; return true; }
            return false;
        }
        default: {
            if constexpr (!cls_has_prim<CLS>(PT_FOG_BOX)) return false;
            if (hit_fog_cold(type, a, b, c, ray, tmin, hit.t, t)) { hit.t = t; hit.prim = i; return true; }
            return false;
        }
    }
}

// plane.rs:42-69
__device__ __forceinline__ bool hit_plane(const PlaneDev& P, const Ray& ray, float tmin, float tmax, float& t) {
    V n = mk(P.n);
    float denom = dot(n, ray.d);
    if (fabsf(denom) < 1e-8f) return false;
    float tt = dot(mk(P.p) - ray.o, n) / denom;
    if (!(tt >= tmin && tt <= tmax)) return false;
    t = tt;
    return true;
}

// ------------------------------------------------------------------------------ traversal
// BVH2 traversal with postponed leaves (the "while-while" organisation of Aila & Laine,
// "Understanding the Efficiency of Ray Traversal on GPUs", HPG 2009), one warp at a time: the
// whole warp runs the two loops below in step, every lane with a walk visiting inner nodes until
// each of them holds a leaf, then all lanes testing their leaves together.  Inner nodes are visited
// near child first.  Stack entries (shared memory, entry k of thread j at
// stack[k * blockDim.x + j]) are inner-node indices (>= 0) or leaf ranges ~(first << 3 |
// count - 1); entry 0 holds kSentinel, so a pop needs no test for the empty stack.
constexpr int kSentinel = 0x7fffffff;

// Bytes of dynamic shared memory of a block's stacks of `depth` entries (and the sentinel).
__host__ __device__ constexpr size_t stack_smem(int depth, int threads) {
    return (size_t)(depth + 1) * threads * sizeof(int);
}
// The thread's stack in the block's dynamic shared memory, its sentinel set.
__device__ __forceinline__ int* lane_stack(int* smem) {
    int* s = smem + threadIdx.x;
    *s = kSentinel;
    return s;
}

// The end of a node visit, given both children's slab intervals: the nearer child hit becomes the
// node, the other one is pushed (or, past `limit`, dropped with the overflow flag); with no child
// hit the node is popped; a node that is a leaf becomes the postponed leaf if there is none, and
// another is popped.  sp: 32-bit shared address of the top entry.  One block of predicated
// instructions: no branches, so the lanes that pop and those that push stay together, and no
// predicate is turned into an integer and back (the integer pipe is the busiest, 63-67%): against
// predicated accesses taking 0/1 operands 20.8 -> 20.3 ms on the sphere field (64 spp), 1% on quads
// and the box room.
__device__ __forceinline__ void visit_children(float en0, float ex0, float en1, float ex1, int link0, int link1,
                                               int& node, int& leaf, uint32_t& sp, uint32_t limit, uint32_t stride,
                                               uint32_t& err) {
    asm volatile(
        "{\n"
        ".reg .pred h0, h1, c1, both, none, room, push, over, post;\n"
        ".reg .b32 n, f;\n"
        "setp.lt.f32 h0, %4, %5;\n"
        "setp.lt.f32 h1, %6, %7;\n"
        "setp.lt.f32 c1, %6, %4;\n"          // child 1 first: h1 && (!h0 || en1 < en0)
        "not.pred none, h0;\n"
        "or.pred c1, c1, none;\n"
        "and.pred c1, c1, h1;\n"
        "and.pred both, h0, h1;\n"
        "or.pred none, h0, h1;\n"
        "not.pred none, none;\n"
        "selp.b32 n, %9, %8, c1;\n"
        "selp.b32 f, %8, %9, c1;\n"
        "setp.lt.u32 room, %2, %10;\n"
        "and.pred push, both, room;\n"
        "not.pred room, room;\n"
        "and.pred over, both, room;\n"
        "@over or.b32 %3, %3, %12;\n"
        "@push add.u32 %2, %2, %11;\n"
        "@push st.shared.b32 [%2], f;\n"
        "@none ld.shared.b32 n, [%2];\n"
        "@none sub.u32 %2, %2, %11;\n"
        "setp.lt.s32 post, n, 0;\n"
        "setp.eq.and.s32 post, %1, 0, post;\n"
        "@post mov.b32 %1, n;\n"
        "@post ld.shared.b32 n, [%2];\n"
        "@post sub.u32 %2, %2, %11;\n"
        "mov.b32 %0, n;\n"
        "}"
        : "=r"(node), "+r"(leaf), "+r"(sp), "+r"(err)
        : "f"(en0), "f"(ex0), "f"(en1), "f"(ex1), "r"(link0), "r"(link1), "r"(limit), "r"(stride),
          "n"((int)LUM_KERR_STACK_OVERFLOW)
        : "memory");
}
__device__ __forceinline__ int load_shared(uint32_t addr) {
    int v;
    asm volatile("ld.shared.b32 %0, [%1];" : "=r"(v) : "r"(addr) : "memory");
    return v;
}

// Two f32 fused multiply-adds in one instruction (each rounded as fmaf rounds).
__device__ __forceinline__ unsigned long long pair_of(float x) {
    unsigned long long r;
    asm("mov.b64 %0, {%1, %1};" : "=l"(r) : "f"(x));
    return r;
}
__device__ __forceinline__ float2 fma_pair(unsigned long long a, unsigned long long b, unsigned long long c) {
    float2 r;
    asm("{\n.reg .b64 t;\nfma.rn.f32x2 t, %2, %3, %4;\nmov.b64 {%0, %1}, t;\n}"
        : "=f"(r.x), "=f"(r.y) : "l"(a), "l"(b), "l"(c));
    return r;
}


// Place of a suspended BVH walk (walk_warp): the next node to visit (an inner node index, or
// kSentinel when the walk is over) and the stack's depth in bytes; the stack entries stay in
// shared memory and the closest hit so far in the caller's Hit.
struct Trav {
    int node;
    int sp;
};

// The BVH walks of a warp, resumable.  Called by all 32 lanes; `act`: the lane has a walk (its
// place in tv, {0, 0} at the start, or kSentinel for a scene without nodes; found as false).
// With SUSPEND > 0 the call returns once at most SUSPEND lanes are still walking (none of them
// holding a leaf): those keep their place in tv, so that the lanes which finished can shade and
// start new rays before the warp walks on (Aila & Laine 2009 replace terminated rays in the same
// spirit: a warp's traversal otherwise runs as long as its longest ray while the finished lanes
// idle).  Returns true for a lane whose walk is complete (planes tested, `found` final).
//
// What bounds it is instruction issue and how many lanes each instruction serves.  So both loops
// are the warp's: their conditions are full-warp votes, which also bring the lanes together
// after every visit and every primitive test; a visit ends without branches (visit_children); a leaf's
// primitives and a second pending leaf follow each other in one loop, so a lane with a short
// leaf takes its next one meanwhile; and the slab tests use the packed f32 FMA.  The earlier form
// (each lane's own loops, which the compiler let diverge: 11.4 lanes per instruction on the box
// room, 7.2 on the mixed scenes) against this one, same box, same images: sphere field 1080p 64
// spp 23.0 -> 21.8 ms, dense mesh 1080p 16 spp 20.2 -> 17.8, quads 512x512 9.77 -> 8.56, box room
// 1.99 -> 1.83, twelve mixed scenes 236 -> 200, adaptive sphere field 34.4 -> 30.7.
// Leaving the node loop once at most 3 lanes lack a leaf gained 1-2% on the sphere field and the
// mesh and lost 7-9% on the room and the materials' scene; leaving it only when no lane can
// walk on (no vote on leaves) lost 4-13%; leaving the leaf loop with 2, 6 or 12 lanes' leaves
// unfinished lost 2-10%; branches instead of predicated stack accesses lost up to 3%.
template <bool COUNT = false, bool SPH = false, int SUSPEND = 0, int CLS = CLS_GROUND>
__device__ __forceinline__ bool walk_warp(const SceneDev& S, const Ray& ray, float tmin, bool any, Hit& hit,
                                          bool& found, Trav& tv, int* stack, uint32_t& err, bool act,
                                          bool fresh, TestTally* tl = nullptr) {
    constexpr unsigned full = 0xffffffffu;
    // Reciprocals of direction components clamped away from zero: the FMA slab form
    // lo*inv - o*inv would give inf - inf = NaN for an axis-parallel ray, while a finite
    // +-1e20 keeps the ordering of the reference's (lo - o) * (1/d) (aabb.rs:23-25).
    const float ix = 1.0f / (fabsf(ray.d.x) > 1e-20f ? ray.d.x : copysignf(1e-20f, ray.d.x));
    const float iy = 1.0f / (fabsf(ray.d.y) > 1e-20f ? ray.d.y : copysignf(1e-20f, ray.d.y));
    const float iz = 1.0f / (fabsf(ray.d.z) > 1e-20f ? ray.d.z : copysignf(1e-20f, ray.d.z));
    const unsigned long long ix2 = pair_of(ix), iy2 = pair_of(iy), iz2 = pair_of(iz);
    const unsigned long long ox2 = pair_of(-ray.o.x * ix), oy2 = pair_of(-ray.o.y * iy), oz2 = pair_of(-ray.o.z * iz);
    // the sphere class divides by |d|^2 once per walk instead of once per sphere test
    float ia_ray = 0.0f;
    if constexpr (SPH && !COUNT) ia_ray = 1.0f / len2(ray.d);
    const ulonglong2* nodes = reinterpret_cast<const ulonglong2*>(S.nodes);
    const uint32_t stride = blockDim.x * 4u;
    const uint32_t base = (uint32_t)__cvta_generic_to_shared(stack);
    const uint32_t limit = base + (uint32_t)S.stack_depth * stride;
    uint32_t sp = base + (uint32_t)tv.sp;      // address of the top entry
    int node = act ? tv.node : kSentinel;      // inner node index, leaf (< 0) or kSentinel
    int leaf = 0;                              // postponed leaf (< 0) or 0
    // The big spheres, for all new walks of the warp at once: in the tree a ground was a leaf that nearly
    // every ray visited and tested in f64 a few lanes at a time.  Found first, it also shortens the
    // ray.  Sphere field (64 spp) 19.9 -> 19.1 ms, adaptive 26.4 -> 25.0, same images; only the builds
    // that meet such scenes carry it (general scenes 2-10% slower with it).
    if constexpr (cls_has_big<CLS>() || SPH || COUNT) {
        for (int k = S.n_prims - S.n_big; k < S.n_prims; ++k) {
            if constexpr (COUNT) tl->prim[PT_SPHERE] += fresh ? 1 : 0;
            const float4 c = ldp(S, k, 0);
            float t;
            if (fresh && !(any && found) &&
                hit_sphere<true>(c, make_float4(0.0f, 0.0f, 0.0f, 0.0f), ray, tmin, hit.t, t, ia_ray)) {
                hit.t = t;
                hit.prim = k;
                found = true;
                if (any) node = kSentinel;
            }
        }
    }
    for (;;) {
        for (;;) {
            if ((unsigned)node < (unsigned)kSentinel) {
                const ulonglong2 n0 = __ldg(nodes + 4 * node + 0), n1 = __ldg(nodes + 4 * node + 1),
                                 n2 = __ldg(nodes + 4 * node + 2);
                const int2 link = __ldg(reinterpret_cast<const int2*>(nodes + 4 * node + 3));
                if constexpr (COUNT) tl->node++;
                // slab tests of both children (aabb.rs:18-56), lo and hi of an axis per pair
                const float2 ax = fma_pair(n0.x, ix2, ox2), ay = fma_pair(n0.y, iy2, oy2), az = fma_pair(n2.x, iz2, oz2);
                const float2 bx = fma_pair(n1.x, ix2, ox2), by = fma_pair(n1.y, iy2, oy2), bz = fma_pair(n2.y, iz2, oz2);
                const float en0 = fmaxf(fmaxf(fminf(ax.x, ax.y), fminf(ay.x, ay.y)), fmaxf(fminf(az.x, az.y), tmin));
                const float ex0 = fminf(fminf(fmaxf(ax.x, ax.y), fmaxf(ay.x, ay.y)), fminf(fmaxf(az.x, az.y), hit.t));
                const float en1 = fmaxf(fmaxf(fminf(bx.x, bx.y), fminf(by.x, by.y)), fmaxf(fminf(bz.x, bz.y), tmin));
                const float ex1 = fminf(fminf(fmaxf(bx.x, bx.y), fmaxf(by.x, by.y)), fminf(fmaxf(bz.x, bz.y), hit.t));
                visit_children(en0, ex0, en1, ex1, link.x, link.y, node, leaf, sp, limit, stride, err);
            }
            // on while some lane that can walk has no leaf yet
            // (builds for large scenes: while more than kSlack such lanes are left, or none holds a leaf)
            const bool on = (unsigned)node < (unsigned)kSentinel && leaf == 0;
            constexpr int kSlack = cls_slack<CLS>();
            if constexpr (kSlack > 0) {
                const unsigned left = __ballot_sync(full, on);
                if (left == 0 || (__popc(left) <= kSlack && __any_sync(full, leaf < 0))) break;
            } else {
                if (!__any_sync(full, on)) break;
            }
        }
        int k = 0, last = -1;                  // primitives of the leaf to test
        if (leaf < 0) {
            k = (~leaf) >> 3;
            last = k + ((~leaf) & 7);
            leaf = 0;
        }
        for (;;) {
            if (k <= last) {
                if (test_prim<COUNT, SPH, CLS>(S, k, ray, tmin, hit, tl, ia_ray)) {
                    found = true;
                    if (any) {                 // the shadow query is answered
                        node = kSentinel;
                        last = -1;
                    }
                }
                ++k;
                if (k > last && node < 0) {    // the next node is a leaf too
                    k = (~node) >> 3;
                    last = k + ((~node) & 7);
                    node = load_shared(sp);
                    sp -= stride;
                }
            }
            if (!__any_sync(full, k <= last)) break;
        }
        if (__popc(__ballot_sync(full, node != kSentinel)) <= SUSPEND) break;
    }
    if (act) {
        tv.node = node;
        tv.sp = (int)(sp - base);
    }
    if (!act || node != kSentinel) return false;
    for (int k = 0; k < S.n_planes && !(any && found); ++k) {              // scene.rs:826-831
        if constexpr (COUNT) tl->plane++;
        float t;
        if (hit_plane(S.planes[k], ray, tmin, hit.t, t)) {
            hit.t = t;
            hit.prim = -2 - k;
            found = true;
        }
    }
    return true;
}

// LUM_SUSPEND_LANES, the SUSPEND of the persistent kernels' walks (half of it in the sphere class):
// lanes still walking the BVH when at most that many of the warp are left keep their place and let
// the finished lanes shade and start new rays first (walk_warp); 0 = every walk runs to its end
// before any lane shades.  Measured on B200 with warp-convergent walks (kernel time per frame,
// images identical), 4 / 8 / 12 lanes: dense mesh 17.2 / 16.7 / 16.8 ms, quads 7.69 / 7.60 / 7.68, mixed
// scenes 147.4 / 145.4 / 145.3, sphere field 18.5 / 18.6 / 19.2 (2 lanes 18.5).
#ifndef LUM_SUSPEND_LANES
#define LUM_SUSPEND_LANES 8
#endif

// Closest hit (any = false) keeps the nearest accepted t; any = true returns at the first
// accepted hit (the shadow query, render.rs:1457-1460).  Unbounded planes follow the BVH
// (scene.rs:826-831).  Called by the whole warp; act: the lane has a ray.
template <bool COUNT = false, bool SPH = false>
__device__ __forceinline__ bool trace(const SceneDev& S, const Ray& ray, float tmin, bool any, Hit& hit, int* stack,
                                      uint32_t& err, bool act, TestTally* tl = nullptr) {
    bool found = false;
    Trav tv{S.n_nodes > 0 ? 0 : kSentinel, 0};
    walk_warp<COUNT, SPH, 0, CLS_GROUND>(S, ray, tmin, any, hit, found, tv, stack, err, act, act, tl);
    return found;
}

// ---------------------------------------------------------------------------- hit details
struct Surface {
    V p, n;          // point, normal facing the ray
    bool front;
    int mat;
};

// Point, outward normal, face orientation and material of a hit (hit.rs:19-43).
template <bool SPH = false, int CLS = CLS_ALL>
__device__ __forceinline__ Surface surface_of(const SceneDev& S, const Ray& ray, const Hit& h) {
    Surface s;
    s.p = fma3(ray.d, h.t, ray.o);
    V on;
    if (h.prim <= -2) {
        const PlaneDev& P = S.planes[-2 - h.prim];
        on = mk(P.n);
        s.mat = P.material;
    } else {
        // material and type: record 2's w, in the L1 since the hit (the sphere class's tests read only
        // record 0)
        const int meta = SPH ? __ldg(S.meta + h.prim) : __float_as_int(ldp(S, h.prim, 2).w);
        int type = SPH ? (int)PT_SPHERE : meta & 15;
        s.mat = meta >> 4;
        float4 a = ldp(S, h.prim, 0);
        switch (type) {
            case PT_SPHERE: {
                if constexpr (!cls_has_prim<CLS>(PT_SPHERE)) break;
                V c = xyz(a);
                if constexpr (!SPH) {
                    float4 b = ldp(S, h.prim, 1);
                    if (b.w != 0.0f) c = fma3(xyz(b) - c, ray.time, c);
                }
                on = (s.p - c) * (1.0f / a.w);
                break;
            }
            case PT_QUAD: {
                if constexpr (!cls_has_prim<CLS>(PT_QUAD)) break;
                float4 d = ldp(S, h.prim, 3);
                on = unit(xyz(d)) * d.w;
                break;
            }
            case PT_TRIANGLE: {
                if constexpr (!cls_has_prim<CLS>(PT_TRIANGLE)) break;
                float4 d = ldp(S, h.prim, 3);
                int si = __float_as_int(d.w);
                if (si >= 0) {
                    const float* sn = S.smooth_n + 9 * si;
                    float w0 = 1.0f - h.b1 - h.b2;
                    on = unit(mk(sn) * w0 + mk(sn + 3) * h.b1 + mk(sn + 6) * h.b2);
                } else {
                    on = xyz(d);
                }
                break;
            }
            case PT_DISK:
                if constexpr (cls_has_prim<CLS>(PT_DISK)) on = xyz(ldp(S, h.prim, 1));
                break;
            default: on = mk(1.0f, 0.0f, 0.0f); break;                 // constant_medium.rs:63
        }
    }
    s.front = dot(ray.d, on) < 0.0f;
    s.n = s.front ? on : -on;
    return s;
}

// ------------------------------------------------------------------------------ shading
static __device__ __noinline__ V checker_cold(const MatDev* mp, V p) {           // texture.rs:19-50
    const MatDev& m = *mp;
    float inv = 1.0f / m.tex_scale;
    long long x = (long long)floorf(p.x * inv), y = (long long)floorf(p.y * inv), z = (long long)floorf(p.z * inv);
    return ((x + y + z) % 2 == 0) ? mk(m.color) : mk(m.color2);
}
__device__ __forceinline__ V tex_value(const MatDev& m, V p) { return m.tex == 0 ? mk(m.color) : checker_cold(&m, p); }

__device__ __forceinline__ V emitted(const MatDev& m, V p) {           // material.rs:241-243
    return m.kind == 4 ? tex_value(m, p) * m.intensity : mk(0.0f, 0.0f, 0.0f);
}

__device__ __forceinline__ float schlick(float cosine, float ref_idx) { // material.rs:138-141
    float r0 = (1.0f - ref_idx) / (1.0f + ref_idx);
    r0 = r0 * r0;
    float m = 1.0f - cosine;
    float m2 = m * m;
    return r0 + (1.0f - r0) * (m2 * m2 * m);
}

__device__ __forceinline__ V fresnel(float cos_t, V f0) {              // material.rs:291-294
    float m = fmaxf(1.0f - cos_t, 0.0f);
    float m2 = m * m;
    float t = m2 * m2 * m;
    return f0 * (1.0f - t) + mk(t, t, t);
}

// material.rs:297-319 with tan(theta) evaluated directly (same angle, no atan/sin/cos); sp, cp: the
// azimuth's sine and cosine.
__device__ __forceinline__ V ggx_normal(V n, float alpha, float r1, float sp, float cp) {
    float tan2 = alpha * alpha * r1 / (1.0f - r1 + 1e-10f);
    float ct = rsqrtf(1.0f + tan2);
    float st = sqrtf(tan2) * ct;
    V up = fabsf(n.y) < 0.999f ? mk(0.f, 1.f, 0.f) : mk(1.f, 0.f, 0.f);
    V tg = unit(cross(up, n));
    V bt = cross(n, tg);
    return unit(tg * (st * cp) + bt * (st * sp) + n * ct);
}

struct Scatter {
    V dir;
    V att;
    V org;   // origin of the scattered ray: the hit point (set by the caller), or Subsurface's exit point
};

enum : int { MAT_BLEND = 7 };

// Blend::scatter's choice (material.rs:408-415): one draw per level, mat_a with probability
// ratio, down to a material that is not a Blend.
__device__ __forceinline__ const MatDev* blend_walk(const MatDev* mats, const MatDev* m, uint32_t key0,
                                                        uint32_t key1, uint32_t pixel, uint32_t stratum,
                                                        uint32_t bounce) {
    const float4 u = draw4_cold(key0, key1, pixel, stratum, bounce, CALL_BLEND);
    const float uu[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
    for (int l = 0; l < kMaxBlendDepth; ++l) {
        if (m->kind != MAT_BLEND) break;
        m = &mats[uu[l] < m->extra[0] ? m->sub[0] : m->sub[1]];
    }
    return m;
}
__device__ __forceinline__ const MatDev& blend_leaf(const SceneDev& S, const MatDev& m, const RenderDev& R,
                                                    uint32_t pixel, uint32_t stratum, uint32_t bounce) {
    return m.kind == MAT_BLEND ? *blend_walk(S.mats, &m, R.key0, R.key1, pixel, stratum, bounce) : m;
}

// Blend::emitted (material.rs:417-420): ratio * emitted(a) + (1 - ratio) * emitted(b),
// evaluated from the blend's flattened list of emissive leaves (no recursion, no call).
__device__ __forceinline__ V emitted_at(const SceneDev& S, int idx, const MatDev& m, V p) {
    if (m.kind != MAT_BLEND) return emitted(m, p);
    V e = mk(0.f, 0.f, 0.f);
    for (int k = 0; k < m.n_emit; ++k) {
        const BlendEmit be = S.blend_emit[m.emit_first + k];
        e = e + emitted(S.mats[be.leaf], p) * be.weight;
    }
    return e;
}

// Iridescent::thin_film_color (material.rs:469-491): sin^2(phase / 2) at 650 / 532 / 450 nm
// with phase = 2 pi opd / lambda, i.e. sin^2(pi opd / lambda).
__device__ __forceinline__ V thin_film(float cos_t, float thickness, float film_ior) {
    float sin_t = sqrtf(fmaxf(1.0f - cos_t * cos_t, 0.0f));
    float sf = sin_t / film_ior;
    float cf = sqrtf(fmaxf(1.0f - sf * sf, 0.0f));
    float opd = 2.0f * thickness * film_ior * cf;
    float r = sinpif(opd / 650.0f), g = sinpif(opd / 532.0f), b = sinpif(opd / 450.0f);
    return mk(r * r, g * g, b * b);
}

// The other materials' scatter (material.rs:408-865).  Keyed draws: CALL_SCATTER slots as
// noted, Subsurface's exit direction from CALL_EXTRA.  Inlined like everything the megakernel
// calls: a device-function call makes every value live across it a spill candidate.
struct ScatterMore {
    V dir, att, org;
    bool ok;
};
__device__ __forceinline__ ScatterMore scatter_more(const MatDev* mp, V rd, V hp, V hn, float4 s, uint32_t key0,
                                                       uint32_t key1, uint32_t pixel, uint32_t stratum,
                                                       uint32_t bounce) {
    const MatDev& m = *mp;
    ScatterMore out;
    out.org = hp;
    out.ok = true;
    struct {
        V p, n;
    } sf{hp, hn};
    struct {
        V d;
    } ray{rd};
    switch (m.kind) {
        case 8: {                                                      // Transparent, material.rs:429-435
            out.dir = ray.d;
            out.att = mk(1.f, 1.f, 1.f);
            return out;
        }
        case 9: {                                                      // Iridescent, material.rs:499-527
            V ud = unit(ray.d);
            float ct = fminf(fabsf(dot(-ud, sf.n)), 1.0f);
            out.att = mul(mk(m.color), thin_film(ct, m.extra[0], m.ior));
            V d = reflect(ud, sf.n);
            if (m.roughness > 0.0f) {
                d = d + in_unit_sphere(s.x, s.y, s.z) * m.roughness;
                if (dot(d, sf.n) <= 0.0f) { out.ok = false; return out; }
            }
            out.dir = d;
            return out;
        }
        case 10: {                                                     // Toon, material.rs:549-577
            V d = sf.n + unit_vector(s.x, s.y);
            if (near_zero(d)) d = sf.n;
            V du = unit(d);
            float ndl = fmaxf(dot(du, sf.n), 0.0f);
            float band = fminf(fmaxf(floorf(ndl * m.extra[0]) / (m.extra[0] - 1.0f), 0.0f), 1.0f);
            V hv = unit(unit(-ray.d) + du);
            float spec = powf(fmaxf(dot(hv, sf.n), 0.0f), m.extra[1] * 100.0f);
            out.dir = d;
            out.att = mk(m.color) * (band + (spec > 0.5f ? 0.3f : 0.0f));
            return out;
        }
        case 11: {                                                     // Anisotropic, material.rs:607-641
            V refl = reflect(unit(ray.d), sf.n);
            const int ax = (int)m.extra[2];
            V wt = ax == 0 ? mk(1.f, 0.f, 0.f) : (ax == 1 ? mk(0.f, 1.f, 0.f) : mk(0.f, 0.f, 1.f));
            V t = unit(wt - sf.n * dot(wt, sf.n));
            V b = cross(sf.n, t);
            float sp, cp;
            sincospif(2.0f * s.x, &sp, &cp);
            float r2 = sqrtf(s.y);
            V sc = unit(refl + t * (cp * r2 * m.extra[0]) + b * (sp * r2 * m.extra[1]));
            if (!(dot(sc, sf.n) > 0.0f)) { out.ok = false; return out; }
            out.dir = sc;
            out.att = mk(m.color);
            return out;
        }
        case 12: {                                                     // Clearcoat, material.rs:664-707
            V ud = unit(ray.d);
            float ct = fminf(fabsf(dot(-ud, sf.n)), 1.0f);
            float r0 = (1.0f - m.ior) / (1.0f + m.ior);
            r0 = r0 * r0;
            float om = 1.0f - ct, om2 = om * om;
            float fr = r0 + (1.0f - r0) * (om2 * om2 * om);
            if (s.x < fr * m.extra[0]) {
                V refl = reflect(ud, sf.n);
                float rough = (1.0f - m.extra[0]) * 0.3f;
                V d = refl;
                if (rough > 0.001f) {
                    V fz = refl + in_unit_sphere(s.y, s.z, s.w) * rough;
                    if (dot(fz, sf.n) > 0.0f) d = fz;
                }
                out.dir = d;
                out.att = mk(1.f, 1.f, 1.f);
                return out;
            }
            V d = sf.n + unit_vector(s.y, s.z);
            if (near_zero(d)) d = sf.n;
            out.dir = d;
            out.att = mk(m.color);
            return out;
        }
        case 13: {                                                     // Velvet, material.rs:724-746
            V d = sf.n + unit_vector(s.x, s.y);
            if (near_zero(d)) d = sf.n;
            float ct = fabsf(dot(-unit(ray.d), sf.n));
            float st = sqrtf(fmaxf(1.0f - ct * ct, 0.0f));
            out.dir = d;
            out.att = mk(m.color) * (1.0f + st * sqrtf(st) * m.extra[0]);
            return out;
        }
        case 14: {                                                     // Translucent, material.rs:769-797
            V d;
            if (s.x < m.extra[0]) {
                V below = -sf.n + unit_vector(s.y, s.z);
                d = unit(ray.d) * (1.0f - m.extra[1]) + below * m.extra[1];
                if (near_zero(d)) d = -sf.n;
            } else {
                d = sf.n + unit_vector(s.y, s.z);
                if (near_zero(d)) d = sf.n;
            }
            out.dir = d;
            out.att = mk(m.color);
            return out;
        }
        case 15: {                                                     // Subsurface, material.rs:823-864
            float fr = schlick(fabsf(dot(unit(ray.d), sf.n)), 1.0f / 1.4f);
            if (s.x < fr) {
                V d = sf.n + unit_vector(s.y, s.z);
                if (near_zero(d)) d = sf.n;
                out.dir = d;
                out.att = mk(m.color);
                return out;
            }
            const float mfp = m.extra[0];
            float step = -mfp * logf(fmaxf(s.y, 1e-10f));
            out.org = sf.p + unit_vector(s.z, s.w) * step;
            float4 ex = draw4_cold(key0, key1, pixel, stratum, bounce, CALL_EXTRA);
            V d = sf.n + unit_vector(ex.x, ex.y);
            out.dir = near_zero(d) ? sf.n : unit(d);
            const float k = -step / mfp;
            out.att = mul(mk(m.color), mk(__expf(k * (1.0f - m.color2[0])), __expf(k * (1.0f - m.color2[1])),
                                          __expf(k * (1.0f - m.color2[2]))));
            return out;
        }
        default:
            { out.ok = false; return out; }
    }
}

// Material::scatter; draws s = (s0..s3) of CALL_SCATTER, extra for dispersion.
// KIND >= 0 fixes the material kind at compile time (the material-sorted shading kernels of
// the wavefront tracer); KIND = -1 dispatches on m.kind.  Both run the same arithmetic.
// EXT = false leaves out the other materials (material.rs:396-865): kernels for scenes
// without them carry none of their code (the megakernel is sensitive to its code size).
// SPH: the scene's materials are Lambertian / Metal / Dielectric / Emissive only.
template <int KIND = -1, bool EXT = true, bool SPH = false, int U = 10>
__device__ __forceinline__ bool scatter(const MatDev& m, const Ray& ray, const Surface& sf, float hit_t, float4 s,
                                        const RenderDev& R, uint32_t pixel, uint32_t stratum, uint32_t bounce,
                                        Scatter& out) {
    if constexpr (SPH) {
        if (KIND < 0 && m.kind > 3) return false;                      // Emissive: no scatter
    }
    // The materials' random unit vector, evaluated once for all lanes of the warp (Lambertian, Metal and
    // Isotropic draw it from s.x, s.y; rough Dielectric and both Microfacet lobes' azimuths from s.y,
    // s.z): each material inlined its own copy, for its own lanes, in kernels bound by instruction
    // fetch and divergence.  Twelve mixed scenes 169 -> 159 ms, dense mesh (16 spp) 17.6 -> 17.2,
    // quads 7.76 -> 7.62, box room 1.66 -> 1.65, sphere field (64 spp) 18.9 -> 18.8.
    const int kind = KIND >= 0 ? KIND : m.kind;
    const bool late = kind == 3 || kind == 5;
    float us, uc;
    sincospif(2.0f * (late ? s.z : s.y), &us, &uc);
    const float uz = 1.0f - 2.0f * (late ? s.y : s.x);
    const float ur = sqrtf(fmaxf(0.0f, 1.0f - uz * uz));
    // n plus the unit vector, fused explicitly (see add_light), and the unit vector times x
    auto about = [&](V n) { return V{fmaf(ur, uc, n.x), fmaf(ur, us, n.y), n.z + uz}; };
    auto times = [&](float x) { return V{ur * uc, ur * us, uz} * x; };
    switch (kind) {
        case 1: {                                                      // material.rs:59-71
            V d = about(sf.n);
            if (near_zero(d)) d = sf.n;
            out.dir = d;
            out.att = tex_value(m, sf.p);
            return true;
        }
        case 2: {                                                      // material.rs:94-106
            V refl = reflect(unit(ray.d), sf.n);
            V sc = refl + times(cbrtf(s.z)) * m.fuzz;
            if (dot(sc, sf.n) > 0.0f) {
                out.dir = sc;
                out.att = mk(m.color);
                return true;
            }
            return false;
        }
        case 3: {                                                      // material.rs:149-213
            float ior = m.ior;
            V chan = mk(1.f, 1.f, 1.f);
            if (m.dispersion > 0.0f) {
                float4 ex = draw4_cold(R.key0, R.key1, pixel, stratum, bounce, CALL_EXTRA);
                uint32_t ch = (uint32_t)(ex.x * 3.0f);
                ior += ch == 0 ? -m.dispersion : (ch == 1 ? 0.0f : m.dispersion);
                chan = ch == 0 ? mk(3.f, 0.f, 0.f) : (ch == 1 ? mk(0.f, 3.f, 0.f) : mk(0.f, 0.f, 3.f));
            }
            float eta = sf.front ? 1.0f / ior : ior;
            V ud = unit(ray.d);
            float ct = fminf(dot(-ud, sf.n), 1.0f);
            float st = sqrtf(1.0f - ct * ct);
            V d;
            if (eta * st > 1.0f || schlick(ct, eta) > s.x) {
                d = reflect(ud, sf.n);
            } else {                                                   // vec3.rs:73-78
                V rp = (ud + sf.n * ct) * eta;
                d = rp + sf.n * -sqrtf(fabsf(1.0f - len2(rp)));
            }
            if (m.roughness > 0.0f) d = d + times(cbrtf(s.w)) * m.roughness;
            V att;
            if (!sf.front && !m.tint_white)
                att = mk(__expf(-(1.0f - m.tint[0]) * hit_t), __expf(-(1.0f - m.tint[1]) * hit_t),
                         __expf(-(1.0f - m.tint[2]) * hit_t));
            else
                att = mk(m.tint);
            if (m.dispersion > 0.0f) att = mul(att, chan);
            out.dir = d;
            out.att = att;
            return true;
        }
        case 5: {                                                      // material.rs:328-390
            float alpha = m.roughness * m.roughness;
            V v = unit(-ray.d);
            V n = sf.n;
            V alb = tex_value(m, sf.p);
            float ndv = fmaxf(dot(n, v), 0.001f);
            V f0 = mk(0.04f, 0.04f, 0.04f) * (1.0f - m.metallic) + alb * m.metallic;
            V fw = fresnel(ndv, f0);
            float sp = fminf(fmaxf((fw.x + fw.y + fw.z) * (1.0f / 3.0f), 0.1f), 0.9f);
            if (s.x < sp) {
                V h = ggx_normal(n, alpha, s.y, us, uc);
                V l = h * (2.0f * dot(v, h)) - v;
                float ndl = dot(n, l);
                if (ndl <= 0.0f) return false;
                float ndh = fmaxf(dot(n, h), 0.0f);
                float vdh = fmaxf(dot(v, h), 0.0f);
                float k = (m.roughness + 1.0f) * (m.roughness + 1.0f) * 0.125f;
                float g = (ndv / (ndv * (1.0f - k) + k)) * (ndl / (ndl * (1.0f - k) + k));
                V f = fresnel(vdh, f0);
                V w = ndh > 0.001f ? f * (g * vdh / (ndv * ndh)) : mk(0.f, 0.f, 0.f);
                out.dir = l;
                out.att = w * (1.0f / sp);
                return true;
            }
            V d = about(n);
            if (near_zero(d)) d = n;
            V kd = (mk(1.f, 1.f, 1.f) - fw) * (1.0f - m.metallic);
            out.dir = d;
            out.att = mul(kd, alb) * (1.0f / (1.0f - sp));
            return true;
        }
        case 6: {                                                      // constant_medium.rs:81-89
            out.dir = times(cbrtf(s.z));
            out.att = mk(m.color);
            return true;
        }
        case 8: case 9: case 10: case 11: case 12: case 13: case 14: case 15: {
            if constexpr (EXT) {
                const ScatterMore r = scatter_more(&m, ray.d, sf.p, sf.n, s, R.key0, R.key1, pixel, stratum, bounce);
                out.dir = r.dir;
                out.att = r.att;
                out.org = r.org;
                return r.ok;
            }
            return false;
        }
        default:                                                       // Emissive: no scatter
            return false;
    }
}

// render.rs:1333-1343 (Frisvad)
__device__ __forceinline__ void build_onb(V n, V& a, V& b) {
    if (n.z < -0.9999999f) {
        a = mk(0.f, -1.f, 0.f);
        b = mk(-1.f, 0.f, 0.f);
        return;
    }
    float aa = 1.0f / (1.0f + n.z);
    float bb = -n.x * n.y * aa;
    a = mk(1.0f - n.x * n.x * aa, bb, -n.x);
    b = mk(bb, 1.0f - n.y * n.y * aa, -n.y);
}

// Samples one light (render.rs:1346-1455).  Returns false when the sample contributes
// nothing before visibility; otherwise the shadow ray and unoccluded contribution.
template <int CLS = CLS_ALL>
__device__ __forceinline__ bool sample_light(const SceneDev& S, V hp, V normal, V albedo, float4 u, Ray& shadow,
                                             float& shadow_tmax, V& contrib) {
    int nl = S.n_lights;
    int idx = min((int)(u.y * (float)nl), nl - 1);
    const LightDev& L = S.lights[idx];
    V lp, ln;
    float area;
    if (!cls_has_light<CLS>(L.kind)) return false;                      // not in this build's class
    if (cls_has_light<CLS>(1) && L.kind == 1) {
        V to_c = mk(L.p0) - hp;
        float d2c = len2(to_c);
        if (d2c < L.radius * L.radius) return false;
        float dc = sqrtf(d2c);
        float stm = L.radius / dc;
        float ctm = sqrtf(fmaxf(1.0f - stm * stm, 0.0f));
        float ct = 1.0f - u.z * (1.0f - ctm);
        float st = sqrtf(fmaxf(1.0f - ct * ct, 0.0f));
        float sp, cp;
        sincospif(2.0f * u.w, &sp, &cp);
        V w = to_c * (1.0f / dc);
        V a, b;
        build_onb(w, a, b);
        V dir = unit(a * (st * cp) + b * (st * sp) + w * ct);
        V oc = hp - mk(L.p0);
        float bc = dot(oc, dir);
        float cc = len2(oc) - L.radius * L.radius;
        float disc = bc * bc - cc;
        float t;
        if (disc > 0.0f) {
            float sq = sqrtf(disc);
            float t1 = -bc - sq;
            t = t1 > 0.001f ? t1 : -bc + sq;
        } else {
            t = dc;
        }
        lp = fma3(dir, t, hp);
        ln = unit(lp - mk(L.p0));
        float solid = 2.0f * CUDART_PI_F * (1.0f - ctm);
        area = solid * t * t / fmaxf(fabsf(dot(-dir, ln)), 0.001f);
    } else if (cls_has_light<CLS>(2) && L.kind == 2) {
        lp = mk(L.p0) + mk(L.u) * u.z + mk(L.v) * u.w;
        area = L.area;
        ln = mk(L.n);
    } else if constexpr (cls_has_light<CLS>(3)) {
        float r = sqrtf(u.z) * L.radius;
        float sp, cp;
        sincospif(2.0f * u.w, &sp, &cp);
        V w = mk(L.n);
        V av = fabsf(w.x) > 0.9f ? mk(0.f, 1.f, 0.f) : mk(1.f, 0.f, 0.f);
        V ut = unit(cross(w, av));
        V vt = cross(w, ut);
        lp = mk(L.p0) + ut * (r * cp) + vt * (r * sp);
        area = L.area;
        ln = w;
    } else {
        return false;
    }
    V tl = lp - hp;
    float d2 = len2(tl);
    float dist = sqrtf(d2);
    V dir = tl * (1.0f / dist);
    float ct = dot(normal, dir);
    if (ct <= 0.0f) return false;
    float ctl = fabsf(dot(-dir, ln));
    if (ctl <= 0.001f) return false;
    shadow.o = hp;
    shadow.d = dir;
    shadow.time = 0.0f;                                                // Ray::new (render.rs:1457)
    shadow_tmax = dist - 0.001f;
    contrib = mul(mk(L.e), albedo) * (ct * ctl * area * (float)nl / (CUDART_PI_F * d2));
    return true;
}

// sample_light out of line for the mesh class (see hit_fog_cold).
template <int CLS>
__device__ __noinline__ bool sample_light_cold(const SceneDev& S, V hp, V normal, V albedo, float4 u, Ray& shadow,
                                               float& shadow_tmax, V& contrib) {
    return sample_light<CLS>(S, hp, normal, albedo, u, shadow, shadow_tmax, contrib);
}

// Background::Starfield (render.rs:86-112): dark blue space plus stars hashed from the
// direction quantised at 500 * density cells per unit.
__device__ __forceinline__ V starfield(float density, float brightness, V ud, float t) {
    V space = mk(0.0f, 0.0f, 0.02f) * (1.0f - t) + mk(0.02f, 0.0f, 0.05f) * t;
    const float scale = 500.0f * density;
    const long long ix = (long long)floorf(ud.x * scale), iy = (long long)floorf(ud.y * scale),
                    iz = (long long)floorf(ud.z * scale);
    const unsigned long long hash = ((unsigned long long)ix * 73856093ull) ^ ((unsigned long long)iy * 19349663ull) ^
                                    ((unsigned long long)iz * 83492791ull);
    const float star = (float)(hash % 10000ull) / 10000.0f;
    if (!(star > 0.997f)) return space;
    const float rh = (float)((hash >> 8) % 100ull) / 100.0f;
    const V c = rh < 0.3f ? mk(1.0f, 0.9f, 0.8f) : (rh < 0.6f ? mk(0.9f, 0.9f, 1.0f) : mk(1.f, 1.f, 1.f));
    return space + c * (star * brightness);
}

// Background::EnvMap (render.rs:113-151): equirectangular lookup, bilinear, times intensity.
__device__ __forceinline__ V envmap(const float* env, uint32_t env_w, uint32_t env_h, float intensity, V ud) {
    if (!env) return mk(0.f, 0.f, 0.f);
    const float theta = acosf(-ud.y);
    const float phi = atan2f(-ud.z, ud.x) + CUDART_PI_F;
    const float fx = phi * (0.5f / CUDART_PI_F) * (float)env_w - 0.5f;
    const float fy = theta * (1.0f / CUDART_PI_F) * (float)env_h - 0.5f;
    const float flx = floorf(fx), fly = floorf(fy);
    const int w = (int)env_w, h = (int)env_h;
    int x0 = (int)flx % w;
    if (x0 < 0) x0 += w;
    const int y0 = (int)fminf(fmaxf(fly, 0.0f), (float)(h - 1));
    const int x1 = (x0 + 1) % w, y1 = min(y0 + 1, h - 1);
    const float tx = fx - flx, ty = fy - fly;
    auto px = [&](int x, int y) { return mk(env + 3 * ((size_t)y * w + x)); };
    const V c = px(x0, y0) * ((1.0f - tx) * (1.0f - ty)) + px(x1, y0) * (tx * (1.0f - ty)) +
                px(x0, y1) * ((1.0f - tx) * ty) + px(x1, y1) * (tx * ty);
    return c * intensity;
}

// The unit direction and the gradients' blend are rounded explicitly (see add_light): an image must
// not depend on which kernel's contraction of y * rsqrt + 1 or a * (1 - t) + b * t it got.
template <bool EXT = true>
__device__ __noinline__ V background_cold(const float* env, uint32_t env_w, uint32_t env_h, const RenderDev& R, V rd) {  // render.rs:73-171
    const float rl = rsqrtf(len2(rd));
    const V ud = V{__fmul_rn(rd.x, rl), __fmul_rn(rd.y, rl), __fmul_rn(rd.z, rl)};
    const float t = 0.5f * __fadd_rn(ud.y, 1.0f), u = __fsub_rn(1.0f, t);
    auto blend = [t, u](V a, V b) {
        return V{fmaf(b.x, t, __fmul_rn(a.x, u)), fmaf(b.y, t, __fmul_rn(a.y, u)), fmaf(b.z, t, __fmul_rn(a.z, u))};
    };
    if (R.background == 2) return blend(mk(R.bg_color), mk(R.bg_color2));
    if (R.background == 3) {
        V sky = blend(mk(1.f, 1.f, 1.f), mk(R.bg_color2));
        float sd = dot(ud, unit(mk(R.bg_dir)));
        if (sd > 0.9995f) return mk(R.bg_color) * R.bg_intensity;
        if (sd > 0.995f) {
            float glow = (sd - 0.995f) / (0.9995f - 0.995f);
            return sky + mk(R.bg_color) * (R.bg_intensity * 0.3f * glow);
        }
        return sky;
    }
    if constexpr (EXT) {
        if (R.background == 4) return starfield(R.star_density, R.star_brightness, ud, t);
        if (R.background == 5) return envmap(env, env_w, env_h, R.bg_intensity, ud);
    }
    return blend(mk(1.f, 1.f, 1.f), mk(0.5f, 0.7f, 1.0f));
}
template <bool EXT = true>
__device__ __forceinline__ V background(const SceneDev& S, const RenderDev& R, const Ray& r) {  // render.rs:73-171
    if (R.background == 1) return mk(R.bg_color);
    if (R.background != 0) return background_cold<EXT>(S.env, S.env_w, S.env_h, R, r.d);
    const float rl = rsqrtf(len2(r.d));
    const float t = 0.5f * __fadd_rn(__fmul_rn(r.d.y, rl), 1.0f), u = __fsub_rn(1.0f, t);
    return V{fmaf(0.5f, t, u), fmaf(0.7f, t, u), fmaf(1.0f, t, u)};
}

// The pixel filter is written with explicitly rounded operations (no FMA contraction): the
// compiler contracts a*b+c per call site, so the same expression could round differently in the
// megakernel and in the wavefront kernels, and the images of both must agree bit for bit.
__device__ __forceinline__ float mitchell_1d(float x) {                // render.rs:220-237
    x = fabsf(x);
    const float b = 1.0f / 3.0f, c = 1.0f / 3.0f;
    const float x2 = __fmul_rn(x, x), x3 = __fmul_rn(x2, x);
    if (x < 1.0f)
        return __fdiv_rn(__fadd_rn(__fadd_rn(__fmul_rn(12.f - 9.f * b - 6.f * c, x3),
                                             __fmul_rn(-18.f + 12.f * b + 6.f * c, x2)),
                                   6.f - 2.f * b), 6.f);
    if (x < 2.0f)
        return __fdiv_rn(__fadd_rn(__fadd_rn(__fadd_rn(__fmul_rn(-b - 6.f * c, x3), __fmul_rn(6.f * b + 30.f * c, x2)),
                                             __fmul_rn(-12.f * b - 48.f * c, x)),
                                   8.f * b + 24.f * c), 6.f);
    return 0.0f;
}
static __device__ __noinline__ float filter_weight_cold(int f, float dx, float dy) {  // render.rs:201-216
    if (f == 1)
        return __fmul_rn(fmaxf(__fsub_rn(1.0f, __fmul_rn(fabsf(dx), 2.0f)), 0.0f),
                         fmaxf(__fsub_rn(1.0f, __fmul_rn(fabsf(dy), 2.0f)), 0.0f));
    if (f == 2) return __expf(__fdiv_rn(-__fadd_rn(__fmul_rn(dx, dx), __fmul_rn(dy, dy)), 2.0f * 0.35f * 0.35f));
    if (f == 3) return __fmul_rn(mitchell_1d(__fmul_rn(dx, 2.0f)), mitchell_1d(__fmul_rn(dy, 2.0f)));
    return 1.0f;
}
__device__ __forceinline__ float filter_weight(int f, float dx, float dy) {
    return f == 0 ? 1.0f : filter_weight_cold(f, dx, dy);
}

// A finished path's contribution to its pixel (render.rs:1692-1701): radiance clamped to
// luminance 100, times the filter weight, and the weight; explicitly rounded like the filter.
__device__ __forceinline__ float4 path_sample(const RenderDev& R, V L, float jx, float jy) {
    const float lum = __fadd_rn(__fadd_rn(__fmul_rn(0.2126f, L.x), __fmul_rn(0.7152f, L.y)), __fmul_rn(0.0722f, L.z));
    const float k = lum > 100.0f ? __fdiv_rn(100.0f, lum) : 1.0f;
    const float w = filter_weight(R.pixel_filter, __fsub_rn(jx, 0.5f), __fsub_rn(jy, 0.5f));
    if (lum > 100.0f) L = V{__fmul_rn(L.x, k), __fmul_rn(L.y, k), __fmul_rn(L.z, k)};
    return make_float4(__fmul_rn(L.x, w), __fmul_rn(L.y, w), __fmul_rn(L.z, w), w);
}

// ------------------------------------------------------------------------------ path state
struct Path {
    Ray ray;
    V beta;        // throughput B_j
    V L;           // accumulated radiance
    float jx, jy;  // stratum jitter (pixel filter)
    uint32_t stratum;
    uint32_t bounce;
    bool skip_emission;
};

__device__ __forceinline__ unsigned long long globaltimer() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

// a / b for a finite a and b = 1, 2, ... with r = 1 / b rounded to nearest: the quotient a * r
// corrected by its exact remainder (Markstein, "Computation of elementary functions on the IBM RISC
// System/6000 processor", IBM J. Res. Dev. 1990).  His theorem 8.1 asks for a first quotient within one
// ulp, and two roundings only give 1.5, so that this is the rounded quotient is checked, not proven:
// no difference for any b below 2^16 and any mantissa of a, nor in 2^30 draws with b up to 2^24.
// r = 0 stands for b = 0: the plain division.
__device__ __forceinline__ float div_by(float a, float b, float r) {
    if (r == 0.0f) return a / b;
    const float q = a * r;
    return fmaf(fmaf(-q, b, a), r, q);
}

// Direction of the equirectangular camera at (uc, vc); out of line, see draw4_cold.
static __device__ __noinline__ V panorama_dir(V fwd, V u, V v, float uc, float vc) {
    // equirectangular (camera.rs:83-90): latitude theta = pi (1 - t), longitude
    // phi = 2 pi s - pi, unit direction; no lens
    // (explicitly rounded: the compiler contracts a * b + c into an FMA per call site, and
    // every kernel must produce the same direction bit for bit)
    float st_, ct_, sp_, cp_;
    sincospif(1.0f - vc, &st_, &ct_);
    sincospif(fmaf(2.0f, uc, -1.0f), &sp_, &cp_);
    const float a_ = __fmul_rn(st_, cp_), b_ = __fmul_rn(st_, sp_);
    return mk(fmaf(fwd.x, a_, fmaf(u.x, b_, __fmul_rn(v.x, ct_))),
                   fmaf(fwd.y, a_, fmaf(u.y, b_, __fmul_rn(v.y, ct_))),
                   fmaf(fwd.z, a_, fmaf(u.z, b_, __fmul_rn(v.z, ct_))));
}

// Camera ray through sub-pixel position (jx, jy) of pixel (gi, gj) for stratum st; c holds
// the stratum's camera draws (z, w: lens) (render.rs:1683-1690, camera.rs:82-102).
template <int U = 10>
__device__ __forceinline__ void start_path_at(const SceneDev& S, const RenderDev& R, uint32_t gi, uint32_t gj,
                                              uint32_t pixel, uint32_t st, float4 c, float jx, float jy, Path& P) {
    P.jx = jx;
    P.jy = jy;
    float y = (float)(R.full_h - 1 - gj);
    const float uc = div_by((float)gi + P.jx, (float)(R.full_w - 1), R.inv_w1);
    const float vc = div_by(y + P.jy, (float)(R.full_h - 1), R.inv_h1);
    const CameraDev& C = S.cam;
    if (C.panorama) {
        const V d = panorama_dir(mk(C.fwd), mk(C.u), mk(C.v), uc, vc);
        P.ray.o = mk(C.origin);
        P.ray.d = d * rsqrtf(len2(d));
    } else {
        V off = mk(0.f, 0.f, 0.f);
        if (C.lens_radius > 0.0f) {
            float r = sqrtf(c.z) * C.lens_radius, sp, cp;
            sincospif(2.0f * c.w, &sp, &cp);
            off = mk(C.u) * (r * cp) + mk(C.v) * (r * sp);
        }
        P.ray.o = mk(C.origin) + off;
        P.ray.d = mk(C.llc) + mk(C.hor) * uc + mk(C.ver) * vc - mk(C.origin) - off;
    }
    // time matters only to moving spheres; a static scene skips the draw (the keyed draws of
    // the other calls do not depend on it)
    P.ray.time = S.moving ? draw4_cold(R.key0, R.key1, pixel, st, 0, CALL_CAMERA2).x : 0.0f;
    P.beta = mk(1.f, 1.f, 1.f);
    P.L = mk(0.f, 0.f, 0.f);
    P.stratum = st;
    P.bounce = 0;
    P.skip_emission = false;
}

// Camera ray of stratum st: stratified jitter (render.rs:1683-1690).  A path start is a tenth of the
// sphere field's time, and its divisions were most of it: the stratum's row comes from a high
// multiply, the image coordinates from div_by, the tile's pixel from shifts (tile_task).  With
// the box filter's constant weights left out of the sums as well: sphere field (64 spp) 20.3 ->
// 20.0 ms, box room 1.69 -> 1.66, quads 7.86 -> 7.75.
template <int U = 10>
__device__ __forceinline__ void start_path(const SceneDev& S, const RenderDev& R, uint32_t gi, uint32_t gj,
                                           uint32_t pixel, uint32_t st, Path& P) {
    const uint32_t sy = R.root_magic ? __umulhi(st, R.root_magic) : st / R.sqrt_spp, sx = st - sy * R.sqrt_spp;
    const float inv_n = R.inv_root;
    float4 c = draw4<U>(R.key0, R.key1, pixel, st, 0, CALL_CAMERA);
    start_path_at<U>(S, R, gi, gj, pixel, st, c, ((float)sx + c.x) * inv_n, ((float)sy + c.y) * inv_n, P);
}

// The one sample of a pixel after the time limit: stratum 0's draws, the pixel centre
// (render.rs:1612-1616).
__device__ __forceinline__ void start_path_centre(const SceneDev& S, const RenderDev& R, uint32_t gi, uint32_t gj,
                                                  uint32_t pixel, Path& P) {
    start_path_at(S, R, gi, gj, pixel, 0, draw4(R.key0, R.key1, pixel, 0, 0, CALL_CAMERA), 0.5f, 0.5f, P);
}

// Path states of the megakernel lanes.
enum : int { ST_IDLE = 0, ST_CLOSEST = 1, ST_SHADOW = 2, ST_DONE = 3 };

// NEE shadow query pending after a bounce: direction from the new hit point, its t range
// end, and the contribution B_j * (E albedo cos cos' A N / (pi d^2)) added if unoccluded.
// The shadow ray starts at the path's origin (P.ray.o), the hit point.  When Subsurface moves
// the next segment's origin to its exit point while a shadow query is pending, shade keeps the
// hit point in P.ray.o, writes the exit point to the caller's stash and negates tmax; the
// caller traces the shadow to |tmax| and then moves P.ray.o to the stashed point
// (shadow_done).
struct Pending {
    V dir;
    float tmax;
    V contrib;
};

// After a shadow query: the deferred Subsurface origin move, if any.
template <bool EXT>
__device__ __forceinline__ void shadow_done(Path& P, Pending& pend, const V* exit_stash) {
    if constexpr (EXT) {
        if (pend.tmax < 0.0f) {
            P.ray.o = *exit_stash;
            pend.tmax = -pend.tmax;
        }
    }
}

// L += B (.) e, fused explicitly: the compiler contracts the product and the sum or not depending on
// the code around them, and every kernel must round a path's radiance alike.
__device__ __forceinline__ void add_light(Path& P, V e) {
    P.L = V{fmaf(P.beta.x, e.x, P.L.x), fmaf(P.beta.y, e.y, P.L.y), fmaf(P.beta.z, e.z, P.L.z)};
}

// Shading after the closest hit of segment j (ray_color, render.rs:1472-1537, iterative):
// L += B_j e_j now, B_{j+1} = B_j att_j rrw_j, the NEE term B_j d_j once its shadow ray is
// known to be unoccluded.  Returns the lane's next state.
// NEE = false builds the shading step of scenes without lights: no light-sampling code in the
// kernel (the megakernel runs ~11% faster on a light-free scene without it: instruction fetch).
template <int KIND = -1, bool EXT = true, bool NEE = true, bool SPH = false, int CLS = CLS_ALL>
__device__ __forceinline__ int shade(const SceneDev& S, const RenderDev& R, uint32_t pixel, Path& P, bool found,
                                     const Hit& h, Pending& pend, V* exit_stash = nullptr) {
    if (!found) {
        add_light(P, background<EXT>(S, R, P.ray));
        return ST_DONE;
    }
    const uint32_t depth = R.max_depth - P.bounce;
    Surface sf = surface_of<SPH, CLS>(S, P.ray, h);
    // A non-finite hit point (e.g. a fog hit at t = inf along a zero-length direction, where
    // the reference's distance test compares against NaN) makes this level's result NaN in
    // the reference, which its guard turns into zero for the level and everything deeper
    // (render.rs:1526-1531).  Ending the path here drops the same terms and keeps NaN rays
    // (whose slab tests pass every box) out of the traversal.
    if (!isfinite(sf.p.x) || !isfinite(sf.p.y) || !isfinite(sf.p.z)) return ST_DONE;
    const MatDev& m = S.mats[sf.mat];
    V e = P.skip_emission ? mk(0.f, 0.f, 0.f)
                          : (EXT && KIND < 0 ? emitted_at(S, sf.mat, m, sf.p) : emitted(m, sf.p));
    float4 su = draw4<philox_unroll<CLS, SPH>()>(R.key0, R.key1, pixel, P.stratum, P.bounce, CALL_SCATTER);
    Scatter sc;
    sc.org = sf.p;
    const MatDev& ms = EXT && KIND < 0 ? blend_leaf(S, m, R, pixel, P.stratum, P.bounce) : m;
    if (!scatter<KIND, EXT, SPH, philox_unroll<CLS, SPH>()>(ms, P.ray, sf, h.t, su, R, pixel, P.stratum, P.bounce, sc)) {
        add_light(P, e);
        return ST_DONE;
    }
    // A zero or non-finite scatter direction (in_unit_sphere at radius 0) would make the
    // next level NaN in the reference (its unit vectors divide by zero): end the path.
    const float dl2 = len2(sc.dir);
    if (!(dl2 > 0.0f) || !isfinite(dl2)) {
        add_light(P, e);
        return ST_DONE;
    }
    // the next segment (its origin and direction are dead past this point otherwise; a path
    // that ends below no longer reads its ray)
    P.ray.o = sc.org;
    P.ray.d = sc.dir;
    float4 nu = draw4<philox_unroll<CLS, SPH>()>(R.key0, R.key1, pixel, P.stratum, P.bounce, CALL_NEE);
    float surv = fminf(fmaxf(fmaxf(fmaxf(sc.att.x, sc.att.y), sc.att.z), 0.05f), 1.0f);
    if (depth < 47 && nu.x > surv) {                                   // Russian roulette
        add_light(P, e);
        return ST_DONE;
    }
    float rrw = depth < 47 ? 1.0f / surv : 1.0f;
    V nb = mul(P.beta, sc.att) * rrw;
    if (has_nan(e) || has_nan(nb)) return ST_DONE;                     // render.rs:1526-1531
    add_light(P, e);
    bool use_nee = NEE && !m.specular && S.n_lights > 0;
    bool shadow = false;
    if (use_nee) {
        Ray sr;
        V contrib;
        const bool lit = cls_is_mesh<CLS>() ? sample_light_cold<CLS>(S, sf.p, sf.n, sc.att, nu, sr, pend.tmax, contrib)
                                         : sample_light<CLS>(S, sf.p, sf.n, sc.att, nu, sr, pend.tmax, contrib);
        if (lit) {
            pend.dir = sr.d;
            pend.contrib = mul(P.beta, contrib);
            shadow = !has_nan(pend.contrib);
        }
    }
    P.beta = nb;
    P.skip_emission = use_nee;
    ++P.bounce;
    if constexpr (EXT) {
        if (shadow && (P.ray.o.x != sf.p.x || P.ray.o.y != sf.p.y || P.ray.o.z != sf.p.z)) {
            *exit_stash = P.ray.o;                     // Subsurface: the shadow starts at the hit point
            P.ray.o = sf.p;
            pend.tmax = -pend.tmax;
        }
    }
    if (shadow) return ST_SHADOW;
    return P.bounce >= R.max_depth ? ST_DONE : ST_CLOSEST;             // depth == 0 -> black
}

}  // namespace lum
