// Plain f64 form of the path integrator: each pixel's samples run in order on
// one lane, continuing the reference's per-pixel RNG stream (src/render.rs:
// 141-158) through radiance() (src/integrator.rs:53-135) with the
// reference's f64 arithmetic.  This translation unit is compiled with
// -fmad=false so a*b+c rounds twice, as in the reference; f64 division and
// sqrt are IEEE-rounded on the GPU.  Transcendentals come from CUDA's libm,
// whose last-bit results can differ from glibc's, so a pixel's stream can
// diverge from the reference's after such a difference flips a branch.
//
// What World::hit returns is defined by the f64 tests of its triangles and
// spheres; which boxes are looked at on the way is not.  So rays walk the
// FP32 forms' trees with FP32 box tests that err on the side of visiting
// (world_trace), and only the primitives that are left run the reference's
// f64 arithmetic.
#include "plain_f64.cuh"
#include "texel.hpp"

#include <algorithm>

namespace tpt {
namespace plain {

constexpr double kPi = 3.14159265358979323846264338327950288;
constexpr double kTau = 6.28318530717958647692528676655900577;
constexpr double kEps = 1e-4;     // RAY_EPSILON (src/constants.rs:4)
constexpr double kTMax = 1e30;    // RAY_T_MAX (src/constants.rs:7)
constexpr int kStack = 64;        // bvh.rs:255 fixed stack

struct V { double x, y, z; };
__device__ __forceinline__ V mk(double x, double y, double z) { return V{x, y, z}; }
__device__ __forceinline__ V ld(const double* p) { return V{p[0], p[1], p[2]}; }
__device__ __forceinline__ V operator+(V a, V b) { return V{a.x + b.x, a.y + b.y, a.z + b.z}; }
__device__ __forceinline__ V operator-(V a, V b) { return V{a.x - b.x, a.y - b.y, a.z - b.z}; }
__device__ __forceinline__ V operator-(V a) { return V{-a.x, -a.y, -a.z}; }
__device__ __forceinline__ V operator*(V a, double s) { return V{a.x * s, a.y * s, a.z * s}; }
__device__ __forceinline__ V operator*(double s, V a) { return a * s; }
__device__ __forceinline__ V operator/(V a, double s) { return V{a.x / s, a.y / s, a.z / s}; }
__device__ __forceinline__ V had(V a, V b) { return V{a.x * b.x, a.y * b.y, a.z * b.z}; }
__device__ __forceinline__ double dot(V a, V b) { return a.x * b.x + a.y * b.y + a.z * b.z; }
__device__ __forceinline__ V cross(V a, V b) { return V{a.y * b.z - a.z * b.y, a.z * b.x - a.x * b.z, a.x * b.y - a.y * b.x}; }
__device__ __forceinline__ double len(V a) { return sqrt(dot(a, a)); }
__device__ __forceinline__ V norm(V a) { double l = fmax(len(a), 1e-30); return a / l; }
__device__ __forceinline__ double lum(V c) { return 0.2126 * c.x + 0.7152 * c.y + 0.0722 * c.z; }
__device__ __forceinline__ V clamp_lum(V c, double m) {             // math.rs:42-49
    double l = lum(c);
    return (l > m && l > 0.0) ? c * (m / l) : c;
}
__device__ __forceinline__ V reflect(V v, V n) { return v - (2.0 * dot(v, n)) * n; }  // math.rs:193
__device__ __forceinline__ double clampd(double x, double a, double b) { return fmin(fmax(x, a), b); }

struct Ray { V o, d; double time; };
struct Hit { double t; V p, n; int mat; };

// ---- src/geometry.rs ------------------------------------------------------
__device__ bool box_hit(const double* bmin, const double* bmax, const Ray& r, V inv, double tmin, double tmax,
                        double* t_enter) {  // Aabb::hit_inv / hit_range_inv (:117-165)
    double t0 = (bmin[0] - r.o.x) * inv.x, t1 = (bmax[0] - r.o.x) * inv.x;
    tmin = fmax(tmin, fmin(t0, t1)); tmax = fmin(tmax, fmax(t0, t1));
    if (tmax <= tmin) return false;
    t0 = (bmin[1] - r.o.y) * inv.y; t1 = (bmax[1] - r.o.y) * inv.y;
    tmin = fmax(tmin, fmin(t0, t1)); tmax = fmin(tmax, fmax(t0, t1));
    if (tmax <= tmin) return false;
    t0 = (bmin[2] - r.o.z) * inv.z; t1 = (bmax[2] - r.o.z) * inv.z;
    tmin = fmax(tmin, fmin(t0, t1)); tmax = fmin(tmax, fmax(t0, t1));
    if (tmax <= tmin) return false;
    if (t_enter) *t_enter = tmin;
    return true;
}

// Triangle::hit (:236-273): the distance, and the edges its normal comes from.
__device__ __forceinline__ bool tri_test(const TriF64& tr, V o, V d, double time, double tmin, double tmax, double& th,
                                         V& e1, V& e2) {
    V v0 = ld(tr.v0) * (1.0 - time) + ld(tr.v0) * time;  // vertices_at (:212-218), static
    V v1 = ld(tr.v1) * (1.0 - time) + ld(tr.v1) * time;
    V v2 = ld(tr.v2) * (1.0 - time) + ld(tr.v2) * time;
    e1 = v1 - v0;
    e2 = v2 - v0;
    V pvec = cross(d, e2);
    double det = dot(e1, pvec);
    if (fabs(det) < 1e-10) return false;
    double inv_det = 1.0 / det;
    V tvec = o - v0;
    double u = dot(tvec, pvec) * inv_det;
    if (u < 0.0 || u > 1.0) return false;
    V qvec = cross(tvec, e1);
    double v = dot(d, qvec) * inv_det;
    if (v < 0.0 || u + v > 1.0) return false;
    th = dot(e2, qvec) * inv_det;
    return !(th < tmin || th > tmax);
}

// Sphere::hit (:174-195): the distance.
__device__ __forceinline__ bool sphere_test(V c, double rad, const Ray& r, double tmin, double tmax, double& t) {
    V oc = r.o - c;
    double a = dot(r.d, r.d);
    double b = dot(oc, r.d);
    double cc = dot(oc, oc) - rad * rad;
    double d = b * b - a * cc;
    if (d <= 0.0) return false;
    double sd = sqrt(d);
    t = (-b - sd) / a;
    if (t < tmin || t > tmax) {
        t = (-b + sd) / a;
        if (t < tmin || t > tmax) return false;
    }
    return true;
}

// ---- src/bvh.rs:248-351 ---------------------------------------------------
// Bvh::hit as the reference walks it: its own tree, box by box in f64.  Kept
// for what depends on the order of that walk (mesh_done below) and for trees
// deeper than its stack.  Returns the triangle (index in S.tris), -1 = none.
__device__ __noinline__ int bvh_hit(const NodeF64* nodes, const TriF64* tris, int* flags, V o, V d, double time,
                                    double tmin, double tmax, double* t_hit) {
    const Ray r{o, d, time};
    V inv = mk(1.0 / r.d.x, 1.0 / r.d.y, 1.0 / r.d.z);
    int stack[kStack];
    int sp = 0;
    stack[sp++] = 0;
    int best = -1;
    while (sp > 0) {
        const NodeF64& n = nodes[stack[--sp]];
        if (!box_hit(n.bmin, n.bmax, r, inv, tmin, tmax, nullptr)) continue;
        if (n.left == -1 && n.right == -1) {
            for (uint32_t k = n.start; k < n.start + n.count; ++k) {
                double th;
                V e1, e2;
                if (tri_test(tris[k], o, d, time, tmin, tmax, th, e1, e2)) { tmax = th; best = (int)k; }
            }
            continue;
        }
        int a_id = n.left, b_id = n.right;
        int push[2];
        int np = 0;
        if (a_id == -1) {
            if (b_id != -1) push[np++] = b_id;
        } else if (b_id == -1) {
            push[np++] = a_id;
        } else {
            double ta, tb;
            bool ha = box_hit(nodes[a_id].bmin, nodes[a_id].bmax, r, inv, tmin, tmax, &ta);
            bool hb = box_hit(nodes[b_id].bmin, nodes[b_id].bmax, r, inv, tmin, tmax, &tb);
            if (ha && hb) {
                if (ta <= tb) { push[np++] = b_id; push[np++] = a_id; }  // far then near
                else { push[np++] = a_id; push[np++] = b_id; }
            } else if (ha) {
                push[np++] = a_id;
            } else if (hb) {
                push[np++] = b_id;
            }
        }
        for (int k = 0; k < np; ++k) {
            if (sp < kStack) stack[sp++] = push[k];
            else raise_flag(flags, TPT_FLAG_STACK_OVERFLOW);
        }
    }
    *t_hit = tmax;
    return best;
}

__device__ V xf_point(const InstanceF64& x, V p) {          // apply_point (transform.rs:75-77)
    const double* a = x.a;
    return mk(a[0] * p.x + a[1] * p.y + a[2] * p.z, a[3] * p.x + a[4] * p.y + a[5] * p.z,
              a[6] * p.x + a[7] * p.y + a[8] * p.z) + ld(x.t);
}
__device__ V mat_vec(const double* a, V p) {
    return mk(a[0] * p.x + a[1] * p.y + a[2] * p.z, a[3] * p.x + a[4] * p.y + a[5] * p.z,
              a[6] * p.x + a[7] * p.y + a[8] * p.z);
}

// ---- World::hit (src/world.rs:81-121) ---------------------------------------
// The FP32 view of a ray for the box tests.  A slab distance (b - o) / d is
// formed as b * idir - o * idir; against the f64 value its error is at most
// a few ulps of the distance itself (the rounding of d, of its reciprocal
// and of the sum) plus the rounding of o and of o * idir, below |o| * 2^-22
// in world units.  The second part, and `pad` (world units), widen the box:
// the near planes' offset is lowered and the far planes' raised by that
// much; the first is covered by kSlack on the far distance.
constexpr float kSlack = 1.0f + 3e-6f;
struct Ray32 {
    float3 idir, near_off, far_off;
};
__device__ __forceinline__ float safe_rcp(float d) {  // within an ulp
    float r;
    asm("rcp.approx.f32 %0, %1;" : "=f"(r) : "f"(fabsf(d) > 1e-20f ? d : copysignf(1e-20f, d)));
    return r;
}
__device__ __forceinline__ void set_axis(double o, double d, float pad, float& idir, float& lo, float& hi) {
    const float of = (float)o;
    idir = safe_rcp((float)d);
    const float c = of * idir, m = (fabsf(of) * 2.4e-7f + pad) * fabsf(idir);
    lo = -c - m;
    hi = -c + m;
}
__device__ __forceinline__ Ray32 ray32(V o, V d, float pad) {
    Ray32 r;
    set_axis(o.x, d.x, pad, r.idir.x, r.near_off.x, r.far_off.x);
    set_axis(o.y, d.y, pad, r.idir.y, r.near_off.y, r.far_off.y);
    set_axis(o.z, d.z, pad, r.idir.z, r.near_off.z, r.far_off.z);
    return r;
}
// Entry distance of the widened box; *hit = false only when no point of the
// box lies on the ray below tmax (a NaN keeps the box).  That no f64 test in the
// box succeeds then rests on the hits lying in their boxes: a triangle's by its
// box's 1e-9 and the widening here, which a ray within about 1e-9 of the
// triangle's plane (det near its bound of 1e-10) may pass by at an edge.
__device__ __forceinline__ float box32(const Ray32& r, float x0, float x1, float y0, float y1, float z0, float z1,
                                       float tmax, bool* hit) {
    const bool sx = r.idir.x < 0.0f, sy = r.idir.y < 0.0f, sz = r.idir.z < 0.0f;
    const float nx = __fmaf_rn(sx ? x1 : x0, r.idir.x, r.near_off.x), fx = __fmaf_rn(sx ? x0 : x1, r.idir.x, r.far_off.x);
    const float ny = __fmaf_rn(sy ? y1 : y0, r.idir.y, r.near_off.y), fy = __fmaf_rn(sy ? y0 : y1, r.idir.y, r.far_off.y);
    const float nz = __fmaf_rn(sz ? z1 : z0, r.idir.z, r.near_off.z), fz = __fmaf_rn(sz ? z0 : z1, r.idir.z, r.far_off.z);
    const float n = fmaxf(fmaxf(nx, ny), fmaxf(nz, 0.0f));
    const float f = fminf(fminf(fx, fy), fminf(fz, tmax)) * kSlack;
    *hit = !(n > f);
    return n;
}

// The closest hit so far in the world.
struct Best {
    double t;        // world distance (the ray's tmax until something is hit)
    double th;       // instances: distance in the mesh's space
    int inst, prim;  // instance and triangle, or -1 and the sphere; prim -1 = nothing
};

// True when the walk of instance `inst` ends in the closest hit: its mesh
// hit taken to the world and compared as world.rs:92-108 does.
__device__ __forceinline__ bool mesh_done(const PlainScene& S, const Ray& r, V o, V d, int inst, int tri, double th,
                                          Best& best) {
    if (tri < 0) return false;
    const V p = xf_point(S.instances[inst], o + d * th);
    const double t_world = dot(p - r.o, r.d);
    // the reference tests instances in index order with a strict comparison
    // and spheres after them: of equal distances the lowest instance stays
    const bool closer = t_world < best.t || (t_world == best.t && best.inst > inst);
    if (!(t_world > kEps && closer)) return false;
    best = Best{t_world, th, inst, tri};
    return true;
}

// A ray that is not a number, beyond the range of the FP32 box tests or not of
// unit length.  (Shadow rays are none of these: a contribution is zero or
// stopped by its cosine where the hit they start from is not a number.)
__device__ __forceinline__ bool unusual(const Ray& r) {
    const float ox = (float)r.o.x, oy = (float)r.o.y, oz = (float)r.o.z;
    const float dx = (float)r.d.x, dy = (float)r.d.y, dz = (float)r.d.z;
    return !(fabsf(dx * dx + dy * dy + dz * dz - 1.0f) < 1e-6f && fabsf(ox + oy + oz) < 1e30f);
}
// World::hit by the reference's own loops, for unusual rays and for scenes with
// geometry out of range.  Every comparison of the reference's tests lets a NaN
// pass, so a NaN ray meets the last sphere and a NaN triangle stops the rays that
// come to its leaf; which ones these are only the order of its loops says.  And
// instances count at dot(p - o, d), spheres at their root: only for a unit
// direction does a box that starts past the one hold no closer other.
__device__ __noinline__ Best world_loops(const PlainScene& S, V ro, V rd, double time, double tmax, int* flags) {
    const Ray r{ro, rd, time};
    Best best{tmax, 0.0, -1, -1};
    for (int i = 0; i < S.n_instances; ++i) {
        const InstanceF64& I = S.instances[i];
        const MeshF64 m = S.meshes[I.mesh_id];
        if (m.n_nodes == 0) continue;
        const V o = mat_vec(I.a_inv, r.o - ld(I.t)), d = norm(mat_vec(I.a_inv, r.d));
        double th;
        const int tri = bvh_hit(S.nodes + m.node_offset, S.tris + m.tri_offset, flags, o, d, r.time, kEps, 1e30, &th);
        mesh_done(S, r, o, d, i, tri < 0 ? -1 : tri + m.tri_offset, th, best);
    }
    for (int i = 0; i < S.n_spheres; ++i) {
        double t;
        if (sphere_test(ld(S.spheres[i].c), S.spheres[i].r, r, kEps, best.t, t)) best = Best{t, 0.0, -1, i};
    }
    return best;
}

// World::hit in a scene of spheres alone: the reference's loop over them.
__device__ __forceinline__ bool spheres_hit(const PlainScene& S, const Ray& r, double tmax, bool any, Best& best) {
    best = Best{tmax, 0.0, -1, -1};
#pragma unroll 1
    for (int i = 0; i < S.n_spheres; ++i) {
        double t;
        if (!sphere_test(ld(S.spheres[i].c), S.spheres[i].r, r, kEps, best.t, t)) continue;
        best = Best{t, 0.0, -1, i};
        if (any) return true;
    }
    return best.prim >= 0;
}

constexpr int kLeaveMesh = ~0;  // stack entry: back to world space (no leaf of a tree has the code 0 / 0)

// World::hit over the top-level tree (spheres and instances) and the mesh
// trees of the FP32 forms.  Bound by the latency of dependent node loads in
// divergent lanes; against the reference's own tree and its linear sphere
// and instance loops in f64 it visits the same primitives' tests with an
// eighth of the f64 work (rates at k_paths below).
//
// Why the result is the reference's, whatever tree is walked:
//  * A primitive's f64 test decides alone whether and where it is hit; the
//    closest one wins.  Equal distances follow the reference's loop order:
//    instances by index, spheres after them, the last sphere.
//  * Bvh::hit reaches a triangle only through its leaf's box.  The f64 box
//    test is monotonic, so a leaf that passes has ancestors that pass; the
//    leaf's own test (box_hit on `leaf`) is therefore the whole condition,
//    and it is run for each triangle that is hit.
//  * What remains depends on the order of the reference's walk: two
//    triangles of one mesh hit at the same distance, or a leaf box entered
//    no earlier than the hit (the box might have been culled by an earlier
//    hit).  Then the mesh is walked again by bvh_hit.
__device__ __forceinline__ bool world_trace(const PlainScene& S, const Ray& r, double tmax, bool any, bool by_loops,
                                            Best& best, int* stack, int* flags) {
    if (by_loops) {
        best = world_loops(S, r.o, r.d, r.time, tmax, flags);
        return best.prim >= 0;
    }
    best = Best{tmax, 0.0, -1, -1};
    if (S.top_root == TPT_REF_NONE) return false;
    Ray32 q = ray32(r.o, r.d, S.top_pad);
    float far = __double2float_ru(tmax);
    V o = r.o, d = r.d;  // the ray in the entered mesh's space
    int inst = -1, tri = -1;
    bool redo = false;
    double th = 1e30;
    int ref = S.top_root, sp = 0;
    for (;;) {
        while (ref >= 0) {
            const float4* np = reinterpret_cast<const float4*>(S.nodes32 + ref);
            const float4 lx = __ldg(np), rx = __ldg(np + 1), zz = __ldg(np + 2);
            const int2 rf = __ldg(reinterpret_cast<const int2*>(np + 3));
            bool hl, hr;
            const float ln = box32(q, lx.x, lx.y, lx.z, lx.w, zz.x, zz.y, far, &hl);
            const float rn = box32(q, rx.x, rx.y, rx.z, rx.w, zz.z, zz.w, far, &hr);
            if (hl && hr) {
                const bool right = rn < ln;
                if (sp < kStack) stack[sp++] = right ? rf.x : rf.y;
                else raise_flag(flags, TPT_FLAG_STACK_OVERFLOW);
                ref = right ? rf.y : rf.x;
            } else if (hl || hr) {
                ref = hl ? rf.x : rf.y;
            } else {
                ref = sp > 0 ? stack[--sp] : TPT_REF_NONE;
            }
        }
        if (ref == TPT_REF_NONE) return best.prim >= 0;
        const uint32_t code = (uint32_t)(~ref), first = code >> 3, count = code & 7u;
        if (ref == kLeaveMesh) {
            if (redo) {
                const MeshF64 m = S.meshes[S.instances[inst].mesh_id];
                tri = bvh_hit(S.nodes + m.node_offset, S.tris + m.tri_offset, flags, o, d, r.time, kEps, 1e30, &th);
                if (tri >= 0) tri += m.tri_offset;
            }
            if (mesh_done(S, r, o, d, inst, tri, th, best) && any) return true;
            inst = -1;
            q = ray32(r.o, r.d, S.top_pad);
            far = __double2float_ru(best.t);
        } else if (count == 7u) {  // enter an instance's mesh
            const InstanceF64& I = S.instances[first];
            const int root = S.meshes32[I.mesh_id].root_ref;
            if (root != TPT_REF_NONE) {
                const V du = mat_vec(I.a_inv, r.d);
                o = mat_vec(I.a_inv, r.o - ld(I.t));
                d = norm(du);
                inst = (int)first;
                tri = -1;
                th = 1e30;
                redo = S.meshes[I.mesh_id].deep != 0;
                q = ray32(o, d, 0.0f);
                // hits past the closest one so far are not needed; one world
                // unit is |A^-1 d| units here (|d|^2 is within 1e-6 of 1), up to the rounding
                // of the two transforms
                const double reach = (best.t * (1.0 + 3e-6) + S.top_pad) * len(du);
                far = reach < 1e30 ? __double2float_ru(reach) : 1e30f;
                if (sp < kStack) stack[sp++] = kLeaveMesh;
                else raise_flag(flags, TPT_FLAG_STACK_OVERFLOW);
                if (!redo) {
                    ref = root;
                    continue;
                }
            }
        } else if (inst >= 0) {
#pragma unroll 1
            for (uint32_t k = first; k < first + count; ++k) {
                const int2 link = __ldg(S.links + k);
                double t;
                V e1, e2;
                if (!tri_test(S.tris[link.x], o, d, r.time, kEps, th, t, e1, e2)) continue;
                const NodeF64& leaf = S.nodes[link.y];
                const V inv = mk(1.0 / d.x, 1.0 / d.y, 1.0 / d.z);
                double enter;
                if (!box_hit(leaf.bmin, leaf.bmax, Ray{o, d, r.time}, inv, kEps, 1e30, &enter)) continue;
                redo = redo || !(enter < t) || (tri >= 0 && t == th);
                th = t;
                tri = link.x;
                far = fminf(far, __double2float_ru(t));
            }
        } else {
#pragma unroll 1
            for (uint32_t k = first; k < first + count; ++k) {
                const int id = __ldg(&S.spheres32[k].orig);
                const SphereF64& s = S.spheres[id];
                double t;
                if (!sphere_test(ld(s.c), s.r, r, kEps, best.t, t)) continue;
                // of equal distances the sphere tested last by the
                // reference's loop, and spheres over instances
                if (t == best.t && best.inst < 0 && best.prim > id) continue;
                best = Best{t, 0.0, -1, id};
                if (any) return true;
                far = __double2float_ru(t);
            }
        }
        ref = sp > 0 ? stack[--sp] : TPT_REF_NONE;
    }
}

// The closest hit's point, normal and material (geometry.rs:174-195, :236-273,
// world.rs:92-108).
__device__ __forceinline__ Hit hit_of(const PlainScene& S, const Ray& r, const Best& b) {
    if (b.inst < 0) {
        const SphereF64& s = S.spheres[b.prim];
        const V p = r.o + r.d * b.t;
        return Hit{b.t, p, (p - ld(s.c)) / s.r, s.mat};
    }
    const InstanceF64& I = S.instances[b.inst];
    const V o = mat_vec(I.a_inv, r.o - ld(I.t)), d = norm(mat_vec(I.a_inv, r.d));
    const TriF64& tr = S.tris[b.prim];
    const V v0 = ld(tr.v0) * (1.0 - r.time) + ld(tr.v0) * r.time;
    const V e1 = (ld(tr.v1) * (1.0 - r.time) + ld(tr.v1) * r.time) - v0;
    const V e2 = (ld(tr.v2) * (1.0 - r.time) + ld(tr.v2) * r.time) - v0;
    return Hit{b.t, xf_point(I, o + d * b.th), norm(mat_vec(I.nmat, norm(cross(e1, e2)))),
               I.mat_override >= 0 ? I.mat_override : tr.mat};
}

// ---- src/material.rs -------------------------------------------------------
__device__ __forceinline__ double pow5(double x) { double x2 = x * x; return x2 * x2 * x; }
__device__ V fresnel_schlick(double c, V f0) {
    double x = 1.0 - fmax(c, 0.0);
    return f0 + (mk(1.0, 1.0, 1.0) - f0) * pow5(x);
}
__device__ double ggx_d(double alpha, double ch) {
    if (ch <= 0.0) return 0.0;
    double a2 = alpha * alpha;
    double den = ch * ch * (a2 - 1.0) + 1.0;
    return a2 / (kPi * den * den);
}
__device__ double ggx_g1(double alpha, double c) {
    if (c <= 0.0) return 0.0;
    double a = alpha * sqrt(fmax(1.0 - c * c, 0.0)) / fmax(c, 1e-6);
    return 2.0 / (1.0 + sqrt(1.0 + a * a));
}
__device__ V ggx_eval(V albedo, double alpha, V n, V wo, V wi) {
    double ci = dot(n, wo), co = dot(n, wi);
    if (ci <= 0.0 || co <= 0.0) return mk(0, 0, 0);
    V m = norm(wo + wi);
    double ch = fmax(dot(n, m), 0.0);
    double d = ggx_d(alpha, ch);
    double g = ggx_g1(alpha, ci) * ggx_g1(alpha, co);
    V f = fresnel_schlick(fabs(dot(wi, m)), albedo);
    double den = 4.0 * ci * co + 1e-6;
    return f * (d * g / den);
}
__device__ double ggx_pdf(double alpha, V n, V wo, V wi) {
    double ci = dot(n, wo), co = dot(n, wi);
    if (ci <= 0.0 || co <= 0.0) return 0.0;
    V m = norm(wo + wi);
    double ch = fmax(dot(n, m), 0.0);
    double d = ggx_d(alpha, ch);
    double g1 = ggx_g1(alpha, ci);
    double pdf_m = d * g1 * ch / fmax(ci, 1e-6);
    double den = 4.0 * fmax(fabs(dot(wi, m)), 1e-6);
    return fmax(pdf_m / den, 0.0);
}
__device__ void tangent_frame(V n, V& t, V& b) {
    V a = fabs(n.x) > 0.9 ? mk(0, 1, 0) : mk(1, 0, 0);
    t = norm(cross(n, a));
    b = cross(t, n);
}
__device__ V cos_hemi(V n, uint64_t& rng) {
    double u = pcg_f64(rng);
    double v = pcg_f64(rng);
    double r = sqrt(u);
    double phi = 2.0 * kPi * v;
    double x = r * cos(phi), y = r * sin(phi), z = sqrt(1.0 - u);
    V t, b;
    tangent_frame(n, t, b);
    return t * x + b * y + n * z;
}
__device__ V vndf(V wo, double alpha, double u1, double u2) {
    V v = norm(mk(alpha * wo.x, alpha * wo.y, wo.z));
    V t1, t2;
    if (v.z < 0.9999) { t1 = norm(mk(-v.y, v.x, 0.0)); t2 = cross(v, t1); }
    else { t1 = mk(1, 0, 0); t2 = mk(0, 1, 0); }
    double r = sqrt(u1);
    double phi = kTau * u2;
    double t1p = r * cos(phi);
    double t2pi = r * sin(phi);
    double s = 0.5 * (1.0 + v.z);
    double t2p = sqrt(1.0 - s) * t2pi + s * sqrt(fmax(1.0 - t1p * t1p, 0.0));
    V nh = norm(t1 * t1p + t2 * t2p + v * sqrt(fmax(1.0 - t1p * t1p - t2p * t2p, 0.0)));
    return norm(mk(alpha * nh.x, alpha * nh.y, nh.z));
}

struct Bsdf { Ray ray; V w; double pdf; bool delta; };

__device__ bool mat_sample(const MaterialF64& m, const Ray& in, const Hit& h, uint64_t& rng, Bsdf& s) {  // :76-201
    bool entering = dot(h.n, in.d) < 0.0;
    V n = entering ? h.n : -h.n;
    V c = ld(m.c);
    switch (m.kind) {
        case TPT_MAT_LAMBERT: {
            V d = cos_hemi(n, rng);
            s = Bsdf{Ray{h.p + kEps * d, d, in.time}, c, fmax(dot(n, d), 0.0) / kPi, false};
            return true;
        }
        case TPT_MAT_METAL: {
            V d = reflect(in.d, n);
            s = Bsdf{Ray{h.p + kEps * d, d, in.time}, c, 0.0, true};
            return true;
        }
        case TPT_MAT_DIELECTRIC: {
            double ior = m.p;
            double eta = entering ? 1.0 / ior : ior;
            double ci = fmax(dot(-in.d, n), 0.0);
            double fq = (ior - 1.0) / (ior + 1.0);
            double f0 = fq * fq;
            double fr = f0 + (1.0 - f0) * pow5(1.0 - ci);
            V beta = mk(1, 1, 1);
            if (!entering) {
                double dist = fmax(h.t, 0.0);
                beta = had(beta, mk(exp(-c.x * dist), exp(-c.y * dist), exp(-c.z * dist)));
            }
            V refl = reflect(in.d, n);
            // refract (math.rs:199-207)
            double cosi = fmin(fmax(dot(-in.d, n), -1.0), 1.0);
            double sin2t = eta * eta * (1.0 - cosi * cosi);
            bool has_refr = !(sin2t >= 1.0);
            V refr = mk(0, 0, 0);
            if (has_refr) {
                double cost = sqrt(1.0 - sin2t);
                refr = eta * in.d + (eta * cosi - cost) * n;
            }
            bool choose_refl = !has_refr || pcg_f64(rng) < fr;
            V d;
            if (choose_refl) {
                beta = beta * (fr / fmax(fr, 1e-6));
                d = refl;
            } else {
                double sc = (1.0 - fr) / fmax(1.0 - fr, 1e-6);
                beta = beta * sc * (eta * eta);
                d = refr;
            }
            s = Bsdf{Ray{h.p + kEps * d, d, in.time}, beta, 0.0, true};
            return true;
        }
        case TPT_MAT_GGX: {
            double av = fmax(m.p, 1e-3);
            V t, b;
            tangent_frame(n, t, b);
            V wo = norm(-in.d);
            V wl = mk(dot(wo, t), dot(wo, b), dot(wo, n));
            if (wl.z <= 0.0) return false;
            double u1 = pcg_f64(rng);
            double u2 = pcg_f64(rng);
            V ml = vndf(wl, av, u1, u2);
            V mh = t * ml.x + b * ml.y + n * ml.z;
            V d = reflect(in.d, mh);
            double co = dot(d, n);
            double ci = dot(-in.d, n);
            if (co <= 1e-6 || ci <= 1e-6) return false;
            double ch = fmax(dot(n, mh), 0.0);
            double dg = ggx_d(av, ch);
            double g = ggx_g1(av, ci) * ggx_g1(av, co);
            V f = fresnel_schlick(fabs(dot(d, mh)), c);
            double den = 4.0 * ci * co + 1e-6;
            V spec = f * (dg * g / den);
            double pdf = ggx_pdf(av, n, wo, d);
            s = Bsdf{Ray{h.p + kEps * d, d, in.time}, spec * (co / fmax(pdf, 1e-6)), pdf, false};
            return true;
        }
        case TPT_MAT_SUBSURFACE: {
            double sc = fmax(m.p, 1e-4);
            double u = fmax(pcg_f64(rng), 1e-12);
            double dist = -log(u) * sc;
            V no = h.n;
            V d = cos_hemi(no, rng);
            V att = c * exp(-dist / sc);
            V o = h.p - no * dist + kEps * d;
            s = Bsdf{Ray{o, d, in.time}, att, fmax(dot(n, d), 0.0) / kPi, false};
            return true;
        }
        default:
            return false;
    }
}

__device__ void mat_eval(const MaterialF64& m, V wo, V wi, V n, V& f, double& pdf) {  // :207-223
    if (m.kind == TPT_MAT_LAMBERT || m.kind == TPT_MAT_SUBSURFACE) {
        double c = fmax(dot(n, wi), 0.0);
        if (c <= 0.0) { f = mk(0, 0, 0); pdf = 0.0; return; }
        f = ld(m.c) * (1.0 / kPi);
        pdf = c / kPi;
        return;
    }
    if (m.kind == TPT_MAT_GGX) {
        double a = fmax(m.p, 1e-3);
        f = ggx_eval(ld(m.c), a, n, wo, wi);
        pdf = ggx_pdf(a, n, wo, wi);
        return;
    }
    f = mk(0, 0, 0);
    pdf = 0.0;
}

// ---- src/env.rs ------------------------------------------------------------
// EnvMap::lookup (:92-121) and, when asked for, the density of the same
// direction (:156-182; both take the same u, v).
__device__ __forceinline__ V env_at(const PlainScene& S, V dir, bool want_pdf, double& pdf) {
    V d = norm(dir);
    double theta = acos(clampd(d.y, -1.0, 1.0));
    double phi = atan2(d.z, d.x);
    if (phi < 0.0) phi += kTau;
    double u = phi / kTau, v = theta / kPi;
    const int W = S.env_w, H = S.env_h;
    double x = u * (double)W;
    double y = v * ((double)H - 1.0);
    int x0 = texel_index(x, W);       // 0 <= u <= 1 or NaN, so x0 % W needs one step
    if (x0 >= W) x0 -= W;
    const int x1 = x0 + 1 < W ? x0 + 1 : 0;
    const int y0 = texel_index(y, H - 1);
    const int y1 = y0 + 1 < H - 1 ? y0 + 1 : H - 1;
    double fx = x - floor(x), fy = y - floor(y);
    const double* D = S.env_data;
    const size_t r0 = (size_t)y0 * W, r1 = (size_t)y1 * W;
    V c00 = ld(D + 3 * (r0 + x0)), c10 = ld(D + 3 * (r0 + x1));
    V c01 = ld(D + 3 * (r1 + x0)), c11 = ld(D + 3 * (r1 + x1));
    V c0 = c00 * (1.0 - fx) + c10 * fx;
    V c1 = c01 * (1.0 - fx) + c11 * fx;
    if (want_pdf) {
        pdf = 1.0 / (4.0 * kPi);
        if (S.env_total > 0.0) {
            const int px = texel_index(u * (double)W, W - 1), py = texel_index(v * (double)H, H - 1);
            double th0 = kPi * (double)py / (double)H, th1 = kPi * (double)(py + 1) / (double)H;
            double st = fmax(sin(theta), 1e-6);
            double rw = fmax(cos(th0) - cos(th1), 0.0);
            double l = fmax(lum(ld(D + 3 * ((size_t)py * W + px))), 0.0);
            double wgt = l * rw;
            pdf = 0.0;
            if (wgt > 0.0) {
                double pdf_uv = (wgt / S.env_total) * (double)W * (double)H;
                pdf = pdf_uv / (2.0 * kPi * kPi * st);
            }
        }
    }
    return c0 * (1.0 - fy) + c1 * fy;
}
// env.rs:185-197, world.rs:324-336.  guide, when given, holds the answers at
// the edges of k equal buckets of the variate u that x is a multiple of: the
// answer for x lies between those of u's bucket.
__device__ size_t cdf_search(const double* cdf, size_t n, double x, const uint16_t* guide = nullptr, int k = 0,
                             double u = 0.0) {
    size_t lo = 0, hi = n == 0 ? 0 : n - 1;
    if (guide) {
        const int b = (int)(u * (double)k);  // u in [0, 1), k a power of two: exact
        lo = guide[b];
        const size_t above = (size_t)guide[b + 1] + 1;
        if (above < hi) hi = above;
    }
#pragma unroll 1
    while (lo + 1 < hi) {
        size_t mid = (lo + hi) / 2;
        if (cdf[mid] <= x) lo = mid; else hi = mid;
    }
    return lo;
}
// EnvMap::sample_dir (:124-152): the direction.  False when it was drawn
// uniformly (:200-210), whose density is 1 / 4 pi.
__device__ bool env_sample_dir(const PlainScene& S, uint64_t& rng, V& dir) {
    const size_t W = (size_t)S.env_w, H = (size_t)S.env_h;
    if (S.env_total > 0.0) {
        const double u0 = pcg_f64(rng), r0 = u0 * S.env_total;
        size_t y = cdf_search(S.env_row_cdf, H + 1, r0, S.env_row_guide, S.env_row_k, u0);
        if (y > H - 1) y = H - 1;
        double row_sum = fmax(S.env_row_cdf[y + 1] - S.env_row_cdf[y], 0.0);
        if (row_sum > 0.0) {
            const double u1 = pcg_f64(rng), r1 = u1 * row_sum;
            const uint16_t* guide = S.env_col_guide ? S.env_col_guide + y * (size_t)(S.env_col_k + 1) : nullptr;
            size_t x = cdf_search(S.env_col_cdf + y * (W + 1), W + 1, r1, guide, S.env_col_k, u1);
            if (x > W - 1) x = W - 1;
            double u = ((double)x + pcg_f64(rng)) / (double)W;
            double v = ((double)y + pcg_f64(rng)) / (double)H;
            double theta = kPi * v, phi = kTau * u;
            double st = sin(theta);
            dir = mk(cos(phi) * st, cos(theta), sin(phi) * st);
            return true;
        }
    }
    double u = pcg_f64(rng), v = pcg_f64(rng);
    double z = 1.0 - 2.0 * u;
    double r = sqrt(fmax(1.0 - z * z, 0.0));
    double phi = kTau * v;
    dir = mk(r * cos(phi), z, r * sin(phi));
    return false;
}

// ---- src/world.rs:171-272 --------------------------------------------------
__device__ bool sample_light(const PlainScene& S, uint64_t& rng, double time, V p, V& pos, V& nrm, V& emit,
                             double& pdf) {
    if (S.light_total <= 0.0 || S.n_lights == 0) return false;
    double r = pcg_f64(rng) * S.light_total;
    size_t idx = cdf_search(S.light_cdf, (size_t)S.n_lights, r);
    if (idx > (size_t)S.n_lights - 1) idx = (size_t)S.n_lights - 1;
    const LightF64& L = S.lights[idx];
    double pdf_sel = L.weight / S.light_total;
    double area;
    if (L.is_sphere) {
        const SphereF64& s = S.spheres[L.sphere];
        double u = pcg_f64(rng), v = pcg_f64(rng);
        double z = 1.0 - 2.0 * u;
        double rr = sqrt(fmax(1.0 - z * z, 0.0));
        double phi = kTau * v;
        V dir = mk(rr * cos(phi), z, rr * sin(phi));
        pos = ld(s.c) + dir * s.r;
        nrm = dir;
        area = 4.0 * kPi * s.r * s.r;
    } else {
        const InstanceF64& inst = S.instances[L.inst];
        V w0 = xf_point(inst, ld(L.v) * (1.0 - time) + ld(L.v) * time);
        V w1 = xf_point(inst, ld(L.v + 3) * (1.0 - time) + ld(L.v + 3) * time);
        V w2 = xf_point(inst, ld(L.v + 6) * (1.0 - time) + ld(L.v + 6) * time);
        double u = pcg_f64(rng), v = pcg_f64(rng);
        double su = sqrt(u);
        double b0 = 1.0 - su, b1 = v * su, b2 = 1.0 - b0 - b1;
        pos = w0 * b0 + w1 * b1 + w2 * b2;
        V nn = cross(w1 - w0, w2 - w0);
        area = 0.5 * len(nn);
        nrm = area > 0.0 ? nn / (2.0 * area) : mk(0.0, 1.0, 0.0);
    }
    if (area <= 0.0) return false;
    V tl = pos - p;
    double d2 = dot(tl, tl);
    if (d2 <= 1e-12) return false;
    double dist = sqrt(d2);
    V wi = tl / dist;
    double cl = fmax(dot(nrm, -wi), 0.0);
    if (cl <= 0.0) return false;
    double pdf_area = 1.0 / area;
    double pdf_omega = pdf_area * d2 / cl;
    pdf = pdf_sel * pdf_omega;
    if (pdf <= 0.0) return false;
    emit = ld(L.emit);
    return true;
}

// ---- src/integrator.rs -----------------------------------------------------
__device__ __forceinline__ V sky(V d) {  // :25-28
    double t = 0.5 * (d.y + 1.0);
    return (1.0 - t) * mk(0.9, 0.95, 1.0) + t * mk(0.6, 0.75, 1.0);
}
__device__ __forceinline__ double mis(double a, double b) {
    double a2 = a * a, b2 = b * b;
    return (a2 + b2 > 0.0) ? a2 / (a2 + b2) : 0.0;
}

__device__ Ray camera_ray(const CameraF64& c, double sx, double sy, uint64_t& rng) {  // ray.rs:91-108
    V u = ld(c.u), v = ld(c.v), w = ld(c.w), o = ld(c.o);
    V dir_base = norm(((-w) + (sx * c.half_w) * u) + (sy * c.half_h) * v);
    V lens = mk(0, 0, 0);
    if (c.lens_radius > 0.0) {
        double dx = 0.0, dy = 0.0;
        // sample_unit_disk (:112-120); the acceptance rate is pi/4, so the
        // 256-try bound is never reached in practice ((1-pi/4)^256 ~ 1e-171).
#pragma unroll 1
        for (int k = 0; k < 256; ++k) {
            dx = 2.0 * pcg_f64(rng) - 1.0;
            dy = 2.0 * pcg_f64(rng) - 1.0;
            if (dx * dx + dy * dy < 1.0) break;
        }
        lens = u * (dx * c.lens_radius) + v * (dy * c.lens_radius);
    }
    V origin = o + lens;
    V focus = o + dir_base * c.focus_dist;
    V dir = norm(focus - origin);
    double time = c.shutter_open + (c.shutter_close - c.shutter_open) * pcg_f64(rng);
    return Ray{origin, dir, time};
}

// Pixels are handed out by tiles of 32, a warp's worth each: 8 x 4, and where
// the film is thinner than that 32 x 1 or 1 x 32.  A film of 2^30 pixels, the
// largest, then has fewer than 3.1e9 ids, so that 32 bits hold them and what the
// last lanes take in vain (64-bit ids cost 2 to 3% of a small scene's render).
struct Tiles {
    int log_w;
    unsigned across, n_ids;
};
__host__ __device__ __forceinline__ Tiles tiles_of(const PlainParams& P) {
    const int log_w = P.n_rows < 4 ? 5 : (P.width < 8 ? 0 : 3);
    const unsigned w = 1u << log_w, h = 32u >> log_w;
    const unsigned across = ((unsigned)P.width + w - 1u) / w;
    return Tiles{log_w, across, across * (((unsigned)P.n_rows + h - 1u) / h) * 32u};
}

// A pixel's sums (src/render.rs:158-191).
struct Sums {
    V c, c2;
    double mean, m2;
    int n;
};
// Adds a sample; true when it was the pixel's last.
__device__ __forceinline__ bool add_sample(const PlainParams& P, Sums& s, V L) {
    s.c = s.c + L;
    s.c2 = s.c2 + had(L, L);
    s.n += 1;
    bool stop = s.n >= P.spp;
    if (P.adaptive) {  // render.rs:160-176
        const int min_spp = min(P.adaptive_min_spp > 1 ? P.adaptive_min_spp : 1, P.spp > 1 ? P.spp : 1);
        double l = lum(L);
        double delta = l - s.mean;
        s.mean += delta / (double)s.n;
        double delta2 = l - s.mean;
        s.m2 += delta * delta2;
        if (s.n >= min_spp) {
            double var = s.n > 1 ? s.m2 / (double)(s.n - 1) : __longlong_as_double(0x7ff0000000000000ll);
            double den = fmax(fabs(s.mean), 1e-4);
            if (sqrt(var) / den < P.adaptive_threshold) stop = true;
        }
    }
    return stop;
}
__device__ __forceinline__ void store_pixel(const PlainParams& P, int x, int row, const Sums& s, double* acc, double* acc_w,
                                            double* acc_sq) {
    const size_t gi = (size_t)row * (size_t)P.width + (size_t)x;
    acc[3 * gi] = s.c.x; acc[3 * gi + 1] = s.c.y; acc[3 * gi + 2] = s.c.z;
    acc_w[gi] = (double)s.n;
    if (acc_sq) { acc_sq[3 * gi] = s.c2.x; acc_sq[3 * gi + 1] = s.c2.y; acc_sq[3 * gi + 2] = s.c2.z; }
}
__device__ __forceinline__ Ray sample_ray(const PlainScene& S, const PlainParams& P, int x, int row, double inv_w,
                                          double inv_h, uint64_t& rng) {  // src/render.rs:151-158
    const int y = P.row_begin + row * P.row_step;
    double jx = pcg_f64(rng);
    double jy = pcg_f64(rng);
    double sx = ((double)x + jx) * inv_w * 2.0 - 1.0;
    double sy = 1.0 - ((double)y + jy) * inv_h * 2.0;
    return camera_ray(S.cam, sx, sy, rng);
}
// Pixel `id` of the film in the order of its tiles; false past the film's edge.
__device__ __forceinline__ bool tile_pixel(const Tiles& T, const PlainParams& P, unsigned id, int& x, int& row) {
    const unsigned tile = id >> 5, in = id & 31u, ty = tile / T.across;
    x = (int)(((tile - ty * T.across) << T.log_w) + (in & ((1u << T.log_w) - 1u)));
    row = (int)((ty << (5 - T.log_w)) + (in >> T.log_w));
    return x < P.width && row < P.n_rows;
}
__device__ __forceinline__ void count_rays(unsigned long long* counters, unsigned long long n_samples,
                                           unsigned long long n_closest, unsigned long long n_shadow) {
    for (int off = 16; off > 0; off >>= 1) {
        n_samples += __shfl_down_sync(0xffffffffu, n_samples, off);
        n_closest += __shfl_down_sync(0xffffffffu, n_closest, off);
        n_shadow += __shfl_down_sync(0xffffffffu, n_shadow, off);
    }
    if ((threadIdx.x & 31u) == 0) {
        atomicAdd(&counters[0], n_samples);
        atomicAdd(&counters[1], n_closest);
        atomicAdd(&counters[2], n_shadow);
    }
}

// What a path waits for before its next bounce.
constexpr int kJobEnv = 1, kJobArea = 2, kJobClosest = 4;

// Every lane runs one pixel's samples, bounce by bounce; a lane whose pixel is
// finished takes the next one.  A round of the block is: shade what the last
// closest-hit rays met (radiance(), src/integrator.rs:53-135, one bounce),
// finish samples and start new ones, then trace -- first the NEE shadow rays
// of the bounce, then its next ray -- until no lane of the warp waits for a
// ray.  The contributions of the shadow rays are formed before the trace and
// added after it, in the reference's order, so a round has one copy of the
// walk and one of the shading code.
//
// Bound by instruction fetch, then by the latency of each pixel's chain of
// bounces (its samples share one stream): the f64 code is some 190 KB, a warp
// alone waits for nearly every line of it ("no instruction" 18 of 23 cycles
// per issue), and no SM has work for more than a few warps at 65,536 pixels.
// Barriers between the stages keep the block's warps on the same lines.
// Measured on one B200, sphere scene 256x256 x 64 spp / mesh scene (327,680
// triangles, 200 spheres, env map) 480x270 x 32 spp, ms: one thread per pixel
// over the reference's tree and linear loops 43.7 / 115; this kernel without
// barriers 21.0 / 17.3; with them 8.5 / 16.2 in blocks of 256, one per SM,
// and 11.8 / 13.8 in blocks of 128, two per SM.  At 128 registers (512 lanes
// per SM) 10.6 / 18.4.  `lanes` lanes of each warp take pixels.  SHORT: samples
// end in the round of their last shadow rays.
template <int BLOCK, int CTAS, bool SHORT>
__global__ void __launch_bounds__(BLOCK, CTAS) k_paths(const __grid_constant__ PlainScene S,
                                                     const __grid_constant__ PlainParams P, double* __restrict__ acc,
                                                     double* __restrict__ acc_w, double* __restrict__ acc_sq,
                                                     unsigned long long* __restrict__ counters, int* flags,
                                                     unsigned lanes) {
    const unsigned lane = threadIdx.x & 31u;
    const bool has_env = S.env_kind == TPT_ENV_MAP;
    const double inv_w = 1.0 / (double)P.width, inv_h = 1.0 / (double)P.height;
    const Tiles T = tiles_of(P);
    int stack[kStack];
    unsigned long long n_samples = 0, n_closest = 0, n_shadow = 0;
    // the pixel
    int x = -1, row = 0;
    uint64_t rng = 0;
    Sums sums{};
    bool exhausted = lane >= lanes;
    // the path
    Ray ray{};
    V L = mk(0, 0, 0), beta = mk(1, 1, 1);
    double last_pdf = 0.0;
    int bounce = 0, jobs = 0;
    bool last_nd = false, ended = false, found = false, odd = false;
    Best best{};
    // shadow rays: direction, contribution when nothing is in the way
    V sh_p = mk(0, 0, 0), env_wi = mk(0, 0, 0), env_c = mk(0, 0, 0), area_wi = mk(0, 0, 0), area_c = mk(0, 0, 0);
    double area_t = 0.0;
    // where a path has ended, its sample ends and the next one starts
    auto next_sample = [&] {
        bool start = false;
        if (x >= 0 && ended && jobs == 0) {  // the sample is complete (src/render.rs:158-191)
            const bool stop = add_sample(P, sums, L);
            if (stop) {
                store_pixel(P, x, row, sums, acc, acc_w, acc_sq);
                n_samples += (unsigned long long)sums.n;
                x = -1;
            }
            start = !stop;
        }
        const bool want = x < 0 && !exhausted;
        const unsigned wm = __ballot_sync(0xffffffffu, want);
        if (wm) {
            unsigned base = 0;
            const int leader = __ffs(wm) - 1;
            if ((int)lane == leader) base = (unsigned)atomicAdd(&counters[3], (unsigned long long)__popc(wm));
            base = __shfl_sync(0xffffffffu, base, leader);
            if (want) {
                const unsigned id = base + __popc(wm & ((1u << lane) - 1u));
                exhausted = id >= T.n_ids;
                int px, py;
                if (!exhausted && tile_pixel(T, P, id, px, py)) {
                    x = px;
                    row = py;
                    sums = Sums{};
                    rng = pixel_seed((uint32_t)x, (uint32_t)(P.row_begin + row * P.row_step), P.seed);
                    start = true;
                }
            }
        }
        if (start) {
            ray = sample_ray(S, P, x, row, inv_w, inv_h, rng);
            L = mk(0, 0, 0);
            beta = mk(1, 1, 1);
            last_pdf = 0.0;
            last_nd = false;
            bounce = 0;
            ended = P.max_bounces <= 0;
            if (!ended) jobs = kJobClosest;
            odd = unusual(ray);
        }
    };
    auto trace = [&](int due) {
        while (__any_sync(0xffffffffu, (jobs & due) != 0)) {
            if ((jobs & due) != 0) {
                const int job = jobs & -jobs;
                Ray r = ray;
                double tmax = kTMax;
                if (job != kJobClosest) {
                    const V wi = job == kJobEnv ? env_wi : area_wi;
                    r = Ray{sh_p + kEps * wi, wi, ray.time};
                    if (job == kJobArea) tmax = area_t;
                }
                Best b;
                const bool h = world_trace(S, r, tmax, job != kJobClosest, S.by_loops || (job == kJobClosest && odd), b, stack, flags);
                if (job == kJobClosest) {
                    best = b;
                    found = h;
                    ++n_closest;
                } else if (!h) {
                    L = L + (job == kJobEnv ? env_c : area_c);
                }
                jobs ^= job;
            }
        }
    };
    for (;;) {
        __syncthreads();
        const bool shade = x >= 0 && !ended;
        V dir = ray.d, nrm = mk(0, 0, 0);
        bool surface = false, want_pdf = last_nd;
        Hit hit{};
        int kind = -1;
        if (shade && found) {
            hit = hit_of(S, ray, best);
            if (bounce >= P.rr_start) {
                double p = fmax(fmin(fmax(fmax(beta.x, beta.y), beta.z), 0.95), 0.05);
                if (pcg_f64(rng) > p) ended = true;
                else beta = beta / p;
            }
            if (!ended) {
                kind = S.mats[hit.mat].kind;
                if (kind == TPT_MAT_DIFFUSE_LIGHT) {
                    L = L + clamp_lum(had(beta, ld(S.mats[hit.mat].c)), 50.0);
                    ended = true;
                } else {
                    surface = true;
                    nrm = dot(hit.n, ray.d) < 0.0 ? hit.n : -hit.n;
                    sh_p = hit.p;
                }
            }
        }
        const bool nee = surface && kind != TPT_MAT_METAL && kind != TPT_MAT_DIELECTRIC;
        __syncthreads();
        if (nee && has_env) want_pdf = env_sample_dir(S, rng, dir);
        V bg = mk(0, 0, 0);
        double pe = 1.0 / (4.0 * kPi);
        __syncthreads();
        // (a black map adds 0 whatever the direction, unless the weight overflows)
        const bool dark = S.env_black && fabs(beta.x) + fabs(beta.y) + fabs(beta.z) < kTMax;
        if (has_env && !dark && shade && (!found || nee)) bg = env_at(S, dir, want_pdf, pe);
        __syncthreads();
        if (shade && !found) {  // miss
            if (!has_env) bg = sky(ray.d);
            V contrib = had(beta, bg);
            if (has_env && last_nd) contrib = contrib * mis(last_pdf, pe);
            L = L + clamp_lum(contrib, 50.0);
            ended = true;
        }
        bool area = false;
        double ca = 0.0, lpdf = 1.0;
        V le = mk(0, 0, 0);
        if (nee) {
            V lp, ln;
            if (sample_light(S, rng, ray.time, hit.p, lp, ln, le, lpdf)) {  // nee_area_light (:178-213)
                V tl = lp - hit.p;
                double d2 = dot(tl, tl);
                double dist = sqrt(d2);
                if (dist > 1e-6) {
                    area_wi = tl / dist;
                    ca = fmax(dot(nrm, area_wi), 0.0);
                    area = ca > 0.0;
                    area_t = fmax(dist - kEps, kEps);
                }
            }
        }
        __syncthreads();
        if (nee) {
            // nee_environment (:148-172), then nee_area_light: one BSDF
            // evaluation each.  A contribution of exactly zero adds nothing,
            // whatever its shadow ray meets.
            const MaterialF64& mat = S.mats[hit.mat];
            const V wo = norm(-ray.d);
            const double ce = has_env ? fmax(dot(nrm, dir), 0.0) : 0.0;
#pragma unroll 1
            for (int k = 0; k < 2; ++k) {
                if (!(k == 0 ? ce > 0.0 && pe > 0.0 : area)) continue;
                const V wi = k == 0 ? dir : area_wi, li = k == 0 ? bg : le;
                const double cs = k == 0 ? ce : ca, pl = k == 0 ? pe : lpdf;
                ++n_shadow;
                if (k == 0 && dark) continue;
                V f;
                double pb;
                mat_eval(mat, wo, wi, nrm, f, pb);
                const V contrib = had(had(beta, f), li) * (cs * mis(pl, pb) / pl);
                if (contrib.x == 0.0 && contrib.y == 0.0 && contrib.z == 0.0) continue;
                if (k == 0) { env_wi = wi; env_c = contrib; jobs |= kJobEnv; }
                else { area_c = contrib; jobs |= kJobArea; }
            }
        }
        __syncthreads();
        if (surface) {
            Bsdf s;
            if (!mat_sample(S.mats[hit.mat], ray, hit, rng, s)) {
                ended = true;
            } else {
                last_pdf = s.pdf;
                last_nd = !s.delta;
                beta = had(beta, s.w);
                ray = s.ray;
                if (++bounce >= P.max_bounces) ended = true;
                else jobs |= kJobClosest;
                odd = unusual(ray);
            }
        }
        __syncthreads();
        if constexpr (SHORT) {
            trace(kJobEnv | kJobArea);
            __syncthreads();
        }
        next_sample();
        if (!__syncthreads_or(x >= 0 || !exhausted)) break;
        trace(kJobEnv | kJobArea | kJobClosest);
    }
    count_rays(counters, n_samples, n_closest, n_shadow);
}

// Scenes of spheres alone (launch_plain): a lane per pixel runs its samples, and
// each sample's path, to the end.  Bound by f64 latency at 12 warps per SM.  The
// loop over the spheres is the same for every lane and the code without trees
// short, so that k_paths' steps only add to each sample's chain: built-in scene
// 1280x720 x 4 spp 2.75 ms in k_paths, 2.27 here, at one bounce 1.15 and 0.49, empty
// scene 960x540 x 16 spp 0.55 and 0.24.
__global__ void __launch_bounds__(128, 3) k_pixels(const __grid_constant__ PlainScene S,
                                                       const __grid_constant__ PlainParams P, double* __restrict__ acc,
                                                       double* __restrict__ acc_w, double* __restrict__ acc_sq,
                                                       unsigned long long* __restrict__ counters, int* flags) {
    const Tiles T = tiles_of(P);
    const unsigned id = blockIdx.x * 128u + threadIdx.x;
    const bool has_env = S.env_kind == TPT_ENV_MAP;
    const double inv_w = 1.0 / (double)P.width, inv_h = 1.0 / (double)P.height;
    int x = 0, row = 0;
    unsigned long long n_samples = 0, n_closest = 0, n_shadow = 0;
    if (id < T.n_ids && tile_pixel(T, P, id, x, row)) {
        uint64_t rng = pixel_seed((uint32_t)x, (uint32_t)(P.row_begin + row * P.row_step), P.seed);
        Sums sums{};
        V L;
        do {
            Ray ray = sample_ray(S, P, x, row, inv_w, inv_h, rng);
            V beta = mk(1, 1, 1);
            double last_pdf = 0.0;
            bool last_nd = false;
            L = mk(0, 0, 0);
#pragma unroll 1
            for (int bounce = 0; bounce < P.max_bounces; ++bounce) {
                ++n_closest;
                Best best;
                if (!spheres_hit(S, ray, kTMax, false, best)) {
                    double pe = 1.0 / (4.0 * kPi);
                    V contrib = had(beta, has_env ? env_at(S, ray.d, last_nd, pe) : sky(ray.d));
                    if (has_env && last_nd) contrib = contrib * mis(last_pdf, pe);
                    L = L + clamp_lum(contrib, 50.0);
                    break;
                }
                if (bounce >= P.rr_start) {
                    const double p = fmax(fmin(fmax(fmax(beta.x, beta.y), beta.z), 0.95), 0.05);
                    if (pcg_f64(rng) > p) break;
                    beta = beta / p;
                }
                const Hit hit = hit_of(S, ray, best);
                const MaterialF64& mat = S.mats[hit.mat];
                if (mat.kind == TPT_MAT_DIFFUSE_LIGHT) {
                    L = L + clamp_lum(had(beta, ld(mat.c)), 50.0);
                    break;
                }
                if (mat.kind != TPT_MAT_METAL && mat.kind != TPT_MAT_DIELECTRIC) {
                    const V nrm = dot(hit.n, ray.d) < 0.0 ? hit.n : -hit.n, wo = norm(-ray.d);
                    // nee_environment (:148-172), then nee_area_light (:178-213)
#pragma unroll 1
                    for (int k = has_env ? 0 : 1; k < 2; ++k) {
                        V wi, li;
                        double pl, tmax = kTMax;
                        if (k == 0) {
                            const bool by_cdf = env_sample_dir(S, rng, wi);
                            pl = 1.0 / (4.0 * kPi);
                            li = env_at(S, wi, by_cdf, pl);
                        } else {
                            V lp, ln;
                            if (!sample_light(S, rng, ray.time, hit.p, lp, ln, li, pl)) continue;
                            const V tl = lp - hit.p;
                            const double dist = sqrt(dot(tl, tl));
                            if (!(dist > 1e-6)) continue;
                            wi = tl / dist;
                            tmax = fmax(dist - kEps, kEps);
                        }
                        const double cs = fmax(dot(nrm, wi), 0.0);
                        if (!(cs > 0.0) || (k == 0 && !(pl > 0.0))) continue;
                        ++n_shadow;
                        V f;
                        double pb;
                        mat_eval(mat, wo, wi, nrm, f, pb);
                        const V contrib = had(had(beta, f), li) * (cs * mis(pl, pb) / pl);
                        if (contrib.x == 0.0 && contrib.y == 0.0 && contrib.z == 0.0) continue;
                        if (!spheres_hit(S, Ray{hit.p + kEps * wi, wi, ray.time}, tmax, true, best)) L = L + contrib;
                    }
                }
                Bsdf s;
                if (!mat_sample(mat, ray, hit, rng, s)) break;
                last_pdf = s.pdf;
                last_nd = !s.delta;
                beta = had(beta, s.w);
                ray = s.ray;
            }
        } while (!add_sample(P, sums, L));
        store_pixel(P, x, row, sums, acc, acc_w, acc_sq);
        n_samples = (unsigned long long)sums.n;
    }
    count_rays(counters, n_samples, n_closest, n_shadow);
}

}  // namespace plain

cudaError_t launch_plain(const PlainScene& S, const PlainParams& P, double* acc, double* acc_w, double* acc_sq,
                         unsigned long long* counters, int* flags, int sm_count, cudaStream_t stream) {
    const plain::Tiles tiles = plain::tiles_of(P);
    // Spheres alone, few enough for the reference's loop over them, or nothing to
    // hit: a lane per pixel on its own.  Over 284 random calls of that kind (films
    // to 1280x720, 1 to 600 spheres, with and without maps and lights) it is 1.29
    // times as fast as k_paths; past some hundred spheres small films lose (200
    // spheres 16x16 x 17 spp 1.9 ms in k_paths, 2.5 here), large ones gain (1280x720 x
    // 2 spp 53 and 17), and 600 lose.  A single triangle brings the meshes' trees in,
    // where lanes on their own fall behind (512x512 x 8 spp at one bounce, ms, in k_paths
    // / lane by lane: 2 triangles 0.60 / 0.87, 5,120 triangles 1.55 / 8.1).
    if (P.max_bounces <= 0 || (S.n_tris == 0 && S.n_spheres <= 256)) {
        const unsigned grid = (tiles.n_ids + 127u) / 128u;
        plain::k_pixels<<<grid, 128, 0, stream>>>(S, P, acc, acc_w, acc_sq, counters, flags);
        return cudaGetLastError();
    }
    // Short walks: one block of 256 per SM, whose warps share the most fetched
    // lines.  Past about a thousand triangles the warps' walks differ so much
    // in length that waiting for the slowest of 8 costs more than fetching for
    // 4, and two blocks of 128 are better (480x270 x 32 spp with 200 spheres
    // and 1,280 / 20,480 / 327,680 triangles, ms: 9.6 / 11.9 / 15.9 in blocks
    // of 256, 9.2 / 10.7 / 14.0 in blocks of 128; sphere scene 8.5 / 11.7).
    // One bounce: a sample's shadow rays are its last, so it ends in their round
    // and the next one's camera ray joins it (512x512 x 8 spp, ms: sphere scene
    // 0.93 -> 0.65, 5,120 triangles 1.7 -> 1.56; with paths of several bounces the
    // extra barrier costs 2 to 8%), and 384 lanes per SM hide more of the short
    // chains' latency than 256 (0.65 -> 0.60).
    const bool brief = P.max_bounces <= 1;
    const int block = brief ? 192 : (S.n_tris < 1024 ? 256 : 128), ctas = brief ? 2 : 256 / block;
    // 256 (384) lanes per SM hold a pixel each.  A film of fewer pixels spreads them
    // over the warps: a warp of a few lanes diverges less, and it is each
    // pixel's own chain of bounces that the render waits for (48x30 x 64 spp:
    // 7.5 ms in full warps, 4.6 spread).
    const long long pixels = tiles.n_ids;  // in whole tiles
    const long long warps = (long long)sm_count * ctas * (block / 32);
    const unsigned lanes = (unsigned)std::min<long long>(32, std::max<long long>(1, (pixels + warps - 1) / warps));
    const long long per_block = (long long)lanes * (block / 32);
    const unsigned grid = (unsigned)std::min<long long>((pixels + per_block - 1) / per_block, warps * 32 / block);
    auto launch = [&](auto kernel) {
        kernel<<<grid, block, 0, stream>>>(S, P, acc, acc_w, acc_sq, counters, flags, lanes);
    };
    if (brief) launch(plain::k_paths<192, 2, true>);
    else if (block == 256) launch(plain::k_paths<256, 1, false>);
    else launch(plain::k_paths<128, 2, false>);
    return cudaGetLastError();
}

}  // namespace tpt
