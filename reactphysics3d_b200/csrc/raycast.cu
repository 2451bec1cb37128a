// Batched world raycast: one lane traces one ray as PhysicsWorld::raycast
// does (reference src/collision/broadphase/DynamicAABBTree.cpp:684-747,
// src/systems/BroadPhaseSystem.cpp:224-240, src/collision/RaycastInfo.cpp:34-49,
// src/collision/Collider.cpp:173-192): the broad-phase tree in its stack order
// with the ray clipped by each accepted hit, the category filter, the ray
// taken into the collider's local space, the shape's own raycast, the hit
// taken back to world space.  Float expression trees follow the reference's
// (no contraction: the library is built with --fmad=false).
#include <cfloat>

#include "raycast_launch.h"
#include "rp3dg_math.cuh"

namespace rp3dg {
namespace {

constexpr int RAY_STACK = 96;
constexpr int RAY_BLOCK = 128;
// Four resident CTAs per SM: with the lanes of a warp kept busy the spills of
// 64 registers cost more than the warps they buy (300,007 rays over a
// 20,000-body terrain: 2.64 ms at 8 CTAs, 2.36 at 6, 2.27 at 4, 2.40 at 3).
#ifndef RAY_MIN_BLOCKS
#define RAY_MIN_BLOCKS 4
#endif

struct LocalHit {
    v3 point, normal;
    float fraction;
};

RD float comp(v3 a, int i) { return i == 0 ? a.x : (i == 1 ? a.y : a.z); }
RD int iclamp(int v, int lo, int hi) {  // clamp(int, int, int): std::min(std::max(v, lo), hi)
    const int m = (v < lo) ? lo : v;
    return (hi < m) ? hi : m;
}

// AABB::testRayIntersect (AABB.h:285-314)
RD bool ray_aabb(float4 lo, float4 hi, v3 o, v3 inv, float maxf) {
    float t1 = (lo.x - o.x) * inv.x;
    float t2 = (hi.x - o.x) * inv.x;
    float tmin = smin(t1, t2);
    float tmax = smax(t1, t2);
    tmax = smin(tmax, maxf);
    t1 = (lo.y - o.y) * inv.y;
    t2 = (hi.y - o.y) * inv.y;
    tmin = smax(tmin, smin(t1, t2));
    tmax = smin(tmax, smax(t1, t2));
    t1 = (lo.z - o.z) * inv.z;
    t2 = (hi.z - o.z) * inv.z;
    tmin = smax(tmin, smin(t1, t2));
    tmax = smin(tmax, smax(t1, t2));
    return tmax >= smax(tmin, 0.0f);
}

// The same for finite bounds and a ray with a finite origin and inverse
// direction: no product is NaN, and of two zeros it does not matter which a
// minimum returns, so the hardware's minimum and maximum give the same answer
// in half the instructions.
RD bool ray_aabb_finite(float4 lo, float4 hi, v3 o, v3 inv, float maxf) {
    const float x1 = (lo.x - o.x) * inv.x, x2 = (hi.x - o.x) * inv.x;
    const float y1 = (lo.y - o.y) * inv.y, y2 = (hi.y - o.y) * inv.y;
    const float z1 = (lo.z - o.z) * inv.z, z2 = (hi.z - o.z) * inv.z;
    const float tmin = fmaxf(fmaxf(fminf(x1, x2), fminf(y1, y2)), fminf(z1, z2));
    const float tmax = fminf(fminf(fminf(fmaxf(x1, x2), maxf), fmaxf(y1, y2)), fmaxf(z1, z2));
    return tmax >= fmaxf(tmin, 0.0f);
}

// SphereShape::raycast (SphereShape.cpp:61-104) and
// CapsuleShape::raycastWithSphereEndCap (CapsuleShape.cpp:243-286): the
// sphere of radius r centred at c.
RD bool ray_sphere_at(v3 p1, v3 p2, v3 c, float maxf, float r, v3& point, float& fraction) {
    const v3 m = vsub(p1, c);
    const float cc = vdot(m, m) - r * r;
    if (cc < 0.0f) return false;
    const v3 d = vsub(p2, p1);
    const float b = vdot(m, d);
    if (b > 0.0f) return false;
    const float len2 = vlen2(d);
    const float disc = b * b - len2 * cc;
    if (disc < 0.0f || len2 < MACHINE_EPSILON) return false;
    float t = -b - sqrtf(disc);
    if (t < maxf * len2) {
        t /= len2;
        fraction = t;
        point = vadd(p1, vmul(d, t));
        return true;
    }
    return false;
}

RD bool ray_sphere(v3 p1, v3 p2, float maxf, float r, LocalHit& h) {
    // the sphere's raycast uses the ray origin itself (m = point1)
    const v3 m = p1;
    const float c = vdot(m, m) - r * r;
    if (c < 0.0f) return false;
    const v3 d = vsub(p2, p1);
    const float b = vdot(m, d);
    if (b > 0.0f) return false;
    const float len2 = vlen2(d);
    const float disc = b * b - len2 * c;
    if (disc < 0.0f || len2 < MACHINE_EPSILON) return false;
    float t = -b - sqrtf(disc);
    if (t < maxf * len2) {
        t /= len2;
        h.fraction = t;
        h.point = vadd(p1, vmul(d, t));
        h.normal = h.point;
        return true;
    }
    return false;
}

// CapsuleShape::raycast (CapsuleShape.cpp:97-240): segment p-q on the y axis
RD bool ray_capsule(v3 p1, v3 p2, float maxf, float r, float hh, LocalHit& h) {
    const v3 n = vsub(p2, p1);
    const float eps = 0.01f;
    const v3 p = V(0.0f, -hh, 0.0f), q = V(0.0f, hh, 0.0f);
    const v3 d = vsub(q, p);
    const v3 m = vsub(p1, p);
    const float mDotD = vdot(m, d), nDotD = vdot(n, d), dDotD = vdot(d, d);
    const float vec1DotD = vdot(vsub(p1, V(0.0f, -hh - r, 0.0f)), d);
    if (vec1DotD < 0.0f && vec1DotD + nDotD < 0.0f) return false;
    const float extra = 2.0f * r * d.y;
    if (vec1DotD > dDotD + extra && vec1DotD + nDotD > dDotD + extra) return false;
    const float nDotN = vdot(n, n), mDotN = vdot(m, n);
    const float a = dDotD * nDotN - nDotD * nDotD;
    const float k = vdot(m, m) - r * r;
    const float c = dDotD * k - mDotD * mDotD;
    auto cap = [&](v3 centre) -> bool {
        v3 hp;
        float hf;
        if (!ray_sphere_at(p1, p2, centre, maxf, r, hp, hf)) return false;
        h.fraction = hf;
        h.point = hp;
        h.normal = vsub(hp, centre);
        return true;
    };
    if (fabsf(a) < eps) {
        if (c > 0.0f) return false;
        if (mDotD < 0.0f) return cap(p);
        if (mDotD > dDotD) return cap(q);
        return false;
    }
    const float b = dDotD * mDotN - nDotD * mDotD;
    const float disc = b * b - a * c;
    if (disc < 0.0f) return false;
    const float t = (-b - sqrtf(disc)) / a;
    const float value = mDotD + t * nDotD;
    if (value < 0.0f) return cap(p);
    if (value > dDotD) return cap(q);
    if (t < 0.0f || t > maxf) return false;
    const v3 lp = vadd(p1, vmul(n, t));
    h.fraction = t;
    h.point = lp;
    const v3 v = vsub(lp, p);
    const v3 w = vmul(d, vdot(v, d) / vlen2(d));
    h.normal = vunit(vsub(lp, vadd(p, w)));
    return true;
}

// BoxShape::raycast (BoxShape.cpp:62-119): slabs, the entering face's
// (unnormalised) normal
RD bool ray_box(v3 p1, v3 p2, float maxf, v3 he, LocalHit& h) {
    const v3 d = vsub(p2, p1);
    float tmin = -FLT_MAX, tmax = FLT_MAX;
    v3 nd = V(0.0f, 0.0f, 0.0f);
    for (int i = 0; i < 3; i++) {
        const float di = comp(d, i), pi = comp(p1, i), hi = comp(he, i);
        if (fabsf(di) < MACHINE_EPSILON) {
            if (pi > hi || pi < -hi) return false;
        } else {
            const float inv = 1.0f / di;
            float t1 = (-hi - pi) * inv;
            float t2 = (hi - pi) * inv;
            v3 cn = V(i == 0 ? -hi : 0.0f, i == 1 ? -hi : 0.0f, i == 2 ? -hi : 0.0f);
            if (t1 > t2) {
                const float tt = t1;
                t1 = t2;
                t2 = tt;
                cn = vneg(cn);
            }
            if (t1 > tmin) {
                tmin = t1;
                nd = cn;
            }
            tmax = smin(tmax, t2);
            if (tmin > maxf) return false;
            if (tmin > tmax) return false;
        }
    }
    if (tmin < 0.0f || tmin > maxf) return false;
    h.point = vadd(p1, vmul(d, tmin));
    h.fraction = tmin;
    h.normal = nd;
    return true;
}

// ConvexMeshShape::raycast (ConvexMeshShape.cpp:107-172): face planes from
// the scaled face normals and the mesh's (unscaled) first vertex of each face
RD bool ray_mesh(v3 p1, v3 p2, float maxf, const MeshHdr* H, const uint32_t* w, LocalHit& h) {
    const v3 d = vsub(p2, p1);
    float tmin = 0.0f, tmax = maxf;
    v3 cn = V(0.0f, 0.0f, 0.0f);
    bool found = false;
    const uint32_t nf = H->nf;
    for (uint32_t f = 0; f < nf; f++) {
        const uint32_t on = H->off_normals + 4 * f;
        const v3 nrm = V(__uint_as_float(w[on]), __uint_as_float(w[on + 1]), __uint_as_float(w[on + 2]));
        const uint32_t v0 = w[H->off_face_verts + w[H->off_face_start + f]];
        const uint32_t ov = H->off_verts + 4 * v0;
        const v3 fp = V(__uint_as_float(w[ov]), __uint_as_float(w[ov + 1]), __uint_as_float(w[ov + 2]));
        const float denom = vdot(nrm, d);
        const float planeD = vdot(nrm, fp);
        const float dist = planeD - vdot(nrm, p1);
        if (denom == 0.0f) {
            if (dist < 0.0f) return false;
        } else {
            const float t = dist / denom;
            if (denom < 0.0f) {
                if (t > tmin) {
                    tmin = t;
                    cn = nrm;
                    found = true;
                }
            } else {
                if (t < tmax) tmax = t;
            }
            if (tmin > tmax) return false;
        }
    }
    if (!found) return false;
    h.point = vadd(p1, vmul(d, tmin));
    h.fraction = tmin;
    h.normal = cn;
    return true;
}

// AABB::raycast (AABB.h:317-357)
RD bool aabb_raycast(v3 mn, v3 mx, v3 p1, v3 p2, v3& hit, float& entry) {
    float tmin = 0.0f, tmax = FLT_MAX;
    const float eps = 0.00001f;
    const v3 d = vsub(p2, p1);
    for (int i = 0; i < 3; i++) {
        const float di = comp(d, i), pi = comp(p1, i), lo = comp(mn, i), hi = comp(mx, i);
        if (fabsf(di) < eps) {
            if (pi < lo || pi > hi) return false;
        } else {
            const float inv = 1.0f / di;
            float t1 = (lo - pi) * inv;
            float t2 = (hi - pi) * inv;
            if (t1 > t2) {
                const float tt = t2;
                t2 = t1;
                t1 = tt;
            }
            tmin = smax(tmin, t1);
            tmax = smin(tmax, t2);
            if (tmin > tmax) return false;
        }
    }
    hit = vadd(p1, vmul(d, tmin));
    entry = tmin;
    return true;
}

// TriangleShape::raycast (TriangleShape.cpp:143-230), FRONT side (the
// ConcaveShape default the height field passes on), from the three signed
// volumes on: none of them is negative.
RD bool ray_triangle_hit(v3 p1, v3 pq, float maxf, v3 a, v3 b, v3 c, float u, float v, float w, LocalHit& h) {
    if (fabsf(u - 0.0f) < MACHINE_EPSILON && fabsf(v - 0.0f) < MACHINE_EPSILON && fabsf(w - 0.0f) < MACHINE_EPSILON)
        return false;
    const float denom = 1.0f / (u + v + w);
    u *= denom;
    v *= denom;
    w *= denom;
    const v3 lp = vadd(vadd(vmul(a, u), vmul(b, v)), vmul(c, w));
    const float hf = vdot(vsub(lp, p1), pq) / vlen2(pq);
    if (hf < 0.0f || hf > maxf) return false;
    v3 nrm = vnormalize(vcross(vsub(b, a), vsub(c, a)));
    nrm = vdot(nrm, pq) > 0.0f ? vneg(nrm) : nrm;
    h.point = lp;
    h.fraction = hf;
    h.normal = nrm;
    return true;
}
RD bool ray_triangle(v3 p1, v3 p2, float maxf, v3 a, v3 b, v3 c, LocalHit& h) {
    const v3 pq = vsub(p2, p1);
    const v3 pa = vsub(a, p1), pb = vsub(b, p1), pc = vsub(c, p1);
    const v3 m = vcross(pq, pc);
    const float u = vdot(pb, m);
    if (u < 0.0f) return false;
    const float v = -vdot(pa, m);
    if (v < 0.0f) return false;
    const float w = vdot(pa, vcross(pq, pb));
    if (w < 0.0f) return false;
    return ray_triangle_hit(p1, pq, maxf, a, b, c, u, v, w, h);
}

// HeightField::getVertexAt (HeightField.cpp:386-393)
RD v3 hf_vertex(const HfDesc& H, int x, int y, float height) {
    return V(-H.width * 0.5f + float(x), H.origin + height, -H.length * 0.5f + float(y));
}

// HeightField::raycast with computeEnteringRayGridCoordinates
// (HeightField.cpp:258-384) on the ray already in the field's unscaled
// space: a grid walk from the cell where the ray enters the bounds, both
// triangles of each cell tested against the unclipped ray, a later hit at an
// equal fraction replacing an earlier one.  The reference's walk does not end
// when the ray's z direction is exactly zero and it enters on a cell
// boundary; this walk stops after as many cells as the grid can cross
// (*limit set).
//
// The reference walks on to the grid's border; this walk also stops where no
// later triangle can be accepted.  A triangle is accepted when none of its
// three signed volumes with the ray's line is negative: the line passes within
// rounding of it, or lies in its plane.  Divided by |p2 - p1|, the volumes are
// off by less than 10 * 2^-24 * D^2 for vertices up to D from p1 (products of
// two differences and the ray), so "within rounding" is less than a sixth of
// noise = 0.05 + 4e-6 D^2 sqrt(1 + 2 H^2) cells, H the field's height range.
//   - Height: from t_exit on, the line is more than H + noise outside the
//     field's height range and leaving.  A later column's triangle is not in
//     the line's plane (its plane reaches at most H beyond the range inside its
//     column), and the line is near it only if the column begins within noise
//     of where the line left the range.
//   - Length: past the parameter maxf + (2 + 2 H + noise) / |p2 - p1| an
//     accepted point's fraction is above maxf, again unless the column begins
//     within noise of where the line was at that parameter.
// So the walk ends when it crosses a cell boundary more than noise beyond the
// earlier of the two (every later column lies behind that boundary).  The
// heights of the next cell are read before the current one is tested.
// Rays over a 170 x 170 field walked 75 cells on average to the border.
RD bool ray_heightfield(v3 p1, v3 p2, float maxf, const HfDesc& H, LocalHit& h, bool* limit) {
    const v3 mn = V(H.bmin[0], H.bmin[1], H.bmin[2]), mx = V(H.bmax[0], H.bmax[1], H.bmax[2]);
    v3 g;
    float entry;
    if (!aabb_raycast(mn, mx, p1, p2, g, entry)) return false;
    const v3 ext = vsub(mx, mn);
    const int ni = int(H.ncol) - 1, nj = int(H.nrow) - 1;
    g = vsub(g, mn);
    const float stepI = ext.x / float(ni), stepJ = ext.z / float(nj);
    int i = iclamp(int(g.x / stepI), 0, ni - 1);
    int j = iclamp(int(g.z / stepJ), 0, nj - 1);
    const v3 d = vsub(p2, p1);
    const int si = d.x > 0.0f ? 1 : (d.x < 0.0f ? -1 : 0);
    const int sj = d.z > 0.0f ? 1 : (d.z < 0.0f ? -1 : 0);
    const float nextI = float(si >= 0 ? i + 1 : i), nextJ = float(sj >= 0 ? j + 1 : j);
    const float sizeI = ext.x / float(ni), sizeJ = ext.z / float(nj);
    float tMaxI = ((nextI * sizeI) - g.x) / d.x;
    float tMaxJ = ((nextJ * sizeJ) - g.z) / d.z;
    const float tDeltaI = sizeI / fabsf(d.x), tDeltaJ = sizeJ / fabsf(d.z);
    float smallest = maxf;
    bool hit = false;
    const int max_cells = ni + nj + 2;
    int cells = 0;
    // where the walk may stop early (see above); a parameter that is not a
    // finite number stops nothing
    const float fx = fmaxf(fabsf(mn.x - p1.x), fabsf(mx.x - p1.x)), fy = fmaxf(fabsf(mn.y - p1.y), fabsf(mx.y - p1.y));
    const float fz = fmaxf(fabsf(mn.z - p1.z), fabsf(mx.z - p1.z));
    const float noise = 0.05f + 4.0e-6f * (fx * fx + fy * fy + fz * fz) * sqrtf(1.0f + 2.0f * ext.y * ext.y);
    const float t_exit = d.y < 0.0f ? (-(ext.y + noise) - g.y) / d.y : (d.y > 0.0f ? (2.0f * ext.y + noise - g.y) / d.y : FLT_MAX);
    const float t_last = maxf - entry + (2.0f + 2.0f * ext.y + noise) / vlen(d);
    const float t_stop = t_last < t_exit ? t_last : t_exit;
    auto at = [&](int x, int y) { return __ldg(H.heights + size_t(y) * H.ncol + size_t(x)); };
    float h1 = at(i, j), h2 = at(i, j + 1), h3 = at(i + 1, j), h4 = at(i + 1, j + 1);
    for (;;) {
        if (cells++ >= max_cells) {
            *limit = true;
            break;
        }
        const int ci = i, cj = j;
        bool more = si != 0 || sj != 0;
        const float te = tMaxI < tMaxJ ? tMaxI : tMaxJ;   // where the ray leaves this cell
        const float da = fabsf(tMaxI < tMaxJ ? d.x : d.z);
        if (tMaxI < tMaxJ) {
            tMaxI += tDeltaI;
            i += si;
        } else {
            tMaxJ += tDeltaJ;
            j += sj;
        }
        more = more && i >= 0 && i < ni && j >= 0 && j < nj;
        if (fabsf(te) <= FLT_MAX && (te - t_stop) * da > noise) more = false;
        const int xi = more ? i : ci, xj = more ? j : cj;
        const float n1 = at(xi, xj), n2 = at(xi, xj + 1), n3 = at(xi + 1, xj), n4 = at(xi + 1, xj + 1);
        const v3 q1 = hf_vertex(H, ci, cj, h1), q2 = hf_vertex(H, ci, cj + 1, h2);
        const v3 q3 = hf_vertex(H, ci + 1, cj, h3), q4 = hf_vertex(H, ci + 1, cj + 1, h4);
        // the signed volumes of triangles (q1, q2, q3) and (q3, q2, q4)
        const v3 e1 = vsub(q1, p1), e2 = vsub(q2, p1), e3 = vsub(q3, p1), e4 = vsub(q4, p1);
        const v3 m1 = vcross(d, e3), m2 = vcross(d, e4), c2 = vcross(d, e2);
        const float u1 = vdot(e2, m1), v1 = -vdot(e1, m1), w1 = vdot(e1, c2);
        const float u2 = vdot(e2, m2), v2 = -vdot(e3, m2), w2 = vdot(e3, c2);
        LocalHit t;
        if (!(u1 < 0.0f) && !(v1 < 0.0f) && !(w1 < 0.0f) && ray_triangle_hit(p1, d, maxf, q1, q2, q3, u1, v1, w1, t) &&
            t.fraction <= smallest) {
            h = t;
            smallest = t.fraction;
            hit = true;
        }
        if (!(u2 < 0.0f) && !(v2 < 0.0f) && !(w2 < 0.0f) && ray_triangle_hit(p1, d, maxf, q3, q2, q4, u2, v2, w2, t) &&
            t.fraction <= smallest) {
            h = t;
            smallest = t.fraction;
            hit = true;
        }
        if (!more) break;
        h1 = n1;
        h2 = n2;
        h3 = n3;
        h4 = n4;
    }
    return hit;
}

// ConcaveMeshShape::raycast (ConcaveMeshShape.cpp:179-274): the ray without
// the mesh's scale walks the mesh's tree (DynamicAABBTree::raycast,
// DynamicAABBTree.cpp:684-747, whose callback collects every leaf it reaches
// and returns the ray's maxFraction, so the walk is never clipped), then each
// collected triangle, scaled, is tested in that order against the unscaled
// ray (TriangleShape::raycast, FRONT side), a hit at a fraction <= the
// smallest so far replacing the current one.
constexpr int MESH_RAY_STACK = 64;
__device__ __noinline__ bool ray_concave_mesh(v3 p1, v3 p2, float maxf, const CmDesc& cm, LocalHit& h, bool* overflow) {
    const v3 is = V(cm.inv_scale[0], cm.inv_scale[1], cm.inv_scale[2]);
    const v3 s1 = vcmul(p1, is), s2 = vcmul(p2, is);
    const v3 d = vsub(s2, s1);
    const v3 dinv = V(1.0f / d.x, 1.0f / d.y, 1.0f / d.z);
    float smallest = maxf;
    bool hit = false;
    int stack[MESH_RAY_STACK];
    int sp = 0;
    stack[sp++] = cm.root;
    while (sp > 0) {
        const int id = stack[--sp];
        if (id < 0) continue;
        const float4 lo = __ldg(&cm.nodes[id].lo), hi = __ldg(&cm.nodes[id].hi);
        if (!ray_aabb(lo, hi, s1, dinv, maxf)) continue;
        const int c0 = __float_as_int(lo.w);
        if (c0 <= -2) {
            const uint32_t tri = uint32_t(-2 - c0);
            const uint32_t i0 = __ldg(cm.tris + 3 * tri), i1 = __ldg(cm.tris + 3 * tri + 1), i2 = __ldg(cm.tris + 3 * tri + 2);
            auto ld = [&](uint32_t v) { return V(__ldg(cm.sverts + 3 * v), __ldg(cm.sverts + 3 * v + 1), __ldg(cm.sverts + 3 * v + 2)); };
            LocalHit th;
            if (ray_triangle(p1, p2, maxf, ld(i0), ld(i1), ld(i2), th) && th.fraction <= smallest) {
                h = th;
                smallest = th.fraction;
                hit = true;
            }
            // the callback's answer is the ray's maxFraction: 0 ends the walk
            if (maxf == 0.0f) break;
        } else {
            if (sp + 2 > MESH_RAY_STACK) {
                *overflow = true;
                break;
            }
            stack[sp++] = c0;
            stack[sp++] = __float_as_int(hi.w);
        }
    }
    return hit;
}

// Collider::raycast: the ray into the collider's local space
// (localToWorld.getInverse() * point), the shape's raycast, the hit point and
// the rotated, normalised normal back in world space.
RD bool collider_raycast(const RayArgs& a, int4 col, v3 p1, v3 p2, float maxf, LocalHit& h, int* flags) {
    const float4 tp = a.c_wpos[col.x], tq = a.c_wori[col.x];
    const quat q = Q(tq.x, tq.y, tq.z, tq.w);
    const quat iq = qinv(q);
    const v3 ip = qrot(iq, V(-tp.x, -tp.y, -tp.z));
    const v3 l1 = vadd(qrot(iq, p1), ip), l2 = vadd(qrot(iq, p2), ip);
    const rp3dg_shape s = a.shapes[col.z];
    bool hit = false;
    switch (s.kind) {
        case RP3DG_SHAPE_SPHERE: hit = ray_sphere(l1, l2, maxf, s.params[0], h); break;
        case RP3DG_SHAPE_CAPSULE: hit = ray_capsule(l1, l2, maxf, s.params[0], s.params[1], h); break;
        case RP3DG_SHAPE_BOX: hit = ray_box(l1, l2, maxf, V(s.params[0], s.params[1], s.params[2]), h); break;
        case RP3DG_SHAPE_CONVEX_MESH:
            hit = ray_mesh(l1, l2, maxf, reinterpret_cast<const MeshHdr*>(a.mesh_words) + s.mesh, a.mesh_words, h);
            break;
        case RP3DG_SHAPE_HEIGHTFIELD: {
            if (s.mesh < 0 || uint32_t(s.mesh) >= a.nb_hfields) break;
            const HfDesc H = a.hfields[s.mesh];
            // HeightFieldShape::raycast (HeightFieldShape.cpp:76-90)
            const v3 is = V(1.0f / H.scale[0], 1.0f / H.scale[1], 1.0f / H.scale[2]);
            bool limit = false;
            hit = ray_heightfield(vcmul(l1, is), vcmul(l2, is), maxf, H, h, &limit);
            if (hit) h.point = vcmul(h.point, V(H.scale[0], H.scale[1], H.scale[2]));
            if (limit) *flags |= 1;
            break;
        }
        case RP3DG_SHAPE_CONCAVE_MESH: {
            if (s.mesh < 0 || uint32_t(s.mesh) >= a.nb_cmeshes) break;
            bool overflow = false;
            hit = ray_concave_mesh(l1, l2, maxf, a.cmeshes[s.mesh], h, &overflow);
            if (overflow) atomicOr(a.error, 1u);
            break;
        }
        default: break;
    }
    if (!hit) return false;
    h.point = vadd(qrot(q, h.point), V(tp.x, tp.y, tp.z));
    h.normal = vnormalize(qrot(q, h.normal));
    return true;
}

// What a lane's ray waits for.
enum RayWait { RAY_NODES = 0, RAY_SHAPE = 1, RAY_TERRAIN = 2, RAY_DONE = 3 };
// Lanes that wait before their phase runs while others still have nodes to
// visit, and before finished lanes take new rays (4 / 4: 3 % less on the
// terrain, but 684 us instead of 521 for 100,000 rays over 512 convex shapes).
constexpr int RAY_GATHER = 8, RAY_REFILL = 4;

// One lane per ray.  The lanes of a warp work in phases, so that a phase's
// instructions serve many of them: tree nodes; the convex shapes of the leaves
// reached, when RAY_GATHER rays wait for one; height-field and triangle-mesh
// walks (tens of cells) likewise; and new rays for the lanes that are done.  A
// ray meets its nodes, its leaves and their clips in the reference's order;
// only the lanes' progress relative to each other changes.  Bound: the node
// steps (245 a ray on the terrain), two dependent reads and ~75 instructions
// each.  Each ray on its own path ran 2.7 lanes an instruction: 300,007 rays
// over a 20,000-body terrain 5.16 ms, here 2.24; 32 rays 844 and 281 us;
// 100,000 rays over 512 convex shapes 1,102 and 521 us.
//
// A node step reads both children of the current node at once and tests them
// against the ray as it is: a child that misses now would miss later, the ray
// only gets shorter; the first child is pushed if it hits and tested again
// when popped.
__global__ void __launch_bounds__(RAY_BLOCK, RAY_MIN_BLOCKS) world_raycast_kernel(const RayArgs a, const uint32_t lanes) {
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t users = lanes == 32u ? 0xffffffffu : (1u << lanes) - 1u;   // lanes that take rays
    uint32_t i = a.n, mask = 0u, count = 0;
    v3 p1 = V(0.0f, 0.0f, 0.0f), p2 = p1, inv = p1;
    float maxf = 0.0f;
    bool finite = true, more = true;
    int wait = RAY_DONE;
    int stack[RAY_STACK];
    int sp = 0;
    int first = -1, second = -1;   // the next nodes to test: `first` and its subtree before `second`
    int leaf = -1;
    int4 col = make_int4(0, 0, 0, 0);
    for (;;) {
        // new rays
        const uint32_t done = __ballot_sync(0xffffffffu, wait == RAY_DONE) & users;
        if (more && (done == users || __popc(done) >= RAY_REFILL)) {
            uint32_t base = 0;
            if (lane == 0) base = atomicAdd(a.queue, uint32_t(__popc(done)));
            base = __shfl_sync(0xffffffffu, base, 0);
            more = base + uint32_t(__popc(done)) < a.n;
            if (done >> lane & 1u) {
                i = base + uint32_t(__popc(done & ((1u << lane) - 1u)));
                if (i < a.n) {
                    const rp3dg_ray R = a.rays[i];
                    p1 = V(R.point1[0], R.point1[1], R.point1[2]);
                    p2 = V(R.point2[0], R.point2[1], R.point2[2]);
                    maxf = R.max_fraction;
                    mask = R.category_mask;
                    const v3 dir = vsub(p2, p1);
                    inv = V(1.0f / dir.x, 1.0f / dir.y, 1.0f / dir.z);
                    // (a NaN fails the comparison)
                    finite = a.finite_nodes && fabsf(inv.x) <= FLT_MAX && fabsf(inv.y) <= FLT_MAX && fabsf(inv.z) <= FLT_MAX &&
                             fabsf(p1.x) <= FLT_MAX && fabsf(p1.y) <= FLT_MAX && fabsf(p1.z) <= FLT_MAX;
                    sp = 0;
                    count = 0;
                    first = a.root;
                    second = -1;
                    wait = RAY_NODES;
                }
            }
        }
        // nodes
        for (;;) {
            const uint32_t at_nodes = __ballot_sync(0xffffffffu, wait == RAY_NODES);
            if (!at_nodes) break;
            if (__popc(__ballot_sync(0xffffffffu, wait == RAY_SHAPE)) >= RAY_GATHER ||
                __popc(__ballot_sync(0xffffffffu, wait == RAY_TERRAIN)) >= RAY_GATHER ||
                (more && __popc(__ballot_sync(0xffffffffu, wait == RAY_DONE) & users) >= RAY_REFILL))
                break;
            if (wait == RAY_NODES) {
                if (first < 0 && sp > 0) first = stack[--sp];
                if (first < 0) {
                    wait = RAY_DONE;
                    a.nb_hits[i] = count;
                } else {
                    const int other = second >= 0 ? second : first;
                    const float4 lo1 = __ldg(&a.nodes[first].lo), hi1 = __ldg(&a.nodes[first].hi);
                    const float4 lo0 = __ldg(&a.nodes[other].lo), hi0 = __ldg(&a.nodes[other].hi);
                    bool hit1, hit0;
                    if (finite) {
                        hit1 = ray_aabb_finite(lo1, hi1, p1, inv, maxf);
                        hit0 = ray_aabb_finite(lo0, hi0, p1, inv, maxf);
                    } else {
                        hit1 = ray_aabb(lo1, hi1, p1, inv, maxf);
                        hit0 = ray_aabb(lo0, hi0, p1, inv, maxf);
                    }
                    hit0 = hit0 && second >= 0;
                    const bool full = hit1 && hit0 && sp == RAY_STACK;
                    if (hit1 && hit0 && !full) stack[sp++] = second;
                    const int c0 = __float_as_int(hit1 ? lo1.w : lo0.w), c1 = __float_as_int(hit1 ? hi1.w : hi0.w);
                    const bool any = hit1 || hit0, inner = any && c0 > -2;
                    // children[1]'s subtree comes before children[0]'s
                    first = inner ? (c1 >= 0 ? c1 : c0) : -1;
                    second = inner && c1 >= 0 ? c0 : -1;
                    if (any && !inner) {
                        leaf = -2 - c0;
                        col = __ldg(&a.colliders[leaf]);
                        if ((mask & uint32_t(col.w) & 0xffffu) != 0u)
                            wait = (col.w >> 16) >= RP3DG_SHAPE_HEIGHTFIELD ? RAY_TERRAIN : RAY_SHAPE;
                    }
                    if (full) {
                        atomicOr(a.error, 1u);
                        wait = RAY_DONE;
                        a.nb_hits[i] = count;
                    }
                }
            }
        }
        // shapes or walks: the larger group
        const int nshape = __popc(__ballot_sync(0xffffffffu, wait == RAY_SHAPE));
        const int nterrain = __popc(__ballot_sync(0xffffffffu, wait == RAY_TERRAIN));
        if (nshape + nterrain == 0) {
            if (!more && !__any_sync(0xffffffffu, wait == RAY_NODES)) break;   // every ray is done
            continue;
        }
        if (wait == (nshape >= nterrain ? RAY_SHAPE : RAY_TERRAIN)) {
            LocalHit h;
            int flags = 0;
            float ret = maxf;   // RaycastTest::raycastAgainstShape without a hit
            if (collider_raycast(a, col, p1, p2, maxf, h, &flags)) {
                rp3dg_raycast_hit rec;
                rec.world_point[0] = h.point.x; rec.world_point[1] = h.point.y; rec.world_point[2] = h.point.z;
                rec.world_normal[0] = h.normal.x; rec.world_normal[1] = h.normal.y; rec.world_normal[2] = h.normal.z;
                rec.hit_fraction = h.fraction;
                rec.body = col.y;
                rec.collider = leaf;
                rec.flags = flags;
                rp3dg_raycast_hit* out = a.hits + size_t(i) * a.max_hits;
                if (a.mode == RP3DG_RAYCAST_ALL) {
                    if (count < a.max_hits) out[count] = rec;
                    ret = 1.0f;
                } else {
                    if (a.max_hits) out[0] = rec;
                    ret = (a.mode == RP3DG_RAYCAST_ANY) ? 0.0f : h.fraction;
                }
                count++;
            }
            wait = RAY_NODES;
            if (ret == 0.0f) {
                wait = RAY_DONE;
                a.nb_hits[i] = count;
            }
            if (ret > 0.0f && ret < maxf) maxf = ret;
        }
    }
}

}  // namespace

cudaError_t launch_world_raycast(const RayArgs& a, int num_sms, cudaStream_t stream) {
    if (a.n == 0) return cudaSuccess;
    // A batch that does not fill the GPU spreads over its warps, whose rays
    // wait for one another: one ray a warp up to 32 warps per SM, then 2, 4,
    // ... 32; past that, lanes take new rays as they finish.
    const uint32_t warps = uint32_t(num_sms) * RAY_MIN_BLOCKS * (RAY_BLOCK / 32);
    uint32_t lanes = 1;
    while (lanes < 32u && a.n > warps * lanes) lanes *= 2;
    const uint32_t need = (a.n + lanes - 1) / lanes, use = need < warps ? need : warps;
    world_raycast_kernel<<<(use + RAY_BLOCK / 32 - 1) / (RAY_BLOCK / 32), RAY_BLOCK, 0, stream>>>(a, lanes);
    return cudaGetLastError();
}

}  // namespace rp3dg
