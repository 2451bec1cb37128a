// Dynamics stage of a world step, after contact creation: world inverse
// inertia, velocity integration, the sequential-impulse contact solver with
// split impulses, position integration and the body / collider state update
// (reference src/engine/PhysicsWorld.cpp:239-318, src/systems/
// DynamicsSystem.cpp:44-183, src/systems/ContactSolverSystem.cpp:66-818).
//
// Five steps: bodies (inertia + velocities), manifolds (solver records, one
// thread per manifold), islands (warm start, iterations, stored impulses: a
// thread, a warp or a CTA per island, the manifolds of every body in the
// reference's order, so each sees exactly the reference's sequence of
// Gauss-Seidel updates), bodies (positions + state), colliders
// (local-to-world).  Every expression keeps the
// reference's operand order; the library is built without FMA contraction,
// so results are bit-identical to the reference's float build.
#include <cuda_runtime.h>
#include <algorithm>
#ifdef RP3DG_PROFILE_GIANT
#include <cstdio>
#endif

#include "broadphase_launch.h"
#include "dynamics_launch.h"
#include "rp3dg_internal.h"
#include "rp3dg_math.cuh"

namespace rp3dg {

namespace {

constexpr float BETA = 0.2f;               // ContactSolverSystem.cpp:43
constexpr float BETA_SPLIT_IMPULSE = 0.2f;  // :44
constexpr float SLOP = 0.01f;              // :45

RD v3 L3(const float4 a) { return V(a.x, a.y, a.z); }
RD float4 F4(v3 a, float w = 0.0f) { return make_float4(a.x, a.y, a.z, w); }

// Matrix3x3 * Vector3 (Matrix3x3.h:324-331), row-major m[9]
RD v3 mv(const float* m, v3 v) {
    return V(m[0] * v.x + m[1] * v.y + m[2] * v.z,
             m[3] * v.x + m[4] * v.y + m[5] * v.z,
             m[6] * v.x + m[7] * v.y + m[8] * v.z);
}

// Quaternion::getMatrix (src/mathematics/Quaternion.cpp:138-165)
RD void quat_matrix(quat q, float* r) {
    const float nQ = q.x * q.x + q.y * q.y + q.z * q.z + q.w * q.w;
    float s = 0.0f;
    if (nQ > 0.0f) s = 2.0f / nQ;
    const float xs = q.x * s, ys = q.y * s, zs = q.z * s;
    const float wxs = q.w * xs, wys = q.w * ys, wzs = q.w * zs;
    const float xxs = q.x * xs, xys = q.x * ys, xzs = q.x * zs;
    const float yys = q.y * ys, yzs = q.y * zs, zzs = q.z * zs;
    r[0] = 1.0f - yys - zzs; r[1] = xys - wzs;        r[2] = xzs + wys;
    r[3] = xys + wzs;        r[4] = 1.0f - xxs - zzs; r[5] = yzs - wxs;
    r[6] = xzs - wys;        r[7] = yzs + wxs;        r[8] = 1.0f - xxs - yys;
}

// RigidBody::computeWorldInertiaTensorInverse (RigidBody.h:246-262):
// out = R * (diag(inv) * R^T), Matrix3x3 product of Matrix3x3.h:302-321
RD void world_inertia(const float* R, v3 inv, float* out) {
    float t[9];
    t[0] = R[0] * inv.x; t[1] = R[3] * inv.x; t[2] = R[6] * inv.x;
    t[3] = R[1] * inv.y; t[4] = R[4] * inv.y; t[5] = R[7] * inv.y;
    t[6] = R[2] * inv.z; t[7] = R[5] * inv.z; t[8] = R[8] * inv.z;
    for (int i = 0; i < 3; i++)
        for (int j = 0; j < 3; j++)
            out[3 * i + j] = R[3 * i + 0] * t[0 + j] + R[3 * i + 1] * t[3 + j] + R[3 * i + 2] * t[6 + j];
}

// v2 + w2 x r2 - v1 - w1 x r1, written out as in ContactSolverSystem.cpp:196-201
RD v3 rel_velocity(v3 v1, v3 w1, v3 v2, v3 w2, v3 r1, v3 r2) {
    return V(v2.x + w2.y * r2.z - w2.z * r2.y - v1.x - w1.y * r1.z + w1.z * r1.y,
             v2.y + w2.z * r2.x - w2.x * r2.z - v1.y - w1.z * r1.x + w1.x * r1.z,
             v2.z + w2.x * r2.y - w2.y * r2.x - v1.z - w1.x * r1.y + w1.y * r1.x);
}

// Vector3::getOneUnitOrthogonalVector (src/mathematics/Vector3.cpp:46-64)
RD v3 unit_orthogonal(v3 v) {
    const v3 a = V(fabsf(v.x), fabsf(v.y), fabsf(v.z));
    const int minElement = (a.x < a.y ? (a.x < a.z ? 0 : 2) : (a.y < a.z ? 1 : 2));
    if (minElement == 0) {
        const float l = sqrtf(v.y * v.y + v.z * v.z);
        return V(0.0f / l, -v.z / l, v.y / l);
    } else if (minElement == 1) {
        const float l = sqrtf(v.x * v.x + v.z * v.z);
        return V(-v.z / l, 0.0f / l, v.x / l);
    }
    const float l = sqrtf(v.x * v.x + v.y * v.y);
    return V(-v.y / l, v.x / l, 0.0f / l);
}

// Enabled bodies / colliders: the first nb_enabled / nc_enabled rows, or the
// rows flagged in b_enabled / c_enabled when those are given (several worlds
// in one batch, each with its own enabled range).
RD bool body_enabled(const DynArgs& a, uint32_t i) { return a.b_enabled ? a.b_enabled[i] != 0 : i < a.nb_enabled; }
RD bool collider_enabled(const DynArgs& a, uint32_t i) { return a.c_enabled ? a.c_enabled[i] != 0 : i < a.nc_enabled; }

// ---- kernel 1: world inverse inertia + velocity integration --------------
__global__ void __launch_bounds__(128) dyn_bodies_pre(const DynArgs a) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= a.nb) return;
    const float4 zero = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    a.sv[i] = zero;
    a.sw[i] = zero;
    if (!body_enabled(a, i)) {
        // read-only body: the solver sees its stored velocity
        a.cv[i] = a.lin_vel[i];
        a.cw[i] = a.ang_vel[i];
        return;
    }
    // PhysicsWorld::updateBodiesInverseWorldInertiaTensors (:310-318)
    const float4 o = a.orientation[i];
    float R[9], I[9];
    quat_matrix(Q(o.x, o.y, o.z, o.w), R);
    world_inertia(R, L3(a.iil[i]), I);
    a.iiw[3 * i + 0] = make_float4(I[0], I[1], I[2], 0.0f);
    a.iiw[3 * i + 1] = make_float4(I[3], I[4], I[5], 0.0f);
    a.iiw[3 * i + 2] = make_float4(I[6], I[7], I[8], 0.0f);
    // DynamicsSystem::integrateRigidBodiesVelocities (DynamicsSystem.cpp:117-183)
    const float dt = a.dt;
    const float4 m = a.mass[i];  // mass, inverse mass, linear damping, angular damping
    const v3 lf = L3(a.llock[i]), af = L3(a.alock[i]);
    const v3 v = L3(a.lin_vel[i]), w = L3(a.ang_vel[i]);
    const v3 F = L3(a.force[i]);
    const float s = dt * m.y;
    v3 cv = V(v.x + s * lf.x * F.x, v.y + s * lf.y * F.y, v.z + s * lf.z * F.z);
    const v3 It = mv(I, L3(a.torque[i]));
    v3 cw = V(w.x + dt * af.x * It.x, w.y + dt * af.y * It.y, w.z + dt * af.z * It.z);
    if (a.gravity_enabled && a.gravity[i]) {
        cv = V(cv.x + s * lf.x * m.x * a.gx, cv.y + s * lf.y * m.x * a.gy, cv.z + s * lf.z * m.x * a.gz);
    }
    const float lin_damp = 1.0f / (1.0f + m.z * dt);
    const float ang_damp = 1.0f / (1.0f + m.w * dt);
    cv = vmul(cv, lin_damp);
    cw = vmul(cw, ang_damp);
    a.cv[i] = F4(cv);
    a.cw[i] = F4(cw);
}

RD bool is_fixed(const DynArgs& a, int32_t b) {
    if (uint32_t(b) >= a.nb || !body_enabled(a, uint32_t(b))) return true;
    const float4 il = a.iil[b];
    return a.mass[b].y == 0.0f && il.x == 0.0f && il.y == 0.0f && il.z == 0.0f;
}

RD float4 F4w(v3 a, float w) { return make_float4(a.x, a.y, a.z, w); }

// ---- island sizes: which islands get a thread each -------------------------
//
// An island on a thread costs kernel 3a a chain of its manifolds, however many
// islands there are, and more the more lanes of a warp are at one; an island on
// a warp costs one of kernel 3b's warps its time, and the warps share the
// islands.  A thread each pays when the warps would have several small islands
// each, so the limit is chosen from the stage's island sizes, by what both sides
// measured (points at random, 888 warps): threads 21, 56, 91, 126, 266 us for
// islands of 1, 2, 3, 4, 8 manifolds when all lanes have one, a warp 10, 17, 23,
// 28, 42 us an island.
// 12,000 islands of one manifold: warps 208 us a stage, threads 97; 2,500
// islands of eight: warps 206, threads 341; 192 captured worlds (6,976
// islands, half of them of one manifold): limit 0 817, 1 804, 8 859; 4,096 of
// them: 0 2,635, 4 1,846, 8 1,785.
constexpr uint32_t BIG_ISLAND = 64;   // queued first: the longest islands start first
constexpr uint32_t SIZE_CLASSES = 8;  // islands of 1 .. 8 manifolds by size
enum IslandSizes { IS_MID = SIZE_CLASSES, IS_MID_MAX, IS_BIG, IS_BIG_SUM, IS_BIG_MAX, IS_WORDS };   // from counters[9]
static_assert(9 + IS_WORDS == DYN_COUNTERS, "counters");

// `longest` the most manifolds of an island, `manifolds` those of all, a stage of `ni` islands
RD uint32_t thread_us(uint32_t longest, uint32_t manifolds, uint32_t ni) {
    return longest ? uint32_t(13.0f * float(longest) + 22.0f * float(manifolds) / float(ni)) - 5u : 0u;
}
RD uint32_t warp_us(uint32_t manifolds) {
    return manifolds <= SIZE_CLASSES ? 7u + 5u * manifolds : 47u + (manifolds - SIZE_CLASSES) * 11u / 4u;
}

// Block `block` counts its 128 islands.
RD void count_island_sizes(const DynArgs& a, uint32_t block) {
    __shared__ uint32_t h[IS_WORDS];
    if (threadIdx.x < IS_WORDS) h[threadIdx.x] = 0;
    __syncthreads();
    const uint32_t is = block * 128u + threadIdx.x;
    const uint32_t cnt = is < a.ni && !(a.i_jcount && a.i_jcount[is]) ? a.i_count[is] : 0u;
    if (cnt != 0 && cnt <= a.nm) {
        if (cnt <= SIZE_CLASSES) {
            atomicAdd(h + cnt - 1, 1u);
        } else if (cnt <= BIG_ISLAND) {
            atomicAdd(h + IS_MID, warp_us(cnt));
            atomicMax(h + IS_MID_MAX, warp_us(cnt));
        } else {
            atomicAdd(h + IS_BIG, 1u);
            atomicAdd(h + IS_BIG_SUM, warp_us(cnt));
            atomicMax(h + IS_BIG_MAX, warp_us(cnt));
        }
    }
    __syncthreads();
    const uint32_t k = threadIdx.x;
    if (k < IS_WORDS && h[k]) {
        if (k == IS_MID_MAX || k == IS_BIG_MAX) atomicMax(a.counters + 9 + k, h[k]);
        else atomicAdd(a.counters + 9 + k, h[k]);
    }
}

// The limit whose estimate is the lowest (of two alike the smaller); lane s of
// a warp estimates limit s.
RD uint32_t small_limit(const DynArgs& a, uint32_t lane) {
    if (!a.small_auto) return a.small_max;
    const uint32_t* h = a.counters + 9;
    const uint32_t warps = a.large_ctas * uint32_t(LARGE_WARPS);
    const bool big = h[IS_BIG] > a.giant_ctas;   // too many for a CTA each
    uint32_t sum = h[IS_MID] + (big ? h[IS_BIG_SUM] : 0u), longest = h[IS_MID_MAX], top = 0, mans = 0;
    if (big && h[IS_BIG_MAX] > longest) longest = h[IS_BIG_MAX];
#pragma unroll
    for (uint32_t c = 1; c <= SIZE_CLASSES; c++) {
        const uint32_t n = h[c - 1];
        if (n && c <= lane) { top = c; mans += n * c; }       // on threads
        if (n && c > lane) longest = warp_us(c) > longest ? warp_us(c) : longest;
        if (c > lane) sum += n * warp_us(c);                 // on warps
    }
    const uint32_t share = (sum + warps - 1) / warps;
    const uint32_t us = thread_us(top, mans, a.ni) + (share > longest ? share : longest);
    const uint32_t key = lane <= a.small_max && lane <= SIZE_CLASSES ? us << 4 | lane : 0xffffffffu;
    return __reduce_min_sync(0xffffffffu, key) & 15u;
}

// ---- kernel 2: ContactSolverSystem::initializeForIsland per manifold ------
// (ContactSolverSystem.cpp:116-318).  Writes the manifold's solver record and
// its points' records (layouts in dynamics_launch.h).
__global__ void __launch_bounds__(128) dyn_manifold_init(const DynArgs a) {
    // the blocks behind the manifolds' count the islands
    const uint32_t mblocks = (a.nm + 127u) / 128u;
    if (blockIdx.x >= mblocks) {
        count_island_sizes(a, blockIdx.x - mblocks);
        return;
    }
    const uint32_t m = blockIdx.x * blockDim.x + threadIdx.x;
    if (m >= a.nm) return;
    float4* __restrict__ q = a.mrec[m].q;
    const int4 id = a.m_ids[m];
    const int32_t b1 = id.x, b2 = id.y;
    const uint32_t nb = a.m_npts[m], ps = a.m_pstart[m];
    if (uint32_t(b1) >= a.nb || uint32_t(b2) >= a.nb || b1 == b2 || uint32_t(id.z) >= a.nc ||
        uint32_t(id.w) >= a.nc || nb == 0 || nb > 4 || ps > a.np || nb > a.np - ps) {
        atomicOr(a.error, 4u);
        q[DQ_IDS] = make_float4(__int_as_float(0), __int_as_float(0), __int_as_float(0), __int_as_float(0));
        q[DQ_MASS] = make_float4(0.0f, 0.0f, 0.0f, 3.0f);  // no points: every pass skips it
        return;
    }
    q[DQ_IDS] = make_float4(__int_as_float(b1), __int_as_float(b2), __int_as_float(int32_t(nb)), __int_as_float(int32_t(ps)));
    const v3 x1 = L3(a.com_world[b1]), x2 = L3(a.com_world[b2]);
    float I1[9], I2[9];
    {
        const float4 r0 = a.iiw[3 * b1], r1 = a.iiw[3 * b1 + 1], r2 = a.iiw[3 * b1 + 2];
        I1[0] = r0.x; I1[1] = r0.y; I1[2] = r0.z; I1[3] = r1.x; I1[4] = r1.y; I1[5] = r1.z;
        I1[6] = r2.x; I1[7] = r2.y; I1[8] = r2.z;
        q[DQ_I1 + 0] = r0; q[DQ_I1 + 1] = r1; q[DQ_I1 + 2] = r2;
    }
    {
        const float4 r0 = a.iiw[3 * b2], r1 = a.iiw[3 * b2 + 1], r2 = a.iiw[3 * b2 + 2];
        I2[0] = r0.x; I2[1] = r0.y; I2[2] = r0.z; I2[3] = r1.x; I2[4] = r1.y; I2[5] = r1.z;
        I2[6] = r2.x; I2[7] = r2.y; I2[8] = r2.z;
        q[DQ_I2 + 0] = r0; q[DQ_I2 + 1] = r1; q[DQ_I2 + 2] = r2;
    }
    const float im1 = a.mass[b1].y, im2 = a.mass[b2].y;
    const float4 mat1 = a.c_mat[id.z], mat2 = a.c_mat[id.w];
    const float friction = mat1.x * mat2.x;                          // computeMixedFrictionCoefficient
    const float restitution = (mat1.y > mat2.y) ? mat1.y : mat2.y;   // computeMixedRestitutionFactor
    const float fixed = float((is_fixed(a, b1) ? 1 : 0) | (is_fixed(a, b2) ? 2 : 0));
    q[DQ_MASS] = make_float4(im1, im2, friction, fixed);
    q[DQ_LF1] = a.llock[b1]; q[DQ_LF2] = a.llock[b2];
    const float4 al1 = a.alock[b1], al2 = a.alock[b2];
    q[DQ_AF1] = al1; q[DQ_AF2] = al2;
    const v3 af1 = L3(al1), af2 = L3(al2);
    const float beta = a.split ? BETA_SPLIT_IMPULSE : BETA;
    const v3 v1 = L3(a.lin_vel[b1]), w1 = L3(a.ang_vel[b1]);
    const v3 v2 = L3(a.lin_vel[b2]), w2 = L3(a.ang_vel[b2]);
    const float4 o1 = a.c_wori[id.z], o2 = a.c_wori[id.w];
    const xform t1 = X(L3(a.c_wpos[id.z]), Q(o1.x, o1.y, o1.z, o1.w));
    const xform t2 = X(L3(a.c_wpos[id.w]), Q(o2.x, o2.y, o2.z, o2.w));
    v3 fp1 = V(0.0f, 0.0f, 0.0f), fp2 = V(0.0f, 0.0f, 0.0f), nsum = V(0.0f, 0.0f, 0.0f);
    for (uint32_t k = 0; k < nb; k++) {
        const uint32_t p = ps + k;
        DynPointRec& r = a.prec[p];
        const float4 nd = a.p_nd[p];
        const v3 n = V(nd.x, nd.y, nd.z);
        const v3 p1 = xapply(t1, L3(a.p_l1[p]));
        const v3 p2 = xapply(t2, L3(a.p_l2[p]));
        const v3 r1 = V(p1.x - x1.x, p1.y - x1.y, p1.z - x1.z);
        const v3 r2 = V(p2.x - x2.x, p2.y - x2.y, p2.z - x2.z);
        const uint8_t resting = a.p_resting[p];
        a.p_resting[p] = 1;
        fp1 = V(fp1.x + p1.x, fp1.y + p1.y, fp1.z + p1.z);
        fp2 = V(fp2.x + p2.x, fp2.y + p2.y, fp2.z + p2.z);
        const v3 dv = rel_velocity(v1, w1, v2, w2, r1, r2);
        const v3 r1n = vcross(r1, n), r2n = vcross(r2, n);
        const v3 i1 = mv(I1, r1n), i2 = mv(I2, r2n);
        const float mp = im1 + im2 + vdot(vcross(i1, r1), n) + vdot(vcross(i2, r2), n);
        const float inv_mass = mp > 0.0f ? 1.0f / mp : 0.0f;
        float bias = 0.0f;
        const float dvn = dv.x * n.x + dv.y * n.y + dv.z * n.z;
        if (dvn < -a.restitution_threshold) bias = restitution * dvn;
        // the penetration bias and the products i * angular lock factor are the
        // same in every pass (solve, :479-759, forms them anew): kept here
        float bias_pen = 0.0f;
        if (nd.w > SLOP) {
            const float excess = nd.w - SLOP;
            bias_pen = -(beta / a.dt) * ((0.0f < excess) ? excess : 0.0f);
        }
        r.q[DP_R1] = F4w(r1, 0.0f);
        r.q[DP_R2] = F4w(r2, inv_mass);
        r.q[DP_N] = F4w(n, a.split ? bias : bias_pen + bias);
        r.q[DP_I1] = F4w(vcmul(i1, af1), bias_pen);
        r.q[DP_I2] = F4w(vcmul(i2, af2), 0.0f);
        r.mut = make_float4(a.p_impulse[p], 0.0f, resting ? 1.0f : 0.0f, 0.0f);
        nsum = V(nsum.x + n.x, nsum.y + n.y, nsum.z + n.z);
    }
    const float fnb = float(nb);
    fp1 = vdivs(fp1, fnb);
    fp2 = vdivs(fp2, fnb);
    const v3 r1f = V(fp1.x - x1.x, fp1.y - x1.y, fp1.z - x1.z);
    const v3 r2f = V(fp2.x - x2.x, fp2.y - x2.y, fp2.z - x2.z);
    q[DQ_OFV1] = a.m_fv1[m];
    q[DQ_OFV2] = a.m_fv2[m];
    const float4 fi = a.m_fimp[m];
    a.mrec[m].mut = make_float4(fi.x, fi.y, fi.z, 0.0f);
    const v3 n = vnormalize(nsum);
    // computeFrictionVectors (:789-818)
    const v3 dvf = rel_velocity(v1, w1, v2, w2, r1f, r2f);
    const float dvfn = vdot(dvf, n);
    const v3 nv = vmul(n, dvfn);
    const v3 tv = V(dvf.x - nv.x, dvf.y - nv.y, dvf.z - nv.z);
    const float lt = vlen(tv);
    const v3 fv1 = lt > MACHINE_EPSILON ? vdivs(tv, lt) : unit_orthogonal(n);
    const v3 fv2 = vcross(n, fv1);
    const v3 r1ct1 = vcross(r1f, fv1), r1ct2 = vcross(r1f, fv2);
    const v3 r2ct1 = vcross(r2f, fv1), r2ct2 = vcross(r2f, fv2);
    const float f1m = im1 + im2 + vdot(vcross(mv(I1, r1ct1), r1f), fv1) + vdot(vcross(mv(I2, r2ct1), r2f), fv1);
    const float f2m = im1 + im2 + vdot(vcross(mv(I1, r1ct2), r1f), fv2) + vdot(vcross(mv(I2, r2ct2), r2f), fv2);
    const float twm = vdot(n, mv(I1, n)) + vdot(n, mv(I2, n));
    q[DQ_N] = F4w(n, twm > 0.0f ? 1.0f / twm : 0.0f);
    q[DQ_R1F] = F4w(r1f, f1m > 0.0f ? 1.0f / f1m : 0.0f);
    q[DQ_R2F] = F4w(r2f, f2m > 0.0f ? 1.0f / f2m : 0.0f);
    q[DQ_FV1] = F4w(fv1, 0.0f);
    q[DQ_FV2] = F4w(fv2, 0.0f);
    q[DQ_R1CT1] = F4w(r1ct1, 0.0f);
    q[DQ_R1CT2] = F4w(r1ct2, 0.0f);
    q[DQ_R2CT1] = F4w(r2ct1, 0.0f);
    q[DQ_R2CT2] = F4w(r2ct2, 0.0f);
}

// A manifold's constant solver data in registers (one 16-byte load per row).
struct Man {
    int32_t b1, b2, nb, pstart;
    float im1, im2, friction;
    uint32_t fixed;
    v3 lf1, lf2, af1, af2;
    float I1[9], I2[9];
    v3 n, r1f, r2f, fv1, fv2, r1ct1, r1ct2, r2ct1, r2ct2;
    float inv_tw, inv_f1, inv_f2;
};

template <bool LDG>
RD float4 ldq(const float4* p) { return LDG ? __ldg(p) : *p; }

template <bool LDG>
RD void rows3(const float4* __restrict__ q, float* I) {
    const float4 r0 = ldq<LDG>(q), r1 = ldq<LDG>(q + 1), r2 = ldq<LDG>(q + 2);
    I[0] = r0.x; I[1] = r0.y; I[2] = r0.z; I[3] = r1.x; I[4] = r1.y; I[5] = r1.z;
    I[6] = r2.x; I[7] = r2.y; I[8] = r2.z;
}

// The records are written by kernel 2 and only read here, so the read-only
// data path may serve them (LDG); the giant-island kernel reads copies staged
// in shared memory (generic loads).
template <bool LDG = true>
RD void load_man_q(const float4* __restrict__ q, Man& c) {
    const float4 ids = ldq<LDG>(q + DQ_IDS), ms = ldq<LDG>(q + DQ_MASS);
    c.b1 = __float_as_int(ids.x); c.b2 = __float_as_int(ids.y);
    c.nb = __float_as_int(ids.z); c.pstart = __float_as_int(ids.w);
    c.im1 = ms.x; c.im2 = ms.y; c.friction = ms.z; c.fixed = uint32_t(ms.w);
    c.lf1 = L3(ldq<LDG>(q + DQ_LF1)); c.lf2 = L3(ldq<LDG>(q + DQ_LF2));
    c.af1 = L3(ldq<LDG>(q + DQ_AF1)); c.af2 = L3(ldq<LDG>(q + DQ_AF2));
    rows3<LDG>(q + DQ_I1, c.I1);
    rows3<LDG>(q + DQ_I2, c.I2);
    const float4 n = ldq<LDG>(q + DQ_N), r1f = ldq<LDG>(q + DQ_R1F), r2f = ldq<LDG>(q + DQ_R2F);
    c.n = L3(n); c.inv_tw = n.w;
    c.r1f = L3(r1f); c.inv_f1 = r1f.w;
    c.r2f = L3(r2f); c.inv_f2 = r2f.w;
    c.fv1 = L3(ldq<LDG>(q + DQ_FV1)); c.fv2 = L3(ldq<LDG>(q + DQ_FV2));
    c.r1ct1 = L3(ldq<LDG>(q + DQ_R1CT1)); c.r1ct2 = L3(ldq<LDG>(q + DQ_R1CT2));
    c.r2ct1 = L3(ldq<LDG>(q + DQ_R2CT1)); c.r2ct2 = L3(ldq<LDG>(q + DQ_R2CT2));
}
RD void load_man(const DynManifoldRec* __restrict__ rec, Man& c) { load_man_q<true>(rec->q, c); }

struct Pt {
    v3 r1, r2, n, i1, i2;          // i1, i2: times the angular lock factors
    float inv_mass, bias, bias_pen;  // bias: of the constrained velocities
};

template <bool LDG = true>
RD void load_pt_q(const float4* __restrict__ q, Pt& p) {
    const float4 a = ldq<LDG>(q + DP_R1), b = ldq<LDG>(q + DP_R2), c = ldq<LDG>(q + DP_N);
    p.r1 = L3(a);
    p.r2 = L3(b); p.inv_mass = b.w;
    p.n = L3(c); p.bias = c.w;
    const float4 d = ldq<LDG>(q + DP_I1);
    p.i1 = L3(d); p.bias_pen = d.w;
    p.i2 = L3(ldq<LDG>(q + DP_I2));
}

// v -= im * imp * lock  /  v += im * imp * lock, per component (Vector3 operators)
RD v3 lin_sub(v3 v, float im, v3 imp, v3 lf) {
    return V(v.x - im * imp.x * lf.x, v.y - im * imp.y * lf.y, v.z - im * imp.z * lf.z);
}
RD v3 lin_add(v3 v, float im, v3 imp, v3 lf) {
    return V(v.x + im * imp.x * lf.x, v.y + im * imp.y * lf.y, v.z + im * imp.z * lf.z);
}
// w -= i * af * s  /  w += i * af * s, per component (the point updates; the
// point rows hold i * af)
RD v3 ang_sub(v3 w, v3 iaf, float s) { return V(w.x - iaf.x * s, w.y - iaf.y * s, w.z - iaf.z * s); }
RD v3 ang_add(v3 w, v3 iaf, float s) { return V(w.x + iaf.x * s, w.y + iaf.y * s, w.z + iaf.z * s); }

// Where the solver reads and writes the velocities (constrained and split)
// of a manifold's two bodies: the global scratch arrays, or a warp's shared
// memory copy for the movable bodies of a large island.
struct BodyVel {
    float4 *v1, *w1, *s1, *t1, *v2, *w2, *s2, *t2;
};

// Where the solver reads a manifold's constant rows and reads / writes its
// impulses: the records in global memory, or copies in shared memory.
// Point k's rows are at pq + k * pq_stride, its impulses at pmut + k * pmut_stride.
struct RecSrc {
    const float4* mq;
    float4* mmut;
    const float4* pq;
    float4* pmut;
    int pq_stride, pmut_stride;
    float2* pm2 = nullptr;   // PRE cores: the impulses (penetration, split), when kept apart from the resting flags in pmut
};
constexpr int PREC_ROWS = int(sizeof(DynPointRec) / sizeof(float4));
RD RecSrc rec_global(const DynArgs& a, uint32_t mi, int32_t pstart) {
    RecSrc r;
    r.mq = a.mrec[mi].q;
    r.mmut = &a.mrec[mi].mut;
    r.pq = a.prec[pstart].q;
    r.pmut = &a.prec[pstart].mut;
    r.pq_stride = PREC_ROWS;
    r.pmut_stride = PREC_ROWS;
    return r;
}

RD BodyVel vel_global(const DynArgs& a, int32_t b1, int32_t b2) {
    BodyVel p;
    p.v1 = a.cv + b1; p.w1 = a.cw + b1; p.s1 = a.sv + b1; p.t1 = a.sw + b1;
    p.v2 = a.cv + b2; p.w2 = a.cw + b2; p.s2 = a.sv + b2; p.t2 = a.sw + b2;
    return p;
}

// warmStart (:324-476) of one manifold: its two bodies' velocities are loaded,
// updated in the reference's statement order and stored back (the two bodies
// are distinct; fixed bodies are never stored).
// A manifold's point impulses held in four registers (PRE cores): loaded
// together before the points are solved and stored after, so that copies in
// global memory cost one round trip; points beyond four (none after the
// manifold step) are read and written in place.
RD float4 pm2_load(const RecSrc& r, int k) {
    const float2 v = r.pm2[k];
    return make_float4(v.x, v.y, r.pmut[k * r.pmut_stride].z, 0.0f);
}
RD void pmv_load(const RecSrc& r, int nb, float4& p0, float4& p1, float4& p2, float4& p3) {
    if (r.pm2) {
        if (nb > 0) p0 = pm2_load(r, 0);
        if (nb > 1) p1 = pm2_load(r, 1);
        if (nb > 2) p2 = pm2_load(r, 2);
        if (nb > 3) p3 = pm2_load(r, 3);
        return;
    }
    if (nb > 0) p0 = r.pmut[0];
    if (nb > 1) p1 = r.pmut[r.pmut_stride];
    if (nb > 2) p2 = r.pmut[2 * r.pmut_stride];
    if (nb > 3) p3 = r.pmut[3 * r.pmut_stride];
}
RD void pmv_store(const RecSrc& r, int nb, const float4& p0, const float4& p1, const float4& p2, const float4& p3) {
    if (r.pm2) {
        if (nb > 0) r.pm2[0] = make_float2(p0.x, p0.y);
        if (nb > 1) r.pm2[1] = make_float2(p1.x, p1.y);
        if (nb > 2) r.pm2[2] = make_float2(p2.x, p2.y);
        if (nb > 3) r.pm2[3] = make_float2(p3.x, p3.y);
        return;
    }
    if (nb > 0) r.pmut[0] = p0;
    if (nb > 1) r.pmut[r.pmut_stride] = p1;
    if (nb > 2) r.pmut[2 * r.pmut_stride] = p2;
    if (nb > 3) r.pmut[3 * r.pmut_stride] = p3;
}
template <bool PRE>
RD float4 pm_get(const RecSrc& r, int k, const float4& p0, const float4& p1, const float4& p2, const float4& p3) {
    if (!PRE) return r.pmut[k * r.pmut_stride];
    return k == 0 ? p0 : k == 1 ? p1 : k == 2 ? p2 : k == 3 ? p3 : r.pmut[k * r.pmut_stride];
}
template <bool PRE>
RD void pm_set(const RecSrc& r, int k, const float4& v, float4& p0, float4& p1, float4& p2, float4& p3) {
    if (!PRE || k > 3) { r.pmut[k * r.pmut_stride] = v; return; }
    if (k == 0) p0 = v;
    else if (k == 1) p1 = v;
    else if (k == 2) p2 = v;
    else p3 = v;
}

template <bool LDG, bool PRE = false>
RD void warm_core(const DynArgs& a, const RecSrc& r, const BodyVel& bv, int32_t nb) {
    if (nb == 0) return;  // rejected by the manifold kernel
    Man c;
    load_man_q<LDG>(r.mq, c);
    const v3 o1 = L3(ldq<LDG>(r.mq + DQ_OFV1)), o2 = L3(ldq<LDG>(r.mq + DQ_OFV2));
    float4 mut = *r.mmut;
    v3 v1 = L3(*bv.v1), w1 = L3(*bv.w1), v2 = L3(*bv.v2), w2 = L3(*bv.w2);
    float4 pv0, pv1, pv2, pv3;
    if (PRE) pmv_load(r, nb, pv0, pv1, pv2, pv3);
    bool resting_any = false;
    for (int k = 0; k < nb; k++) {
        float4 pm = pm_get<PRE>(r, k, pv0, pv1, pv2, pv3);
        if (pm.z != 0.0f) {
            resting_any = true;
            Pt p;
            load_pt_q<LDG>(r.pq + k * r.pq_stride, p);
            const float pi = pm.x;
            const v3 ip = V(p.n.x * pi, p.n.y * pi, p.n.z * pi);
            v1 = lin_sub(v1, c.im1, ip, c.lf1);
            w1 = ang_sub(w1, p.i1, pi);
            v2 = lin_add(v2, c.im2, ip, c.lf2);
            w2 = ang_add(w2, p.i2, pi);
        } else {
            pm.x = 0.0f;
            pm_set<PRE>(r, k, pm, pv0, pv1, pv2, pv3);
        }
    }
    if (PRE) pmv_store(r, nb, pv0, pv1, pv2, pv3);
    float f1 = mut.x, f2 = mut.y, ftw = mut.z;
    if (resting_any) {
        const v3 ofi = V(f1 * o1.x + f2 * o2.x, f1 * o1.y + f2 * o2.y, f1 * o1.z + f2 * o2.z);
        f1 = vdot(ofi, c.fv1);
        f2 = vdot(ofi, c.fv2);
        // first friction constraint
        v3 ai1 = V(-c.r1ct1.x * f1, -c.r1ct1.y * f1, -c.r1ct1.z * f1);
        v3 li2 = V(c.fv1.x * f1, c.fv1.y * f1, c.fv1.z * f1);
        v3 ai2 = V(c.r2ct1.x * f1, c.r2ct1.y * f1, c.r2ct1.z * f1);
        v1 = lin_sub(v1, c.im1, li2, c.lf1);
        w1 = vadd(w1, vcmul(c.af1, mv(c.I1, ai1)));
        v2 = lin_add(v2, c.im2, li2, c.lf2);
        w2 = vadd(w2, vcmul(c.af2, mv(c.I2, ai2)));
        // second friction constraint
        ai1 = V(-c.r1ct2.x * f2, -c.r1ct2.y * f2, -c.r1ct2.z * f2);
        li2 = V(c.fv2.x * f2, c.fv2.y * f2, c.fv2.z * f2);
        ai2 = V(c.r2ct2.x * f2, c.r2ct2.y * f2, c.r2ct2.z * f2);
        v1 = lin_sub(v1, c.im1, li2, c.lf1);
        w1 = vadd(w1, vcmul(c.af1, mv(c.I1, ai1)));
        v2 = lin_add(v2, c.im2, li2, c.lf2);
        w2 = vadd(w2, vcmul(c.af2, mv(c.I2, ai2)));
        // twist friction constraint (the reference applies the body-2
        // angular impulse to both bodies a second time, :461-465)
        ai1 = V(-c.n.x * ftw, -c.n.y * ftw, -c.n.z * ftw);
        ai2 = V(c.n.x * ftw, c.n.y * ftw, c.n.z * ftw);
        w1 = vadd(w1, vcmul(c.af1, mv(c.I1, ai1)));
        w2 = vadd(w2, vcmul(c.af2, mv(c.I2, ai2)));
        w1 = vsub(w1, vcmul(c.af1, mv(c.I1, ai2)));
        w2 = vadd(w2, vcmul(c.af2, mv(c.I2, ai2)));
    } else {
        f1 = 0.0f; f2 = 0.0f; ftw = 0.0f;
    }
    *r.mmut = make_float4(f1, f2, ftw, mut.w);
    if (!(c.fixed & 1)) { *bv.v1 = F4(v1); *bv.w1 = F4(w1); }
    if (!(c.fixed & 2)) { *bv.v2 = F4(v2); *bv.w2 = F4(w2); }
}
RD void warm_manifold(const DynArgs& a, uint32_t mi, const BodyVel& bv, int32_t nb, int32_t pstart) {
    warm_core<true>(a, rec_global(a, mi, pstart), bv, nb);
}

// One solve pass (:479-759) over one manifold.
template <bool LDG, bool PRE = false>
RD void solve_core(const DynArgs& a, const RecSrc& r, const BodyVel& bv, int32_t nb) {
    if (nb == 0) return;
    Man c;
    load_man_q<LDG>(r.mq, c);
    float4 mut = *r.mmut;
    v3 v1 = L3(*bv.v1), w1 = L3(*bv.w1), v2 = L3(*bv.v2), w2 = L3(*bv.w2);
    v3 s1 = L3(*bv.s1), t1 = L3(*bv.t1), s2 = L3(*bv.s2), t2 = L3(*bv.t2);
    float4 pv0, pv1, pv2, pv3;
    if (PRE) pmv_load(r, nb, pv0, pv1, pv2, pv3);
    float sum_pen = 0.0f;
    for (int k = 0; k < nb; k++) {
        Pt p;
        load_pt_q<LDG>(r.pq + k * r.pq_stride, p);
        float4 pm = pm_get<PRE>(r, k, pv0, pv1, pv2, pv3);
        const v3 n = p.n;
        const v3 dv = rel_velocity(v1, w1, v2, w2, p.r1, p.r2);
        const float Jv = dv.x * n.x + dv.y * n.y + dv.z * n.z;
        float dl = -(Jv + p.bias) * p.inv_mass;
        const float lt = pm.x;
        const float sum = pm.x + dl;
        pm.x = (sum < 0.0f) ? 0.0f : sum;
        dl = pm.x - lt;
        const v3 li = V(n.x * dl, n.y * dl, n.z * dl);
        v1 = lin_sub(v1, c.im1, li, c.lf1);
        w1 = ang_sub(w1, p.i1, dl);
        v2 = lin_add(v2, c.im2, li, c.lf2);
        w2 = ang_add(w2, p.i2, dl);
        sum_pen += pm.x;
        if (a.split) {
            const v3 dvs = rel_velocity(s1, t1, s2, t2, p.r1, p.r2);
            const float Jvs = dvs.x * n.x + dvs.y * n.y + dvs.z * n.z;
            float dls = -(Jvs + p.bias_pen) * p.inv_mass;
            const float lts = pm.y;
            const float ss = pm.y + dls;
            pm.y = (ss < 0.0f) ? 0.0f : ss;
            dls = pm.y - lts;
            const v3 lis = V(n.x * dls, n.y * dls, n.z * dls);
            s1 = lin_sub(s1, c.im1, lis, c.lf1);
            t1 = ang_sub(t1, p.i1, dls);
            s2 = lin_add(s2, c.im2, lis, c.lf2);
            t2 = ang_add(t2, p.i2, dls);
        }
        pm_set<PRE>(r, k, pm, pv0, pv1, pv2, pv3);
    }
    if (PRE) pmv_store(r, nb, pv0, pv1, pv2, pv3);
    float f1 = mut.x, f2 = mut.y, ftw = mut.z;
    // first friction constraint
    {
        const v3 dv = rel_velocity(v1, w1, v2, w2, c.r1f, c.r2f);
        const float Jv = dv.x * c.fv1.x + dv.y * c.fv1.y + dv.z * c.fv1.z;
        float dl = -Jv * c.inv_f1;
        const float limit = c.friction * sum_pen;
        const float lt = f1;
        f1 = smax(-limit, smin(f1 + dl, limit));
        dl = f1 - lt;
        const v3 ai1 = V(-c.r1ct1.x * dl, -c.r1ct1.y * dl, -c.r1ct1.z * dl);
        const v3 li2 = V(c.fv1.x * dl, c.fv1.y * dl, c.fv1.z * dl);
        const v3 ai2 = V(c.r2ct1.x * dl, c.r2ct1.y * dl, c.r2ct1.z * dl);
        v1 = lin_sub(v1, c.im1, li2, c.lf1);
        w1 = vadd(w1, vcmul(c.af1, mv(c.I1, ai1)));
        v2 = lin_add(v2, c.im2, li2, c.lf2);
        w2 = vadd(w2, vcmul(c.af2, mv(c.I2, ai2)));
    }
    // second friction constraint
    {
        const v3 dv = rel_velocity(v1, w1, v2, w2, c.r1f, c.r2f);
        const float Jv = dv.x * c.fv2.x + dv.y * c.fv2.y + dv.z * c.fv2.z;
        float dl = -Jv * c.inv_f2;
        const float limit = c.friction * sum_pen;
        const float lt = f2;
        f2 = smax(-limit, smin(f2 + dl, limit));
        dl = f2 - lt;
        const v3 ai1 = V(-c.r1ct2.x * dl, -c.r1ct2.y * dl, -c.r1ct2.z * dl);
        const v3 li2 = V(c.fv2.x * dl, c.fv2.y * dl, c.fv2.z * dl);
        const v3 ai2 = V(c.r2ct2.x * dl, c.r2ct2.y * dl, c.r2ct2.z * dl);
        v1 = lin_sub(v1, c.im1, li2, c.lf1);
        w1 = vadd(w1, vcmul(c.af1, mv(c.I1, ai1)));
        v2 = lin_add(v2, c.im2, li2, c.lf2);
        w2 = vadd(w2, vcmul(c.af2, mv(c.I2, ai2)));
    }
    // twist friction constraint
    {
        const v3 dw = vsub(w2, w1);
        const float Jv = dw.x * c.n.x + dw.y * c.n.y + dw.z * c.n.z;
        float dl = -Jv * c.inv_tw;
        const float limit = c.friction * sum_pen;
        const float lt = ftw;
        ftw = smax(-limit, smin(ftw + dl, limit));
        dl = ftw - lt;
        const v3 ai2 = V(c.n.x * dl, c.n.y * dl, c.n.z * dl);
        w1 = vsub(w1, vcmul(c.af1, mv(c.I1, ai2)));
        w2 = vadd(w2, vcmul(c.af2, mv(c.I2, ai2)));
    }
    *r.mmut = make_float4(f1, f2, ftw, mut.w);
    if (!(c.fixed & 1)) { *bv.v1 = F4(v1); *bv.w1 = F4(w1); *bv.s1 = F4(s1); *bv.t1 = F4(t1); }
    if (!(c.fixed & 2)) { *bv.v2 = F4(v2); *bv.w2 = F4(w2); *bv.s2 = F4(s2); *bv.t2 = F4(t2); }
}
RD void solve_manifold(const DynArgs& a, uint32_t mi, const BodyVel& bv, int32_t nb, int32_t pstart) {
    solve_core<true>(a, rec_global(a, mi, pstart), bv, nb);
}

// storeImpulses (:763-785) of one manifold.
RD void store_manifold(const DynArgs& a, uint32_t mi) {
    Man c;
    load_man(a.mrec + mi, c);
    if (c.nb == 0) return;
    for (int k = 0; k < c.nb; k++) a.p_impulse[c.pstart + k] = a.prec[c.pstart + k].mut.x;
    const float4 mut = a.mrec[mi].mut;
    a.m_fimp[mi] = make_float4(mut.x, mut.y, mut.z, 0.0f);
    a.m_fv1[mi] = F4(c.fv1);
    a.m_fv2[mi] = F4(c.fv2);
}

// ---- kernel 3: warm start, velocity iterations, stored impulses ----------
//
// The reference runs the manifolds of an island strictly in order; manifold j
// only reads and writes the velocities of its two bodies, and islands share
// only fixed bodies (static or kinematic: never written here).  So islands
// are independent, and inside an island any schedule that keeps, for every
// movable body, the order of the manifolds touching it gives bit-identical
// results.
//
// 3a: one thread per island queues the islands by size and solves those of up
//     to small_limit manifolds itself, in the reference's order.
// 3b: persistent warps take the queued islands.  The warp gives each manifold
//     a level (1 + the highest level of an earlier manifold sharing a movable
//     body) and sorts the island's manifolds by level; every pass (warm
//     start, each velocity iteration) then runs level after level, __syncwarp
//     (which orders the lanes' memory accesses) between them: four manifolds at
//     a time on eight lanes each, or 32 on a lane each where the levels are
//     wide.  An island of up to STAGE_MANIFOLDS manifolds and STAGE_BODIES
//     bodies (fixed ones too) keeps its schedule and its bodies' velocities in
//     the warp's shared memory; larger ones use the same schedule built in
//     global scratch, one lane a manifold, velocities in global memory.
// 3c: one CTA per island, staged in up to the whole opt-in shared memory of a
//     CTA: the islands above giant_min manifolds, and those above BIG_ISLAND
//     when there is a CTA for each (big_on_ctas).  When there are more giant
//     islands than CTAs, 3b takes those that fit a warp (giants_on_warps).
// 3d: the islands that do not fit 3c, streamed through global memory.
// (small_max, 8 by default, and giant_min, 256 by default, come from DynTuning.)
constexpr uint32_t ISLAND_DONE = 0xffffffffu;   // entry of giant_list solved by kernel 3b

RD int4 man_ids(const DynArgs& a, uint32_t mi) {
    const float4 q = __ldg(a.mrec[mi].q + DQ_IDS);
    return make_int4(__float_as_int(q.x), __float_as_int(q.y), __float_as_int(q.z), __float_as_int(q.w));
}
RD uint32_t man_fixed(const DynArgs& a, uint32_t mi) { return uint32_t(__ldg(a.mrec[mi].q + DQ_MASS).w); }

__global__ void __launch_bounds__(128) dyn_islands_small(const DynArgs a) {
    __shared__ uint32_t s_limit;
    if (threadIdx.x < 32) {
        const uint32_t limit = small_limit(a, threadIdx.x);
        if (threadIdx.x == 0) s_limit = limit;
    }
    __syncthreads();
    const uint32_t is = blockIdx.x * blockDim.x + threadIdx.x;
    if (is >= a.ni) return;
    const uint32_t m0 = a.i_start[is], cnt = a.i_count[is];
    if (m0 > a.nm || cnt > a.nm - m0) {
        atomicOr(a.error, 4u);
        return;
    }
    if (a.i_jcount && a.i_jcount[is]) return;  // kernel 3e
    if (cnt == 0) return;
    if (cnt > s_limit) {
        // big islands fill the list from the front, the others from the back
        if (cnt > a.giant_min) a.giant_list[atomicAdd(a.counters + 3, 1u)] = is;
        else if (cnt > BIG_ISLAND) a.large_list[atomicAdd(a.counters, 1u)] = is;
        else a.large_list[a.ni - 1 - atomicAdd(a.counters + 2, 1u)] = is;
        return;
    }
    const unsigned here = __activemask();
    if ((threadIdx.x & 31u) == uint32_t(__ffs(here)) - 1u) atomicAdd(a.counters + 7, uint32_t(__popc(here)));
    const uint32_t m1 = m0 + cnt;
    for (uint32_t mi = m0; mi < m1; mi++) {
        const int4 id = man_ids(a, mi);
        warm_manifold(a, mi, vel_global(a, id.x, id.y), id.z, id.w);
    }
    for (int it = 0; it < a.iterations; it++)
        for (uint32_t mi = m0; mi < m1; mi++) {
            const int4 id = man_ids(a, mi);
            solve_manifold(a, mi, vel_global(a, id.x, id.y), id.z, id.w);
        }
    for (uint32_t mi = m0; mi < m1; mi++) store_manifold(a, mi);
}

// ---- a manifold on eight lanes --------------------------------------------
//
// An island's manifolds form a chain of levels of two or three manifolds
// each, so a warp that gives every manifold one lane issues the ~1,400
// instructions of a four-point manifold for two or three active lanes and is
// bound by its own issue rate.  Here eight lanes share a manifold.  Lanes 0-3
// solve its constrained velocities and lanes 4-7 its split-impulse velocities
// (two independent chains until the bodies are stored); in each half lane
// c < 3 keeps component c of the linear velocities and components c + 1, c + 2
// of the angular ones (lane 3 repeats lane 0 and stores nothing).  Component c
// of v + w x r needs exactly those, so the only exchange is the three products
// of a dot product, read with shuffles and added in the reference's order by
// every lane: each value goes through the same operations in the same order
// as in warm_core / solve_core, bit for bit.  Measured on a chain of one
// manifold a level, cycles a level with 1 / 4 points: one CTA an island
// 1,562 / 2,392 with a lane a manifold, 1,273 / 1,841 here; one warp an island
// 2,277 / 4,319 and 1,697 / 2,141 (1,981 / 2,478 while its copies and loads of
// the next chunk were conditional: a dozen divergent branches).  4,096
// captured worlds: 5.28 -> 1.76 ms.
constexpr uint32_t LANES_PER_MANIFOLD = 8, WARP_MANIFOLDS = 32 / LANES_PER_MANIFOLD;
// A manifold's rows staged in shared memory: its record's constant rows, then
// its points' records (the impulse rows among them are the values at staging
// time; only their resting flags are read).
struct __align__(16) LaneSlot {
    float4 mq[DQ_ROWS];
    float4 pq[4 * PREC_ROWS];
};

RD void cp_async16(void* smem, const void* gmem) {
    const unsigned sa = static_cast<unsigned>(__cvta_generic_to_shared(smem));
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(sa), "l"(gmem) : "memory");
}
RD void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N>
RD void cp_async_wait() { asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory"); }

// Predicated stores, written out, where a nest of C++ conditionals becomes a
// chain of divergent branches.
RD void st_shared_if(bool ok, float* p, float v) {
    const unsigned sa = static_cast<unsigned>(__cvta_generic_to_shared(p));
    asm volatile("{\n .reg .pred q;\n setp.ne.s32 q, %2, 0;\n @q st.shared.f32 [%0], %1;\n}\n" ::"r"(sa), "f"(v), "r"(int(ok)) : "memory");
}
RD void st_global_if(bool ok, float* p, float v) {
    asm volatile("{\n .reg .pred q;\n setp.ne.s32 q, %2, 0;\n @q st.global.f32 [%0], %1;\n}\n" ::"l"(p), "f"(v), "r"(int(ok)) : "memory");
}

struct LaneId {
    uint32_t group;     // manifold of the warp's four
    uint32_t role;      // 0 constrained, 1 split velocities
    uint32_t c, c1, c2; // component and the two after it
    uint32_t q;         // lane of the half
    bool writer;
};
RD LaneId lane_id(uint32_t lane) {
    LaneId id;
    id.group = lane >> 3;
    id.role = (lane >> 2) & 1u;
    const uint32_t c = lane & 3u;
    id.writer = c < 3;
    id.q = c;
    id.c = c < 3 ? c : 0u;
    id.c1 = id.c == 2 ? 0u : id.c + 1;
    id.c2 = id.c == 0 ? 2u : id.c - 1;
    return id;
}
// (x + y) + z of the three components' products, the same in every lane
RD float lanes_sum(float p) {
    const float x = __shfl_sync(0xffffffffu, p, 0, 4), y = __shfl_sync(0xffffffffu, p, 1, 4);
    const float z = __shfl_sync(0xffffffffu, p, 2, 4);
    return x + y + z;
}
// the same where lane c holds the product of component c + 1
RD float lanes_sum_next(float p) {
    const float x = __shfl_sync(0xffffffffu, p, 2, 4), y = __shfl_sync(0xffffffffu, p, 0, 4);
    const float z = __shfl_sync(0xffffffffu, p, 1, 4);
    return x + y + z;
}
// row of Matrix3x3 * Vector3
RD float row_dot(const float4& m, v3 v) { return m.x * v.x + m.y * v.y + m.z * v.z; }

// This lane's share of the two bodies' velocities.
struct LaneVel { float v1, w1a, w1b, v2, w2a, w2b; };
// b1 / b2: the bodies' rows of the lane's role, the angular row `wofs` floats
// behind the linear one.
RD LaneVel lane_vel_load(const float* b1, const float* b2, uint32_t wofs, const LaneId& id) {
    return LaneVel{b1[id.c], b1[wofs + id.c1], b1[wofs + id.c2], b2[id.c], b2[wofs + id.c1], b2[wofs + id.c2]};
}
// Every component is stored by one lane (its angular share by c + 1); the
// rows are in shared memory.
RD void lane_vel_store(float* b1, float* b2, uint32_t wofs, const LaneId& id, bool ok, uint32_t fixed, const LaneVel& u) {
    const bool s1 = ok && !(fixed & 1u), s2 = ok && !(fixed & 2u);
    st_shared_if(s1, b1 + id.c, u.v1);
    st_shared_if(s1, b1 + wofs + id.c1, u.w1a);
    st_shared_if(s2, b2 + id.c, u.v2);
    st_shared_if(s2, b2 + wofs + id.c1, u.w2a);
}
// A half's four lanes hold the same impulses: each stores one point's and one
// friction impulse.
RD float lane_pick(uint32_t q, const float (&x)[4]) {
    const float lo = q & 1u ? x[1] : x[0], hi = q & 1u ? x[3] : x[2];
    return q & 2u ? hi : lo;
}

// warm_core on eight lanes; the whole warp calls it, `nbw` is the largest
// point count of the warp's manifolds.  imp[k] is point k's penetration
// impulse, f the friction impulses (all lanes of the half agree).
RD void lanes_warm(const float* mq, const float* pq, uint32_t nb, uint32_t nbw, bool active, const LaneId& id,
                   float* b1, float* b2, uint32_t wofs, float (&imp)[4], float (&f)[3]) {
    const float4* q = reinterpret_cast<const float4*>(mq);
    const float4 ms = q[DQ_MASS];
    const uint32_t fixed = uint32_t(ms.w);
    const float lf1 = mq[4 * DQ_LF1 + id.c], lf2 = mq[4 * DQ_LF2 + id.c];
    const float af1a = mq[4 * DQ_AF1 + id.c1], af1b = mq[4 * DQ_AF1 + id.c2];
    const float af2a = mq[4 * DQ_AF2 + id.c1], af2b = mq[4 * DQ_AF2 + id.c2];
    LaneVel u = lane_vel_load(b1, b2, wofs, id);
    bool resting_any = false;
#pragma unroll
    for (uint32_t k = 0; k < 4; k++) {
        if (k >= nbw) break;
        const float* p = pq + k * 4 * PREC_ROWS;
        const bool resting = p[4 * DP_ROWS + 2] != 0.0f;   // mut.z
        const float pi = imp[k];
        const float ip = p[4 * DP_N + id.c] * pi;
        LaneVel t;
        t.v1 = u.v1 - ms.x * ip * lf1;
        t.w1a = u.w1a - p[4 * DP_I1 + id.c1] * pi;
        t.w1b = u.w1b - p[4 * DP_I1 + id.c2] * pi;
        t.v2 = u.v2 + ms.y * ip * lf2;
        t.w2a = u.w2a + p[4 * DP_I2 + id.c1] * pi;
        t.w2b = u.w2b + p[4 * DP_I2 + id.c2] * pi;
        if (k < nb && resting) {
            u = t;
            resting_any = true;
        }
        if (k < nb && !resting) imp[k] = 0.0f;
    }
    if (__any_sync(0xffffffffu, resting_any)) {
        const LaneVel u0 = u;
        const v3 o1 = L3(q[DQ_OFV1]), o2 = L3(q[DQ_OFV2]);
        const v3 fv1 = L3(q[DQ_FV1]), fv2 = L3(q[DQ_FV2]), n = L3(q[DQ_N]);
        const v3 r1ct1 = L3(q[DQ_R1CT1]), r1ct2 = L3(q[DQ_R1CT2]), r2ct1 = L3(q[DQ_R2CT1]), r2ct2 = L3(q[DQ_R2CT2]);
        const float4 I1a = q[DQ_I1 + id.c1], I1b = q[DQ_I1 + id.c2], I2a = q[DQ_I2 + id.c1], I2b = q[DQ_I2 + id.c2];
        const v3 ofi = V(f[0] * o1.x + f[1] * o2.x, f[0] * o1.y + f[1] * o2.y, f[0] * o1.z + f[1] * o2.z);
        f[0] = vdot(ofi, fv1);
        f[1] = vdot(ofi, fv2);
        const float f1 = f[0], f2 = f[1], ftw = f[2];
        // first friction constraint
        v3 ai1 = V(-r1ct1.x * f1, -r1ct1.y * f1, -r1ct1.z * f1);
        float li2 = mq[4 * DQ_FV1 + id.c] * f1;
        v3 ai2 = V(r2ct1.x * f1, r2ct1.y * f1, r2ct1.z * f1);
        u.v1 = u.v1 - ms.x * li2 * lf1;
        u.w1a = u.w1a + af1a * row_dot(I1a, ai1); u.w1b = u.w1b + af1b * row_dot(I1b, ai1);
        u.v2 = u.v2 + ms.y * li2 * lf2;
        u.w2a = u.w2a + af2a * row_dot(I2a, ai2); u.w2b = u.w2b + af2b * row_dot(I2b, ai2);
        // second friction constraint
        ai1 = V(-r1ct2.x * f2, -r1ct2.y * f2, -r1ct2.z * f2);
        li2 = mq[4 * DQ_FV2 + id.c] * f2;
        ai2 = V(r2ct2.x * f2, r2ct2.y * f2, r2ct2.z * f2);
        u.v1 = u.v1 - ms.x * li2 * lf1;
        u.w1a = u.w1a + af1a * row_dot(I1a, ai1); u.w1b = u.w1b + af1b * row_dot(I1b, ai1);
        u.v2 = u.v2 + ms.y * li2 * lf2;
        u.w2a = u.w2a + af2a * row_dot(I2a, ai2); u.w2b = u.w2b + af2b * row_dot(I2b, ai2);
        // twist friction constraint (both bodies a second time, as warm_core)
        ai1 = V(-n.x * ftw, -n.y * ftw, -n.z * ftw);
        ai2 = V(n.x * ftw, n.y * ftw, n.z * ftw);
        u.w1a = u.w1a + af1a * row_dot(I1a, ai1); u.w1b = u.w1b + af1b * row_dot(I1b, ai1);
        u.w2a = u.w2a + af2a * row_dot(I2a, ai2); u.w2b = u.w2b + af2b * row_dot(I2b, ai2);
        u.w1a = u.w1a - af1a * row_dot(I1a, ai2); u.w1b = u.w1b - af1b * row_dot(I1b, ai2);
        u.w2a = u.w2a + af2a * row_dot(I2a, ai2); u.w2b = u.w2b + af2b * row_dot(I2b, ai2);
        if (!resting_any) u = u0;
    }
    if (!resting_any) f[0] = f[1] = f[2] = 0.0f;
    __syncwarp();   // every lane has read its share (lanes_solve: its shuffles)
    lane_vel_store(b1, b2, wofs, id, active && id.writer && id.role == 0, fixed, u);
}

// A point's rows as one lane needs them.
struct LanePt { float n, r1a, r1b, r2a, r2b, i1a, i1b, i2a, i2b, inv_mass, bias; };
RD LanePt lane_pt(const float* p, const LaneId& id) {
    LanePt t;
    t.r1a = p[4 * DP_R1 + id.c1]; t.r1b = p[4 * DP_R1 + id.c2];
    t.r2a = p[4 * DP_R2 + id.c1]; t.r2b = p[4 * DP_R2 + id.c2];
    t.n = p[4 * DP_N + id.c];
    t.bias = p[id.role ? 4 * DP_I1 + 3 : 4 * DP_N + 3];
    t.inv_mass = p[4 * DP_R2 + 3];
    t.i1a = p[4 * DP_I1 + id.c1]; t.i1b = p[4 * DP_I1 + id.c2];
    t.i2a = p[4 * DP_I2 + id.c1]; t.i2b = p[4 * DP_I2 + id.c2];
    return t;
}

// solve_core on eight lanes (split: the stage's split-impulse switch); imp[k]
// is the lane's role's impulse of point k.  A point's rows are read while the
// one before it is solved (a LaneSlot has rows for four points: those of
// points the manifold does not have are read and discarded).
RD void lanes_solve(bool split, const float* mq, const float* pq, uint32_t nb, uint32_t nbw, bool active,
                    const LaneId& id, float* b1, float* b2, uint32_t wofs, float (&imp)[4], float (&f)[3]) {
    const float4* q = reinterpret_cast<const float4*>(mq);
    LaneVel u = lane_vel_load(b1, b2, wofs, id);
    LanePt next = lane_pt(pq, id);
    const float4 ms = q[DQ_MASS];
    const uint32_t fixed = uint32_t(ms.w);
    const float lf1 = mq[4 * DQ_LF1 + id.c], lf2 = mq[4 * DQ_LF2 + id.c];
    float sum_pen = 0.0f;
#pragma unroll
    for (uint32_t k = 0; k < 4; k++) {
        if (k >= nbw) break;
        const LanePt p = next;
        const float dv = u.v2 + u.w2a * p.r2b - u.w2b * p.r2a - u.v1 - u.w1a * p.r1b + u.w1b * p.r1a;
        const float Jv = lanes_sum(dv * p.n);
        // (behind the shuffles, whose queue the reads share)
        if (k < 3) next = lane_pt(pq + (k + 1) * 4 * PREC_ROWS, id);
        float dl = -(Jv + p.bias) * p.inv_mass;
        const float sum = imp[k] + dl;
        const float now = (sum < 0.0f) ? 0.0f : sum;
        dl = now - imp[k];
        const float li = p.n * dl;
        LaneVel t;
        t.v1 = u.v1 - ms.x * li * lf1;
        t.w1a = u.w1a - p.i1a * dl; t.w1b = u.w1b - p.i1b * dl;
        t.v2 = u.v2 + ms.y * li * lf2;
        t.w2a = u.w2a + p.i2a * dl; t.w2b = u.w2b + p.i2b * dl;
        if (k < nb) {
            u = t;
            imp[k] = now;
            sum_pen += now;
        }
    }
    // the split half ends here: what it computes below is discarded
    const float af1a = mq[4 * DQ_AF1 + id.c1], af1b = mq[4 * DQ_AF1 + id.c2];
    const float af2a = mq[4 * DQ_AF2 + id.c1], af2b = mq[4 * DQ_AF2 + id.c2];
    const float t1 = mq[4 * DQ_FV1 + id.c], t2 = mq[4 * DQ_FV2 + id.c], nt = mq[4 * DQ_N + id.c1];
    const v3 r1ct1 = L3(q[DQ_R1CT1]), r1ct2 = L3(q[DQ_R1CT2]), r2ct1 = L3(q[DQ_R2CT1]), r2ct2 = L3(q[DQ_R2CT2]);
    const float4 I1a = q[DQ_I1 + id.c1], I1b = q[DQ_I1 + id.c2], I2a = q[DQ_I2 + id.c1], I2b = q[DQ_I2 + id.c2];
    const float f1a = mq[4 * DQ_R1F + id.c1], f1b = mq[4 * DQ_R1F + id.c2], inv_f1 = mq[4 * DQ_R1F + 3];
    const float f2a = mq[4 * DQ_R2F + id.c1], f2b = mq[4 * DQ_R2F + id.c2], inv_f2 = mq[4 * DQ_R2F + 3];
    const float4 nq = q[DQ_N];
    const LaneVel us = u;
    const float limit = ms.z * sum_pen;
    // first friction constraint
    {
        const float dv = u.v2 + u.w2a * f2b - u.w2b * f2a - u.v1 - u.w1a * f1b + u.w1b * f1a;
        float dl = -lanes_sum(dv * t1) * inv_f1;
        const float lt = f[0];
        f[0] = smax(-limit, smin(lt + dl, limit));
        dl = f[0] - lt;
        const v3 ai1 = V(-r1ct1.x * dl, -r1ct1.y * dl, -r1ct1.z * dl), ai2 = V(r2ct1.x * dl, r2ct1.y * dl, r2ct1.z * dl);
        const float li2 = t1 * dl;
        u.v1 = u.v1 - ms.x * li2 * lf1;
        u.w1a = u.w1a + af1a * row_dot(I1a, ai1); u.w1b = u.w1b + af1b * row_dot(I1b, ai1);
        u.v2 = u.v2 + ms.y * li2 * lf2;
        u.w2a = u.w2a + af2a * row_dot(I2a, ai2); u.w2b = u.w2b + af2b * row_dot(I2b, ai2);
    }
    // second friction constraint
    {
        const float dv = u.v2 + u.w2a * f2b - u.w2b * f2a - u.v1 - u.w1a * f1b + u.w1b * f1a;
        float dl = -lanes_sum(dv * t2) * inv_f2;
        const float lt = f[1];
        f[1] = smax(-limit, smin(lt + dl, limit));
        dl = f[1] - lt;
        const v3 ai1 = V(-r1ct2.x * dl, -r1ct2.y * dl, -r1ct2.z * dl), ai2 = V(r2ct2.x * dl, r2ct2.y * dl, r2ct2.z * dl);
        const float li2 = t2 * dl;
        u.v1 = u.v1 - ms.x * li2 * lf1;
        u.w1a = u.w1a + af1a * row_dot(I1a, ai1); u.w1b = u.w1b + af1b * row_dot(I1b, ai1);
        u.v2 = u.v2 + ms.y * li2 * lf2;
        u.w2a = u.w2a + af2a * row_dot(I2a, ai2); u.w2b = u.w2b + af2b * row_dot(I2b, ai2);
    }
    // twist friction constraint
    {
        const float Jv = lanes_sum_next((u.w2a - u.w1a) * nt);
        float dl = -Jv * nq.w;
        const float lt = f[2];
        f[2] = smax(-limit, smin(lt + dl, limit));
        dl = f[2] - lt;
        const v3 ai2 = V(nq.x * dl, nq.y * dl, nq.z * dl);
        u.w1a = u.w1a - af1a * row_dot(I1a, ai2); u.w1b = u.w1b - af1b * row_dot(I1b, ai2);
        u.w2a = u.w2a + af2a * row_dot(I2a, ai2); u.w2b = u.w2b + af2b * row_dot(I2b, ai2);
    }
    if (id.role) u = us;
    lane_vel_store(b1, b2, wofs, id, active && id.writer && (id.role == 0 || split), fixed, u);
}

// ---- level schedule of one island (one warp) --------------------------------
//
// A manifold's level is one more than the latest level of its movable bodies;
// every body of the island gets a slot for its velocities (fixed bodies too:
// their slots are read, never written back).  32 manifolds at a time: the
// lanes look their bodies up in a shared hash (compare-and-swap insertion; a
// slot's number follows the races, which decides where a velocity is staged
// and nothing else), then a 32-step shuffle scan settles the levels in
// manifold order, then a stable counting sort by level.  (One lane doing this
// serially took ~250 cycles a manifold.)
struct IslandSched {
    int32_t* hkey;        // H entries: body (-1 empty)
    uint32_t* hval;       // slot << 16 | last level
    int32_t* slot_body;   // nbmax: body of each slot, -1 - body when fixed
    short2* slot;         // per manifold: slot of body 1 / body 2
    uint16_t *klev, *order, *lev;   // level, level order, start of each level (lev[depth] = cnt)
    uint32_t H, nbmax;
    uint32_t* nslots;     // shared counter
};

RD uint32_t sched_find(const IslandSched& S, int32_t b, bool fixed, bool& ok) {
    uint32_t h = (uint32_t(b) * 2654435761u >> 12) & (S.H - 1);
    for (uint32_t probe = 0; probe < S.H; probe++, h = (h + 1) & (S.H - 1)) {
        const int32_t k = atomicCAS(S.hkey + h, -1, b);
        if (k == b) return h;
        if (k < 0) {
            const uint32_t s = atomicAdd(S.nslots, 1u);
            if (s >= S.nbmax) { ok = false; return h; }
            S.hval[h] = s << 16;
            S.slot_body[s] = fixed ? -1 - b : b;
            return h;
        }
    }
    ok = false;
    return 0;
}

// False (nothing written to global memory) when the island has more bodies
// than slots.
RD bool island_schedule(const DynArgs& a, uint32_t m0, uint32_t cnt, const IslandSched& S, uint32_t lane, uint32_t& depth) {
    for (uint32_t h = lane; h < S.H; h += 32) S.hkey[h] = -1;
    if (lane == 0) *S.nslots = 0;
    __syncwarp();
    depth = 0;
    bool ok = true;
    for (uint32_t base = 0; base < cnt; base += 32) {
        const uint32_t k = base + lane;
        int32_t b1 = -1, b2 = -1;   // movable bodies (the scan's keys)
        uint32_t h1 = 0, h2 = 0;
        bool used = false;
        if (k < cnt) {
            const int4 id = man_ids(a, m0 + k);
            if (id.z != 0) {
                const uint32_t fixed = man_fixed(a, m0 + k);
                used = true;
                h1 = sched_find(S, id.x, (fixed & 1u) != 0, ok);
                h2 = sched_find(S, id.y, (fixed & 2u) != 0, ok);
                b1 = (fixed & 1u) ? -1 : id.x;
                b2 = (fixed & 2u) ? -1 : id.y;
            }
        }
        if (__any_sync(0xffffffffu, !ok)) return false;
        __syncwarp();
        const uint32_t e1 = used ? S.hval[h1] : 0u, e2 = used ? S.hval[h2] : 0u;
        uint32_t l1 = b1 >= 0 ? e1 & 0xffffu : 0u, l2 = b2 >= 0 ? e2 & 0xffffu : 0u, L = 1;
        bool last1 = true, last2 = true;
        const uint32_t steps = cnt - base < 32 ? cnt - base : 32u;
        for (uint32_t j = 0; j < steps; j++) {
            if (lane == j) L = 1 + (l1 > l2 ? l1 : l2);
            const uint32_t Lj = __shfl_sync(0xffffffffu, L, int(j));
            const int32_t c1 = __shfl_sync(0xffffffffu, b1, int(j)), c2 = __shfl_sync(0xffffffffu, b2, int(j));
            const bool m1 = b1 >= 0 && (b1 == c1 || b1 == c2), m2 = b2 >= 0 && (b2 == c1 || b2 == c2);
            if (lane > j) {
                if (m1) l1 = Lj;
                if (m2) l2 = Lj;
            } else if (lane < j) {
                if (m1) last1 = false;
                if (m2) last2 = false;
            }
        }
        if (k < cnt) {
            if (b1 >= 0 && last1) S.hval[h1] = (e1 & 0xffff0000u) | L;
            if (b2 >= 0 && last2) S.hval[h2] = (e2 & 0xffff0000u) | L;
            S.slot[k] = used ? make_short2(short(e1 >> 16), short(e2 >> 16)) : make_short2(0, 0);
            S.klev[k] = uint16_t(L);
            depth = L > depth ? L : depth;
        }
        __syncwarp();
    }
    depth = __reduce_max_sync(0xffffffffu, depth);
    for (uint32_t L = lane; L <= depth; L += 32) S.lev[L] = 0;
    __syncwarp();
    const uint32_t lt = (1u << lane) - 1u;
    // manifolds per level (the lowest lane of a level's peers adds them), scan, scatter
    for (uint32_t base = 0; base < cnt; base += 32) {
        const uint32_t k = base + lane;
        const uint32_t L = k < cnt ? S.klev[k] : 0u;
        const uint32_t peers = __match_any_sync(0xffffffffu, L);
        if (k < cnt && (peers & lt) == 0) S.lev[L - 1] = uint16_t(S.lev[L - 1] + __popc(peers));
        __syncwarp();
    }
    uint32_t run = 0;
    for (uint32_t base = 0; base < depth; base += 32) {
        const uint32_t L = base + lane;
        const uint32_t v = L < depth ? S.lev[L] : 0u;
        uint32_t inc = v;
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t t = __shfl_up_sync(0xffffffffu, inc, o);
            if (lane >= uint32_t(o)) inc += t;
        }
        if (L < depth) S.lev[L] = uint16_t(run + inc - v);
        run += __shfl_sync(0xffffffffu, inc, 31);
    }
    __syncwarp();
    for (uint32_t base = 0; base < cnt; base += 32) {
        const uint32_t k = base + lane;
        const uint32_t L = k < cnt ? S.klev[k] : 0u;
        const uint32_t peers = __match_any_sync(0xffffffffu, L);
        const uint32_t at = k < cnt ? S.lev[L - 1] : 0u;
        __syncwarp();
        if (k < cnt) {
            S.order[at + __popc(peers & lt)] = uint16_t(k);
            if ((peers & lt) == 0) S.lev[L - 1] = uint16_t(at + __popc(peers));
        }
        __syncwarp();
    }
    // lev[L] is now the end of level L: shift to the starts
    for (uint32_t top = depth; top > 0;) {
        const uint32_t n = top < 32 ? top : 32u;   // positions top - n + 1 .. top take their predecessors' ends
        const uint32_t p = top - n + 1 + lane;
        const uint16_t v = lane < n ? S.lev[p - 1] : uint16_t(0);
        __syncwarp();
        if (lane < n) S.lev[p] = v;
        __syncwarp();
        top -= n;
    }
    if (lane == 0) S.lev[0] = 0;
    __syncwarp();
    return true;
}

// Shared memory of one warp of kernel 3b.
constexpr uint32_t STAGE_HASH = 512;   // open addressing over at most STAGE_BODIES bodies
struct __align__(16) WarpStage {
    float4 vel[4][STAGE_BODIES];        // constrained v, w and split v, w of the island's bodies
    union {
        struct {
            int32_t hkey[STAGE_HASH];
            uint32_t hval[STAGE_HASH];
            uint16_t klev[STAGE_MANIFOLDS];
            short2 slot[STAGE_MANIFOLDS];
        } s;                                 // while the schedule is built
        LaneSlot ring[2][WARP_MANIFOLDS];    // while it is solved
    };
    int4 desc[STAGE_MANIFOLDS];         // by level: slot 1 | slot 2 << 16, points, manifold (island index), first point
    uint16_t order[STAGE_MANIFOLDS];    // island manifolds sorted by level
    uint16_t lev[STAGE_MANIFOLDS + 8];  // start of each level
    int32_t slot_body[STAGE_BODIES];    // body of each slot (-1 - body: fixed)
    uint32_t nslots;
};
static_assert(sizeof(WarpStage) <= LARGE_WARP_SMEM, "warp stage");

// A level's manifolds are taken four at a time (a chunk: order[pos .. end)).
struct LaneChunk { uint32_t pos, end, L; };
RD LaneChunk chunk_next(const WarpStage* st, const LaneChunk& c, uint32_t depth, uint32_t& wrapped) {
    const bool level = c.pos + WARP_MANIFOLDS >= c.end;
    const uint32_t L = c.L + (level ? 1u : 0u);
    wrapped = L == depth ? 1u : 0u;
    LaneChunk n;
    n.L = wrapped ? 0u : L;
    const uint32_t first = st->lev[n.L];
    n.pos = level ? first : c.pos + WARP_MANIFOLDS;
    n.end = st->lev[n.L + 1];
    return n;
}
// A lane group's manifold of a chunk (desc row; no points: none) and its
// impulses, read one chunk ahead (only the manifold itself writes them): lane
// q of a half holds point q's and friction impulse q (q < 3).
struct LaneJob {
    int4 d;
    float imp, f;
};
// A group without a manifold gets the chunk's first one with no points: its
// loads and copies are valid and what they bring is discarded (no branches).
RD int4 chunk_desc(const WarpStage* st, const LaneChunk& c, const LaneId& id) {
    const uint32_t at = c.pos + id.group;
    int4 d = st->desc[at < c.end ? at : c.pos];
    d.y = at < c.end ? d.y : 0;
    return d;
}
RD void job_load(const DynArgs& a, uint32_t m0, const int4& d, const LaneId& id, LaneJob& j) {
    j.d = d;
    const uint32_t k = id.q < uint32_t(d.y) ? id.q : 0u;
    j.imp = reinterpret_cast<const float*>(&a.prec[uint32_t(d.w) + k].mut)[id.role];
    j.f = reinterpret_cast<const float*>(&a.mrec[m0 + uint32_t(d.z)].mut)[id.c];
}
// Each lane group stages its own manifold's rows (a lane past the last row
// copies the last row again).
RD void chunk_stage(const DynArgs& a, uint32_t m0, LaneSlot* slot, const int4& d, uint32_t lane) {
    const uint32_t sub = lane & 7u;
    const float4* mq = a.mrec[m0 + uint32_t(d.z)].q;
#pragma unroll
    for (uint32_t r = 0; r < DQ_ROWS; r += 8) {
        const uint32_t row = r + sub < DQ_ROWS ? r + sub : DQ_ROWS - 1;
        cp_async16(&slot->mq[row], mq + row);
    }
    const float4* pq = a.prec[d.w].q;
    const uint32_t last = (d.y ? uint32_t(d.y) : 1u) * PREC_ROWS - 1;
#pragma unroll
    for (uint32_t r = 0; r < 4 * PREC_ROWS; r += 8) {
        const uint32_t row = r + sub < last ? r + sub : last;
        cp_async16(&slot->pq[row], pq + row);
    }
    cp_async_commit();
}

// Whether an island's levels are wide: a warp takes four manifolds at a time
// with eight lanes each, 32 with one each, and such a round takes 2.2 times as
// long.  200 islands of 200 manifolds in two levels: 541 us with eight lanes,
// 339 with one; in 12 levels of 17: 591 and 452; 1,000 of 60 manifolds in ten
// levels (18 chunks of four): 403 with eight lanes, 514 with one.
RD bool wide_levels(const WarpStage* st, uint32_t depth, uint32_t lane) {
    uint32_t fours = 0, rounds = 0;
    for (uint32_t L = lane; L < depth; L += 32) {
        const uint32_t width = uint32_t(st->lev[L + 1]) - uint32_t(st->lev[L]);
        fours += (width + WARP_MANIFOLDS - 1) / WARP_MANIFOLDS;
        rounds += (width + 31u) / 32u;
    }
    return __reduce_add_sync(0xffffffffu, fours) > 2u * __reduce_add_sync(0xffffffffu, rounds);
}
// One lane a manifold, level after level, the rows from global memory.
RD void solve_staged_wide(const DynArgs& a, uint32_t m0, WarpStage* st, uint32_t lane, uint32_t depth) {
    for (int pass = 0; pass <= a.iterations; pass++)
        for (uint32_t L = 0; L < depth; L++) {
            for (uint32_t k = st->lev[L] + lane; k < st->lev[L + 1]; k += 32) {
                const int4 d = st->desc[k];
                const uint32_t s1 = uint32_t(d.x) & 0xffffu, s2 = uint32_t(d.x) >> 16;
                BodyVel bv;
                bv.v1 = &st->vel[0][s1]; bv.w1 = &st->vel[1][s1]; bv.s1 = &st->vel[2][s1]; bv.t1 = &st->vel[3][s1];
                bv.v2 = &st->vel[0][s2]; bv.w2 = &st->vel[1][s2]; bv.s2 = &st->vel[2][s2]; bv.t2 = &st->vel[3][s2];
                const RecSrc r = rec_global(a, m0 + uint32_t(d.z), d.w);
                if (pass == 0) warm_core<true>(a, r, bv, d.y);
                else solve_core<true>(a, r, bv, d.y);
            }
            __syncwarp();
        }
}
RD void staged_write_back(const DynArgs& a, const WarpStage* st, uint32_t lane) {
    for (uint32_t s = lane; s < st->nslots; s += 32) {
        const int32_t b = st->slot_body[s];
        if (b < 0) continue;
        a.cv[b] = st->vel[0][s]; a.cw[b] = st->vel[1][s];
        a.sv[b] = st->vel[2][s]; a.sw[b] = st->vel[3][s];
    }
}

// Solves a scheduled island from the warp's stage: the rows of the next
// chunk arrive by cp.async while a chunk is solved.
RD void solve_staged(const DynArgs& a, uint32_t m0, uint32_t cnt, WarpStage* st, uint32_t lane, uint32_t depth) {
    const uint32_t nslots = st->nslots;
    for (uint32_t s = lane; s < nslots; s += 32) {
        const int32_t e = st->slot_body[s], b = e < 0 ? -1 - e : e;
        st->vel[0][s] = a.cv[b]; st->vel[1][s] = a.cw[b];
        st->vel[2][s] = a.sv[b]; st->vel[3][s] = a.sw[b];
    }
    for (uint32_t k = lane; k < cnt; k += 32) {
        const uint32_t kk = st->order[k];
        const int4 id = man_ids(a, m0 + kk);
        const short2 sl = st->s.slot[kk];
        st->desc[k] = make_int4(int(uint32_t(uint16_t(sl.x)) | (uint32_t(uint16_t(sl.y)) << 16)), id.z, int(kk), id.w);
    }
    __syncwarp();   // the schedule's part of the union is free now
    if (wide_levels(st, depth, lane)) {
        solve_staged_wide(a, m0, st, lane, depth);
        staged_write_back(a, st, lane);
        return;
    }
    const LaneId id = lane_id(lane);
    float* vel = reinterpret_cast<float*>(st->vel[2 * id.role]);
    constexpr uint32_t wofs = 4 * STAGE_BODIES;
    LaneChunk c{0, st->lev[1], 0};
    // a pass of one chunk reads its impulses after they are stored
    const bool single = depth == 1 && cnt <= WARP_MANIFOLDS;
    int pass = 0;
    uint32_t buf = 0;
    LaneJob job, nxt;
    job_load(a, m0, chunk_desc(st, c, id), id, job);
    chunk_stage(a, m0, &st->ring[0][id.group], job.d, lane);
    uint32_t wrapped;
    c = chunk_next(st, c, depth, wrapped);
    int pass_n = int(wrapped);             // pass of the next chunk
    int4 dn = chunk_desc(st, c, id);       // its manifolds
    cp_async_wait<0>();
    __syncwarp();
    for (;;) {
        const bool more = pass_n <= a.iterations;
        if (more) chunk_stage(a, m0, &st->ring[buf ^ 1][id.group], dn, lane);
        if (more && !single) job_load(a, m0, dn, id, nxt);
        // the chunk after it, looked up while this one is solved
        c = chunk_next(st, c, depth, wrapped);
        const int pass_nn = pass_n + int(wrapped);
        const int4 dnn = chunk_desc(st, c, id);
        const LaneSlot* sl = &st->ring[buf][id.group];
        const float *mq = reinterpret_cast<const float*>(sl->mq), *pq = reinterpret_cast<const float*>(sl->pq);
        const uint32_t nb = uint32_t(job.d.y);
        const bool active = nb != 0;
        float *b1 = vel + 4 * (job.d.x & 0xffff), *b2 = vel + 4 * int(uint32_t(job.d.x) >> 16);
        float imp[4], f[3];
#pragma unroll
        for (int k = 0; k < 4; k++) imp[k] = __shfl_sync(0xffffffffu, job.imp, k, 4);
#pragma unroll
        for (int k = 0; k < 3; k++) f[k] = __shfl_sync(0xffffffffu, job.f, k, 4);
        const uint32_t nbw = __reduce_max_sync(0xffffffffu, nb);
        if (pass == 0) lanes_warm(mq, pq, nb, nbw, active, id, b1, b2, wofs, imp, f);
        else lanes_solve(a.split != 0, mq, pq, nb, nbw, active, id, b1, b2, wofs, imp, f);
        const bool keep = active && (id.role == 0 || (pass != 0 && a.split));
        st_global_if(keep && id.q < nb, reinterpret_cast<float*>(&a.prec[uint32_t(job.d.w) + id.q].mut) + id.role, lane_pick(id.q, imp));
        st_global_if(active && id.writer && id.role == 0, reinterpret_cast<float*>(&a.mrec[m0 + uint32_t(job.d.z)].mut) + id.c,
                     id.c == 0 ? f[0] : (id.c == 1 ? f[1] : f[2]));
        cp_async_wait<0>();
        __syncwarp();
        if (!more) break;
        if (single) job_load(a, m0, dn, id, nxt);
        pass = pass_n;
        pass_n = pass_nn;
        dn = dnn;
        buf ^= 1;
        job = nxt;
    }
    staged_write_back(a, st, lane);
}

RD bool schedule_staged(const DynArgs& a, uint32_t m0, uint32_t cnt, WarpStage* st, uint32_t lane, uint32_t& depth) {
    IslandSched S;
    S.hkey = st->s.hkey; S.hval = st->s.hval; S.H = STAGE_HASH;
    S.slot_body = st->slot_body; S.nbmax = STAGE_BODIES;
    S.slot = st->s.slot; S.klev = st->s.klev; S.order = st->order; S.lev = st->lev;
    S.nslots = &st->nslots;
    return island_schedule(a, m0, cnt, S, lane, depth);
}

// Islands too large for the stage: the same schedule in global scratch.
RD void solve_global(const DynArgs& a, uint32_t m0, uint32_t cnt, uint32_t lane) {
    uint32_t* __restrict__ ord = a.order + m0;
    uint32_t* __restrict__ lev = a.level + m0;
    uint32_t* __restrict__ blev = a.body_level;
    for (uint32_t k = lane; k < cnt; k += 32) {
        const int4 id = man_ids(a, m0 + k);
        if (id.z == 0) continue;
        const uint32_t fixed = man_fixed(a, m0 + k);
        if (!(fixed & 1)) blev[id.x] = 0;
        if (!(fixed & 2)) blev[id.y] = 0;
    }
    __syncwarp();
    uint32_t depth = 0;
    if (lane == 0) {
        for (uint32_t k = 0; k < cnt; k++) {
            const int4 id = man_ids(a, m0 + k);
            uint32_t L = 1;
            if (id.z != 0) {
                const uint32_t fixed = man_fixed(a, m0 + k);
                const uint32_t l1 = (fixed & 1) ? 0u : blev[id.x];
                const uint32_t l2 = (fixed & 2) ? 0u : blev[id.y];
                L = 1 + (l1 > l2 ? l1 : l2);
                if (!(fixed & 1)) blev[id.x] = L;
                if (!(fixed & 2)) blev[id.y] = L;
            }
            ord[k] = L;  // the level, until the scatter below
            depth = L > depth ? L : depth;
        }
        for (uint32_t L = 0; L < depth; L++) lev[L] = 0;
        for (uint32_t k = 0; k < cnt; k++) lev[ord[k] - 1]++;
        uint32_t run = 0;
        for (uint32_t L = 0; L < depth; L++) { run += lev[L]; lev[L] = run; }
        // keep the levels in the records' spare word while scattering
        for (uint32_t k = 0; k < cnt; k++) a.mrec[m0 + k].mut.w = __int_as_float(int32_t(ord[k]));
        for (uint32_t k = cnt; k-- > 0;) {
            const uint32_t L = uint32_t(__float_as_int(a.mrec[m0 + k].mut.w));
            ord[--lev[L - 1]] = k;
        }
    }
    depth = __shfl_sync(0xffffffffu, depth, 0);
    __syncwarp();
    for (int pass = 0; pass <= a.iterations; pass++) {
        for (uint32_t L = 0; L < depth; L++) {
            const uint32_t b = lev[L];
            const uint32_t e = (L + 1 < depth) ? lev[L + 1] : cnt;
            for (uint32_t k = b + lane; k < e; k += 32) {
                const uint32_t mi = m0 + ord[k];
                const int4 id = man_ids(a, mi);
                if (pass == 0) warm_manifold(a, mi, vel_global(a, id.x, id.y), id.z, id.w);
                else solve_manifold(a, mi, vel_global(a, id.x, id.y), id.z, id.w);
            }
            __syncwarp();
        }
    }
}

// Whether the islands of more than BIG_ISLAND manifolds go to kernel 3c with
// the giant ones: when there is a CTA for each of them.  A CTA takes a level
// of up to 16 manifolds in one round (a warp four a round) and a chain's level
// in 1,273-1,841 cycles (a warp 1,697-2,141).
RD bool big_on_ctas(const DynArgs& a) {
    return a.giant_auto && a.giant_smem && a.counters[3] + a.counters[0] <= a.giant_ctas;
}
// Whether the giant islands that fit a warp's stage go to kernel 3b: when there
// are more of them than CTAs of kernel 3c (one each): 300 chains of 300
// manifolds took 6.4 ms as CTAs (three rounds of 148), 2.7 ms as warps; 148 or
// fewer are faster as CTAs.
RD bool giants_on_warps(const DynArgs& a) { return a.giant_auto && a.counters[3] > a.giant_ctas; }

__global__ void __launch_bounds__(LARGE_WARPS * 32, 2) dyn_islands_large(const DynArgs a) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const uint32_t wid = threadIdx.x >> 5, lane = threadIdx.x & 31;
    WarpStage* st = reinterpret_cast<WarpStage*>(smem_raw + size_t(wid) * LARGE_WARP_SMEM);
    // the longest work first
    const uint32_t n_giant = giants_on_warps(a) ? a.counters[3] : 0u;
    const uint32_t n_big = big_on_ctas(a) ? 0u : a.counters[0], n_mid = a.counters[2];
    uint32_t solved = 0;
    for (;;) {
        uint32_t k = 0;
        if (lane == 0) k = atomicAdd(a.counters + 1, 1u);
        k = __shfl_sync(0xffffffffu, k, 0);
        if (k >= n_giant + n_big + n_mid) break;
        const bool giant = k < n_giant;
        const uint32_t j = k - n_giant;
        const uint32_t is = giant ? a.giant_list[k] : (j < n_big ? a.large_list[j] : a.large_list[a.ni - 1 - (j - n_big)]);
        const uint32_t m0 = a.i_start[is], cnt = a.i_count[is];
        uint32_t depth = 0;
        if (cnt <= STAGE_MANIFOLDS && schedule_staged(a, m0, cnt, st, lane, depth)) {
            solve_staged(a, m0, cnt, st, lane, depth);
            if (giant && lane == 0) a.giant_list[k] = ISLAND_DONE;
        } else if (giant) {
            __syncwarp();
            continue;   // kernel 3c takes it
        } else {
            solve_global(a, m0, cnt, lane);
        }
        __syncwarp();
        for (uint32_t i = lane; i < cnt; i += 32) store_manifold(a, m0 + i);
        solved++;
        __syncwarp();
    }
    if (lane == 0 && solved) atomicAdd(a.counters + 8, solved);
}


}  // namespace
}  // namespace rp3dg
#include "joints.cuh"
namespace rp3dg {
namespace {

// ---- kernel 3e: islands with joints --------------------------------------
//
// One thread per island, in the reference's order: the contact warm start
// (ContactSolverSystem::init), the joints' warm start
// (ConstraintSolverSystem::initialize: ball-and-socket, then hinge), then per
// velocity iteration the joints (solveVelocityConstraints) before the
// contacts (ContactSolverSystem::solve), and storeImpulses.
// The island of a thread when a warp takes `lanes` islands (items_per_warp),
// or none.  643 islands on 643 warps instead of 21: the solver's kernel 256 ->
// 94 us, the position correction 246 -> 164 us.
RD uint32_t joint_island(uint32_t lanes) {
    const uint32_t lane = threadIdx.x & 31u;
    return lane < lanes ? (blockIdx.x * 2u + (threadIdx.x >> 5)) * lanes + lane : 0xffffffffu;
}
__global__ void __launch_bounds__(128) dyn_joints_init(const DynArgs a) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < a.nj) joint_init(a, a.j_list[i]);
}

__global__ void __launch_bounds__(64) dyn_islands_joint(const DynArgs a, uint32_t lanes) {
    const uint32_t k = joint_island(lanes);
    if (k >= a.nji) return;
    const uint32_t is = a.ji_island[k];
    const uint32_t m0 = a.i_start[is], cnt = a.i_count[is];
    const uint32_t j0 = a.i_jstart[is], jn = a.i_jcount[is];
    if (m0 > a.nm || cnt > a.nm - m0 || j0 > a.nj || jn > a.nj - j0) {
        atomicOr(a.error, 4u);
        return;
    }
    for (uint32_t mi = m0; mi < m0 + cnt; mi++) {
        const int4 id = man_ids(a, mi);
        warm_manifold(a, mi, vel_global(a, id.x, id.y), id.z, id.w);
    }
    for (uint32_t j = j0; j < j0 + jn; j++) joint_warm(a, a.j_list[j]);
    for (int it = 0; it < a.iterations; it++) {
        for (uint32_t j = j0; j < j0 + jn; j++) joint_solve(a, a.j_list[j]);
        for (uint32_t mi = m0; mi < m0 + cnt; mi++) {
            const int4 id = man_ids(a, mi);
            solve_manifold(a, mi, vel_global(a, id.x, id.y), id.z, id.w);
        }
    }
    for (uint32_t mi = m0; mi < m0 + cnt; mi++) store_manifold(a, mi);
}

// ---- kernel 4b: position correction of the joints (solvePositionCorrection,
// PhysicsWorld.cpp:348-360) and updateBodiesState (DynamicsSystem.cpp:74-110)
// of the islands with joints.
__global__ void __launch_bounds__(64) dyn_joints_position(const DynArgs a, uint32_t lanes) {
    const uint32_t k = joint_island(lanes);
    if (k >= a.nji) return;
    const uint32_t is = a.ji_island[k];
    const uint32_t j0 = a.i_jstart[is], jn = a.i_jcount[is];
    if (j0 > a.nj || jn > a.nj - j0) return;
    for (int it = 0; it < a.position_iterations; it++)
        for (uint32_t j = j0; j < j0 + jn; j++) joint_position(a, a.j_list[j]);
    for (uint32_t r = a.ji_bstart[k]; r < a.ji_bstart[k] + a.ji_bcount[k]; r++) {
        const int32_t i = a.ji_rows[r];
        const v3 cp = L3(a.xc[i]);
        const float4 c4 = a.qc[i];
        const quat co = Q(c4.x, c4.y, c4.z, c4.w);
        a.com_world[i] = F4(cp);
        const float len = sqrtf(co.x * co.x + co.y * co.y + co.z * co.z + co.w * co.w);
        const quat u = Q(co.x / len, co.y / len, co.z / len, co.w / len);
        a.orientation[i] = make_float4(u.x, u.y, u.z, u.w);
        const v3 rr = qrot(u, L3(a.com_local[i]));
        a.position[i] = F4(V(cp.x - rr.x, cp.y - rr.y, cp.z - rr.z));
    }
}

// ---- kernel 3c: large islands, a CTA each ---------------------------------
//
// One CTA of five warps takes one island at a time with the CTA's whole opt-in
// shared memory: the bodies' velocities, every manifold's and point's impulses,
// the manifold table and the level schedule (island_schedule, by warp 0) stay
// on chip for the warm start and all velocity iterations.  Warp 0 then stages
// the constant rows of the first GIANT_RING manifolds (and their points) of
// level t + 2 into a three-level ring with cp.async, with a compact descriptor
// per manifold, while warps 1 to 4 solve level t, four manifolds each on eight
// lanes a manifold (lanes_warm / lanes_solve); manifolds of a level beyond the
// ring go one a lane with their rows from global memory (warm_core /
// solve_core).  The warps meet at one named barrier per level.  An island that
// does not fit, or whose points are not one range, is queued for kernel 3d.
// The first solver warp, which every level needs, does not share the staging
// warp's scheduler (the fourth does).
constexpr uint32_t GIANT_SOLVERS = 4;
constexpr uint32_t GIANT_RING = GIANT_SOLVERS * WARP_MANIFOLDS;   // manifolds of a level staged (the first 16)
constexpr uint32_t GIANT_LEVELS = 3;   // levels in the ring
constexpr uint32_t GIANT_THREADS = (GIANT_SOLVERS + 1) * 32;
struct __align__(16) GiantSlot {
    int4 desc;                         // 16 * slot 1, 16 * slot 2, points | manifold (island index) << 8, first point
    LaneSlot rows;
};
// named barrier 1 over the CTA's warps
template <uint32_t THREADS>
RD void cta_bar() { asm volatile("bar.sync 1, %0;\n" ::"n"(THREADS) : "memory"); }

// A level of the ring: its first position in the level order and its width,
// the largest point count of each solver warp's manifolds (0: nothing to do).
struct __align__(16) GiantLevel {
    uint32_t first, width, pad[2];
    uint32_t nbw[GIANT_SOLVERS];
    GiantSlot slot[GIANT_RING];
};

// The CTA's dynamic shared memory at a byte offset.
template <class T>
RD T* gsh(uint32_t off) {
    extern __shared__ __align__(16) unsigned char gsm[];
    return reinterpret_cast<T*>(gsm + off);
}
// Byte offsets of an island's arrays in the CTA's shared memory (offsets, not
// pointers: every access is then a shared-memory access to the compiler).
struct GiantStage {
    uint32_t vel;          // float4 x 4 nbmax: constrained v, w, split v, w
    uint32_t mmut;         // float4 a manifold: friction impulses
    uint32_t pmut;         // float2 a point: penetration impulse, split impulse
    uint32_t ring;         // GiantLevel x GIANT_LEVELS
    uint32_t hkey, hval, slot_body;
    uint32_t slot;         // short2: slots of body 1 / body 2
    uint32_t order, klev, lev;   // uint16
    uint32_t pofs;         // uint32: first point of each manifold, relative to the island's first point
    uint32_t npt;          // uint8
    uint32_t H, nbmax;
};

RD bool giant_layout(const DynArgs& a, uint32_t cnt, uint32_t np, GiantStage& g) {
    if (cnt > 65535u) return false;
    g.nbmax = 2 * cnt < a.nb ? 2 * cnt : a.nb;
    if (g.nbmax > 32767u) return false;
    g.H = 1;
    while (g.H < 2 * g.nbmax) g.H <<= 1;
    size_t off = 0;
    auto take = [&](size_t bytes) { const size_t o = off; off = (off + bytes + 15) & ~size_t(15); return uint32_t(o); };
    g.vel = take(size_t(4) * g.nbmax * 16);
    g.mmut = take(size_t(cnt) * 16);
    g.pmut = take(size_t(np) * 8);
    g.ring = take(size_t(GIANT_LEVELS) * sizeof(GiantLevel));
    g.hkey = take(size_t(g.H) * 4);
    g.hval = take(size_t(g.H) * 4);
    g.slot_body = take(size_t(g.nbmax) * 4);
    g.slot = take(size_t(cnt) * 4);
    g.order = take(size_t(cnt) * 2);
    g.klev = take(size_t(cnt) * 2);
    g.lev = take(size_t(cnt + 1) * 2);
    g.pofs = take(size_t(cnt) * 4);
    g.npt = take(size_t(cnt));
    return off <= a.giant_smem;
}

// Schedule an island (warp 0); false (nothing written to global memory) when
// it does not fit or its points are not one contiguous range.
RD bool giant_schedule(const DynArgs& a, uint32_t m0, uint32_t cnt, GiantStage& g,
                       uint32_t lane, uint32_t& depth, uint32_t* nslots, uint32_t& p0) {
    const int4 f = man_ids(a, m0), l = man_ids(a, m0 + cnt - 1);
    p0 = uint32_t(f.w);
    const int64_t end = int64_t(l.w) + int64_t(l.z);
    if (f.w < 0 || end < int64_t(p0) || end > int64_t(a.np)) return false;
    const uint32_t np = uint32_t(end - int64_t(p0));
    if (!giant_layout(a, cnt, np, g)) return false;
    uint32_t expect = 0;
    for (uint32_t base = 0; base < cnt; base += 32) {
        const uint32_t k = base + lane;
        uint32_t pofs = 0, npt = 0;
        if (k < cnt) {
            const int4 id = man_ids(a, m0 + k);
            pofs = uint32_t(id.w) - p0;
            npt = uint32_t(id.z < 0 ? 0 : (id.z > 255 ? 255 : id.z));
            gsh<uint32_t>(g.pofs)[k] = pofs;
            gsh<uint8_t>(g.npt)[k] = uint8_t(npt);
        }
        uint32_t inc = npt;
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t t = __shfl_up_sync(0xffffffffu, inc, o);
            if (lane >= uint32_t(o)) inc += t;
        }
        if (__any_sync(0xffffffffu, k < cnt && (npt > 4 || pofs != expect + inc - npt))) return false;
        expect += __shfl_sync(0xffffffffu, inc, 31);
    }
    if (expect != np) return false;
    IslandSched S;
    S.hkey = gsh<int32_t>(g.hkey); S.hval = gsh<uint32_t>(g.hval); S.H = g.H;
    S.slot_body = gsh<int32_t>(g.slot_body); S.nbmax = g.nbmax;
    S.slot = gsh<short2>(g.slot); S.klev = gsh<uint16_t>(g.klev); S.order = gsh<uint16_t>(g.order); S.lev = gsh<uint16_t>(g.lev);
    S.nslots = nslots;
    return island_schedule(a, m0, cnt, S, lane, depth);
}

// Staging warp: the next level of the linearised passes x levels (cursor S)
// into its ring level.  Lane s < 16 looks its manifold up; then the whole warp
// copies slot after slot, two rows a lane.
struct GiantCursor { uint32_t t, L, ring; };
RD void giant_stage_level(const DynArgs& a, const GiantStage& g, uint32_t m0, uint32_t p0, uint32_t depth,
                          uint32_t total, GiantCursor& S, uint32_t lane) {
    if (S.t < total) {
        const uint16_t* lev = gsh<uint16_t>(g.lev);
        const uint32_t first = lev[S.L], width = lev[S.L + 1] - first;
        GiantLevel* R = gsh<GiantLevel>(g.ring) + S.ring;
        uint32_t kk = 0, np = 0, pofs = 0;
        if (lane < GIANT_RING && lane < width) {
            kk = gsh<uint16_t>(g.order)[first + lane];
            const short2 bs = gsh<short2>(g.slot)[kk];
            np = gsh<uint8_t>(g.npt)[kk];
            pofs = gsh<uint32_t>(g.pofs)[kk];
            R->slot[lane].desc = make_int4(16 * int(bs.x), 16 * int(bs.y), int(np | kk << 8), int(pofs));
        }
        const uint32_t n = width < GIANT_RING ? width : GIANT_RING;
        for (uint32_t s = 0; s < n; s++) {
            const uint32_t ks = __shfl_sync(0xffffffffu, kk, int(s)), ns = __shfl_sync(0xffffffffu, np, int(s));
            const uint32_t ps = __shfl_sync(0xffffffffu, pofs, int(s));
            const float4* mq = a.mrec[m0 + ks].q;
            const float4* pq = a.prec[ns ? p0 + ps : 0u].q;
            float4* dst = R->slot[s].rows.mq;   // the point rows follow the manifold's
            const uint32_t rows = DQ_ROWS + ns * PREC_ROWS;
            // (a lane past the last row copies the last row again)
            const uint32_t r0 = lane < rows ? lane : rows - 1, r1 = lane + 32 < rows ? lane + 32 : rows - 1;
            cp_async16(dst + r0, r0 < DQ_ROWS ? mq + r0 : pq + (r0 - DQ_ROWS));
            cp_async16(dst + r1, r1 < DQ_ROWS ? mq + r1 : pq + (r1 - DQ_ROWS));
        }
        uint32_t w = np;
        for (int o = 1; o < int(WARP_MANIFOLDS); o <<= 1) {
            const uint32_t v = __shfl_xor_sync(0xffffffffu, w, o);
            w = v > w ? v : w;
        }
        if (lane < GIANT_RING && lane % WARP_MANIFOLDS == 0) R->nbw[lane / WARP_MANIFOLDS] = w;
        if (lane == 0) { R->first = first; R->width = width; }
        S.t++;
        if (++S.L == depth) S.L = 0;
        if (++S.ring == GIANT_LEVELS) S.ring = 0;
    }
    cp_async_commit();
}

// A lane group's staged manifold of a level, its impulses in shared memory.
RD void giant_manifold(const DynArgs& a, const GiantStage& g, const LaneId& id, bool warm, const GiantSlot* sl,
                       int4 d, bool active, uint32_t nbw) {
    d.x = active ? d.x : 0; d.y = active ? d.y : 0; d.z = active ? d.z : 0; d.w = active ? d.w : 0;
    const uint32_t nb = uint32_t(d.z) & 255u;
    active = nb != 0;
    const uint32_t vel = g.vel + 32 * g.nbmax * id.role;
    float *b1 = gsh<float>(vel + uint32_t(d.x)), *b2 = gsh<float>(vel + uint32_t(d.y));
    const uint32_t wofs = 4 * g.nbmax;
    float* pm = gsh<float>(g.pmut + 8 * uint32_t(d.w) + 4 * id.role);
    float* mm = gsh<float>(g.mmut + (uint32_t(d.z) >> 8 << 4));
    const float *mq = reinterpret_cast<const float*>(sl->rows.mq), *pq = reinterpret_cast<const float*>(sl->rows.pq);
    float imp[4], f[3];
    // a point's impulse behind the island's last is the next array's: read and discarded
#pragma unroll
    for (uint32_t k = 0; k < 4; k++) imp[k] = pm[2 * k];
    f[0] = mm[0]; f[1] = mm[1]; f[2] = mm[2];
    if (warm) lanes_warm(mq, pq, nb, nbw, active, id, b1, b2, wofs, imp, f);
    else lanes_solve(a.split != 0, mq, pq, nb, nbw, active, id, b1, b2, wofs, imp, f);
    const bool keep = active && (id.role == 0 || (!warm && a.split));
    st_shared_if(keep && id.q < nb, pm + 2 * id.q, lane_pick(id.q, imp));
    st_shared_if(active && id.writer && id.role == 0, mm + id.c, id.c == 0 ? f[0] : (id.c == 1 ? f[1] : f[2]));
}

// All warps: stage, solve and write back one island.
RD void giant_solve(const DynArgs& a, uint32_t m0, uint32_t cnt, const GiantStage& g, uint32_t warp,
                    uint32_t lane, uint32_t depth, uint32_t nslots, uint32_t p0) {
    const uint32_t np = gsh<uint32_t>(g.pofs)[cnt - 1] + gsh<uint8_t>(g.npt)[cnt - 1];
    const uint32_t tid = warp * 32 + lane;
    float4 *vel = gsh<float4>(g.vel), *mmut = gsh<float4>(g.mmut);
    float2* pmut = gsh<float2>(g.pmut);
    const int32_t* slot_body = gsh<int32_t>(g.slot_body);
    for (uint32_t s = tid; s < nslots; s += GIANT_THREADS) {
        const int32_t e = slot_body[s], b = e < 0 ? -1 - e : e;
        vel[s] = a.cv[b];
        vel[g.nbmax + s] = a.cw[b];
        vel[2 * g.nbmax + s] = a.sv[b];
        vel[3 * g.nbmax + s] = a.sw[b];
    }
    for (uint32_t k = tid; k < cnt; k += GIANT_THREADS) mmut[k] = a.mrec[m0 + k].mut;
    for (uint32_t p = tid; p < np; p += GIANT_THREADS) {
        const float4 v = a.prec[p0 + p].mut;
        pmut[p] = make_float2(v.x, v.y);
    }
    const uint32_t total = uint32_t(a.iterations + 1) * depth;
    if (warp == 0) {
        GiantCursor S{0, 0, 0};
        giant_stage_level(a, g, m0, p0, depth, total, S, lane);
        giant_stage_level(a, g, m0, p0, depth, total, S, lane);
        cp_async_wait<1>();
        cta_bar<GIANT_THREADS>();          // level 0 staged, stage loads done
        for (uint32_t t = 0; t < total; t++) {
            giant_stage_level(a, g, m0, p0, depth, total, S, lane);   // level t + 2
            cp_async_wait<1>();            // level t + 1 staged
            cta_bar<GIANT_THREADS>();      // end of level t
        }
        cp_async_wait<0>();
    } else {
        const LaneId id = lane_id(lane);
        const uint32_t solver = warp - 1;
        cta_bar<GIANT_THREADS>();
        uint32_t ring = 0;
        for (uint32_t t = 0; t < total; t++) {
            const bool warm = t < depth;
            const GiantLevel* R = gsh<GiantLevel>(g.ring) + ring;
            const uint32_t at = solver * WARP_MANIFOLDS + id.group;
            const uint32_t nbw = R->nbw[solver], b = R->first, width = R->width, e = b + width;
            const int4 d = R->slot[at].desc;
            if (nbw) giant_manifold(a, g, id, warm, &R->slot[at], d, at < width, nbw);
            // a level's manifolds beyond the staged ones: one a lane, their rows
            // from global memory
            if (width > GIANT_RING)
            for (uint32_t j = b + GIANT_RING + solver * 32 + lane; j < e; j += GIANT_SOLVERS * 32) {
                const uint32_t kk = gsh<uint16_t>(g.order)[j], npt = gsh<uint8_t>(g.npt)[kk], pofs = gsh<uint32_t>(g.pofs)[kk];
                const short2 bs = gsh<short2>(g.slot)[kk];
                BodyVel bv;
                const uint32_t n = g.nbmax;
                bv.v1 = vel + bs.x; bv.w1 = bv.v1 + n; bv.s1 = bv.w1 + n; bv.t1 = bv.s1 + n;
                bv.v2 = vel + bs.y; bv.w2 = bv.v2 + n; bv.s2 = bv.w2 + n; bv.t2 = bv.s2 + n;
                RecSrc r = rec_global(a, m0 + kk, int32_t(npt ? p0 + pofs : 0u));
                r.mmut = mmut + kk;
                r.pm2 = pmut + pofs;
                if (warm) warm_core<true, true>(a, r, bv, int32_t(npt));
                else solve_core<true, true>(a, r, bv, int32_t(npt));
            }
            __syncwarp();
            cta_bar<GIANT_THREADS>();
            if (++ring == GIANT_LEVELS) ring = 0;
        }
    }
    __syncthreads();
    for (uint32_t s = tid; s < nslots; s += GIANT_THREADS) {
        const int32_t b = slot_body[s];
        if (b < 0) continue;
        a.cv[b] = vel[s];
        a.cw[b] = vel[g.nbmax + s];
        a.sv[b] = vel[2 * g.nbmax + s];
        a.sw[b] = vel[3 * g.nbmax + s];
    }
    for (uint32_t k = tid; k < cnt; k += GIANT_THREADS) a.mrec[m0 + k].mut = mmut[k];
    for (uint32_t p = tid; p < np; p += GIANT_THREADS) {
        float* mut = reinterpret_cast<float*>(&a.prec[p0 + p].mut);
        const float2 v = pmut[p];
        mut[0] = v.x;
        mut[1] = v.y;
    }
    __syncthreads();
}

// ---- islands too large for shared memory: streamed ---------------------
//
// The level schedule is built by warp 0 in global scratch, 32 manifolds at a
// time: the lanes load their manifolds' bodies and the bodies' last levels in
// parallel, then a 32-step shuffle scan settles the dependencies inside the
// chunk in manifold order (a manifold's level is one more than the latest
// level of its movable bodies, exactly as the sequential rule).  A stable
// counting sort by level follows (histogram, scan, scatter with per-level
// ranks from __match_any_sync).  The solve is the giant pipeline with the
// island state left in global memory: warp 1 stages the constant rows of up
// to 32 manifolds per level two levels ahead, warp 0 solves each level from
// the ring with the velocities and impulses read from and written to global
// memory; both warps meet at the named barrier once per level.
constexpr uint32_t STREAM_RING = 32;
constexpr uint32_t STREAM_THREADS = 64;
using StreamSlot = GiantSlot;          // desc: unused, points, manifold (island index), first point

// Warp 0: levels and the level-ordered manifolds of an island.  Writes
// a.order[m0 + i] (island-relative manifold indices in level order) and
// a.level[m0 + L] = end of level L in that order; returns the depth.
RD uint32_t stream_schedule(const DynArgs& a, uint32_t m0, uint32_t cnt, uint32_t lane) {
    uint32_t* __restrict__ ord = a.order + m0;
    uint32_t* __restrict__ lev = a.level + m0;
    uint32_t* __restrict__ blev = a.body_level;
    for (uint32_t k = lane; k < cnt; k += 32) {
        const int4 id = man_ids(a, m0 + k);
        if (id.z == 0) continue;
        const uint32_t fixed = man_fixed(a, m0 + k);
        if (!(fixed & 1)) blev[id.x] = 0;
        if (!(fixed & 2)) blev[id.y] = 0;
    }
    __syncwarp();
    uint32_t depth = 0;
    for (uint32_t base = 0; base < cnt; base += 32) {
        const uint32_t k = base + lane;
        int32_t b1 = -1, b2 = -1;
        if (k < cnt) {
            const int4 id = man_ids(a, m0 + k);
            if (id.z != 0) {
                const uint32_t fixed = man_fixed(a, m0 + k);
                b1 = (fixed & 1) ? -1 : id.x;
                b2 = (fixed & 2) ? -1 : id.y;
            }
        }
        uint32_t l1 = b1 >= 0 ? blev[b1] : 0u, l2 = b2 >= 0 ? blev[b2] : 0u, L = 1;
        bool last1 = true, last2 = true;
        for (uint32_t j = 0; j < 32; j++) {
            if (lane == j) L = 1 + (l1 > l2 ? l1 : l2);
            const uint32_t Lj = __shfl_sync(0xffffffffu, L, int(j));
            const int32_t c1 = __shfl_sync(0xffffffffu, b1, int(j)), c2 = __shfl_sync(0xffffffffu, b2, int(j));
            const bool m1 = b1 >= 0 && (b1 == c1 || b1 == c2), m2 = b2 >= 0 && (b2 == c1 || b2 == c2);
            if (lane > j) {
                if (m1) l1 = Lj;
                if (m2) l2 = Lj;
            } else if (lane < j) {
                if (m1) last1 = false;
                if (m2) last2 = false;
            }
        }
        if (k < cnt) {
            if (b1 >= 0 && last1) blev[b1] = L;
            if (b2 >= 0 && last2) blev[b2] = L;
            // the level, kept in the record's spare word until the scatter
            a.mrec[m0 + k].mut.w = __int_as_float(int32_t(L));
            depth = L > depth ? L : depth;
        }
        __syncwarp();
    }
    for (int o = 16; o > 0; o >>= 1) {
        const uint32_t d = __shfl_xor_sync(0xffffffffu, depth, o);
        depth = d > depth ? d : depth;
    }
    // counting sort by level, stable in manifold order
    for (uint32_t L = lane; L < depth; L += 32) lev[L] = 0;
    __syncwarp();
    for (uint32_t k = lane; k < cnt; k += 32)
        atomicAdd(lev + (uint32_t(__float_as_int(a.mrec[m0 + k].mut.w)) - 1), 1u);
    __syncwarp();
    uint32_t run = 0;
    for (uint32_t base = 0; base < depth; base += 32) {
        const uint32_t L = base + lane;
        const uint32_t v = L < depth ? lev[L] : 0u;
        uint32_t inc = v;
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t t = __shfl_up_sync(0xffffffffu, inc, o);
            if (lane >= uint32_t(o)) inc += t;
        }
        if (L < depth) lev[L] = run + inc - v;   // first position of level L
        run += __shfl_sync(0xffffffffu, inc, 31);
    }
    __syncwarp();
    const uint32_t lt = (1u << lane) - 1u;
    for (uint32_t base = 0; base < cnt; base += 32) {
        const uint32_t k = base + lane;
        const uint32_t L = k < cnt ? uint32_t(__float_as_int(a.mrec[m0 + k].mut.w)) : 0u;
        const uint32_t key = k < cnt ? L : (0x80000000u | lane);
        const uint32_t peers = __match_any_sync(0xffffffffu, key);
        const uint32_t pos = k < cnt ? lev[L - 1] + uint32_t(__popc(peers & lt)) : 0u;
        __syncwarp();
        if (k < cnt) {
            ord[pos] = k;
            // the lowest lane of a level advances its cursor past the chunk's peers
            if ((peers & lt) == 0) lev[L - 1] += uint32_t(__popc(peers));
        }
        __syncwarp();
    }
    // lev[L] is now the end of level L
    return depth;
}

// Warp 1's staging pipeline: for linearised level x (passes x levels) it
// loads the level's bounds three steps ahead, the lanes' manifold indices two
// steps ahead and their id rows one step ahead, and issues the cp.async
// copies of the rows at x, so that no stage waits on a load issued in the
// same step; the registers then shift by one level.
struct StreamPipe {
    int2 b0, b1, b2;   // bounds of levels x, x + 1, x + 2
    uint32_t k0, k1;   // the lane's manifold of levels x, x + 1 (~0u: none)
    int4 i0;           // the id row of k0
};
RD int2 stream_bounds(const DynArgs& a, uint32_t m0, uint32_t depth, int64_t total, int64_t x) {
    if (x < 0 || x >= total) return make_int2(0, 0);
    const uint32_t L = uint32_t(x) % depth;
    return make_int2(int(L ? a.level[m0 + L - 1] : 0u), int(a.level[m0 + L]));
}
RD uint32_t stream_kk(const DynArgs& a, uint32_t m0, int2 bd, uint32_t lane) {
    const uint32_t j = uint32_t(bd.x) + lane;
    return (lane < STREAM_RING && j < uint32_t(bd.y)) ? a.order[m0 + j] : ~0u;
}

// One pipeline step for level x (negative in the prologue: loads only); the
// header of level x (its bounds) goes to hdr[x % 3] for warp 0.
RD void stream_stage_step(const DynArgs& a, StreamSlot* ring, int2* hdr, StreamPipe& P, uint32_t m0, uint32_t depth,
                          int64_t total, int64_t x, uint32_t lane) {
    const int2 nb3 = stream_bounds(a, m0, depth, total, x + 3);
    const uint32_t nk2 = stream_kk(a, m0, P.b2, lane);
    int4 ni1 = make_int4(0, 0, 0, 0);
    if (P.k1 != ~0u) ni1 = man_ids(a, m0 + P.k1);
    if (x >= 0 && x < total) {
        if (lane == 0) hdr[uint32_t(x) % GIANT_LEVELS] = P.b0;
        if (P.k0 != ~0u) {
            const uint32_t np = P.i0.z < 0 ? 0u : (P.i0.z > 4 ? 4u : uint32_t(P.i0.z));
            StreamSlot* sl = ring + (uint32_t(x) % GIANT_LEVELS) * STREAM_RING + lane;
            sl->desc = make_int4(0, int(np), int(P.k0), P.i0.w);
            const float4* src = a.mrec[m0 + P.k0].q;
            for (int r = 0; r < DQ_ROWS; r++) cp_async16(&sl->rows.mq[r], src + r);
            const float4* ps = a.prec[P.i0.w].q;
            for (uint32_t r = 0; r < np * PREC_ROWS; r++) cp_async16(&sl->rows.pq[r], ps + r);
        }
    }
    if (x >= 0) cp_async_commit();
    P.b0 = P.b1;
    P.b1 = P.b2;
    P.b2 = nb3;
    P.k0 = P.k1;
    P.k1 = nk2;
    P.i0 = ni1;
}

// Both warps: warm start and velocity iterations of a scheduled island.
RD void stream_solve(const DynArgs& a, uint32_t m0, StreamSlot* ring, uint32_t warp, uint32_t lane, uint32_t depth) {
    const uint32_t total = uint32_t(a.iterations + 1) * depth;
    int2* hdr = reinterpret_cast<int2*>(ring + GIANT_LEVELS * STREAM_RING);
    if (warp == 1) {
        StreamPipe P;
        P.b0 = P.b1 = P.b2 = make_int2(0, 0);
        P.k0 = P.k1 = ~0u;
        P.i0 = make_int4(0, 0, 0, 0);
        for (int64_t x = -3; x <= 1; x++) stream_stage_step(a, ring, hdr, P, m0, depth, total, x, lane);
        cp_async_wait<1>();
        cta_bar<STREAM_THREADS>();
        for (uint32_t t = 0; t < total; t++) {
            stream_stage_step(a, ring, hdr, P, m0, depth, total, int64_t(t) + 2, lane);
            cp_async_wait<1>();
            cta_bar<STREAM_THREADS>();
        }
        cp_async_wait<0>();
    } else {
        cta_bar<STREAM_THREADS>();
        for (uint32_t t = 0; t < total; t++) {
            const bool warm = t < depth;
            const int2 bd = hdr[t % GIANT_LEVELS];
            const uint32_t b = uint32_t(bd.x), e = uint32_t(bd.y);
            if (lane < STREAM_RING && b + lane < e) {
                const StreamSlot* sl = ring + (t % GIANT_LEVELS) * STREAM_RING + lane;
                const int4 d = sl->desc;
                const float4 ids = sl->rows.mq[DQ_IDS];
                const BodyVel bv = vel_global(a, __float_as_int(ids.x), __float_as_int(ids.y));
                RecSrc r;
                r.mq = sl->rows.mq;
                r.pq = sl->rows.pq;
                r.pq_stride = PREC_ROWS;
                r.mmut = &a.mrec[m0 + uint32_t(d.z)].mut;
                r.pmut = &a.prec[d.w].mut;
                r.pmut_stride = PREC_ROWS;
                if (warm) warm_core<false, true>(a, r, bv, d.y);
                else solve_core<false, true>(a, r, bv, d.y);
            }
            // manifolds of a level beyond the ring read their rows from global memory
            for (uint32_t j = b + STREAM_RING + lane; j < e; j += 32) {
                const uint32_t mi = m0 + a.order[m0 + j];
                const int4 id = man_ids(a, mi);
                const BodyVel bv = vel_global(a, id.x, id.y);
                if (warm) warm_core<true, true>(a, rec_global(a, mi, id.w), bv, id.z);
                else solve_core<true, true>(a, rec_global(a, mi, id.w), bv, id.z);
            }
            __syncwarp();
            cta_bar<STREAM_THREADS>();
        }
    }
    __syncthreads();
}

__global__ void __launch_bounds__(GIANT_THREADS, 1) dyn_islands_giant(const DynArgs a) {
    __shared__ uint32_t s_island, s_ok, s_depth, s_nslots, s_p0;
    constexpr uint32_t SCHED_WARP = 0;
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t n_giant = a.counters[3], n_big = big_on_ctas(a) ? a.counters[0] : 0u;
    for (;;) {
        if (threadIdx.x == 0) s_island = atomicAdd(a.counters + 4, 1u);
        __syncthreads();
        const uint32_t k = s_island;
        if (k >= n_giant + n_big) break;
        const uint32_t is = k < n_giant ? a.giant_list[k] : a.large_list[k - n_giant];
        if (is == ISLAND_DONE) {
            __syncthreads();
            continue;
        }
        const uint32_t m0 = a.i_start[is], cnt = a.i_count[is];
        GiantStage g;
        if (warp == SCHED_WARP) {
            uint32_t depth = 0, p0 = 0;
            const bool ok = giant_schedule(a, m0, cnt, g, lane, depth, &s_nslots, p0);
            if (lane == 0) { s_ok = ok ? 1u : 0u; s_depth = depth; s_p0 = p0; }
        }
        __syncthreads();
        if (s_ok) {
            if (warp != SCHED_WARP) {
                // the same layout (a pure function of the island's sizes)
                const int4 l = man_ids(a, m0 + cnt - 1);
                giant_layout(a, cnt, uint32_t(int64_t(l.w) + int64_t(l.z) - int64_t(s_p0)), g);
            }
            giant_solve(a, m0, cnt, g, warp, lane, s_depth, s_nslots, s_p0);
        } else if (size_t(GIANT_LEVELS) * STREAM_RING * sizeof(StreamSlot) + GIANT_LEVELS * sizeof(int2) <= a.giant_smem) {
            // streamed by dyn_islands_stream (giant_list may still hold untaken
            // islands up to its end)
            if (threadIdx.x == 0) a.stream_list[atomicAdd(a.counters + 5, 1u)] = is;
            __syncthreads();
            continue;
        } else if (warp == 0) {
            solve_global(a, m0, cnt, lane);
        }
        __syncthreads();
        for (uint32_t j = threadIdx.x; j < cnt; j += GIANT_THREADS) store_manifold(a, m0 + j);
        __syncthreads();
    }
}

// ---- kernel 3d: islands streamed through global memory -------------------
__global__ void __launch_bounds__(STREAM_THREADS, 1) dyn_islands_stream(const DynArgs a) {
    extern __shared__ __align__(16) unsigned char ssm[];
    __shared__ uint32_t s_island, s_depth;
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t n_stream = a.counters[5];
    for (;;) {
        if (threadIdx.x == 0) s_island = atomicAdd(a.counters + 6, 1u);
        __syncthreads();
        const uint32_t k = s_island;
        if (k >= n_stream) break;
        const uint32_t is = a.stream_list[k];
        const uint32_t m0 = a.i_start[is], cnt = a.i_count[is];
        if (warp == 0) {
            const uint32_t depth = stream_schedule(a, m0, cnt, lane);
            if (lane == 0) s_depth = depth;
        }
        __syncthreads();
        stream_solve(a, m0, reinterpret_cast<StreamSlot*>(ssm), warp, lane, s_depth);
        for (uint32_t j = threadIdx.x; j < cnt; j += STREAM_THREADS) store_manifold(a, m0 + j);
        __syncthreads();
    }
}

// ---- kernel 4: integrateRigidBodiesPositions + updateBodiesState ----------
__global__ void __launch_bounds__(128) dyn_bodies_post(const DynArgs a) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= a.nb || !body_enabled(a, i)) return;
    const float dt = a.dt;
    const float f = a.split ? 1.0f : 0.0f;
    const v3 cv = L3(a.cv[i]), cw = L3(a.cw[i]);
    const v3 sv = L3(a.sv[i]), sw = L3(a.sw[i]);
    const v3 nl = V(cv.x + f * sv.x, cv.y + f * sv.y, cv.z + f * sv.z);
    const v3 na = V(cw.x + f * sw.x, cw.y + f * sw.y, cw.z + f * sw.z);
    const v3 x = L3(a.com_world[i]);
    const float4 o4 = a.orientation[i];
    const quat q = Q(o4.x, o4.y, o4.z, o4.w);
    const v3 cp = V(x.x + dt * nl.x, x.y + dt * nl.y, x.z + dt * nl.z);
    const quat dq = qmul(Q(na.x, na.y, na.z, 0.0f), q);
    const quat sq = Q(dt * (0.5f * dq.x), dt * (0.5f * dq.y), dt * (0.5f * dq.z), dt * (0.5f * dq.w));
    const quat co = Q(q.x + sq.x, q.y + sq.y, q.z + sq.z, q.w + sq.w);
    if (a.xc) {
        // mConstrainedPositions / mConstrainedOrientations, read by the joints' position correction
        a.xc[i] = F4(cp);
        a.qc[i] = make_float4(co.x, co.y, co.z, co.w);
    }
    // updateBodiesState
    a.lin_vel[i] = F4(cv);
    a.ang_vel[i] = F4(cw);
    a.com_world[i] = F4(cp);
    const float len = sqrtf(co.x * co.x + co.y * co.y + co.z * co.z + co.w * co.w);
    const quat u = Q(co.x / len, co.y / len, co.z / len, co.w / len);
    a.orientation[i] = make_float4(u.x, u.y, u.z, u.w);
    const v3 r = qrot(u, L3(a.com_local[i]));
    a.position[i] = F4(V(cp.x - r.x, cp.y - r.y, cp.z - r.z));
}

// ---- kernel 5: collider local-to-world transforms ------------------------
__global__ void __launch_bounds__(128) dyn_colliders(const DynArgs a) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= a.nc || !collider_enabled(a, i)) return;
    const int32_t b = a.c_body[i];
    if (uint32_t(b) >= a.nb) {
        atomicOr(a.error, 4u);
        return;
    }
    const float4 bo = a.orientation[b], lo = a.c_lori[i];
    const xform t = xmul(X(L3(a.position[b]), Q(bo.x, bo.y, bo.z, bo.w)), X(L3(a.c_lpos[i]), Q(lo.x, lo.y, lo.z, lo.w)));
    a.c_wpos[i] = F4(t.p);
    a.c_wori[i] = make_float4(t.q.x, t.q.y, t.q.z, t.q.w);
}

uint32_t blocks(uint32_t n) { return (n + 127) / 128; }

// ---- graph-coloured solver -------------------------------------------------
//
// Not the drop-in (the drop-in is the exact-order solver above): for very
// large worlds, where one island of 10^5 manifolds is a chain of 10^4
// dependency levels, the manifolds' conflict graph (two manifolds conflict
// when they share a movable body) is coloured on the GPU and every pass (warm
// start, each velocity iteration) runs colour after colour, the manifolds of
// one colour in parallel.  No two manifolds of a colour share a movable body,
// so each manifold still reads the latest velocities of its bodies and the
// per-manifold arithmetic is the reference's (ContactSolverSystem.cpp:
// 324-759); only the order of the manifolds differs, so the results differ
// from the reference's and the solver is reported by its constraint residual
// and energy, next to the exact solver on the same world.
//
// Colouring: speculative greedy rounds.  Each uncoloured manifold takes the
// lowest colour none of its coloured neighbours has; of two neighbours that
// took the same colour in a round, the one with the lower index keeps it and
// the other tries again in the next round.  Decisions depend on the previous
// round only, so the colouring is deterministic.
constexpr uint8_t NO_COLOR = 0xff;

RD uint32_t movable_mask(const DynArgs& a, uint32_t mi) { return ~man_fixed(a, mi) & 3u; }

__global__ void __launch_bounds__(128) color_degree(const DynArgs a, uint32_t* __restrict__ deg) {
    const uint32_t mi = blockIdx.x * blockDim.x + threadIdx.x;
    if (mi >= a.nm) return;
    const int4 id = man_ids(a, mi);
    const uint32_t mv = movable_mask(a, mi);
    if (mv & 1u) atomicAdd(deg + id.x, 1u);
    if (mv & 2u) atomicAdd(deg + id.y, 1u);
}

__global__ void __launch_bounds__(128) color_adjacency(const DynArgs a, const uint32_t* __restrict__ start,
                                                       uint32_t* __restrict__ fill, uint32_t* __restrict__ adj) {
    const uint32_t mi = blockIdx.x * blockDim.x + threadIdx.x;
    if (mi >= a.nm) return;
    const int4 id = man_ids(a, mi);
    const uint32_t mv = movable_mask(a, mi);
    if (mv & 1u) adj[start[id.x] + atomicAdd(fill + id.x, 1u)] = mi;
    if (mv & 2u) adj[start[id.y] + atomicAdd(fill + id.y, 1u)] = mi;
}

__global__ void __launch_bounds__(128) color_tentative(const DynArgs a, ColorScratch c) {
    const uint32_t mi = blockIdx.x * blockDim.x + threadIdx.x;
    if (mi >= a.nm) return;
    if (c.color[mi] != NO_COLOR) { c.tent[mi] = NO_COLOR; return; }
    const int4 id = man_ids(a, mi);
    const uint32_t mv = movable_mask(a, mi);
    unsigned long long used[2] = {0ull, 0ull};
    for (int side = 0; side < 2; side++) {
        if (!(mv & (1u << side))) continue;
        const int32_t b = side ? id.y : id.x;
        for (uint32_t k = c.start[b]; k < c.start[b + 1]; k++) {
            const uint8_t nc = c.color[c.adj[k]];
            if (nc != NO_COLOR) used[nc >> 6] |= 1ull << (nc & 63u);
        }
    }
    uint8_t t = NO_COLOR;
    if (~used[0]) t = uint8_t(__ffsll(static_cast<long long>(~used[0])) - 1);
    else if (~used[1]) t = uint8_t(64 + __ffsll(static_cast<long long>(~used[1])) - 1);
    c.tent[mi] = t;   // NO_COLOR: every colour is taken (the caller falls back)
}

// Priority of a manifold in the conflict resolution: a hash of its index
// (ties by index).  Index order itself follows the islands, i.e. space, so a
// pile would chain "lower index wins" decisions over hundreds of rounds; a
// hashed order resolves every round's conflicts independently of position
// (a few rounds to colour the 100k-body terrain's island).
RD uint64_t color_priority(uint32_t mi) {
    uint32_t h = mi * 0x9E3779B1u;
    h ^= h >> 16;
    h *= 0x85EBCA6Bu;
    h ^= h >> 13;
    return (uint64_t(h) << 32) | mi;
}

__global__ void __launch_bounds__(128) color_resolve(const DynArgs a, ColorScratch c) {
    const uint32_t mi = blockIdx.x * blockDim.x + threadIdx.x;
    if (mi >= a.nm) return;
    const uint8_t t = c.tent[mi];
    if (t == NO_COLOR) {
        if (c.color[mi] == NO_COLOR) atomicAdd(c.count + COLOR_MAX, 1u);
        return;
    }
    const int4 id = man_ids(a, mi);
    const uint32_t mv = movable_mask(a, mi);
    for (int side = 0; side < 2; side++) {
        if (!(mv & (1u << side))) continue;
        const int32_t b = side ? id.y : id.x;
        for (uint32_t k = c.start[b]; k < c.start[b + 1]; k++) {
            const uint32_t n = c.adj[k];
            if (n != mi && c.tent[n] == t && color_priority(n) < color_priority(mi)) {
                atomicAdd(c.count + COLOR_MAX, 1u);
                return;
            }
        }
    }
    c.color[mi] = t;
}

__global__ void __launch_bounds__(128) color_count(const DynArgs a, ColorScratch c) {
    const uint32_t mi = blockIdx.x * blockDim.x + threadIdx.x;
    if (mi < a.nm) atomicAdd(c.count + c.color[mi], 1u);
}

// Manifolds grouped by colour (the order inside a colour does not matter:
// its manifolds share no movable body).
__global__ void __launch_bounds__(128) color_scatter(const DynArgs a, ColorScratch c) {
    const uint32_t mi = blockIdx.x * blockDim.x + threadIdx.x;
    if (mi < a.nm) c.order[atomicAdd(c.offset + c.color[mi], 1u)] = mi;
}

template <int PASS>   // 0 warm start, 1 velocity iteration
__global__ void __launch_bounds__(128) colored_pass(const DynArgs a, const uint32_t* __restrict__ order, uint32_t off,
                                                    uint32_t cnt) {
    const uint32_t k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= cnt) return;
    const uint32_t mi = order[off + k];
    const int4 id = man_ids(a, mi);
    if (PASS == 0) warm_manifold(a, mi, vel_global(a, id.x, id.y), id.z, id.w);
    else solve_manifold(a, mi, vel_global(a, id.x, id.y), id.z, id.w);
}

__global__ void __launch_bounds__(128) colored_store(const DynArgs a) {
    const uint32_t mi = blockIdx.x * blockDim.x + threadIdx.x;
    if (mi < a.nm) store_manifold(a, mi);
}

// Velocity constraint residual of every contact point after the solve, on
// the constrained velocities (either solver).
__global__ void __launch_bounds__(128) solver_residual(const DynArgs a) {
    const uint32_t mi = blockIdx.x * blockDim.x + threadIdx.x;
    float sq = 0.0f, mx = 0.0f;
    uint32_t np = 0;
    if (mi < a.nm) {
        const int4 id = man_ids(a, mi);
        const v3 v1 = L3(a.cv[id.x]), w1 = L3(a.cw[id.x]), v2 = L3(a.cv[id.y]), w2 = L3(a.cw[id.y]);
        for (int k = 0; k < id.z; k++) {
            const DynPointRec& pr = a.prec[id.w + k];
            const v3 r1 = L3(pr.q[DP_R1]), r2 = L3(pr.q[DP_R2]), n = L3(pr.q[DP_N]);
            const float jv = vdot(rel_velocity(v1, w1, v2, w2, r1, r2), n);
            const float lambda = pr.mut.x;
            const float r = lambda > 0.0f ? fabsf(jv) : (jv < 0.0f ? -jv : 0.0f);
            sq += r * r;
            mx = fmaxf(mx, r);
            np++;
        }
    }
    for (int o = 16; o; o >>= 1) {
        sq += __shfl_xor_sync(0xffffffffu, sq, o);
        mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
        np += __shfl_xor_sync(0xffffffffu, np, o);
    }
    if ((threadIdx.x & 31u) == 0 && np) {
        atomicAdd(&a.stats->residual_sq_sum, double(sq));
        atomicMax(&a.stats->residual_max_bits, __float_as_uint(mx));
        atomicAdd(&a.stats->points, np);
    }
}

// Energies of the enabled dynamic bodies after the stage.
__global__ void __launch_bounds__(128) body_energy(const DynArgs a) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    double ke = 0.0, pe = 0.0;
    if (i < a.nb && body_enabled(a, i)) {
        const float4 m = a.mass[i];   // mass, inverse mass, dampings
        if (m.y > 0.0f) {
            const v3 v = L3(a.lin_vel[i]), w = L3(a.ang_vel[i]);
            const float4 o = a.orientation[i];
            const v3 wl = qrot(qinv(Q(o.x, o.y, o.z, o.w)), w);   // angular velocity in the body frame
            const v3 ii = L3(a.iil[i]);
            double rot = 0.0;
            if (ii.x > 0.0f) rot += double(wl.x) * wl.x / ii.x;
            if (ii.y > 0.0f) rot += double(wl.y) * wl.y / ii.y;
            if (ii.z > 0.0f) rot += double(wl.z) * wl.z / ii.z;
            ke = 0.5 * double(m.x) * (double(v.x) * v.x + double(v.y) * v.y + double(v.z) * v.z) + 0.5 * rot;
            if (a.gravity_enabled && a.gravity[i]) {
                const float4 x = a.com_world[i];
                pe = -double(m.x) * (double(a.gx) * x.x + double(a.gy) * x.y + double(a.gz) * x.z);
            }
        }
    }
    for (int o = 16; o; o >>= 1) {
        ke += __shfl_xor_sync(0xffffffffu, ke, o);
        pe += __shfl_xor_sync(0xffffffffu, pe, o);
    }
    if ((threadIdx.x & 31u) == 0) {
        atomicAdd(&a.stats->kinetic, ke);
        atomicAdd(&a.stats->potential, pe);
    }
}

// Colours every manifold and runs the passes; false when the colouring does
// not finish (every colour taken around some manifold, or too many rounds):
// the caller then runs the exact solver.  Synchronizes the stream.
bool colored_islands(const DynArgs& a, cudaStream_t s, uint64_t* launches) {
    ColorScratch c = *a.color;
    const uint32_t nm = a.nm;
    cudaMemsetAsync(c.start, 0, (size_t(a.nb) + 1) * 4, s);
    cudaMemsetAsync(c.fill, 0, size_t(a.nb) * 4, s);
    cudaMemsetAsync(c.color, NO_COLOR, nm, s);
    color_degree<<<blocks(nm), 128, 0, s>>>(a, c.start);
    launch_exclusive_scan(c.start, a.nb + 1, nullptr, s);
    color_adjacency<<<blocks(nm), 128, 0, s>>>(a, c.start, c.fill, c.adj);
    *launches += 3;
    uint32_t rounds = 0, remaining = nm;
    while (remaining > 0) {
        if (++rounds > 256) return false;
        cudaMemsetAsync(c.count + COLOR_MAX, 0, 4, s);
        color_tentative<<<blocks(nm), 128, 0, s>>>(a, c);
        color_resolve<<<blocks(nm), 128, 0, s>>>(a, c);
        *launches += 2;
        if (cudaMemcpyAsync(&remaining, c.count + COLOR_MAX, 4, cudaMemcpyDeviceToHost, s) != cudaSuccess ||
            cudaStreamSynchronize(s) != cudaSuccess)
            return false;
        // (a manifold whose neighbours hold every colour never gets one: the
        // round limit ends the loop)
    }
    uint32_t cnt[COLOR_MAX];
    cudaMemsetAsync(c.count, 0, COLOR_MAX * 4, s);
    color_count<<<blocks(nm), 128, 0, s>>>(a, c);
    *launches += 1;
    if (cudaMemcpyAsync(cnt, c.count, sizeof(cnt), cudaMemcpyDeviceToHost, s) != cudaSuccess ||
        cudaStreamSynchronize(s) != cudaSuccess)
        return false;
    uint32_t off[COLOR_MAX], ncol = 0, run = 0;
    for (uint32_t k = 0; k < COLOR_MAX; k++) {
        off[k] = run;
        run += cnt[k];
        if (cnt[k]) ncol = k + 1;
    }
    cudaMemcpyAsync(c.offset, off, sizeof(off), cudaMemcpyHostToDevice, s);
    color_scatter<<<blocks(nm), 128, 0, s>>>(a, c);
    *launches += 1;
    for (uint32_t k = 0; k < ncol; k++)
        if (cnt[k]) { colored_pass<0><<<blocks(cnt[k]), 128, 0, s>>>(a, c.order, off[k], cnt[k]); (*launches)++; }
    for (int it = 0; it < a.iterations; it++)
        for (uint32_t k = 0; k < ncol; k++)
            if (cnt[k]) { colored_pass<1><<<blocks(cnt[k]), 128, 0, s>>>(a, c.order, off[k], cnt[k]); (*launches)++; }
    colored_store<<<blocks(nm), 128, 0, s>>>(a);
    (*launches)++;
    if (a.stats) {
        uint32_t cr[2] = {ncol, rounds};
        cudaMemcpyAsync(&a.stats->colors, cr, sizeof(cr), cudaMemcpyHostToDevice, s);
        // the pageable source is read before the function returns
        cudaStreamSynchronize(s);
    }
    return true;
}

}  // namespace

cudaError_t launch_dynamics(const DynArgs& a, cudaStream_t s, uint64_t* launches) {
    // islands with joints, one thread each: giant_ctas is the number of SMs
    const uint32_t joint_lanes = items_per_warp(a.nji, int(a.giant_ctas));
    const uint32_t joint_blocks = (a.nji + 2 * joint_lanes - 1) / std::max(2 * joint_lanes, 1u);
    if (a.ni) cudaMemsetAsync(a.counters, 0, DYN_COUNTERS * sizeof(uint32_t), s);
    if (a.nb) { dyn_bodies_pre<<<blocks(a.nb), 128, 0, s>>>(a); (*launches)++; }
    if (a.nm) { dyn_manifold_init<<<blocks(a.nm) + (a.small_auto ? blocks(a.ni) : 0u), 128, 0, s>>>(a); (*launches)++; }
    if (a.nj) { dyn_joints_init<<<blocks(a.nj), 128, 0, s>>>(a); (*launches)++; }
    if (a.stats) cudaMemsetAsync(a.stats, 0, sizeof(SolverStats), s);
    // the graph-coloured solver takes every island when the stage has no
    // joints (joint islands keep the exact order); it falls back to the exact
    // solver if the colouring does not finish
    bool colored_done = false;
    if (a.colored && a.color && a.nj == 0 && a.nm) colored_done = colored_islands(a, s, launches);
    if (a.ni && !colored_done) {
        dyn_islands_small<<<blocks(a.ni), 128, 0, s>>>(a);
        (*launches)++;
        const size_t smem = size_t(LARGE_WARPS) * LARGE_WARP_SMEM;
        cudaFuncSetAttribute(dyn_islands_large, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem));
        dyn_islands_large<<<a.large_ctas, LARGE_WARPS * 32, smem, s>>>(a);
        (*launches)++;
        if (a.giant_smem) {
            cudaFuncSetAttribute(dyn_islands_giant, cudaFuncAttributeMaxDynamicSharedMemorySize, int(a.giant_smem));
            dyn_islands_giant<<<a.giant_ctas, GIANT_THREADS, a.giant_smem, s>>>(a);
            (*launches)++;
            const size_t ring = size_t(GIANT_LEVELS) * STREAM_RING * sizeof(StreamSlot) + GIANT_LEVELS * sizeof(int2);
            cudaFuncSetAttribute(dyn_islands_stream, cudaFuncAttributeMaxDynamicSharedMemorySize, int(ring));
            dyn_islands_stream<<<a.giant_ctas, STREAM_THREADS, ring, s>>>(a);
            (*launches)++;
        }
        if (a.nji) { dyn_islands_joint<<<joint_blocks, 64, 0, s>>>(a, joint_lanes); (*launches)++; }
    }
    if (a.stats && a.nm) { solver_residual<<<blocks(a.nm), 128, 0, s>>>(a); (*launches)++; }
    const uint32_t nbp = a.b_enabled ? a.nb : a.nb_enabled, ncp = a.c_enabled ? a.nc : a.nc_enabled;
    if (nbp) { dyn_bodies_post<<<blocks(nbp), 128, 0, s>>>(a); (*launches)++; }
    if (a.stats && a.nb) { body_energy<<<blocks(a.nb), 128, 0, s>>>(a); (*launches)++; }
    if (a.nji) { dyn_joints_position<<<joint_blocks, 64, 0, s>>>(a, joint_lanes); (*launches)++; }
    if (ncp) { dyn_colliders<<<blocks(ncp), 128, 0, s>>>(a); (*launches)++; }
    return cudaGetLastError();
}

}  // namespace rp3dg
