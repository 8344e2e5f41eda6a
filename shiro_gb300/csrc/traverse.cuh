// traverse.cuh - BVH traversal with the reference's hit semantics.
//
// The reference (without Embree) intersects every triangle with
// Moller-Trumbore (CpuPathTracer.cpp:386-429) and keeps a new hit only when
// strictly closer, so among equal distances the first (mesh, primitive) wins
// (:431-466).  Here the triangles are reached through a BVH and a hit replaces
// the best one when (t, global index) is lexicographically smaller, which
// selects the same triangle.  The triangle test uses the same operations in
// the same order (compiled without FMA contraction), so t, u, v are
// bit-identical.  Child boxes are inflated at build time by a margin far above
// the rounding error of the box test, so a box is never culled while it holds
// a triangle the exhaustive test would report.
//
// Each traversal loop is bounded by kMaxVisits node visits; past that the
// error word is set and the ray is reported as a miss (a corrupt BVH can never
// hang the kernel).
#pragma once

#include "common.cuh"
#include "lanes.cuh"
#include "scene.cuh"

namespace shiro_gpu {


constexpr uint32_t kMaxVisits = 1u << 22;

// Work counters of the roofline probe (shiro_gpu_count_work).  NullCounter
// compiles every increment away in the render kernels.
struct NullCounter {
    __device__ __forceinline__ void node() {}
    __device__ __forceinline__ void tri() {}
    __device__ __forceinline__ void onode() {}
    __device__ __forceinline__ void otri() {}
    __device__ __forceinline__ void closest() {}
    __device__ __forceinline__ void occlusion() {}
    __device__ __forceinline__ void hit() {}
    __device__ __forceinline__ void env_eval(uint32_t n = 1) {}
    __device__ __forceinline__ void env_sample(uint32_t n = 1) {}
    __device__ __forceinline__ void bsdf_eval() {}
    __device__ __forceinline__ void bsdf_pdf() {}
};
struct LocalCounter {
    uint32_t nodes = 0, tris = 0, onodes = 0, otris = 0, closestRays = 0, occlusionRays = 0, hits = 0, envEvals = 0,
             envSamples = 0, bsdfEvals = 0, bsdfPdfs = 0;
    __device__ __forceinline__ void node() { ++nodes; }
    __device__ __forceinline__ void tri() { ++tris; }
    __device__ __forceinline__ void onode() { ++onodes; }
    __device__ __forceinline__ void otri() { ++otris; }
    __device__ __forceinline__ void closest() { ++closestRays; }
    __device__ __forceinline__ void occlusion() { ++occlusionRays; }
    __device__ __forceinline__ void hit() { ++hits; }
    __device__ __forceinline__ void env_eval(uint32_t n = 1) { envEvals += n; }
    __device__ __forceinline__ void env_sample(uint32_t n = 1) { envSamples += n; }
    __device__ __forceinline__ void bsdf_eval() { ++bsdfEvals; }
    __device__ __forceinline__ void bsdf_pdf() { ++bsdfPdfs; }
};

struct HitRec {
    float t, u, v;
    uint32_t gid;  // global triangle index (meshes in order), 0xffffffff on a miss
};

struct RayInv {
    V3 inv, ood;
};

__device__ __forceinline__ RayInv ray_inv(const V3& o, const V3& d) {
    RayInv r;
    const float dx = fabsf(d.x) > 1.0e-20f ? d.x : copysignf(1.0e-20f, d.x);
    const float dy = fabsf(d.y) > 1.0e-20f ? d.y : copysignf(1.0e-20f, d.y);
    const float dz = fabsf(d.z) > 1.0e-20f ? d.z : copysignf(1.0e-20f, d.z);
    r.inv = V3{1.0f / dx, 1.0f / dy, 1.0f / dz};
    r.ood = V3{o.x * r.inv.x, o.y * r.inv.y, o.z * r.inv.z};
    return r;
}

// Three-input minimum / maximum (PTX min.f32 / max.f32 with three sources,
// sm_100 and later); for non-NaN inputs equal to two nested fminf / fmaxf.
__device__ __forceinline__ float fmin3(float a, float b, float c) {
    float r;
    asm("min.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
    return r;
}
__device__ __forceinline__ float fmax3(float a, float b, float c) {
    float r;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
    return r;
}

// Two fused multiply-adds with one instruction (fma.rn.f32x2, sm_100 and
// later): (x, y) * a + b on register pairs, each half rounded as __fmaf_rn.
__device__ __forceinline__ uint64_t pack2(float a, float b) {
    uint64_t r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ void fma2(uint32_t x, uint32_t y, uint64_t a, uint64_t b, float* r0, float* r1) {
    uint64_t r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(pack2(__uint_as_float(x), __uint_as_float(y))), "l"(a), "l"(b));
    asm("mov.b64 {%0, %1}, %2;" : "=f"(*r0), "=f"(*r1) : "l"(r));
}

// Entry / exit of both child boxes of a node (slab test, fused form).
__device__ __forceinline__ void node_boxes(const float4& n0, const float4& n1, const float4& n2, const RayInv& r,
                                           float tmax, float* t0, float* t1, bool* h0, bool* h1) {
    const float ax = __fmaf_rn(n0.x, r.inv.x, -r.ood.x), bx = __fmaf_rn(n0.y, r.inv.x, -r.ood.x);
    const float ay = __fmaf_rn(n0.z, r.inv.y, -r.ood.y), by = __fmaf_rn(n0.w, r.inv.y, -r.ood.y);
    const float az = __fmaf_rn(n2.x, r.inv.z, -r.ood.z), bz = __fmaf_rn(n2.y, r.inv.z, -r.ood.z);
    const float cx = __fmaf_rn(n1.x, r.inv.x, -r.ood.x), dx = __fmaf_rn(n1.y, r.inv.x, -r.ood.x);
    const float cy = __fmaf_rn(n1.z, r.inv.y, -r.ood.y), dy = __fmaf_rn(n1.w, r.inv.y, -r.ood.y);
    const float cz = __fmaf_rn(n2.z, r.inv.z, -r.ood.z), dz = __fmaf_rn(n2.w, r.inv.z, -r.ood.z);
    const float lo0 = fmax3(fminf(ax, bx), fminf(ay, by), fmaxf(fminf(az, bz), 0.0f));
    const float hi0 = fmin3(fmaxf(ax, bx), fmaxf(ay, by), fminf(fmaxf(az, bz), tmax));
    const float lo1 = fmax3(fminf(cx, dx), fminf(cy, dy), fmaxf(fminf(cz, dz), 0.0f));
    const float hi1 = fmin3(fmaxf(cx, dx), fmaxf(cy, dy), fminf(fmaxf(cz, dz), tmax));
    *t0 = lo0;
    *t1 = lo1;
    *h0 = lo0 <= hi0;
    *h1 = lo1 <= hi1;
}

// Moller-Trumbore, IntersectTriangle (CpuPathTracer.cpp:386-429).
__device__ __forceinline__ bool tri_test(const V3& o, const V3& d, float tMin, float tMax, const float4& a,
                                         const float4& b, const float4& c, float* t, float* u, float* v) {
    const V3 p0 = f4xyz(a), e1 = f4xyz(b), e2 = f4xyz(c);
    const V3 pvec = cross(d, e2);
    const float det = dot(e1, pvec);
    if (fabsf(det) < 1.0e-8f) return false;
    const float inv = 1.0f / det;
    const V3 tvec = o - p0;
    const float uu = dot(tvec, pvec) * inv;
    if (uu < 0.0f || uu > 1.0f) return false;
    const V3 qvec = cross(tvec, e1);
    const float vv = dot(d, qvec) * inv;
    if (vv < 0.0f || uu + vv > 1.0f) return false;
    const float tt = dot(e2, qvec) * inv;
    if (tt < tMin || tt > tMax) return false;
    *t = tt;
    *u = uu;
    *v = vv;
    return true;
}

// ---- compressed 8-wide BVH (layout in bvh_build.h) -------------------------


// Children of wide node `node` hit within [0, tmax]: internal ones as bits
// (slot ^ octInv) of *inner (nearest first = lowest bit), leaf slots (one
// triangle each) as bits 0-7 of *tris with the node's leaf mask in bits 8-15
// (wide_tri takes the triangles off it).
//
// A quantised plane q of an axis lies at t = (origin + q * scale - o) * inv
// = (2^23 + q) * A + (B - 2^23 * A) with A = scale * inv (exact: scale is a
// power of two) and B = origin * inv - o * inv.  A byte permute turns q into
// the float 2^23 + q, and the bias B - 2^23 * A is formed once per node, so a
// plane costs one permute and one FMA; the bias rounds to within half a
// quantisation step, which the builder covers by widening every child box by
// one step.  The near and far plane of an axis share A and B and go through
// one packed FMA; the children's outcomes are gathered as sign bits.  The test
// is bound by instruction issue and the integer / min-max pipe (ncu: 68 % of
// issue slots, 57 % of that pipe): packed FMAs, sign gathering and the
// one-operation scale and mask words took the 1080p field frame from 111.6 to
// 107.9 ms.  Empty slots hold an inverted box (q_lo = 255, q_hi = 0), which
// can only pass when rounding collapses all its planes to one distance; they
// are in neither mask.
__device__ __forceinline__ void wide_node(const DevScene& s, uint32_t node, const RayInv& r, float tmax, uint32_t octInv,
                                          uint32_t* childBase, uint32_t* imask, uint32_t* inner, uint32_t* triBase,
                                          uint32_t* tris) {
    const float4* np = s.nodes8 + 5 * static_cast<size_t>(node);
    const float4 a = __ldg(np), b = __ldg(np + 1);
    const float4 q0 = __ldg(np + 2), q1 = __ldg(np + 3), q2 = __ldg(np + 4);
    const uint32_t eb = __float_as_uint(a.w), exy = __float_as_uint(b.w);
    const float sx = __uint_as_float(exy & 0xffff0000u), sy = __uint_as_float(exy << 16),
                sz = __uint_as_float(eb & 0xffff0000u);
    const float ax = sx * r.inv.x, ay = sy * r.inv.y, az = sz * r.inv.z;
    const float bx = __fmaf_rn(-8388608.0f, ax, __fmaf_rn(a.x, r.inv.x, -r.ood.x));
    const float by = __fmaf_rn(-8388608.0f, ay, __fmaf_rn(a.y, r.inv.y, -r.ood.y));
    const float bz = __fmaf_rn(-8388608.0f, az, __fmaf_rn(a.z, r.inv.z, -r.ood.z));
    const uint32_t im = eb & 0xffu;
    // near / far plane words per axis: a negative direction enters through
    // the upper planes (inv < 0 makes their distances the smaller ones)
    const bool nx = r.inv.x < 0.0f, ny = r.inv.y < 0.0f, nz = r.inv.z < 0.0f;
    const uint32_t lx0 = __float_as_uint(q0.x), lx1 = __float_as_uint(q0.y), ly0 = __float_as_uint(q0.z),
                   ly1 = __float_as_uint(q0.w), lz0 = __float_as_uint(q1.x), lz1 = __float_as_uint(q1.y),
                   hx0 = __float_as_uint(q1.z), hx1 = __float_as_uint(q1.w), hy0 = __float_as_uint(q2.x),
                   hy1 = __float_as_uint(q2.y), hz0 = __float_as_uint(q2.z), hz1 = __float_as_uint(q2.w);
    const uint32_t nw[6] = {nx ? hx0 : lx0, nx ? hx1 : lx1, ny ? hy0 : ly0, ny ? hy1 : ly1, nz ? hz0 : lz0, nz ? hz1 : lz1};
    const uint32_t fw[6] = {nx ? lx0 : hx0, nx ? lx1 : hx1, ny ? ly0 : hy0, ny ? ly1 : hy1, nz ? lz0 : hz0, nz ? lz1 : hz1};
    const uint64_t axx = pack2(ax, ax), ayy = pack2(ay, ay), azz = pack2(az, az);
    const uint64_t bxx = pack2(bx, bx), byy = pack2(by, by), bzz = pack2(bz, bz);
    uint32_t miss = 0;  // bit i: child i is missed
#pragma unroll
    for (int i = 7; i >= 0; --i) {
        const int h = i >> 2;
        const uint32_t sel = static_cast<uint32_t>(i & 3) | 0x7540u;  // byte i -> float 2^23 + q
        float x0, x1, y0, y1, z0, z1;
        fma2(__byte_perm(nw[0 + h], 0x4b000000u, sel), __byte_perm(fw[0 + h], 0x4b000000u, sel), axx, bxx, &x0, &x1);
        fma2(__byte_perm(nw[2 + h], 0x4b000000u, sel), __byte_perm(fw[2 + h], 0x4b000000u, sel), ayy, byy, &y0, &y1);
        fma2(__byte_perm(nw[4 + h], 0x4b000000u, sel), __byte_perm(fw[4 + h], 0x4b000000u, sel), azz, bzz, &z0, &z1);
        const float lo = fmax3(x0, y0, fmaxf(z0, 0.0f));
        const float hi = fmin3(x1, y1, fminf(z1, tmax));
        // the sign of hi - lo (never rounded to the other sign) shifts in
        miss = __funnelshift_l(__float_as_uint(hi - lo), miss, 1);
    }
    // internal children: bit i moves to bit i ^ octInv
    uint32_t in = im & ~miss;
    if (octInv & 1u) in = ((in & 0x55u) << 1) | ((in >> 1) & 0x55u);
    if (octInv & 2u) in = ((in & 0x33u) << 2) | ((in >> 2) & 0x33u);
    if (octInv & 4u) in = ((in & 0x0fu) << 4) | ((in >> 4) & 0x0fu);
    *childBase = __float_as_uint(b.x);
    *triBase = __float_as_uint(b.y);
    *imask = im;
    *inner = in;
    *tris = __float_as_uint(b.z) & ~miss;
}

// Whether a node's triangle word (wide_node) still holds triangles to test.
__device__ __forceinline__ bool wide_has_tri(uint32_t bits) { return (bits & 0xffu) != 0u; }

// Takes the next triangle off a node's triangle word: its index in the wide
// order (the leaf slots' triangles lie one after another from triBase on).
__device__ __forceinline__ uint32_t wide_tri(uint32_t triBase, uint32_t& bits) {
    const uint32_t low = bits & (0u - bits);  // the lowest slot left (bits 0-7 are not all clear)
    bits ^= low;
    return triBase + static_cast<uint32_t>(__popc((bits >> 8) & (low - 1u)));
}

__device__ __forceinline__ uint32_t ray_oct_inv(const V3& d) {
    return 7u ^ ((d.x < 0.0f ? 1u : 0u) | (d.y < 0.0f ? 2u : 0u) | (d.z < 0.0f ? 4u : 0u));
}

constexpr uint32_t kNoNode = 0xffffffffu;

// Wide-BVH traversal as resumable state, so that a caller may interleave rays
// (the wavefront stages refill a lane with a new ray as soon as its ray
// finishes) and choose when a node's triangles are tested.  Stack entries are
// groups of sibling wide nodes still to visit: (childBase, remaining inner
// bits << 8 | imask); the caller owns the stack array.  A ray is finished when
// neither a node nor a triangle is left.
struct WideTrav {
    V3 o, d;
    RayInv r;
    uint32_t octInv;
    float tmax;                 // closest: the best distance so far; occlusion: maxDist
    float bu, bv;
    uint32_t bestGid;           // closest: 0xffffffff while nothing is hit
    uint32_t node;              // next node to visit, kNoNode when none is left
    uint32_t tBase, tBits;      // triangles of the visited node not tested yet
    int sp;
    uint32_t visits;
};

__device__ __forceinline__ void wide_init(WideTrav& t, const V3& o, const V3& d, float tmax) {
    t.o = o;
    t.d = d;
    t.r = ray_inv(o, d);
    t.octInv = ray_oct_inv(d);
    t.tmax = tmax;
    t.bu = 0.0f;
    t.bv = 0.0f;
    t.bestGid = 0xffffffffu;
    t.node = 0;
    t.tBase = 0;
    t.tBits = 0;
    t.sp = 0;
    t.visits = 0;
}

// Ends a ray whose bounds check failed: the error word is set, the ray hits
// nothing.
__device__ __forceinline__ void wide_abort(const DevScene& s, WideTrav& t, uint32_t err) {
    atomicOr(s.error, err);
    t.bestGid = 0xffffffffu;
    t.node = kNoNode;
    t.tBits = 0;
}

// Moves to the next node of the traversal (kNoNode when none is left).
__device__ __forceinline__ void wide_next(const DevScene& s, WideTrav& t, uint2* stack, uint32_t gBase, uint32_t gImask,
                                          uint32_t gInner) {
    if (gInner == 0u) {
        if (t.sp == 0) {
            t.node = kNoNode;
            return;
        }
        --t.sp;
        gBase = stack[t.sp].x;
        gInner = stack[t.sp].y >> 8;
        gImask = stack[t.sp].y & 0xffu;
    }
    const uint32_t slot = static_cast<uint32_t>(__ffs(gInner) - 1) ^ t.octInv;
    gInner &= gInner - 1u;
    t.node = gBase + __popc(gImask & ((1u << slot) - 1u));
    if (gInner) {
        if (t.sp >= kStackWide) {
            wide_abort(s, t, kErrStackOverflow);
            return;
        }
        stack[t.sp++] = make_uint2(gBase, (gInner << 8) | gImask);
    }
}

// Visits t.node (its triangles go to tBase / tBits) and moves to the next.
__device__ __forceinline__ void wide_visit(const DevScene& s, WideTrav& t, uint2* stack) {
    if (++t.visits > kMaxVisits) {
        wide_abort(s, t, kErrTraversalLimit);
        return;
    }
    uint32_t gBase, gImask, gInner;
    wide_node(s, t.node, t.r, t.tmax, t.octInv, &gBase, &gImask, &gInner, &t.tBase, &t.tBits);
    wide_next(s, t, stack, gBase, gImask, gInner);
}

// Tests one pending triangle; keeps the closest hit (ties: the lower global
// index).
__device__ __forceinline__ void wide_test_closest(const DevScene& s, WideTrav& t) {
    const float4* tp = s.tris + 3 * static_cast<size_t>(wide_tri(t.tBase, t.tBits));
    const float4 ta = __ldg(tp), tb = __ldg(tp + 1), tc = __ldg(tp + 2);
    float tt, u, v;
    if (!tri_test(t.o, t.d, kRayEpsilon, FLT_MAX, ta, tb, tc, &tt, &u, &v)) return;
    const uint32_t gid = __float_as_uint(ta.w);
    if (tt < t.tmax || (tt == t.tmax && gid < t.bestGid)) {
        t.tmax = tt;
        t.bestGid = gid;
        t.bu = u;
        t.bv = v;
    }
}

// Tests one pending triangle for any hit in [1e-4, t.tmax].
__device__ __forceinline__ bool wide_test_any(const DevScene& s, WideTrav& t) {
    const float4* tp = s.tris + 3 * static_cast<size_t>(wide_tri(t.tBase, t.tBits));
    const float4 ta = __ldg(tp), tb = __ldg(tp + 1), tc = __ldg(tp + 2);
    float tt, u, v;
    return tri_test(t.o, t.d, kRayEpsilon, t.tmax, ta, tb, tc, &tt, &u, &v);
}

// One step of a warp's wide-BVH traversal: every lane that has a node and no
// triangle pending visits it; pending triangles wait until kTriLanes lanes
// hold some (or no lane has a node to visit) and are then tested by those
// lanes together until fewer than kTriStop hold any (postponed leaves, Ylitie,
// Karras and Laine 2017).  Tested as soon as a lane finds them, a warp ran its
// triangle tests for the one or two lanes that had just reached a leaf; on the
// 1080p field frame nodes are now visited by 24.5 of 32 lanes and triangles
// tested by 10.4, and the frame takes 112.3 ms instead of 117.9 (kTriLanes 5:
// 113.3, 12: 113.6, 16: 116.1, 20: 120.1; kTriStop 4: 116.4, 8: 127.9 - lanes
// left with triangles visit no node).  Holding a second node's triangles per
// lane, so that fewer wait, costs more registers than it gains (110 against
// 107.9 ms).  False when no lane has anything left.  Warp-uniform call.
constexpr int kTriLanes = 8;
constexpr int kTriStop = 2;

template <typename Visit, typename Test>
__device__ __forceinline__ bool trav_step(WideTrav& t, Visit&& visit, Test&& test) {
    if (t.node != kNoNode && !wide_has_tri(t.tBits)) visit();
    uint32_t pend = __ballot_sync(kFull, wide_has_tri(t.tBits));
    const uint32_t run = __ballot_sync(kFull, t.node != kNoNode && !wide_has_tri(t.tBits));
    if (run == 0u && pend == 0u) return false;
    if (__popc(pend) >= kTriLanes || run == 0u) {
        do {
            if (wide_has_tri(t.tBits)) test();
            pend = __ballot_sync(kFull, wide_has_tri(t.tBits));
        } while (__popc(pend) >= kTriStop);
    }
    return true;
}

// The one-thread forms test a node's triangles before they move on: with the
// move first, lanes without triangles ran ahead of the others and the warp
// fell apart (90 instead of 31 ms for the 961x541 15-spp field frame).
template <typename Ctr>
__device__ bool trace_closest_wide(const DevScene& s, const V3& o, const V3& d, HitRec* out, Ctr& ctr) {
    WideTrav t;
    uint2 stack[kStackWide];
    wide_init(t, o, d, FLT_MAX);
    for (;;) {
        if (++t.visits > kMaxVisits) {
            wide_abort(s, t, kErrTraversalLimit);
            break;
        }
        ctr.node();
        uint32_t gBase, gImask, gInner;
        wide_node(s, t.node, t.r, t.tmax, t.octInv, &gBase, &gImask, &gInner, &t.tBase, &t.tBits);
        while (wide_has_tri(t.tBits)) {
            ctr.tri();
            wide_test_closest(s, t);
        }
        wide_next(s, t, stack, gBase, gImask, gInner);
        if (t.node == kNoNode) break;
    }
    out->t = t.tmax;
    out->u = t.bu;
    out->v = t.bv;
    out->gid = t.bestGid;
    return t.bestGid != 0xffffffffu;
}

template <typename Ctr>
__device__ bool trace_occluded_wide(const DevScene& s, const V3& o, const V3& d, float maxDist, Ctr& ctr) {
    WideTrav t;
    uint2 stack[kStackWide];
    wide_init(t, o, d, maxDist);
    for (;;) {
        if (++t.visits > kMaxVisits) {
            wide_abort(s, t, kErrTraversalLimit);
            return false;
        }
        ctr.onode();
        uint32_t gBase, gImask, gInner;
        wide_node(s, t.node, t.r, t.tmax, t.octInv, &gBase, &gImask, &gInner, &t.tBase, &t.tBits);
        while (wide_has_tri(t.tBits)) {
            ctr.otri();
            if (wide_test_any(s, t)) return true;
        }
        wide_next(s, t, stack, gBase, gImask, gInner);
        if (t.node == kNoNode) return false;
    }
}

template <typename Ctr>
__device__ __noinline__ bool trace_closest(const DevScene& s, const V3 o, const V3 d, HitRec* out, Ctr& ctr) {
    ctr.closest();
    if (s.nodes8) return trace_closest_wide(s, o, d, out, ctr);
    const RayInv r = ray_inv(o, d);
    float bestT = FLT_MAX;
    uint32_t bestGid = 0xffffffffu;
    float bu = 0.0f, bv = 0.0f;
    int stackNode[kStack];
    float stackT[kStack];
    int sp = 0;
    int node = 0;
    uint32_t visits = 0;
    for (;;) {
        if (++visits > kMaxVisits) {
            atomicOr(s.error, kErrTraversalLimit);
            bestGid = 0xffffffffu;
            break;
        }
        if (node >= 0) {
            ctr.node();
            const float4* np = s.nodes + 4 * static_cast<size_t>(node);
            const float4 n0 = __ldg(np), n1 = __ldg(np + 1), n2 = __ldg(np + 2), n3 = __ldg(np + 3);
            float t0, t1;
            bool h0, h1;
            node_boxes(n0, n1, n2, r, bestT, &t0, &t1, &h0, &h1);
            const int c0 = __float_as_int(n3.x), c1 = __float_as_int(n3.y);
            if (h0 && h1) {
                const bool swap = t1 < t0;
                if (sp >= kStack) {
                    atomicOr(s.error, kErrStackOverflow);
                    bestGid = 0xffffffffu;
                    break;
                }
                stackNode[sp] = swap ? c0 : c1;
                stackT[sp] = swap ? t0 : t1;
                ++sp;
                node = swap ? c1 : c0;
                continue;
            }
            if (h0) {
                node = c0;
                continue;
            }
            if (h1) {
                node = c1;
                continue;
            }
        } else {
            const uint32_t enc = ~static_cast<uint32_t>(node);
            const uint32_t first = enc >> 3, cnt = (enc & 7u) + 1u;
            for (uint32_t k = first; k < first + cnt; ++k) {
                ctr.tri();
                const float4* tp = s.tris + 3 * static_cast<size_t>(k);
                const float4 a = __ldg(tp), b = __ldg(tp + 1), c = __ldg(tp + 2);
                float t, u, v;
                if (!tri_test(o, d, kRayEpsilon, FLT_MAX, a, b, c, &t, &u, &v)) continue;
                const uint32_t gid = __float_as_uint(a.w);
                if (t < bestT || (t == bestT && gid < bestGid)) {
                    bestT = t;
                    bestGid = gid;
                    bu = u;
                    bv = v;
                }
            }
        }
        // pop the next entry still in range
        bool found = false;
        while (sp > 0) {
            --sp;
            if (stackT[sp] <= bestT) {
                node = stackNode[sp];
                found = true;
                break;
            }
        }
        if (!found) break;
    }
    out->t = bestT;
    out->u = bu;
    out->v = bv;
    out->gid = bestGid;
    return bestGid != 0xffffffffu;
}

// Any hit with t in [1e-4, maxDist] (Occluded, CpuPathTracer.cpp:468-475).
template <typename Ctr>
__device__ __noinline__ bool trace_occluded(const DevScene& s, const V3 o, const V3 d, float maxDist, Ctr& ctr) {
    ctr.occlusion();
    if (s.nodes8) return trace_occluded_wide(s, o, d, maxDist, ctr);
    const RayInv r = ray_inv(o, d);
    int stackNode[kStack];
    int sp = 0;
    int node = 0;
    uint32_t visits = 0;
    for (;;) {
        if (++visits > kMaxVisits) {
            atomicOr(s.error, kErrTraversalLimit);
            return false;
        }
        if (node >= 0) {
            ctr.onode();
            const float4* np = s.nodes + 4 * static_cast<size_t>(node);
            const float4 n0 = __ldg(np), n1 = __ldg(np + 1), n2 = __ldg(np + 2), n3 = __ldg(np + 3);
            float t0, t1;
            bool h0, h1;
            node_boxes(n0, n1, n2, r, maxDist, &t0, &t1, &h0, &h1);
            const int c0 = __float_as_int(n3.x), c1 = __float_as_int(n3.y);
            if (h0 && h1) {
                if (sp >= kStack) {
                    atomicOr(s.error, kErrStackOverflow);
                    return false;
                }
                const bool swap = t1 < t0;
                stackNode[sp++] = swap ? c0 : c1;
                node = swap ? c1 : c0;
                continue;
            }
            if (h0) {
                node = c0;
                continue;
            }
            if (h1) {
                node = c1;
                continue;
            }
        } else {
            const uint32_t enc = ~static_cast<uint32_t>(node);
            const uint32_t first = enc >> 3, cnt = (enc & 7u) + 1u;
            for (uint32_t k = first; k < first + cnt; ++k) {
                ctr.otri();
                const float4* tp = s.tris + 3 * static_cast<size_t>(k);
                const float4 a = __ldg(tp), b = __ldg(tp + 1), c = __ldg(tp + 2);
                float t, u, v;
                if (tri_test(o, d, kRayEpsilon, maxDist, a, b, c, &t, &u, &v)) return true;
            }
        }
        if (sp == 0) return false;
        node = stackNode[--sp];
    }
}

// ---- warp forms ----
//
// A warp's rays traced side by side: all 32 lanes call, `on` marks the lanes
// that have a ray, and the results are those of trace_closest and
// trace_occluded (a lane takes the same steps in the same order).  Left to the
// compiler, lanes whose traversals take different branches stay apart and the
// warp runs them one by one; here the ballots of every step bring the lanes
// together again.  Binary leaves wait until kBinLeafLanes lanes have reached
// one or no lane has a node left (1: 18.8 ms for the 961x541 15-spp field frame
// in the plain form, 4: 18.6, 8: 18.7).  The two trees have functions of their
// own: one function with both keeps the registers and the stack of the larger,
// 15.8 instead of 13.6 ms.
constexpr int kBinLeafLanes = 4;
constexpr int kBinDone = static_cast<int>(0x80000000u);  // no node (no leaf is encoded so)

template <bool kAny>
__device__ __forceinline__ uint32_t warp_binary(const DevScene& s, bool on, const V3& o, const V3& d, float maxDist,
                                                HitRec* out) {
    const RayInv r = ray_inv(o, d);
    float bestT = maxDist;
    uint32_t bestGid = 0xffffffffu;
    float bu = 0.0f, bv = 0.0f;
    int stackNode[kStack];
    float stackT[kAny ? 1 : kStack];
    int sp = 0;
    int node = on ? 0 : kBinDone;
    uint32_t visits = 0;
    for (;;) {
        const uint32_t leaves = __ballot_sync(kFull, node < 0 && node != kBinDone);
        const uint32_t inner = __ballot_sync(kFull, node >= 0);
        if ((leaves | inner) == 0u) break;
        const bool testLeaves = __popc(leaves) >= kBinLeafLanes || inner == 0u;
        bool pop = false;
        if (node >= 0) {
            if (++visits > kMaxVisits) {
                atomicOr(s.error, kErrTraversalLimit);
                bestGid = 0xffffffffu;
                node = kBinDone;
            } else {
                const float4* np = s.nodes + 4 * static_cast<size_t>(node);
                const float4 n0 = __ldg(np), n1 = __ldg(np + 1), n2 = __ldg(np + 2), n3 = __ldg(np + 3);
                float t0, t1;
                bool h0, h1;
                node_boxes(n0, n1, n2, r, bestT, &t0, &t1, &h0, &h1);
                const int c0 = __float_as_int(n3.x), c1 = __float_as_int(n3.y);
                const bool swap = h1 && (!h0 || t1 < t0);
                node = swap ? c1 : c0;
                if (h0 && h1) {
                    if (sp < kStack) {
                        stackNode[sp] = swap ? c0 : c1;
                        if constexpr (!kAny) stackT[sp] = swap ? t0 : t1;
                        ++sp;
                    } else {
                        atomicOr(s.error, kErrStackOverflow);
                        bestGid = 0xffffffffu;
                        node = kBinDone;
                    }
                }
                pop = !(h0 || h1);
            }
        } else if (testLeaves && node != kBinDone) {
            const uint32_t enc = ~static_cast<uint32_t>(node);
            const uint32_t first = enc >> 3, cnt = (enc & 7u) + 1u;
            pop = true;
            for (uint32_t k = first; k < first + cnt; ++k) {
                const float4* tp = s.tris + 3 * static_cast<size_t>(k);
                const float4 a = __ldg(tp), b = __ldg(tp + 1), c = __ldg(tp + 2);
                float t, u, v;
                if (!tri_test(o, d, kRayEpsilon, kAny ? maxDist : FLT_MAX, a, b, c, &t, &u, &v)) continue;
                if constexpr (kAny) {
                    bestGid = 0u;
                    sp = 0;
                    break;
                } else {
                    const uint32_t gid = __float_as_uint(a.w);
                    if (t < bestT || (t == bestT && gid < bestGid)) {
                        bestT = t;
                        bestGid = gid;
                        bu = u;
                        bv = v;
                    }
                }
            }
        }
        if (pop) {  // the next entry still in range
            node = kBinDone;
            while (sp > 0) {
                --sp;
                if (kAny || stackT[kAny ? 0 : sp] <= bestT) {
                    node = stackNode[sp];
                    break;
                }
            }
        }
    }
    if constexpr (!kAny) *out = HitRec{bestT, bu, bv, bestGid};
    return bestGid;
}

static __device__ __noinline__ bool warp_closest_wide(const DevScene& s, bool on, const V3 o, const V3 d, HitRec* out) {
    WideTrav t;
    uint2 stack[kStackWide];
    wide_init(t, o, d, FLT_MAX);
    if (!on) t.node = kNoNode;
    while (trav_step(t, [&] { wide_visit(s, t, stack); }, [&] { wide_test_closest(s, t); })) {
    }
    *out = HitRec{t.tmax, t.bu, t.bv, t.bestGid};
    return t.bestGid != 0xffffffffu;
}

static __device__ __noinline__ bool warp_occluded_wide(const DevScene& s, bool on, const V3 o, const V3 d, float maxDist) {
    WideTrav t;
    uint2 stack[kStackWide];
    wide_init(t, o, d, maxDist);
    if (!on) t.node = kNoNode;
    bool hit = false;
    const auto test = [&] {
        if (!wide_test_any(s, t)) return;
        hit = true;
        t.node = kNoNode;
        t.tBits = 0u;
    };
    while (trav_step(t, [&] { wide_visit(s, t, stack); }, test)) {
    }
    return hit;
}

static __device__ __noinline__ bool warp_closest_binary(const DevScene& s, bool on, const V3 o, const V3 d, HitRec* out) {
    return warp_binary<false>(s, on, o, d, FLT_MAX, out) != 0xffffffffu;
}

static __device__ __noinline__ bool warp_occluded_binary(const DevScene& s, bool on, const V3 o, const V3 d, float maxDist) {
    return warp_binary<true>(s, on, o, d, maxDist, nullptr) != 0xffffffffu;
}

// trace_closest of the lanes with `on`; the others get false.
__device__ __forceinline__ bool warp_closest(const DevScene& s, bool on, const V3& o, const V3& d, HitRec* out) {
    __syncwarp();
    return s.nodes8 ? warp_closest_wide(s, on, o, d, out) : warp_closest_binary(s, on, o, d, out);
}

// trace_occluded of the lanes with `on`; the others get false.
__device__ __forceinline__ bool warp_occluded(const DevScene& s, bool on, const V3& o, const V3& d, float maxDist) {
    __syncwarp();
    return s.nodes8 ? warp_occluded_wide(s, on, o, d, maxDist) : warp_occluded_binary(s, on, o, d, maxDist);
}

}  // namespace shiro_gpu
