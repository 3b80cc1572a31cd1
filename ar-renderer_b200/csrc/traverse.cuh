// BVH traversal for sm_100a: closest-hit and any-hit queries over the caller's binary BVH, with
// results bit-identical to the reference CPU routines pr::BVH::Intersect / IntersectP
// (src/geometry/bvh.cpp:137-232) and pr::Triangle::Intersect (src/geometry/shape.cpp:202-222).
//
// Layout (built on the device from the v4 node array by convert_nodes in accel.cu):
//   WNode, 64 B, one per INTERIOR reference node: both children's boxes plus their references,
//   so one node visit issues four 16-byte loads that bring both child boxes at once. A child
//   reference >= 0 names an interior WNode; < 0 is a leaf whose first leaf slot is ~ref.
//   LeafPrim, 48 B per leaf slot (primOrder order): triangle p0 | e1 = p1 - p0 | e2 = p2 - p0 and
//   the original primitive index; spheres store centre and radius (64-bit test, as the CPU).
//   The last slot of every leaf carries an end mark, so a stack entry is just (ref, entry t).
//
// Parity. The reference pops a node, tests its own box against the CURRENT tMax, and pushes the
// far child before descending into the near one (near = by the sign of the split axis). Here a
// parent tests both child boxes at once, but only the tMax-independent part of the far child's
// test is evaluated early: its entry distance is pushed with it and compared against the tMax
// current at pop time, exactly the reference's final `tMin < tMax` clause. Every arithmetic step
// is an explicitly rounded IEEE operation (__fadd_rn/__fmul_rn/__fdiv_rn, never contracted into
// an FMA), so box decisions, visit order, tMax updates and hits match bit for bit.
#pragma once

#include "common.cuh"

namespace prb {

struct __align__(16) WNode {
    float4 a;  // c0.min.x c0.min.y c0.min.z c0.max.x
    float4 b;  // c0.max.y c0.max.z c1.min.x c1.min.y
    float4 c;  // c1.min.z c1.max.x c1.max.y c1.max.z
    int4 r;    // ref0, ref1, axis, unused
};

struct __align__(16) LeafPrim {
    float4 v0;  // triangle: p0, prim index (int bits); sphere: centre, prim index
    float4 v1;  // triangle: e1, kind 0; sphere: radius, 0, 0, kind 1
    float4 v2;  // triangle: e2, end-of-leaf mark (int bits 1 on a leaf's last slot, else 0)
};

// 4-wide node, collapsed on the host from the binary tree: the four child boxes stored per axis
// (child i in component i of each float4) and the four child references; 128 bytes, one L2 line.
// Unused child slots carry an inverted box (+inf / -inf), which the slab test always rejects.
struct __align__(16) QNode {
    float4 lox, loy, loz, hix, hiy, hiz;
    int4 child;  // >= 0: interior QNode; < 0: leaf whose first slot is ~child
    int4 pad;
};
// The any-hit traversal addresses the plane vectors by byte offset (slab2).
static_assert(offsetof(QNode, lox) == 0 && offsetof(QNode, loy) == 16 && offsetof(QNode, loz) == 32 &&
                  offsetof(QNode, hix) == 48 && offsetof(QNode, hiy) == 64 && offsetof(QNode, hiz) == 80 &&
                  sizeof(QNode) == 128,
              "QNode layout");

constexpr int kStackSize = 64;
// 1 + 2 * 1.2e-7f * 3 evaluated in float, the far-distance widening of bvh.cpp:143-151.
constexpr float kWiden = 0x1.00000cp+0f;

struct TraceRay {
    V3 o, d, inv;
    int neg[3];
    bool infInv;  // a direction component is +-0: some slab tests can produce NaN
};

__device__ __forceinline__ TraceRay make_trace_ray(V3 o, V3 d) {
    TraceRay r;
    r.o = o;
    r.d = d;
    r.inv = {__fdiv_rn(1.f, d.x), __fdiv_rn(1.f, d.y), __fdiv_rn(1.f, d.z)};
    r.neg[0] = r.inv.x < 0.f;
    r.neg[1] = r.inv.y < 0.f;
    r.neg[2] = r.inv.z < 0.f;
    r.infInv = isinf(r.inv.x) || isinf(r.inv.y) || isinf(r.inv.z);
    return r;
}

// The tMax-independent part of the reference slab test (bvh.cpp:137-156): returns false when the
// box is rejected for every tMax; otherwise writes the entry distance tMin, and the box is hit
// iff tMin < tMax. Comparison order follows the reference so NaN cases resolve the same way.
__device__ __forceinline__ bool box_entry(const TraceRay &r, float lox, float loy, float loz, float hix, float hiy,
                                          float hiz, float *tEntry) {
    float nx = r.neg[0] ? hix : lox, fx = r.neg[0] ? lox : hix;
    float ny = r.neg[1] ? hiy : loy, fy = r.neg[1] ? loy : hiy;
    float nz = r.neg[2] ? hiz : loz, fz = r.neg[2] ? loz : hiz;
    float tMin = __fmul_rn(__fsub_rn(nx, r.o.x), r.inv.x);
    float tMaxX = __fmul_rn(__fsub_rn(fx, r.o.x), r.inv.x);
    float tyMin = __fmul_rn(__fsub_rn(ny, r.o.y), r.inv.y);
    float tyMax = __fmul_rn(__fsub_rn(fy, r.o.y), r.inv.y);
    tMaxX = __fmul_rn(tMaxX, kWiden);
    tyMax = __fmul_rn(tyMax, kWiden);
    if (tMin > tyMax || tyMin > tMaxX) return false;
    if (tyMin > tMin) tMin = tyMin;
    if (tyMax < tMaxX) tMaxX = tyMax;
    float tzMin = __fmul_rn(__fsub_rn(nz, r.o.z), r.inv.z);
    float tzMax = __fmul_rn(__fsub_rn(fz, r.o.z), r.inv.z);
    tzMax = __fmul_rn(tzMax, kWiden);
    if (tMin > tzMax || tzMin > tMaxX) return false;
    if (tzMin > tMin) tMin = tzMin;
    if (tzMax < tMaxX) tMaxX = tzMax;
    *tEntry = tMin;
    return tMaxX > 0.f;
}

// The same slab test without branches, for rays whose reciprocal direction is finite: the same
// products, and max of the entries / min of the (widened) exits. For such rays every entry is at
// most its own slab's exit unless that exit is negative, so "max entry <= min exit" is the
// reference's pairwise tests and the results (accept, entry distance) are identical; rays with an
// infinite reciprocal use box_entry (its NaN handling differs from fminf / fmaxf).
__device__ __forceinline__ bool box_entry_nb(const TraceRay &r, float lox, float loy, float loz, float hix, float hiy,
                                             float hiz, float *tEntry) {
    float nx = r.neg[0] ? hix : lox, fx = r.neg[0] ? lox : hix;
    float ny = r.neg[1] ? hiy : loy, fy = r.neg[1] ? loy : hiy;
    float nz = r.neg[2] ? hiz : loz, fz = r.neg[2] ? loz : hiz;
    float t0 = fmaxf(fmaxf(__fmul_rn(__fsub_rn(nx, r.o.x), r.inv.x), __fmul_rn(__fsub_rn(ny, r.o.y), r.inv.y)),
                     __fmul_rn(__fsub_rn(nz, r.o.z), r.inv.z));
    float t1 = fminf(fminf(__fmul_rn(__fmul_rn(__fsub_rn(fx, r.o.x), r.inv.x), kWiden),
                           __fmul_rn(__fmul_rn(__fsub_rn(fy, r.o.y), r.inv.y), kWiden)),
                     __fmul_rn(__fmul_rn(__fsub_rn(fz, r.o.z), r.inv.z), kWiden));
    *tEntry = t0;
    return t0 <= t1 && t1 > 0.f;
}

// Two floats in one 64-bit register, for the paired FP32 instructions of sm_100 (each half is its own
// correctly rounded operation, so results are those of the scalar instructions at half the issue slots).
__device__ __forceinline__ uint64_t pair_of(float lo, float hi) {
    uint64_t p;
    asm("mov.b64 %0, {%1, %2};" : "=l"(p) : "f"(lo), "f"(hi));
    return p;
}
__device__ __forceinline__ void unpair(uint64_t p, float &lo, float &hi) {
    asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(p));
}
__device__ __forceinline__ uint64_t add2(uint64_t a, uint64_t b) {
    uint64_t p;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(p) : "l"(a), "l"(b));
    return p;
}
__device__ __forceinline__ uint64_t mul2(uint64_t a, uint64_t b) {
    uint64_t p;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(p) : "l"(a), "l"(b));
    return p;
}
__device__ __forceinline__ float max3(float a, float b, float c) {
    float d;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
    return d;
}
__device__ __forceinline__ float min3(float a, float b, float c) {
    float d;
    asm("min.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
    return d;
}

// box_entry_nb of two boxes at once, with the near and far planes already chosen by the ray's octant
// (QNode layout: lo x, y, z at bytes 0, 16, 32, hi at 48, 64, 80): the same products and comparisons,
// folded with the tMax test; +inf when a box is rejected or entered at or after tMax. The exits are
// widened after their minimum: rounding is monotone, so that is the minimum of the widened exits.
// A node step is bound by issue slots: pairs, three-operand min / max and one widening a box take about
// 50 instructions for four boxes instead of 84. Ray-query benchmark (2^24 rays, ms, closest / any hit):
// 4.25 / 2.96 -> 4.20 / 2.92; 4,096-triangle soup, 2^22 rays: 0.838 / 0.611 -> 0.804 / 0.594.
__device__ __forceinline__ void slab2(const TraceRay &r, uint64_t nx, uint64_t fx, uint64_t ny, uint64_t fy,
                                      uint64_t nz, uint64_t fz, float tMax, float &tA, float &tB) {
    const uint64_t ox = pair_of(-r.o.x, -r.o.x), oy = pair_of(-r.o.y, -r.o.y), oz = pair_of(-r.o.z, -r.o.z);
    const uint64_t ix = pair_of(r.inv.x, r.inv.x), iy = pair_of(r.inv.y, r.inv.y), iz = pair_of(r.inv.z, r.inv.z);
    float xa, xb, ya, yb, za, zb;
    unpair(mul2(add2(nx, ox), ix), xa, xb);
    unpair(mul2(add2(ny, oy), iy), ya, yb);
    unpair(mul2(add2(nz, oz), iz), za, zb);
    const float na = max3(xa, ya, za), nb = max3(xb, yb, zb);
    unpair(mul2(add2(fx, ox), ix), xa, xb);
    unpair(mul2(add2(fy, oy), iy), ya, yb);
    unpair(mul2(add2(fz, oz), iz), za, zb);
    const float ea = __fmul_rn(min3(xa, ya, za), kWiden), eb = __fmul_rn(min3(xb, yb, zb), kWiden);
    const float inf = __int_as_float(0x7f800000);
    tA = na <= ea && ea > 0.f && na < tMax ? na : inf;
    tB = nb <= eb && eb > 0.f && nb < tMax ? nb : inf;
}

// slab2 of one box.
__device__ __forceinline__ float slab_nf(const TraceRay &r, float nx, float fx, float ny, float fy, float nz, float fz,
                                         float tMax) {
    const float t0 = max3(__fmul_rn(__fsub_rn(nx, r.o.x), r.inv.x), __fmul_rn(__fsub_rn(ny, r.o.y), r.inv.y),
                          __fmul_rn(__fsub_rn(nz, r.o.z), r.inv.z));
    const float t1 = __fmul_rn(min3(__fmul_rn(__fsub_rn(fx, r.o.x), r.inv.x), __fmul_rn(__fsub_rn(fy, r.o.y), r.inv.y),
                                    __fmul_rn(__fsub_rn(fz, r.o.z), r.inv.z)),
                               kWiden);
    return t0 <= t1 && t1 > 0.f && t0 < tMax ? t0 : __int_as_float(0x7f800000);
}

// Möller-Trumbore in the reference's exact operation order (shape.cpp:202-222).
__device__ __forceinline__ float dot_rn(float ax, float ay, float az, float bx, float by, float bz) {
    return __fadd_rn(__fadd_rn(__fmul_rn(ax, bx), __fmul_rn(ay, by)), __fmul_rn(az, bz));
}
__device__ __forceinline__ bool hit_triangle(const TraceRay &r, float4 v0, float4 v1, float4 v2, float tMax, float *tHit,
                                             float *bu, float *bv) {
    // pvec = d x e2
    float px = __fsub_rn(__fmul_rn(r.d.y, v2.z), __fmul_rn(r.d.z, v2.y));
    float py = __fsub_rn(__fmul_rn(r.d.z, v2.x), __fmul_rn(r.d.x, v2.z));
    float pz = __fsub_rn(__fmul_rn(r.d.x, v2.y), __fmul_rn(r.d.y, v2.x));
    float det = dot_rn(v1.x, v1.y, v1.z, px, py, pz);
    if (det == 0.f || !isfinite(det)) return false;
    float inv = __fdiv_rn(1.f, det);
    float tx = __fsub_rn(r.o.x, v0.x), ty = __fsub_rn(r.o.y, v0.y), tz = __fsub_rn(r.o.z, v0.z);
    float u = __fmul_rn(dot_rn(tx, ty, tz, px, py, pz), inv);
    if (u < 0.f || u > 1.f) return false;
    // qvec = tvec x e1
    float qx = __fsub_rn(__fmul_rn(ty, v1.z), __fmul_rn(tz, v1.y));
    float qy = __fsub_rn(__fmul_rn(tz, v1.x), __fmul_rn(tx, v1.z));
    float qz = __fsub_rn(__fmul_rn(tx, v1.y), __fmul_rn(ty, v1.x));
    float v = __fmul_rn(dot_rn(r.d.x, r.d.y, r.d.z, qx, qy, qz), inv);
    if (v < 0.f || __fadd_rn(u, v) > 1.f) return false;
    float t = __fmul_rn(dot_rn(v2.x, v2.y, v2.z, qx, qy, qz), inv);
    if (t <= 0.f || t >= tMax) return false;
    *tHit = t;
    *bu = u;
    *bv = v;
    return true;
}

// Robust sphere quadratic in double precision, as pr::Sphere::Intersect (shape.cpp:42-61).
__device__ __forceinline__ bool hit_sphere(const TraceRay &r, float4 v0, float4 v1, float tMax, float *tHit) {
    // The origin offset is a float subtraction widened afterwards, as in the reference.
    double ox = __fsub_rn(r.o.x, v0.x), oy = __fsub_rn(r.o.y, v0.y), oz = __fsub_rn(r.o.z, v0.z);
    double dx = r.d.x, dy = r.d.y, dz = r.d.z;
    double rad = v1.x;
    double a = __dadd_rn(__dadd_rn(__dmul_rn(dx, dx), __dmul_rn(dy, dy)), __dmul_rn(dz, dz));
    double b = __dadd_rn(__dadd_rn(__dmul_rn(ox, dx), __dmul_rn(oy, dy)), __dmul_rn(oz, dz));
    double c = __dsub_rn(__dadd_rn(__dadd_rn(__dmul_rn(ox, ox), __dmul_rn(oy, oy)), __dmul_rn(oz, oz)),
                         __dmul_rn(rad, rad));
    double k = __ddiv_rn(b, a);
    double lx = __dsub_rn(ox, __dmul_rn(k, dx)), ly = __dsub_rn(oy, __dmul_rn(k, dy)),
           lz = __dsub_rn(oz, __dmul_rn(k, dz));
    double disc = __dsub_rn(__dmul_rn(rad, rad),
                            __dadd_rn(__dadd_rn(__dmul_rn(lx, lx), __dmul_rn(ly, ly)), __dmul_rn(lz, lz)));
    if (disc < 0.0) return false;
    double q = __dsub_rn(-b, copysign(__dsqrt_rn(__dmul_rn(a, disc)), b));
    double t0 = __ddiv_rn(c, q), t1 = __ddiv_rn(q, a);
    if (t0 > t1) {
        double s = t0;
        t0 = t1;
        t1 = s;
    }
    double t = t0;
    if (t <= 0.0) t = t1;
    if (t <= 0.0 || t >= double(tMax)) return false;
    *tHit = float(t);
    return true;
}

struct Hit {
    float t, u, v;
    int prim;  // original primitive index, -1 = none
};

// Closest hit (kAny = false) or any hit (kAny = true) with t in (0, tMax). Spheres are tested only
// when kSpheres. rootRef describes the root (interior WNode 0, or a single leaf), rootBox its
// bounds. Sets *overflow (and stops) when the traversal stack would overflow.
template <bool kAny, bool kSpheres>
__device__ __forceinline__ bool traverse(const WNode *__restrict__ nodes, const LeafPrim *__restrict__ prims,
                                         const float *__restrict__ rootBox, int rootRef, const TraceRay &r,
                                         float tMax, Hit *hit, bool *overflow) {
    int stackRef[kStackSize];
    float stackT[kStackSize];
    int sp = 0;
    bool found = false;
    float tEntry;
    if (!box_entry(r, rootBox[0], rootBox[1], rootBox[2], rootBox[3], rootBox[4], rootBox[5], &tEntry) ||
        !(tEntry < tMax))
        return false;
    int ref = rootRef;
    while (true) {
        if (ref >= 0) {
            const WNode *n = nodes + ref;
            float4 a = __ldg(&n->a), b = __ldg(&n->b), c = __ldg(&n->c);
            int4 rr = __ldg(&n->r);
            float t0, t1;
            bool h0 = box_entry(r, a.x, a.y, a.z, a.w, b.x, b.y, &t0);
            bool h1 = box_entry(r, b.z, b.w, c.x, c.y, c.z, c.w, &t1);
            // Near child by the sign of the split axis (bvh.cpp:184-190): the second child first
            // when the ray runs towards -axis.
            bool secondFirst = r.neg[rr.z];
            int nRef = secondFirst ? rr.y : rr.x, fRef = secondFirst ? rr.x : rr.y;
            bool nHit = secondFirst ? h1 : h0, fHit = secondFirst ? h0 : h1;
            float nT = secondFirst ? t1 : t0, fT = secondFirst ? t0 : t1;
            if (fHit) {
                if (sp >= kStackSize) {
                    *overflow = true;
                    return found;
                }
                stackRef[sp] = fRef;
                stackT[sp] = fT;
                ++sp;
            }
            if (nHit && nT < tMax) {
                ref = nRef;
                continue;
            }
        } else {
            const LeafPrim *p = prims + ~ref;
            for (bool last = false; !last; ++p) {
                float4 v0 = __ldg(&p->v0), v1 = __ldg(&p->v1), v2 = __ldg(&p->v2);
                last = __float_as_int(v2.w) != 0;
                float t, u = 0.f, v = 0.f;
                bool h;
                if (kSpheres && __float_as_int(v1.w) == 1)
                    h = hit_sphere(r, v0, v1, tMax, &t);
                else
                    h = hit_triangle(r, v0, v1, v2, tMax, &t, &u, &v);
                if (h) {
                    if (kAny) return true;
                    tMax = t;
                    hit->t = t;
                    hit->u = u;
                    hit->v = v;
                    hit->prim = __float_as_int(v0.w);
                    found = true;
                }
            }
        }
        // Pop: a deferred far child is visited only if its entry is still before tMax.
        bool next = false;
        while (sp > 0) {
            --sp;
            if (stackT[sp] < tMax) {
                ref = stackRef[sp];
                next = true;
                break;
            }
        }
        if (!next) break;
    }
    return found;
}

// The same traversal cut into steps (one interior node or one leaf per call), for persistent
// warps that hand a finished lane a new ray at once instead of waiting for the warp's longest
// ray. Visit order, box and triangle arithmetic are those of traverse(), so results are
// identical. Returns true when the ray's traversal is finished.
struct TravState {
    int ref, sp;
    float tMax;
    bool found;
    bool crossed;  // kSkipTransparent: a transparent primitive was intersected before tMax
    Hit hit;
};

// Bit of a primitive's class byte marking it transparent to shadow rays (a medium interface).
constexpr uint8_t kTransparentBit = 0x80;

template <bool kAny, bool kSpheres>
__device__ __forceinline__ bool traverse_step(const WNode *__restrict__ nodes, const LeafPrim *__restrict__ prims,
                                              const TraceRay &r, TravState &s, int *stackRef, float *stackT,
                                              bool *overflow) {
    if (s.ref >= 0) {
        const WNode *n = nodes + s.ref;
        float4 a = __ldg(&n->a), b = __ldg(&n->b), c = __ldg(&n->c);
        int4 rr = __ldg(&n->r);
        float t0, t1;
        bool h0 = box_entry(r, a.x, a.y, a.z, a.w, b.x, b.y, &t0);
        bool h1 = box_entry(r, b.z, b.w, c.x, c.y, c.z, c.w, &t1);
        bool secondFirst = r.neg[rr.z];
        int nRef = secondFirst ? rr.y : rr.x, fRef = secondFirst ? rr.x : rr.y;
        bool nHit = secondFirst ? h1 : h0, fHit = secondFirst ? h0 : h1;
        float nT = secondFirst ? t1 : t0, fT = secondFirst ? t0 : t1;
        if (fHit) {
            if (s.sp >= kStackSize) {
                *overflow = true;
                return true;
            }
            stackRef[s.sp] = fRef;
            stackT[s.sp] = fT;
            ++s.sp;
        }
        if (nHit && nT < s.tMax) {
            s.ref = nRef;
            return false;
        }
    } else {
        const LeafPrim *p = prims + ~s.ref;
        for (bool last = false; !last; ++p) {
            float4 v0 = __ldg(&p->v0), v1 = __ldg(&p->v1), v2 = __ldg(&p->v2);
            last = __float_as_int(v2.w) != 0;
            float t, u = 0.f, v = 0.f;
            bool h;
            if (kSpheres && __float_as_int(v1.w) == 1)
                h = hit_sphere(r, v0, v1, s.tMax, &t);
            else
                h = hit_triangle(r, v0, v1, v2, s.tMax, &t, &u, &v);
            if (h) {
                s.found = true;
                if (kAny) return true;
                s.tMax = t;
                s.hit.t = t;
                s.hit.u = u;
                s.hit.v = v;
                s.hit.prim = __float_as_int(v0.w);
            }
        }
    }
    while (s.sp > 0) {
        --s.sp;
        if (stackT[s.sp] < s.tMax) {
            s.ref = stackRef[s.sp];
            return false;
        }
    }
    return true;
}

// The step traversal over the 4-wide tree: the children a node's slab tests accept (entry before
// tMax) are visited nearest first, the others pushed with their entry distance, farthest first.
// Box and triangle arithmetic are those of the binary traversal, so a hit's primitive and
// distance are the reference's; only among hits at exactly equal distances, or closer together than
// the rounding of a box's entry, can the visit order tell (the binary traversal reproduces the
// reference's order for those).
__device__ __forceinline__ void cswap(float &ta, int &ra, float &tb, int &rb) {
    if (tb < ta) {
        float t = ta;
        ta = tb;
        tb = t;
        int q = ra;
        ra = rb;
        rb = q;
    }
}

// Sorting network for 4 (5 compare-exchanges); misses sort last at +inf. Not stable: which of two children
// entered at the same distance comes first is the network's doing, and part of the visit order.
__device__ __forceinline__ void sort4(float &t0, int &r0, float &t1, int &r1, float &t2, int &r2, float &t3, int &r3) {
    cswap(t0, r0, t1, r1);
    cswap(t2, r2, t3, r3);
    cswap(t0, r0, t2, r2);
    cswap(t1, r1, t3, r3);
    cswap(t1, r1, t2, r2);
}

// The traversal stack as two per-thread arrays (local memory).
struct LocalStack {
    int *ref;
    float *t;
    __device__ __forceinline__ void put(int i, int r, float d) {
        ref[i] = r;
        t[i] = d;
    }
    __device__ __forceinline__ float dist(int i) const { return t[i]; }
    __device__ __forceinline__ int node(int i) const { return ref[i]; }
};

// The bottom kShort entries of a thread's stack in shared memory, the rest in local memory. `sh`
// points at the thread's column of its block's [kShort][kThreads] array, so that the lanes of a
// warp touch consecutive words (no bank conflicts); traversals rarely go deeper than kShort, so
// the local-memory part, which shares the L1 with the node and leaf loads, is rarely touched.
template <int kShort, int kThreads>
struct HybridStack;

// Stack entries per thread in shared memory for the 4-wide traversals: 16 x 8 B x 256 threads =
// 32 KiB per block, 128 KiB per SM at 4 resident blocks (measured on the ray-query benchmark:
// 4 -> 3.27, 8 -> 3.53, 16 -> 3.83, 24 -> 3.79 Grays/s, against 3.36 with the whole stack in local
// memory).
constexpr int kShortStack = 16;

// Persistent traversal kernels refill a warp's idle lanes with new rays once this many lanes are
// idle (or none is busy). The refill (ray load, reciprocal direction, root-box test, the finished
// rays' result stores) run whenever a single lane finished executed with one or two lanes active
// in almost every iteration. Measured on the ray-query benchmark (closest / any hit, Mrays/s):
// 1 lane 3,491 / 4,770, 4 lanes 3,704 / 5,110, 8 lanes 3,829 / 5,319, 16 lanes 3,562 / 4,960.
// Results are unchanged: only the iteration at which a lane starts its next ray moves.
constexpr int kRefillLanes = 8;

template <int kShort, int kThreads>
struct HybridStack {
    static constexpr int kRowStride = kThreads;
    int2 *sh;
    int ref[kStackSize - kShort];
    float t[kStackSize - kShort];
    __device__ __forceinline__ void put(int i, int r, float d) {
        if (i < kShort) {
            sh[i * kThreads] = make_int2(r, __float_as_int(d));
        } else {
            ref[i - kShort] = r;
            t[i - kShort] = d;
        }
    }
    __device__ __forceinline__ float dist(int i) const {
        return i < kShort ? __int_as_float(sh[i * kThreads].y) : t[i - kShort];
    }
    __device__ __forceinline__ int node(int i) const { return i < kShort ? sh[i * kThreads].x : ref[i - kShort]; }
};

// Takes the next deferred child whose entry is still before tMax; false: the traversal is finished.
template <class Stack> __device__ __forceinline__ bool traverse4_pop(TravState &s, Stack &stack) {
    while (s.sp > 0) {
        --s.sp;
        if (stack.dist(s.sp) < s.tMax) {
            s.ref = stack.node(s.sp);
            return true;
        }
    }
    return false;
}

// One interior node (s.ref >= 0). Returns true when the ray's traversal is finished.
// kDeferUV (closest hit): a hit records only its leaf slot (s.hit.prim) and distance (s.tMax);
// the caller repeats the winning primitive's test once at the end (finish_hit), which gives the
// same t, u, v bit for bit. Fewer live registers in the loop let the slab planes be selected by
// address as for any hit (ray-query benchmark, closest hit: 3,821 -> 3,926 Mrays/s; either change
// alone was slower: 3,730 and 3,667).
template <bool kAny, bool kDeferUV, class Stack>
__device__ __forceinline__ bool traverse4_node(const QNode *__restrict__ nodes, const TraceRay &r, TravState &s,
                                               Stack &stack, bool *overflow) {
    const QNode *n = nodes + s.ref;
    float t0, t1, t2, t3;
    const float inf = __int_as_float(0x7f800000);
    int4 ch;
    if constexpr (kAny || kDeferUV) {
        ch = __ldg(&n->child);
        if (!r.infInv) {
            // The near and far planes chosen by address from the ray's octant (six loads, no
            // per-child selects). Measured on the ray-query benchmark: any hit 5,314 -> 5,689
            // Mrays/s; closest hit only together with kDeferUV (see above); the closest-hit
            // form that keeps t, u, v live loads all six plane vectors below.
            const char *nb = reinterpret_cast<const char *>(n);
            const int ox = r.neg[0] ? 48 : 0, oy = r.neg[1] ? 48 : 0, oz = r.neg[2] ? 48 : 0;
            const ulonglong2 nx = __ldg(reinterpret_cast<const ulonglong2 *>(nb + ox));
            const ulonglong2 fx = __ldg(reinterpret_cast<const ulonglong2 *>(nb + 48 - ox));
            const ulonglong2 ny = __ldg(reinterpret_cast<const ulonglong2 *>(nb + 16 + oy));
            const ulonglong2 fy = __ldg(reinterpret_cast<const ulonglong2 *>(nb + 64 - oy));
            const ulonglong2 nz = __ldg(reinterpret_cast<const ulonglong2 *>(nb + 32 + oz));
            const ulonglong2 fz = __ldg(reinterpret_cast<const ulonglong2 *>(nb + 80 - oz));
            slab2(r, nx.x, fx.x, ny.x, fy.x, nz.x, fz.x, s.tMax, t0, t1);
            slab2(r, nx.y, fx.y, ny.y, fy.y, nz.y, fz.y, s.tMax, t2, t3);
        } else {
            const float4 lx = __ldg(&n->lox), ly = __ldg(&n->loy), lz = __ldg(&n->loz);
            const float4 hx = __ldg(&n->hix), hy = __ldg(&n->hiy), hz = __ldg(&n->hiz);
            t0 = box_entry(r, lx.x, ly.x, lz.x, hx.x, hy.x, hz.x, &t0) && t0 < s.tMax ? t0 : inf;
            t1 = box_entry(r, lx.y, ly.y, lz.y, hx.y, hy.y, hz.y, &t1) && t1 < s.tMax ? t1 : inf;
            t2 = box_entry(r, lx.z, ly.z, lz.z, hx.z, hy.z, hz.z, &t2) && t2 < s.tMax ? t2 : inf;
            t3 = box_entry(r, lx.w, ly.w, lz.w, hx.w, hy.w, hz.w, &t3) && t3 < s.tMax ? t3 : inf;
        }
    } else {
        const float4 lx = __ldg(&n->lox), ly = __ldg(&n->loy), lz = __ldg(&n->loz);
        const float4 hx = __ldg(&n->hix), hy = __ldg(&n->hiy), hz = __ldg(&n->hiz);
        ch = __ldg(&n->child);
        if (!r.infInv) {
            t0 = box_entry_nb(r, lx.x, ly.x, lz.x, hx.x, hy.x, hz.x, &t0) && t0 < s.tMax ? t0 : inf;
            t1 = box_entry_nb(r, lx.y, ly.y, lz.y, hx.y, hy.y, hz.y, &t1) && t1 < s.tMax ? t1 : inf;
            t2 = box_entry_nb(r, lx.z, ly.z, lz.z, hx.z, hy.z, hz.z, &t2) && t2 < s.tMax ? t2 : inf;
            t3 = box_entry_nb(r, lx.w, ly.w, lz.w, hx.w, hy.w, hz.w, &t3) && t3 < s.tMax ? t3 : inf;
        } else {
            t0 = box_entry(r, lx.x, ly.x, lz.x, hx.x, hy.x, hz.x, &t0) && t0 < s.tMax ? t0 : inf;
            t1 = box_entry(r, lx.y, ly.y, lz.y, hx.y, hy.y, hz.y, &t1) && t1 < s.tMax ? t1 : inf;
            t2 = box_entry(r, lx.z, ly.z, lz.z, hx.z, hy.z, hz.z, &t2) && t2 < s.tMax ? t2 : inf;
            t3 = box_entry(r, lx.w, ly.w, lz.w, hx.w, hy.w, hz.w, &t3) && t3 < s.tMax ? t3 : inf;
        }
    }
    int r0 = ch.x, r1 = ch.y, r2 = ch.z, r3 = ch.w;
    sort4(t0, r0, t1, r1, t2, r2, t3, r3);
    if (t0 < inf) {
        const int extra = (t1 < inf) + (t2 < inf) + (t3 < inf);
        if (s.sp + extra > kStackSize) {
            *overflow = true;
            return true;
        }
        if (t3 < inf) stack.put(s.sp++, r3, t3);
        if (t2 < inf) stack.put(s.sp++, r2, t2);
        if (t1 < inf) stack.put(s.sp++, r1, t1);
        s.ref = r0;
        return false;
    }
    return !traverse4_pop(s, stack);
}

// One leaf (s.ref < 0). Returns true when the ray's traversal is finished.
// kSkipTransparent: primitives whose class byte (cls) has kTransparentBit do not count as hits;
// intersecting one sets s.crossed.
template <bool kAny, bool kSpheres, bool kSkipTransparent, bool kDeferUV, class Stack>
__device__ __forceinline__ bool traverse4_leaf(const LeafPrim *__restrict__ prims, const TraceRay &r, TravState &s,
                                               Stack &stack, const uint8_t *__restrict__ cls = nullptr) {
    const LeafPrim *p = prims + ~s.ref;
    for (bool last = false; !last; ++p) {
        float4 v0 = __ldg(&p->v0), v1 = __ldg(&p->v1), v2 = __ldg(&p->v2);
        last = __float_as_int(v2.w) != 0;
        float t, u = 0.f, v = 0.f;
        bool h;
        if (kSpheres && __float_as_int(v1.w) == 1)
            h = hit_sphere(r, v0, v1, s.tMax, &t);
        else
            h = hit_triangle(r, v0, v1, v2, s.tMax, &t, &u, &v);
        if (h) {
            if (kSkipTransparent && (__ldg(cls + __float_as_int(v0.w)) & kTransparentBit)) {
                s.crossed = true;
                continue;
            }
            s.found = true;
            if (kAny) return true;
            s.tMax = t;
            if constexpr (kDeferUV) {
                s.hit.prim = int(p - prims);
            } else {
                s.hit.t = t;
                s.hit.u = u;
                s.hit.v = v;
                s.hit.prim = __float_as_int(v0.w);
            }
        }
    }
    return !traverse4_pop(s, stack);
}

template <bool kAny, bool kSpheres, bool kSkipTransparent = false, bool kDeferUV = false, class Stack>
__device__ __forceinline__ bool traverse4_step_st(const QNode *__restrict__ nodes, const LeafPrim *__restrict__ prims,
                                                  const TraceRay &r, TravState &s, Stack &stack, bool *overflow,
                                                  const uint8_t *__restrict__ cls = nullptr) {
    if (s.ref >= 0) return traverse4_node<kAny, kDeferUV>(nodes, r, s, stack, overflow);
    return traverse4_leaf<kAny, kSpheres, kSkipTransparent, kDeferUV>(prims, r, s, stack, cls);
}

// The hit of a kDeferUV traversal: the winning leaf slot's test repeated (no tMax bound), which
// reproduces the distance and barycentrics the traversal computed; prim = the original index.
template <bool kSpheres>
__device__ __forceinline__ Hit finish_hit(const LeafPrim *__restrict__ prims, const TraceRay &r, const TravState &s) {
    Hit h{0.f, 0.f, 0.f, -1};
    if (!s.found) return h;
    const LeafPrim *p = prims + s.hit.prim;
    const float4 v0 = __ldg(&p->v0), v1 = __ldg(&p->v1);
    const float inf = __int_as_float(0x7f800000);
    if (kSpheres && __float_as_int(v1.w) == 1)
        hit_sphere(r, v0, v1, inf, &h.t);
    else
        hit_triangle(r, v0, v1, __ldg(&p->v2), inf, &h.t, &h.u, &h.v);
    h.prim = __float_as_int(v0.w);
    return h;
}

// Cooperative form of the 4-wide traversal: a warp finishes the at most eight rays its lanes still
// hold. The time of a query is at least that of its longest ray, and one lane takes a step per node or
// leaf, each a dependent load and a chain of arithmetic: on the benchmark soups a launch of a few
// thousand rays took 70 to 110 us, and every larger launch ended in such a tail. Here groups of four
// lanes take entries off the rays' stacks (one entry per ray and step with more than four rays left, up
// to eight with one), each lane tests one child box or one of a leaf's triangles, and what is hit goes
// back on the stack, so a ray takes a step per level of the tree rather than per node. Measured (B200,
// closest hit, us, one lane a ray to the end / this): 1,000 rays, 4,096 triangles 85 / 32; 4,096 rays,
// 100,003 triangles 119 / 57; 1.5M rays, 100,003 triangles 456 / 421.
//
// The result is that of the one-lane walk bit for bit, so it does not depend on which rays a warp was left
// with. Box and triangle arithmetic are those of the other traversals, and for a closest hit the walk's
// order is kept: an entry above another on a stack comes with all it leads to before it. Nodes may be
// opened ahead of their turn (an entry is tested against tMax again when it is taken, and tMax only falls;
// a child lies within its node's box and so is entered no earlier, see kLooseBound; the children are sorted by the one-lane walk's own network, in which entries that fall away later, being
// farther than all that stay, do not change the order of the rest), and a leaf tested ahead of its turn is
// done with if nothing in it is hit, but else waits until all entries above it are leaves that end in the
// same step. Of those the hits count in order: a leaf entered
// at or beyond an earlier leaf's hit is not visited (rounding can put a hit before its own box's entry, so
// a later hit may be the nearer one and still not count), and equal distances go to the first. What the
// order of one step cannot settle is handed back (true in its lane) for the one-lane traversal to start
// over: a nearer hit in such a leaf, an accepted distance that is not a number (a determinant whose
// reciprocal overflows), and a sphere tied with another hit (its distance is compared in doubles).
// Any-hit queries take entries in any order: their outcome does not depend on it.
//
// The rays' own lanes keep r and st; stacks move in place from the lanes' columns to regions of 64
// entries (4 columns of the warp's 32, entry e in row e / 4). `bound` is the most entries a depth-first
// walk of the tree holds at a time; a step takes more than one entry of a ray only while its region
// then still has room for such a walk, so a region cannot overflow.
constexpr int kCoopRays = 8, kRayLanes = 4;
constexpr int kLeafPad = kRayLanes - 1;  // records past the leaf array that the lanes of a group may load
// Trees with a larger bound are left to the one-lane traversal. A ray is handed over with at most
// kShortStack + 1 entries, and its region must hold the walk on top of them, which 47 would still do; 24
// leave room to open two entries a step from the first step on. Trees between the two are not measured.
constexpr int kCoopBound = kStackSize - 24;
static_assert(kShortStack + 1 + kCoopBound <= kStackSize, "a ray's region holds what it brings and a walk");

struct CoopState {
    TravState s;
    bool redo;
};

// Out of line: inlined into the persistent kernels it cost their loops registers (closest hits of the
// 2^24-ray benchmark 4.20 -> 4.71 ms). Hence only rays whose stack is within the shared columns.
template <bool kAny, bool kSpheres, bool kSkipTransparent, bool kBatch, int kRow>
__device__ __noinline__ CoopState traverse4_coop(const QNode *nodes, const LeafPrim *prims, const uint8_t *cls,
                                                 int bound, V3 o, V3 d, TravState st, bool active, int2 *column) {
    static_assert(kShortStack * 32 == kCoopRays * kStackSize, "the regions fill the warp's columns");
    __builtin_assume(__isShared(column));
    const unsigned full = 0xffffffffu;
    const float inf = __int_as_float(0x7f800000);
    const int lane = threadIdx.x & 31, sub = lane & (kRayLanes - 1), group = lane / kRayLanes;
    int2 *warpStack = column - lane;  // column 0 of this warp
    const TraceRay r = make_trace_ray(o, d);
    unsigned rays = __ballot_sync(full, active);
    const int region = __popc(rays & ((1u << lane) - 1u));
    // The loop's last stores to the columns come before what is written below into other lanes' columns;
    // the votes alone order no memory, and with empty stacks the loop below has no barrier of its own.
    __syncwarp();
    // In place: row e is read by every ray before entry e lands in row e / 4.
    for (int e = 0; __any_sync(full, active && e < st.sp); ++e) {
        int2 v = make_int2(0, 0);
        if (active && e < st.sp) v = column[e * kRow];
        __syncwarp();
        if (active && e < st.sp) warpStack[(e >> 2) * kRow + 4 * region + (e & 3)] = v;
        __syncwarp();
    }
    if (active) {
        warpStack[(st.sp >> 2) * kRow + 4 * region + (st.sp & 3)] = make_int2(st.ref, __float_as_int(-inf));
        ++st.sp;
    }
    __syncwarp();
    bool redo = false;
    unsigned assigned = 0;
    // The ray this lane works for: its own lane, its region, its data.
    int home = 0, myRegion = 0, perRay = 1;
    bool mine = false;
    TraceRay q = r;
    while (rays) {
        if (rays != assigned) {
            assigned = rays;
            const int m = __popc(rays);
            perRay = m > 4 ? 1 : (m > 2 ? 2 : (m > 1 ? 4 : 8));
            const int i = group / perRay;
            mine = i < m;
            unsigned left = rays;
            for (int k = 0; k < i; ++k) left &= left - 1u;
            home = mine ? __ffs(left) - 1 : 0;
            myRegion = __shfl_sync(full, region, home);
            q.o = {__shfl_sync(full, r.o.x, home), __shfl_sync(full, r.o.y, home), __shfl_sync(full, r.o.z, home)};
            q.d = {__shfl_sync(full, r.d.x, home), __shfl_sync(full, r.d.y, home), __shfl_sync(full, r.d.z, home)};
            q.inv = {__shfl_sync(full, r.inv.x, home), __shfl_sync(full, r.inv.y, home),
                     __shfl_sync(full, r.inv.z, home)};
            q.neg[0] = q.inv.x < 0.f;
            q.neg[1] = q.inv.y < 0.f;
            q.neg[2] = q.inv.z < 0.f;
            q.infInv = isinf(q.inv.x) || isinf(q.inv.y) || isinf(q.inv.z);
        }
        const QNode *qn = nodes;
        const LeafPrim *lp = prims;
        const uint8_t *pc = cls;
        int qb = bound;
        if (kBatch) {
            qn = reinterpret_cast<const QNode *>(__shfl_sync(full, reinterpret_cast<unsigned long long>(nodes), home));
            lp = reinterpret_cast<const LeafPrim *>(__shfl_sync(full, reinterpret_cast<unsigned long long>(prims), home));
            if (kSkipTransparent)
                pc = reinterpret_cast<const uint8_t *>(__shfl_sync(full, reinterpret_cast<unsigned long long>(cls), home));
            qb = __shfl_sync(full, bound, home);
        }
        int sp = __shfl_sync(full, st.sp, home);
        float tMax = __shfl_sync(full, st.tMax, home);
        const int take = min(min(perRay, sp), max(1, (kStackSize - qb - sp) / 3));
        const int turn = group & (perRay - 1);  // 0 takes the topmost entry
        int2 *reg = warpStack + 4 * myRegion;
        const int quad = lane & ~(kRayLanes - 1);
        const unsigned lanesOfRay = (perRay == 8 ? full : (1u << (kRayLanes * perRay)) - 1u)
                                    << (lane & ~(kRayLanes * perRay - 1));
        const unsigned earlier = lanesOfRay & ((1u << quad) - 1u);  // lanes at entries above this lane's
        int ref = 0;
        float entry = inf;
        bool work = mine && turn < take;
        if (work) {
            const int e = sp - 1 - turn;
            const int2 v = reg[(e >> 2) * kRow + (e & 3)];
            ref = v.x;
            entry = __int_as_float(v.y);
            work = entry < tMax;
        }
        __syncwarp();
        float t = inf;   // entry distance of the child, or the leaf's own for its next four triangles
        int next = 0;
        bool hit = false, last = false, nan = false, wall = false, sphere = false, goesOn = false;
        float th = inf;
        if (work) {
            if (ref >= 0) {
                const char *nb = reinterpret_cast<const char *>(qn + ref) + 4 * sub;
                const int ox = q.neg[0] ? 48 : 0, oy = q.neg[1] ? 48 : 0, oz = q.neg[2] ? 48 : 0;
                const float nx = __ldg(reinterpret_cast<const float *>(nb + ox));
                const float fx = __ldg(reinterpret_cast<const float *>(nb + 48 - ox));
                const float ny = __ldg(reinterpret_cast<const float *>(nb + 16 + oy));
                const float fy = __ldg(reinterpret_cast<const float *>(nb + 64 - oy));
                const float nz = __ldg(reinterpret_cast<const float *>(nb + 32 + oz));
                const float fz = __ldg(reinterpret_cast<const float *>(nb + 80 - oz));
                next = __ldg(reinterpret_cast<const int *>(nb + 96));
                if (!q.infInv) {
                    t = slab_nf(q, nx, fx, ny, fy, nz, fz, tMax);
                } else {
                    const bool bx = q.neg[0], by = q.neg[1], bz = q.neg[2];
                    float te;
                    t = box_entry(q, bx ? fx : nx, by ? fy : ny, bz ? fz : nz, bx ? nx : fx, by ? ny : fy, bz ? nz : fz,
                                  &te) && te < tMax ? te : inf;
                }
            } else {
                // Slots past the leaf's last belong to other leaves or are padding: loaded, not tested.
                const LeafPrim *p = lp + ~ref + sub;
                const float4 v0 = __ldg(&p->v0), v1 = __ldg(&p->v1), v2 = __ldg(&p->v2);
                last = __float_as_int(v2.w) != 0;
                const unsigned ends = (__ballot_sync(0xfu << quad, last) >> quad) & 0xfu;
                if (ends == 0u || sub < __ffs(ends)) {
                    float u, v;
                    sphere = kSpheres && __float_as_int(v1.w) == 1;
                    if (sphere)
                        hit = hit_sphere(q, v0, v1, tMax, &th);
                    else
                        hit = hit_triangle(q, v0, v1, v2, tMax, &th, &u, &v);
                    if (kSkipTransparent && hit && (__ldg(pc + __float_as_int(v0.w)) & kTransparentBit)) {
                        wall = true;
                        hit = false;
                    }
                    nan = hit && !(th == th);
                }
                goesOn = ends == 0u;
                if (goesOn && sub == 0) {
                    t = -inf;
                    next = ref - kRayLanes;  // ~(slot + 4)
                }
            }
        }
        __syncwarp();
        const int myFirst = __popc(rays & ((1u << lane) - 1u)) * kRayLanes * perRay;  // of the ray this lane owns
        const bool own = (rays >> lane) & 1u;
        const unsigned ownLanes = own ? (perRay == 8 ? full : (1u << (kRayLanes * perRay)) - 1u) << myFirst : 0u;
        unsigned hits = __ballot_sync(full, hit);
        bool inTurn = true;
        if (!kAny && perRay > 1) {
            // A leaf below a node, or below one that goes on, with a hit in it: back as it is; without: done,
            // or its next four triangles under the leaf's own entry.
            inTurn = !(__ballot_sync(full, work && (ref >= 0 || goesOn)) & earlier);
            if (work && ref < 0 && !inTurn) {
                const bool again = (hits >> quad) & 0xfu;
                hit = nan = false;
                t = (again || goesOn) && sub == 0 ? entry : inf;
                if (again) next = ref;
            }
            if (hits) hits = __ballot_sync(full, hit);
        }
        if (hits) {
            if (!kAny) {
                // The least distance of each group, of the groups up to it, and of the ray's.
                float best = hit ? th : inf;
                for (int k = 1; k < kRayLanes; k <<= 1) best = fminf(best, __shfl_xor_sync(full, best, k));
                bool back = nan;
                if (perRay > 1) {
                    for (int k = kRayLanes; k < kRayLanes * perRay; k <<= 1) {
                        const float o = __shfl_up_sync(full, best, k);
                        if ((lane & (kRayLanes * perRay - 1)) >= k) best = fminf(best, o);
                    }
                    const float above = __shfl_up_sync(full, best, kRayLanes);
                    const float atTurn = turn > 0 ? fminf(tMax, above) : tMax;  // tMax when the walk comes to this leaf
                    best = __shfl_sync(full, best, lane | (kRayLanes * perRay - 1));
                    if (work && ref < 0 && inTurn && !(entry < atTurn)) {  // not visited
                        back |= hit && th < atTurn;
                        hit = false;
                        t = inf;
                    }
                }
                const unsigned win = __ballot_sync(full, hit && th == best);
                if (kSpheres) back |= sphere && hit && th == best && (win & lanesOfRay & ((1u << lane) - 1u));
                const unsigned w = win & ownLanes;
                const int src = w ? __ffs(w) - 1 : 0;
                const float tb = __shfl_sync(full, th, src);
                const int rb = __shfl_sync(full, ref, src);
                if (w) {
                    st.tMax = tb;
                    st.hit.prim = ~rb + (src & (kRayLanes - 1));
                    st.found = true;
                }
                tMax = best < tMax ? best : tMax;
                if (!(t < tMax)) t = inf;
                if (__ballot_sync(full, back) & ownLanes) redo = true;
            } else {
                if (hits & ownLanes) st.found = true;
            }
        }
        if (kSkipTransparent && (__ballot_sync(full, wall) & ownLanes)) st.crossed = true;
        // Push: the later turns' children below the earlier ones', within a group farthest first.
        int rank = 0;
        bool tie = false;
#pragma unroll
        for (int k = 1; k < kRayLanes; ++k) {
            const float o = __shfl_xor_sync(full, t, k);
            rank += o < t || (kAny && o == t && (sub ^ k) < sub);
            tie |= o == t;
        }
        if (!kAny && __any_sync(full, tie && t < inf)) {
            float t0 = __shfl_sync(full, t, quad), t1 = __shfl_sync(full, t, quad + 1);
            float t2 = __shfl_sync(full, t, quad + 2), t3 = __shfl_sync(full, t, quad + 3);
            int i0 = 0, i1 = 1, i2 = 2, i3 = 3;
            sort4(t0, i0, t1, i1, t2, i2, t3, i3);
            rank = sub == i1 ? 1 : (sub == i2 ? 2 : (sub == i3 ? 3 : 0));
        }
        const unsigned push = __ballot_sync(full, t < inf);
        if (t < inf) {
            const unsigned mask = push & lanesOfRay;
            const int below = __popc(mask & ~((2u << (lane | 3)) - 1u));
            const int inGroup = __popc(mask & (0xfu << (lane & ~3)));
            const int e = sp - take + below + inGroup - 1 - rank;
            reg[(e >> 2) * kRow + (e & 3)] = make_int2(next, __float_as_int(t));
        }
        if (own) {
            const int b = kBatch ? bound : qb;
            const int took = min(min(perRay, st.sp), max(1, (kStackSize - b - st.sp) / 3));
            st.sp += __popc(push & ownLanes) - took;
        }
        __syncwarp();
        rays = __ballot_sync(full, own && st.sp > 0 && !redo && !(kAny && st.found));
    }
    return CoopState{st, redo};
}

template <bool kAny, bool kSpheres, bool kSkipTransparent = false>
__device__ __forceinline__ bool traverse4_step(const QNode *__restrict__ nodes, const LeafPrim *__restrict__ prims,
                                               const TraceRay &r, TravState &s, int *stackRef, float *stackT,
                                               bool *overflow, const uint8_t *__restrict__ cls = nullptr) {
    LocalStack st{stackRef, stackT};
    return traverse4_step_st<kAny, kSpheres, kSkipTransparent>(nodes, prims, r, s, st, overflow, cls);
}

// A whole depth-first traversal by one lane, for the rare ray that traverse4_coop hands back. Out of
// line, with its own copies, so that the kernels' loops keep their registers.
template <bool kAny, bool kSpheres, bool kSkipTransparent>
__device__ __noinline__ TravState traverse4_alone(const QNode *nodes, const LeafPrim *prims, const uint8_t *cls,
                                                  int rootRef, V3 o, V3 d, float tMax, bool *overflow) {
    int stackRef[kStackSize];
    float stackT[kStackSize];
    LocalStack stack{stackRef, stackT};
    const TraceRay r = make_trace_ray(o, d);
    TravState s{};
    s.ref = rootRef;
    s.tMax = tMax;
    s.hit.prim = -1;
    while (!traverse4_step_st<kAny, kSpheres, kSkipTransparent, true>(nodes, prims, r, s, stack, overflow, cls)) {
    }
    return s;
}

// Whether a warp whose queue has run dry should stop its loop and finish its rays (busy: the lanes that
// hold one) with traverse4_finish: few enough rays, their stacks within shared memory. The caller has
// checked the tree's bound.
__device__ __forceinline__ bool coop_ready(unsigned busy, bool active, int sp) {
    return __popc(busy) <= kCoopRays && __all_sync(0xffffffffu, !active || sp <= kShortStack);
}

// A warp's step is either a node for the lanes at a node or a leaf for those at a leaf: with both in
// every step, the leaf code ran with two or three lanes. Lanes at a leaf wait until kLeafLanes do, or
// until no lane is at a node. From 1 / 4 / 8 / 12 lanes on: 2^24 rays, 1M triangles, closest 4.69 / 4.15 /
// 3.97 / 3.97 ms, any hit 3.25 / 2.89 / 2.76 / 2.75; leaves of up to four of 100,003 triangles, 1.5M any-hit
// rays 338 / 309 / 302 / 312 us, 200,003 closest 160 / 153 / 155 / 161; renders, ms: box 16.6 / 15.7 / 15.4 /
// 15.5, fog 8.28 / 8.13 / 8.06 / 8.10, guided 8.25 / 8.13 / 8.05 / 8.11.
constexpr int kLeafLanes = 8;
__device__ __forceinline__ bool leaf_turn(unsigned busy, unsigned leaves) {
    return __popc(leaves) >= kLeafLanes || leaves == busy;
}

// The end of a persistent traversal kernel: the warp's last rays (lanes with active) traced to their
// end, `tMax` being what each began with. Returns true when a one-lane traversal ran out of stack.
template <bool kAny, bool kSpheres, bool kSkipTransparent, bool kBatch, class Stack>
__device__ __forceinline__ bool traverse4_finish(const QNode *nodes, const LeafPrim *prims, const uint8_t *cls,
                                                 int bound, int rootRef, const TraceRay &r, TravState &st, bool active,
                                                 Stack &stack, float tMax) {
    bool overflow = false;
    const CoopState c = traverse4_coop<kAny, kSpheres, kSkipTransparent, kBatch, Stack::kRowStride>(
        nodes, prims, cls, bound, r.o, r.d, st, active, stack.sh);
    st = c.s;
    if (c.redo)
        st = traverse4_alone<kAny, kSpheres, kSkipTransparent>(nodes, prims, cls, rootRef, r.o, r.d, tMax, &overflow);
    return overflow;
}

} // namespace prb
