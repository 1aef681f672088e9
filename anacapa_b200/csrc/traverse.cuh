// Closest-hit and any-hit traversal of the triangle BVH2 and the curve BVH2.
//
// Hit-identity parity: the triangle test restates BVHBackend::intersectTriangle
// (src/accel/BVHBackend.cpp:264-283) with every operation rounded on its own
// (no FMA), so (t, u, v) equal the reference's float results compiled without
// contraction; the box tests restate intersectAABB (BVHBackend.cpp:249-262):
// ray tMin/tMax, the dirNeg slab selection and the `tMax <= tMin` rejection,
// plus the caller's `tNear > closestT` cull; the curve path restates
// CurveBrute::trace's aabbHit and the ray-ribbon subdivide
// (src/accel/CurveBrute.cpp:85-234, 478-498).
#pragma once
#include <type_traits>
#include "dmath.cuh"
#include "layout.h"
#include "motion.cuh"

namespace ana {

struct Ray {
    float3 o, d;
    float tmin, tmax;
    float time;  // normalized shutter time (motion-blurred meshes)
};

// BVHBackend::makeRay4 (BVHBackend.cpp:233-247): invDir = 1/safe(d) where
// safe(v) = |v| > 1e-9 ? v : 1e-9 (the sign of tiny components is dropped),
// and the triangle test rebuilds dir = 1/invDir.
struct TriRay {
    float3 o, inv;
    float tmin, tmax;
    uint32_t neg;  // bit i: direction component i is negative
};

__device__ __forceinline__ float safe_comp(float v) { return fabsf(v) > 1e-9f ? v : 1e-9f; }

__device__ __forceinline__ TriRay make_tri_ray(const Ray& r) {
    TriRay q;
    q.o = r.o;
    q.inv = f3(xdiv(1.f, safe_comp(r.d.x)), xdiv(1.f, safe_comp(r.d.y)), xdiv(1.f, safe_comp(r.d.z)));
    q.tmin = r.tmin;
    q.tmax = r.tmax;
    q.neg = (r.d.x < 0.f ? 1u : 0u) | (r.d.y < 0.f ? 2u : 0u) | (r.d.z < 0.f ? 4u : 0u);
    return q;
}
__device__ __forceinline__ float3 tri_dir(const TriRay& q) {
    return f3(xdiv(1.f, q.inv.x), xdiv(1.f, q.inv.y), xdiv(1.f, q.inv.z));
}

// (p - o) * inv of two boxes' planes of one axis, each operation rounded on
// its own (packed single precision: two boxes per instruction).
__device__ __forceinline__ float2 plane_pair(float p, float q, float o, float inv) {
    float2 r;
    asm("{\n .reg .b64 a, b, c;\n mov.b64 a, {%2, %3};\n mov.b64 b, {%4, %4};\n mov.b64 c, {%5, %5};\n"
        " add.rn.f32x2 a, a, b;\n mul.rn.f32x2 a, a, c;\n mov.b64 {%0, %1}, a;\n}"
        : "=f"(r.x), "=f"(r.y)
        : "f"(p), "f"(q), "f"(-o), "f"(inv));
    return r;
}

// Slab distances of four child boxes (lo / hi: the boxes' planes by axis): the
// entries (from the ray's tmin) and the exits (from its tmax). A box's near
// plane is its high one where the direction is negative.
__device__ __forceinline__ void box_slabs(const TriRay& r, const float (&lo)[3][4], const float (&hi)[3][4],
                                          float (&tn)[4], float (&tf)[4]) {
    const float o[3] = {r.o.x, r.o.y, r.o.z}, inv[3] = {r.inv.x, r.inv.y, r.inv.z};
#pragma unroll
    for (int k = 0; k < 4; k += 2) {
        float2 n[3], f[3];
#pragma unroll
        for (int i = 0; i < 3; ++i) {
            const bool neg = r.neg & (1u << i);
            n[i] = plane_pair(neg ? hi[i][k] : lo[i][k], neg ? hi[i][k + 1] : lo[i][k + 1], o[i], inv[i]);
            f[i] = plane_pair(neg ? lo[i][k] : hi[i][k], neg ? lo[i][k + 1] : hi[i][k + 1], o[i], inv[i]);
        }
        tn[k] = fmaxf(fmaxf(fmaxf(r.tmin, n[0].x), n[1].x), n[2].x);
        tn[k + 1] = fmaxf(fmaxf(fmaxf(r.tmin, n[0].y), n[1].y), n[2].y);
        tf[k] = fminf(fminf(fminf(r.tmax, f[0].x), f[1].x), f[2].x);
        tf[k + 1] = fminf(fminf(fminf(r.tmax, f[0].y), f[1].y), f[2].y);
    }
}

// Moller-Trumbore, BVHBackend::intersectTriangle.
__device__ __forceinline__ bool tri_hit(float3 o, float3 dir, float tmin, float3 v0, float3 e1, float3 e2, float tmax,
                                        float& t, float& u, float& v) {
    float3 h = xcross(dir, e2);
    float a = xdot(e1, h);
    if (fabsf(a) < 1e-9f) return false;
    float f = xdiv(1.f, a);
    float3 s = xsub3(o, v0);
    u = xmul(f, xdot(s, h));
    if (u < 0.f || u > 1.f) return false;
    float3 q = xcross(s, e1);
    v = xmul(f, xdot(dir, q));
    if (v < 0.f || xadd(u, v) > 1.f) return false;
    t = xmul(f, xdot(e2, q));
    return t >= tmin && t <= tmax;
}

// Stack entry: interior node index, or a leaf (bit 31) with count-1 in bits
// 25..30 and the first primitive in bits 0..24.
__device__ __forceinline__ uint32_t leaf_entry(uint32_t off, uint32_t cnt) {
    return 0x80000000u | ((cnt - 1u) << 25) | off;
}

struct TriHit {
    float t, u, v;
    int32_t tri;  // leaf-order index, -1 on miss
};

struct Counters {
    uint32_t nodes, prims, segs, cnodes;  // triangle nodes, triangles, segments, curve nodes
};

// ---------------------------------------------------------------------------
// Persistent-warp triangle traversal. Each lane owns one ray at a time; a
// warp loops over
//   1. refill: once enough lanes are without a ray (kRefill*), they take the
//      next queue entries together (one warp-aggregated atomicAdd on the
//      stage's fetch counter);
//   2. interior phase: lanes descend interior nodes until they reach a
//      leaf; the phase ends when no lane can take another interior step, when
//      every lane has parked a leaf or has nothing left, or when at most
//      kLeafPhaseLanes (any hit: kLeafPhaseLanesAny) lanes still descend
//      while others wait with a leaf, so lanes stay converged on the
//      node-test code. Any-hit queries can be speculative (kPark; Aila and
//      Laine, "Understanding the efficiency of ray traversal on GPUs", 2009):
//      a lane that reaches a leaf parks it and keeps descending from its next
//      stack entry. Closest-hit queries do not speculate: a leaf tested early
//      shortens the ray and culls later nodes (measured on the throughput
//      frame: speculation cost closest hit 3 %, saved any hit 8-12 % with
//      one-lane refills; with grouped refills it costs the triangle shadow
//      and MIS kernels too, and only the occlusion queries of ana_trace_batch
//      on triangles park);
//   3. leaf phase: the parked leaf's (else the current leaf's) triangles; curve
//      leaves begin and walk their segments in steps of their own.
// A lane whose stack is used up (or, for occlusion, that found a blocker)
// reports its ray and picks up a new one at the next refill, so finished rays
// do not idle the warp until its slowest ray completes. Box and triangle
// tests are the same functions as above, so results are identical.
// ---------------------------------------------------------------------------
// Interior phases end once this few lanes still descend (and a lane has a
// leaf). On the 1920x1080x64 throughput frame the extend stage took 142.0 ms
// when the phase ran until no lane descended, 118.4 ms at 4 lanes, 117.2 ms at
// 8 and 124.6 ms at 16; the any-hit shadow + MIS stages, parking leaves and
// refilling one lane at a time, 146.5 ms, 137.0 at 4, 132.8 at 8, 128.1 at 16,
// 129.8 at 24 and 191.2 at 32. Any-hit kernels that test leaves as reached use
// the closest-hit count (shadow + MIS 107.0 ms at 8, 111.4 at 4, 108.1 at 12,
// 111.9 at 16); the parked count serves the kernels that still park
// (occlusion queries of ana_trace_batch on triangles). Kernels with
// motion-blurred meshes, whose leaf tests may invert interpolated matrices, keep
// the phase until no lane descends (1280x720x16 motion frame: 13.3 ms against
// 13.9 at 8 lanes). Hits and occlusion answers are unchanged.
constexpr uint32_t kLeafPhaseLanes = 8;      // closest hit, any hit without parking
constexpr uint32_t kLeafPhaseLanesAny = 16;  // any hit (parked leaves)

// Curve leaves: lanes with a segment to begin do so together, lanes inside a
// ribbon walk step together once kWalkLanes of them wait (or nothing else is
// left to do), and the phase ends when at most kBeginLanes segments wait to
// begin. A lane that walked its segment alone held the warp for up to 64 leaves
// of the walk, with 4 of 32 lanes active. 1280x720x8 hair frame, closest-hit
// stage: 145.9 ms a whole segment per lane at a time, 130.6 one node per lane
// and phase; with most segments rejected before their walk (ribbon_far) 102.2,
// and 98.7 with begin and walk steps apart (kWalkLanes 4: 100.5, 6: 98.7, 8:
// 98.7, 12: 102.2; kBeginLanes 4: 101.4 and 12: 99.3; interior phases ending
// at 6 or 10 lanes instead of 8: 100.5, 98.0).
constexpr int kWalkLanes = 6;
constexpr int kBeginLanes = 8;

// Refill thresholds: idle lanes take new rays only once at least this many
// lanes of the warp are idle (or the queue is drained and every lane is).
// Queue entries in path order are the samples of one pixel, so lanes that
// start together trace neighbouring rays and stay converged, where one lane
// refilled at a time starts at the root beside lanes deep in the tree. On the
// 1920x1080x64 throughput frame (closest hit / any hit thresholds): extend
// 115.7 ms at 1, 114.6 at 4, 111.0 at 8, 108.8 at 12, 108.3 at 14, 107.7 at
// 16, 108.2 at 18, 108.4 at 20, 112.4 at 24, 122.5 at 28, 140.5 at 32; shadow +
// MIS 128.3 ms at 1, 127.3 at 8, 126.8 at 12, 127.2 at 16, 134.6 at 20. The
// curve kernels' ribbon walks diverge anyway and want smaller groups: the
// 1280x720x32 hair frame's extend stage 647.5 ms at 1, 634.2 at 4, 636.7 at 6,
// 642.9 at 8, 649.3 at 10, 657.7 at 12; its shadow stage 376.6 ms at 1, 370.4
// at 2, 369.6 at 3, 371.0 at 4, 376.4 at 6, 384.0 at 8.
constexpr int kRefillLanes = 16;
constexpr int kRefillLanesAny = 12;
constexpr int kRefillLanesCurves = 4;
constexpr int kRefillLanesCurvesAny = 4;

struct Traversal {
    TriRay r;        // curve stage: r.inv is the exact 1/d
    float closest;
    uint32_t prim;   // closest hit so far: leaf-order triangle, 0x80000000 | segment, or kNoPrim
    uint32_t cur;
    int sp;
    int rs;          // curve stage: nodes on the stack of the current segment's ribbon walk
    // curve stage (scenes with curves): the triangle BVH is traversed first,
    // then the curve BVH from the triangle hit distance (CurveBrute::trace)
    bool curve;      // the curve BVH is being traversed
    bool unit;       // the direction has unit length (ribbon_far's margin)
    float margin;    // ribbon_far's, of the current segment
    bool flat;       // a direction component is below CurveBrute::aabbHit's 1e-9
    // filled from the frame when the ray is reported
    float u, v, tseg;
    float3 tang;
};
constexpr uint32_t kNoPrim = 0xFFFFFFFFu;

// A lane's local memory: kFrame slots, then the traversal stack. The slots
// below stack[0] hold what the node steps never read, so that the registers
// hold the interior loop's own values: with all of the ray's state in
// registers the compiler spilled some of those instead and reloaded them at
// every node (1920x1080x64 throughput frame: extend stage 108.0 -> 103.2 ms;
// 1280x720x8 hair frame 264.5 -> 260.0 ms).
//   -1 (u, v) of the closest triangle hit     -2, -3.x direction of the
//   -3.y queue entry                             primitive tests
//   -4, -5.x exact direction, -5.y curve root (triangle stage); from the curve
//   stage on -4 .. -6 the ray frame's x and y axes
//   -7, -8 (tangent, strand parameter) of the closest ribbon hit
//   -9.x ray time, -9.y, -10 exact direction (motion)
//   -11.x motion mesh of the object ray in -11.y .. -14.x (origin, direction)
constexpr int kFrame = 14;

__device__ __forceinline__ uint2 pair(float a, float b) { return make_uint2(__float_as_uint(a), __float_as_uint(b)); }
__device__ __forceinline__ float lo(uint2 p) { return __uint_as_float(p.x); }
__device__ __forceinline__ float hi(uint2 p) { return __uint_as_float(p.y); }
__device__ __forceinline__ float3 frame_dir(const uint2* stack) {
    const uint2 a = stack[-2];
    return f3(lo(a), hi(a), lo(stack[-3]));
}

// Starts a traversal at a scene's root (kNoRoot: the scene has no triangles).
// Closest hit keeps the nearest accepted triangle; ties (t == closest) go to
// the later-tested triangle, as `t <= r.tMax` does in the reference; any hit
// (kAny) stops at the first accepted triangle (BVHBackend::occluded,
// BVHBackend.cpp:409-444).
template <bool kCurves, bool kMotion>
__device__ __forceinline__ void trav_init(Traversal& T, const Ray& ray, uint32_t root, uint32_t segRoot, uint32_t idx,
                                          uint2* stack) {
    T.r = make_tri_ray(ray);
    T.closest = ray.tmax;
    T.prim = kNoPrim;
    T.cur = root;
    T.sp = 1;
    stack[0] = make_uint2(kEmptyChild, __float_as_uint(-INFINITY));
    T.rs = 0;
    T.curve = false;
    T.flat = false;
    const float3 d = tri_dir(T.r);
    stack[-2] = pair(d.x, d.y);
    stack[-3] = make_uint2(__float_as_uint(d.z), idx);
    if (kCurves) {
        stack[-4] = pair(ray.d.x, ray.d.y);
        stack[-5] = make_uint2(__float_as_uint(ray.d.z), segRoot);
    }
    if (kMotion) {
        stack[-9] = pair(ray.time, ray.d.x);
        stack[-10] = pair(ray.d.y, ray.d.z);
        stack[-11].x = kNoPrim;
    }
}

// The closest hit's parameters, for the report.
template <bool kCurves>
__device__ __forceinline__ void trav_finish(Traversal& T, const uint2* stack) {
    const uint2 a = stack[-1];
    T.u = lo(a);
    T.v = hi(a);
    if (kCurves) {
        const uint2 b = stack[-7], c = stack[-8];
        T.tang = f3(lo(b), hi(b), lo(c));
        T.tseg = hi(c);
    }
}

// Takes the next stack entry; stack[0] is an entry that is never culled and
// ends the traversal (cur = kEmptyChild), so a pop tests no stack depth and a
// lane's state is its current entry alone: an interior node (bit 31 clear), a
// leaf, or kEmptyChild for nothing left or no ray (1280x720x8 hair frame 260.0
// -> 250.0 ms, 1279x719x16 glass frame 11.55 -> 11.34 ms against flags).
// Traversal stack entry (thread-local memory): x = node or leaf entry, y = the
// entry distance's bits (closest hit; any hit writes x only). One 64-bit
// access per push and pop instead of two 32-bit ones: the throughput frame's
// extend stage 116.4 -> 115.7 ms, the 1920x1080x64 hair frame 4549 -> 4505 ms.
template <bool kAny = false>
__device__ __forceinline__ void trav_pop(Traversal& T, const uint2* stack) {
    if (kAny) {  // an any-hit query ends at its first hit: nothing on the stack is culled
        T.cur = stack[--T.sp].x;
        return;
    }
    uint2 e;
    do e = stack[--T.sp];
    while (__uint_as_float(e.y) > T.closest);
    T.cur = e.x;
}

// Interior step: one 128-byte node fetch and four child-box tests. The
// children entered are ordered by entry distance with a 4-key sorting
// network; the nearest becomes the current node, the others are pushed
// farthest first (popped nearest first, and skipped once a closer hit is
// known). Any-hit queries skip the sort and the entry distances: the children
// entered are taken in stored order, and nothing is culled at a pop because
// the query ends at its first hit. On the 1920x1080x64 throughput frame that
// cut the shadow and MIS stages from 72.9 and 125.7 ms to 60.2 and 85.1 ms;
// near first without keys (the shortcuts below) measured 66.6 and 113.3 ms,
// so the stored order (the SAH build's lower side of each split first) finds
// blockers sooner there. The curve BVH keeps near-first any-hit steps, which
// measured faster on the hair frame.
__device__ __forceinline__ void cswap(float& ka, uint32_t& va, float& kb, uint32_t& vb) {
    if (kb < ka) {
        const float k = ka;
        ka = kb;
        kb = k;
        const uint32_t v = va;
        va = vb;
        vb = v;
    }
}

// Enters the children a closest-hit step found (key: entry distance, +inf
// for a child not entered): the nearest becomes the current node, the others
// are pushed farthest first (popped nearest first, and skipped once a closer
// hit is known). Children entered are ordered with a 4-key sorting network,
// which keeps equal keys in stored order; one or two children entered (most
// steps of incoherent rays) skip the network with the same result (extend
// stage of the throughput frame: 146.6 -> 141.9 ms). Shared by the triangle
// and the curve BVH steps.
__device__ __forceinline__ void enter_near_first(Traversal& T, float (&key)[4], uint32_t (&ref)[4], uint2* stack, uint32_t* err) {
    const int n = int(key[0] < INFINITY) + int(key[1] < INFINITY) + int(key[2] < INFINITY) + int(key[3] < INFINITY);
    if (n == 0) {
        trav_pop(T, stack);
        return;
    }
    if (n == 1) {  // one child entered: it becomes the current node
        T.cur = key[0] < INFINITY ? ref[0] : key[1] < INFINITY ? ref[1] : key[2] < INFINITY ? ref[2] : ref[3];
        return;
    }
    if (n == 2) {  // two entered: the first and the last in stored order, nearer first
        const bool h0 = key[0] < INFINITY, h1 = key[1] < INFINITY;
        const bool g3 = key[3] < INFINITY, g2 = key[2] < INFINITY;
        float ka = h0 ? key[0] : h1 ? key[1] : key[2];
        uint32_t ra = h0 ? ref[0] : h1 ? ref[1] : ref[2];
        float kb = g3 ? key[3] : g2 ? key[2] : key[1];
        uint32_t rb = g3 ? ref[3] : g2 ? ref[2] : ref[1];
        if (T.sp > int(kMaxStack4)) {
            atomicOr(err, 1u);
            T.cur = kEmptyChild;
            return;
        }
        cswap(ka, ra, kb, rb);
        stack[T.sp] = make_uint2(rb, __float_as_uint(kb));
        ++T.sp;
        T.cur = ra;
        return;
    }
    // misses carry key +inf, so the n children entered come first
    cswap(key[0], ref[0], key[1], ref[1]);
    cswap(key[2], ref[2], key[3], ref[3]);
    cswap(key[0], ref[0], key[2], ref[2]);
    cswap(key[1], ref[1], key[3], ref[3]);
    cswap(key[1], ref[1], key[2], ref[2]);
    if (T.sp + n - 2 > int(kMaxStack4)) {
        atomicOr(err, 1u);
        T.cur = kEmptyChild;
        return;
    }
#pragma unroll
    for (int k = 3; k >= 1; --k) {
        if (k < n) {
            stack[T.sp] = make_uint2(ref[k], __float_as_uint(key[k]));
            ++T.sp;
        }
    }
    T.cur = ref[0];
}

// BVHBackend::makeObjectSpaceRay4: the world ray (origin, exact direction)
// taken to the object space of motion mesh `mm` at the ray's time. The origin
// and the triangle tests' direction go to the lane's frame with the mesh: the
// ray keeps them until it meets a leaf of another motion mesh (the reference
// recomputes the same values per triangle). 1280x720x16 motion frame, with the
// matrix interpolated and inverted at every leaf: extend 9.39 ms, shadow 6.04;
// once per ray and run of leaves of a mesh: 5.48 and 3.55.
__device__ __noinline__ void object_ray(const DevScene& S, uint32_t mm, float3 o, uint2* stack) {
    M4 o2w, w2o;
    const uint2 a = stack[-9], b = stack[-10];
    o2w_at(S, mm, lo(a), o2w);
    m4_inverse(o2w, w2o);
    Ray r;
    r.o = m4_point(w2o, o);
    r.d = m4_vector(w2o, f3(hi(a), lo(b), hi(b)));
    r.tmin = r.tmax = r.time = 0.f;
    const TriRay q = make_tri_ray(r);
    const float3 d = tri_dir(q);
    stack[-11] = make_uint2(mm, __float_as_uint(q.o.x));
    stack[-12] = pair(q.o.y, q.o.z);
    stack[-13] = pair(d.x, d.y);
    stack[-14] = pair(d.z, 0.f);
}

// Tests the triangles of leaf entry `leaf`; true when an any-hit query found
// its blocker. kMotion: triangles flagged object-space (bit 31 of the index
// word) meet the ray in their mesh's object space at the ray's time.
template <bool kAny, bool kCount, bool kMotion = false>
__device__ __forceinline__ bool leaf_test(Traversal& T, const DevScene& S, uint32_t leaf, uint2* stack, Counters* cnt) {
    const float3 dir = frame_dir(stack);
    const uint32_t off = leaf & 0x01FFFFFFu, c = ((leaf >> 25) & 63u) + 1u;
    uint32_t held = kNoPrim;  // motion mesh of (oo, od)
    float3 oo, od;
    for (uint32_t i = off; i < off + c; ++i) {
        const float4* tp = S.tri_isect + 3 * size_t(i);
        float4 a = ldg4(tp), b = ldg4(tp + 1), e = ldg4(tp + 2);
        if (kCount) cnt->prims++;
        float t, u, v;
        const float tmax = kAny ? T.r.tmax : T.closest;
        const bool moving = kMotion && (__float_as_uint(a.w) & 0x80000000u);
        if (moving) {
            const uint32_t mm = __float_as_uint(b.w);
            if (mm != held) {
                if (stack[-11].x != mm) object_ray(S, mm, T.r.o, stack);
                const uint2 p = stack[-12], q = stack[-13];
                oo = f3(hi(stack[-11]), lo(p), hi(p));
                od = f3(lo(q), hi(q), lo(stack[-14]));
                held = mm;
            }
        }
        const bool h = tri_hit(moving ? oo : T.r.o, moving ? od : dir, T.r.tmin, f3(a), f3(b), f3(e), tmax, t, u, v);
        if (h) {
            T.closest = t;
            T.prim = i;
            if (kAny) return true;
            stack[-1] = pair(u, v);
        }
    }
    return false;
}

// ===========================================================================
// Curves
// ===========================================================================

// CurveBrute::aabbHit (CurveBrute.cpp:478-498).
__device__ __noinline__ float curve_key_flat(float3 ro, float3 rd, float3 inv, float tmin, float maxT,
                                              const float* box) {
    float tmn = tmin, tmx = maxT;
    const float lo[3] = {box[0], box[8], box[16]}, hi[3] = {box[4], box[12], box[20]};
    const float o[3] = {ro.x, ro.y, ro.z}, d[3] = {rd.x, rd.y, rd.z}, iv[3] = {inv.x, inv.y, inv.z};
#pragma unroll 1
    for (int i = 0; i < 3; ++i) {
        if (fabsf(d[i]) < 1e-9f) {
            if (o[i] < lo[i] || o[i] > hi[i]) return INFINITY;
            continue;
        }
        float t0 = xmul(xsub(lo[i], o[i]), iv[i]);
        float t1 = xmul(xsub(hi[i], o[i]), iv[i]);
        if (iv[i] < 0.f) {
            float tt = t0;
            t0 = t1;
            t1 = tt;
        }
        tmn = fmaxf(tmn, t0);
        tmx = fminf(tmx, t1);
        if (tmx < tmn) return INFINITY;
    }
    return tmn;
}

// The four keys of a curve node for a ray with a direction component below
// 1e-9, whose slab that component does not divide by.
__device__ __forceinline__ void curve_keys_flat(const Traversal& T, const uint2* stack, const float4* np,
                                                float (&key)[4]) {
    const float* f = reinterpret_cast<const float*>(np);
    const float3 d = frame_dir(stack);
#pragma unroll
    for (int k = 0; k < 4; ++k)
        key[k] = __float_as_uint(f[24 + k]) == kEmptyChild
                     ? INFINITY
                     : curve_key_flat(T.r.o, d, T.r.inv, T.r.tmin, T.closest, f + k);
}

// One node of either BVH: one 128-byte read in four loads (a warp's lanes read
// different nodes, so every load costs the L1 one tag lookup per active lane;
// with one 32-byte load per axis instead of two of 16 bytes a node takes four
// lookups instead of seven: 1920x1080x64 throughput frame, extend stage 114.7
// -> 109.2 ms, shadow 52.6 -> 48.7, MIS 67.4 -> 64.1). Triangle boxes (BVHBackend::intersectAABB) are
// entered when tMin..tMax of the slabs is not empty and starts no later than
// the closest hit; curve boxes (CurveBrute::aabbHit) when the slabs' interval
// up to the closest hit is not reversed. Both stages share one copy of the
// loads and slab tests, so lanes in different stages step together; curve boxes
// tested axis by axis with an early exit took the 1280x720x8 hair frame 297.5
// ms against 264.5 without branches. The slab tests run packed, two boxes per
// instruction (glass frame 11.34 -> 11.20 ms, throughput 289.5 -> 288.5 ms).
template <bool kAny, bool kCount, bool kCurves>
__device__ __forceinline__ void node_step(Traversal& T, const DevScene& S, uint2* stack, uint32_t* err, Counters* cnt) {
    const bool curve = kCurves && T.curve;
    const float4* np = reinterpret_cast<const float4*>((curve ? S.seg_nodes : S.tri_nodes) + T.cur);
    float4 lx, hx, ly, hy, lz, hz;
    ldg8(np, lx, hx);
    ldg8(np + 2, ly, hy);
    ldg8(np + 4, lz, hz);
    const float4 rf = ldg4(np + 6);
    if (kCount) {
        if (curve) cnt->cnodes++;
        else cnt->nodes++;
    }
    const float cull = kAny ? T.r.tmax : T.closest;
    float key[4];
    uint32_t ref[4] = {fbits_u(rf.x), fbits_u(rf.y), fbits_u(rf.z), fbits_u(rf.w)};
    {
        const float blo[3][4] = {{lx.x, lx.y, lx.z, lx.w}, {ly.x, ly.y, ly.z, ly.w}, {lz.x, lz.y, lz.z, lz.w}};
        const float bhi[3][4] = {{hx.x, hx.y, hx.z, hx.w}, {hy.x, hy.y, hy.z, hy.w}, {hz.x, hz.y, hz.z, hz.w}};
        float tn[4], tf[4];
        box_slabs(T.r, blo, bhi, tn, tf);
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const bool in = curve ? !(fminf(tf[k], cull) < tn[k]) : (tf[k] > tn[k] && tn[k] <= cull);
            key[k] = ref[k] != kEmptyChild && in ? tn[k] : INFINITY;
        }
    }
    if (kCurves && curve && T.flat) curve_keys_flat(T, stack, np, key);
    if (kAny && !curve) {  // any hit: children entered in stored order, no distance sort
        const int n = int(key[0] < INFINITY) + int(key[1] < INFINITY) + int(key[2] < INFINITY) + int(key[3] < INFINITY);
        if (n == 0) {
            trav_pop<kAny>(T, stack);
            return;
        }
        if (T.sp + n - 2 > int(kMaxStack4)) {
            atomicOr(err, 1u);
            T.cur = kEmptyChild;
            return;
        }
        uint32_t first = kEmptyChild;
#pragma unroll
        for (int k = 3; k >= 0; --k) {
            if (key[k] < INFINITY) {
                if (first != kEmptyChild) stack[T.sp++].x = first;
                first = ref[k];
            }
        }
        T.cur = first;
        return;
    }
    enter_near_first(T, key, ref, stack, err);
}


// Ray-space frame of makeRayFrame (CurveBrute.cpp:29-47): z = direction, x/y
// from buildOrthonormalBasis (Types.h:108-114).
struct RayFrame {
    float3 o, x, y, z;
};

__device__ __forceinline__ void onb_exact(float3 n, float3& t, float3& b) {
    float sign = copysignf(1.f, n.z);
    float a = xdiv(-1.f, xadd(sign, n.z));
    float bb = xmul(xmul(n.x, n.y), a);
    t = f3(xadd(1.f, xmul(xmul(xmul(sign, n.x), n.x), a)), xmul(sign, bb), -xmul(sign, n.x));
    b = f3(bb, xadd(sign, xmul(xmul(n.y, n.y), a)), -n.y);
}

__device__ __forceinline__ RayFrame make_frame(const Ray& r) {
    RayFrame f;
    f.o = r.o;
    f.z = r.d;
    onb_exact(r.d, f.x, f.y);
    return f;
}

__device__ __forceinline__ float3 project(const RayFrame& f, float3 p) {
    float3 q = xsub3(p, f.o);
    return f3(xdot(q, f.x), xdot(q, f.y), xdot(q, f.z));
}

__device__ __forceinline__ float3 xmid(float3 a, float3 b) { return xmul3(xadd3(a, b), 0.5f); }

// bezierTangent (CurveBrute.cpp:59-64)
__device__ __forceinline__ float3 bezier_tangent(float3 P0, float3 P1, float3 P2, float3 P3, float t) {
    float mt = xsub(1.f, t);
    float3 a = xmul3(xsub3(P1, P0), xmul(xmul(3.f, mt), mt));
    float3 b = xmul3(xsub3(P2, P1), xmul(xmul(6.f, mt), t));
    float3 c = xmul3(xsub3(P3, P2), xmul(xmul(3.f, t), t));
    return xadd3(xadd3(a, b), c);
}

__device__ __forceinline__ float min4(float a, float b, float c, float d) {
    return fminf(fminf(a, b), fminf(c, d));
}
__device__ __forceinline__ float max4(float a, float b, float c, float d) {
    return fmaxf(fmaxf(a, b), fmaxf(c, d));
}

// The bounds tests of subdivide (CurveBrute.cpp:97-117) on projected control
// points: depth range against [tmin, bestT], and the projected box's distance
// from the ray axis against the larger half-width. zlo receives zMin - maxHalfW.
__device__ __forceinline__ bool ribbon_bounds(float3 c0, float3 c1, float3 c2, float3 c3, float hw0, float hw3,
                                              float tmin, float bestT, float& zlo) {
    const float maxHalfW = fmaxf(hw0, hw3);
    const float zMin = min4(c0.z, c1.z, c2.z, c3.z), zMax = max4(c0.z, c1.z, c2.z, c3.z);
    zlo = xsub(zMin, maxHalfW);
    if (zlo > bestT) return false;
    if (xadd(zMax, maxHalfW) < tmin) return false;
    const float xMin = min4(c0.x, c1.x, c2.x, c3.x), xMax = max4(c0.x, c1.x, c2.x, c3.x);
    const float yMin = min4(c0.y, c1.y, c2.y, c3.y), yMax = max4(c0.y, c1.y, c2.y, c3.y);
    const float cx = (0.f < xMin) ? xMin : (0.f > xMax ? xMax : 0.f);
    const float cy = (0.f < yMin) ? yMin : (0.f > yMax ? yMax : 0.f);
    return !(xadd(xmul(cx, cx), xmul(cy, cy)) > xmul(maxHalfW, maxHalfW));
}

struct SubSeg {
    float3 P0, P1, P2, P3;  // world-space control points
    float zlo;              // zMin - maxHalfW: the test that depends on bestT
    uint32_t dp;            // depth (bits 0-2, 6 = root) | path from the root (bits 3-8, 1 = right)
};

// The half-widths, and the strand-parameter interval, of the node (depth,
// path) below a segment's: the splits' own updates (CurveBrute.cpp:152-176)
// replayed from the root.
__device__ __forceinline__ void ribbon_widths(uint32_t dp, float hw0r, float hw3r, float& hw0, float& hw3) {
    hw0 = hw0r;
    hw3 = hw3r;
    for (int k = 5 - int(dp & 7u); k >= 0; --k) {
        const float hm = xmul(xadd(hw0, hw3), 0.5f);
        if ((dp >> (3 + k)) & 1u) hw0 = hm;
        else hw3 = hm;
    }
}
__device__ __forceinline__ void ribbon_interval(uint32_t dp, float toffr, float tscr, float& toff, float& tscale) {
    toff = toffr;
    tscale = tscr;
    for (int k = 5 - int(dp & 7u); k >= 0; --k) {
        const float half = xmul(tscale, 0.5f);
        if ((dp >> (3 + k)) & 1u) toff = xadd(toff, half);
        tscale = half;
    }
}

// subdivide (CurveBrute.cpp:85-176): depth-6 de Casteljau subdivision in ray
// space, the left half first, updating bestT on a closer hit. The reference
// projects a node's four control points when it visits the node; a child
// shares two of them with its parent and one with its sibling, so here a split
// projects the five new points once (the same world points give the same
// projections), both children are bounds-tested at once and only survivors are
// pushed. The one test that depends on bestT (which only decreases) is
// repeated when a child is popped, so every node is accepted or culled, and
// every leaf evaluated, exactly as in the recursion and in the same order.
// A stack entry keeps the node's four world points, that test's bound and its
// (depth, path); the end points' projections are recomputed at a pop and the
// half-widths and parameter interval replayed along the path with the same
// operations (56 instead of 100 bytes per entry: hair frame's shadow stage
// 398.6 -> 379.3 ms). (A walk that kept no points at all, rebuilding each
// right half from the segment's four points along its path, measured slower:
// extend 1024 against 842 ms at leaves of four.)
constexpr int kRibbonStack = 8;

// Whether no leaf of the walk below a node can be hit: its projected control
// points all lie on one side of the ray axis, further from it than r along the
// normal of the chord, so does their hull, and so every chord of a leaf. r is
// the larger half-width plus a margin for the rounding of the walk's own
// arithmetic: its midpoints round 18 times on coordinates up to |P|, a
// projection 6 times on |P| + |o|, the leaf's distance a few times more, in all
// below 4e-6 (|P| + |o|) for a direction of unit length; the margin is 1e-5 of
// it. A rejected segment therefore never had a hit to report, and results are
// unchanged. The walk's own bounds (a box in ray space, axis-aligned) pass two
// thirds of the segments that a ray meets, though a strand's segment is thin
// and lies at any angle: with this test before them a ray of the hair frame
// walks 13 nodes instead of 82.
__device__ __forceinline__ bool ribbon_far(float3 c0, float3 c1, float3 c2, float3 c3, float r) {
    const float ux = c3.x - c0.x, uy = c3.y - c0.y;
    const float s0 = c0.y * ux - c0.x * uy, s1 = c1.y * ux - c1.x * uy, s2 = c2.y * ux - c2.x * uy,
                s3 = c3.y * ux - c3.x * uy;
    const float d = fmaxf(min4(s0, s1, s2, s3), -max4(s0, s1, s2, s3));
    const float rl = r * r * (ux * ux + uy * uy);
    return d > 0.f && rl > 1e-30f && d * d > rl;
}
__device__ __forceinline__ float norm1(float3 p) { return fabsf(p.x) + fabsf(p.y) + fabsf(p.z); }

// The ray frame (ray origin, x and y axes, direction) from the lane's frame.
__device__ __forceinline__ RayFrame ray_frame(const Traversal& T, const uint2* stack) {
    const uint2 a = stack[-4], b = stack[-5], c = stack[-6];
    return RayFrame{T.r.o, f3(lo(a), hi(a), lo(b)), f3(hi(b), lo(c), hi(c)), frame_dir(stack)};
}

// Begins the current leaf's first segment: a survivor of the tests of the whole
// segment is the walk's first node.
__device__ __forceinline__ void ribbon_start(Traversal& T, const DevScene& S, const uint2* stack, SubSeg* st) {
    const RayFrame fr = ray_frame(T, stack);
    const float4* sp4 = S.segs + 5 * size_t(T.cur & 0x01FFFFFFu);
    const float4 a = ldg4(sp4), b = ldg4(sp4 + 1), e = ldg4(sp4 + 2), g = ldg4(sp4 + 3);
    const float3 P0 = f3(a), P1 = f3(b), P2 = f3(e), P3 = f3(g);
    T.margin = T.unit ? 1e-5f * (max4(norm1(P0), norm1(P1), norm1(P2), norm1(P3)) + norm1(fr.o)) : INFINITY;
    T.rs = 0;
    // fused arithmetic: the margin covers it, and most segments end here
    // without the walk's separately rounded projections (1280x720x8 hair frame:
    // closest-hit stage 130.6 -> 102.2 ms, 107.2 with the test after those)
    const float3 q0 = P0 - fr.o, q1 = P1 - fr.o, q2 = P2 - fr.o, q3 = P3 - fr.o;
    if (ribbon_far(f3(dot(q0, fr.x), dot(q0, fr.y), 0.f), f3(dot(q1, fr.x), dot(q1, fr.y), 0.f),
                   f3(dot(q2, fr.x), dot(q2, fr.y), 0.f), f3(dot(q3, fr.x), dot(q3, fr.y), 0.f),
                   fmaxf(fabsf(a.w), fabsf(b.w)) * 1.00001f + T.margin))
        return;
    const float3 c0 = project(fr, P0), c1 = project(fr, P1), c2 = project(fr, P2), c3 = project(fr, P3);
    float zlo;
    if (ribbon_bounds(c0, c1, c2, c3, a.w, b.w, T.r.tmin, T.closest, zlo))
        st[T.rs++] = SubSeg{P0, P1, P2, P3, zlo, 6u};
}

// One node of the walk of the current leaf's first segment. True when it is a
// closer hit (recorded).
template <bool kAny>
__device__ __forceinline__ bool ribbon_step(Traversal& T, const DevScene& S, uint2* stack, SubSeg* st) {
    const SubSeg s = st[--T.rs];
    if (s.zlo > T.closest) return false;
    const RayFrame fr = ray_frame(T, stack);
    const uint32_t seg = T.cur & 0x01FFFFFFu;
    const float* sw = reinterpret_cast<const float*>(S.segs + 5 * size_t(seg)) + 3;
    float hw0, hw3;
    ribbon_widths(s.dp, __ldg(sw), __ldg(sw + 4), hw0, hw3);
    const float3 c0 = project(fr, s.P0), c3 = project(fr, s.P3);
    if ((s.dp & 7u) == 0u) {
        const float ax = c0.x, ay = c0.y, bx = c3.x, by = c3.y;
        const float dx = xsub(bx, ax), dy = xsub(by, ay);
        const float lenSq = xadd(xmul(dx, dx), xmul(dy, dy));
        float tLine;
        if (lenSq < 1e-12f) tLine = 0.f;
        else
            tLine = fmaxf(0.f, fminf(1.f, xdiv(xsub(xmul(-ax, dx), xmul(ay, dy)), lenSq)));
        const float px = xadd(ax, xmul(dx, tLine)), py = xadd(ay, xmul(dy, tLine));
        const float dist2 = xadd(xmul(px, px), xmul(py, py));
        const float halfW = xadd(xmul(hw0, xsub(1.f, tLine)), xmul(hw3, tLine));
        if (dist2 > xmul(halfW, halfW)) return false;
        const float tRay = xadd(c0.z, xmul(xsub(c3.z, c0.z), tLine));
        if (tRay < T.r.tmin || tRay >= T.closest) return false;
        T.closest = tRay;
        T.prim = 0x80000000u | seg;
        if (kAny) return true;
        float3 tg = bezier_tangent(s.P0, s.P1, s.P2, s.P3, tLine);
        if (xdot(tg, tg) < 1e-12f) tg = xsub3(s.P3, s.P0);
        const float len = __fsqrt_rn(xdot(tg, tg));
        tg = len > 1e-8f ? xmul3(tg, xdiv(1.f, len)) : f3(0.f, 0.f, 1.f);
        float toff, tscale;
        ribbon_interval(s.dp, __ldg(sw + 8), __ldg(sw + 12), toff, tscale);
        stack[-7] = pair(tg.x, tg.y);
        stack[-8] = pair(tg.z, xadd(toff, xmul(tLine, tscale)));
        return true;
    }
    const float3 Q01 = xmid(s.P0, s.P1), Q12 = xmid(s.P1, s.P2), Q23 = xmid(s.P2, s.P3);
    const float3 R01 = xmid(Q01, Q12), R12 = xmid(Q12, Q23), M = xmid(R01, R12);
    const float3 cq01 = project(fr, Q01), cr01 = project(fr, R01), cm = project(fr, M), cr12 = project(fr, R12),
                 cq23 = project(fr, Q23);
    const float hwMid = xmul(xadd(hw0, hw3), 0.5f);
    float zl, zr;
    bool okL = ribbon_bounds(c0, cq01, cr01, cm, hw0, hwMid, T.r.tmin, T.closest, zl);
    bool okR = ribbon_bounds(cm, cr12, cq23, c3, hwMid, hw3, T.r.tmin, T.closest, zr);
    const uint32_t cd = (s.dp & 7u) - 1u, cp = (s.dp >> 3) << 1;
    if (!kAny) {  // closest hit 109.1 -> 107.1 ms; any hit, which ends at its first leaf, 65.6 -> 69.6
        const float rf = fmaxf(fabsf(hw0), fabsf(hw3)) * 1.00001f + T.margin;
        okL = okL && !ribbon_far(c0, cq01, cr01, cm, rf);
        okR = okR && !ribbon_far(cm, cr12, cq23, c3, rf);
    }
    if (okR) st[T.rs++] = SubSeg{M, R12, Q23, s.P3, zr, cd | ((cp | 1u) << 3)};
    if (okL) st[T.rs++] = SubSeg{s.P0, Q01, R01, M, zl, cd | (cp << 3)};
    return false;
}

// The segment's walk is over: on to the leaf's next segment, else the next
// stack entry.
template <bool kAny>
__device__ __forceinline__ void ribbon_next(Traversal& T, const uint2* stack) {
    if (((T.cur >> 25) & 63u) != 0u) T.cur = T.cur - (1u << 25) + 1u;
    else trav_pop<kAny>(T, stack);
}

// ---------------------------------------------------------------------------
// Curve stage of a traversal (CurveBrute::trace's curve pass,
// CurveBrute.cpp:398-440): after the triangle BVH, the curve BVH is traversed
// from the triangle hit distance, keeping only strictly closer ribbon hits.
// Node and leaf steps mirror the triangle ones, so both stages share the
// converged interior / leaf phases and the stack.
// ---------------------------------------------------------------------------
__device__ __forceinline__ void curve_begin(Traversal& T, uint2* stack) {
    const uint2 a = stack[-4], b = stack[-5];
    const float3 d = f3(lo(a), hi(a), lo(b));
    const uint32_t segRoot = b.y;
    float3 fx, fy;
    onb_exact(d, fx, fy);
    T.curve = true;
    T.flat = fabsf(d.x) < 1e-9f || fabsf(d.y) < 1e-9f || fabsf(d.z) < 1e-9f;
    T.unit = fabsf(dot(d, d) - 1.f) < 1e-3f;
    T.r.inv = f3(xdiv(1.f, d.x), xdiv(1.f, d.y), xdiv(1.f, d.z));
    T.cur = segRoot;
    T.sp = 1;  // stack[0] still ends the stack
    stack[-2] = pair(d.x, d.y);
    stack[-3].x = __float_as_uint(d.z);
    stack[-4] = pair(fx.x, fx.y);
    stack[-5] = pair(fx.z, fy.x);
    stack[-6] = pair(fy.y, fy.z);
}

// A whole leaf at once, and the step after it (one-thread-per-ray schedule;
// triangle leaves of the persistent one).
template <bool kAny, bool kCount, bool kCurves, bool kMotion = false>
__device__ __forceinline__ void leaf_step(Traversal& T, const DevScene& S, uint2* stack, SubSeg* st, Counters* cnt) {
    if (kCurves && T.curve) {
        if (kCount) cnt->segs++;
        ribbon_start(T, S, stack, st);
        while (T.rs > 0) {
            if (ribbon_step<kAny>(T, S, stack, st) && kAny) {
                T.cur = kEmptyChild;
                return;
            }
        }
        ribbon_next<kAny>(T, stack);
    } else if (leaf_test<kAny, kCount, kMotion>(T, S, T.cur, stack, cnt)) {
        T.cur = kEmptyChild;
    } else {
        trav_pop<kAny>(T, stack);
    }
}

// A lane whose triangle traversal ended moves on to the curve BVH (unless an
// any-hit query already found a blocker). Returns true when the ray is done.
template <bool kAny, bool kCurves>
__device__ __forceinline__ bool stage_done(Traversal& T, uint2* stack) {
    if (kCurves && !T.curve && !(kAny && T.prim != kNoPrim)) curve_begin(T, stack);
    return T.cur == kEmptyChild;
}

// Done(i, T) consumes a finished traversal; Done(i, T, next) -> bool may
// instead ask for entry i to be traced again along `next` (same direction:
// a ray stepping through a transmissive surface) by returning true.
template <class Done>
__device__ __forceinline__ bool trace_again(Done& done, uint32_t i, const Traversal& T, Ray& next) {
    if constexpr (std::is_invocable_r_v<bool, Done&, uint32_t, const Traversal&, Ray&>) {
        return done(i, T, next);
    } else {
        done(i, T);
        return false;
    }
}

// Runs the persistent loop. Load(i, ray, root, segRoot) reads queue entry i
// and its scene's triangle and curve BVH roots; Done consumes the finished
// traversal of entry i (a lane-local call, see trace_again: a lane asked to
// trace again keeps its entry). With kCurves a lane that finishes the
// triangle BVH continues with the curve BVH in the same phases.
// kPark: any-hit lanes park the first leaf they reach and keep descending
// (speculative); false: any-hit lanes test each leaf as they reach it.
template <bool kAny, bool kCount, bool kCurves, bool kMotion, bool kPark, class Load, class Done>
__device__ __forceinline__ void persistent_traverse(const DevScene& S, uint32_t n, uint32_t* fetch, uint32_t* err,
                                                    Counters* cnt, Load load, Done done) {
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t ltmask = (1u << lane) - 1u;
    uint2 local[kFrame + kMaxStack4 + 1];
    uint2* const stack = local + kFrame;
    SubSeg ribbon[kCurves ? kRibbonStack : 1];
    Traversal T;
    T.rs = 0;
    T.curve = false;
    T.cur = kEmptyChild;  // of a lane without a ray, and of one whose traversal ended
    bool active = false, drained = false;
    uint32_t parked = kEmptyChild;
    // A queue shorter than the grid's lanes is dealt out evenly over all warps
    // instead of 32 entries to the first ones: late bounces and small queries
    // wait for their slowest warp, and a warp of few rays runs their diverging
    // walks sooner than a full one. With at least 32 entries per warp nothing
    // changes. 1280x720x8 hair frame: MIS stage (7 k rays per launch) 21.0 ->
    // 12.2 ms; 960x540x1 pass of 938 spheres: 3.94 -> 3.29 ms; a query of 64
    // rays 104 -> 78 us. Sharing what is left of a longer queue the same way
    // (entries left / warps per refill) cost its extra atomics: Cornell
    // 256x256x16 1.55 ms against 1.52.
    const uint32_t warps = gridDim.x * (blockDim.x >> 5);
    const uint32_t share = (n - 1u) / warps + 1u;  // n = 0: any, nothing is fetched
    while (true) {
        // 1. refill idle lanes
        if (!drained) {
            uint32_t need = __ballot_sync(0xFFFFFFFFu, !active);
            constexpr int kRefill = kCurves ? (kAny ? kRefillLanesCurvesAny : kRefillLanesCurves)
                                            : (kAny ? kRefillLanesAny : kRefillLanes);
            if (__popc(need) >= kRefill) {
                const uint32_t leader = __ffs(need) - 1u, take = min(uint32_t(__popc(need)), share);
                uint32_t base = 0;
                if (lane == leader) base = atomicAdd(fetch, take);
                base = __shfl_sync(0xFFFFFFFFu, base, leader);
                if (base >= n) drained = true;
                if (!active) {
                    const uint32_t rank = __popc(need & ltmask), idx = base + rank;
                    if (rank < take && idx < n) {
                        Ray ray;
                        uint32_t root, segRoot;
                        load(idx, ray, root, segRoot);
                        trav_init<kCurves, kMotion>(T, ray, root, segRoot, idx, stack);
                        active = true;
                    }
                }
            }
        }
        if (!__any_sync(0xFFFFFFFFu, active)) break;
        // 2. interior phase (speculative)
        while (true) {
            if (kPark && int(T.cur) < 0 && T.cur != kEmptyChild && parked == kEmptyChild) {
                parked = T.cur;
                trav_pop<kAny>(T, stack);
            }
            const bool want = int(T.cur) >= 0;
            const uint32_t wantMask = __ballot_sync(0xFFFFFFFFu, want);
            if (!wantMask) break;
            const bool leaf = kPark ? parked != kEmptyChild : !want && T.cur != kEmptyChild;
            if (kPark && __all_sync(0xFFFFFFFFu, T.cur == kEmptyChild || leaf)) break;
            // Once at most kPhaseLanes lanes still descend and another lane
            // holds a leaf (any hit: a parked one), the phase ends and the
            // leaves are tested (the descending lanes resume in the next
            // interior phase), so few lanes do not hold the warp in the node
            // loop. A lane with a leaf must exist, so every pass makes progress.
            constexpr int kPhaseLanes = kMotion && !kCurves ? 0 : (kPark ? kLeafPhaseLanesAny : kLeafPhaseLanes);
            if (kPhaseLanes > 0 && __popc(wantMask) <= kPhaseLanes && __any_sync(0xFFFFFFFFu, leaf)) break;
            if (want) node_step<kAny, kCount, kCurves>(T, S, stack, err, cnt);
        }
        // 3. leaf phase: one triangle leaf per lane
        if (kPark && parked != kEmptyChild) {
            if (leaf_test<kAny, kCount, kMotion>(T, S, parked, stack, cnt)) T.cur = kEmptyChild;
            parked = kEmptyChild;
        } else if (int(T.cur) < 0 && T.cur != kEmptyChild && !(kCurves && T.curve)) {
            leaf_step<kAny, kCount, false, kMotion>(T, S, stack, nullptr, cnt);
        }
        // curve leaves: every lane with a segment starts it or walks one node
        if (kCurves) {
            bool acted = false;  // every phase begins or walks at least once
            while (true) {
                const bool leaf = T.curve && int(T.cur) < 0 && T.cur != kEmptyChild;
                const bool walk = T.rs > 0, begin = leaf && !walk;
                const uint32_t beginMask = __ballot_sync(0xFFFFFFFFu, begin);
                const int walks = __popc(__ballot_sync(0xFFFFFFFFu, walk));
                if (acted && walks < kWalkLanes && __popc(beginMask) <= kBeginLanes) break;
                if (walks >= kWalkLanes || !beginMask) {
                    if (walk) {
                        if (ribbon_step<kAny>(T, S, stack, ribbon) && kAny) {
                            T.rs = 0;
                            T.cur = kEmptyChild;
                        } else if (T.rs == 0) {
                            ribbon_next<kAny>(T, stack);
                        }
                    }
                } else if (begin) {
                    if (kCount) cnt->segs++;
                    ribbon_start(T, S, stack, ribbon);
                    if (T.rs == 0) ribbon_next<kAny>(T, stack);
                }
                acted = true;
            }
        }
        if (active && T.cur == kEmptyChild && parked == kEmptyChild) {
            if (stage_done<kAny, kCurves>(T, stack)) {  // else the curve BVH follows
                trav_finish<kCurves>(T, stack);
                const uint32_t idx = stack[-3].y;
                Ray next;
                if (trace_again(done, idx, T, next)) {
                    Ray ray;
                    uint32_t root, segRoot;
                    load(idx, ray, root, segRoot);
                    trav_init<kCurves, kMotion>(T, next, root, segRoot, idx, stack);
                } else {
                    active = false;
                }
            }
        }
    }
}

}  // namespace ana
