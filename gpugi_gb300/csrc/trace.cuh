// Ray walks over the scene's hierarchy and their intersection tests (device
// code). All return trace_ray's results bit for bit:
//   trace_ray     one thread per ray, stackless (escape pointers): the
//                 reference's walk, which the others are held against
//   walk_step     the same one test at a time, for warps that refill lanes
//   group_walks   4, 8 or 16 lanes walk one ray together, stackless
//   wide_walks    a depth-first stack over the four-wide copy of a box
//                 hierarchy (wide.cu), a lane or a warp per ray
//   lane_walks    the escape walk with leaves tested by eight lanes each, for
//                 hierarchies without that copy
//
// Same walk as gpugi's TraceRay/TraceRayAnyHit (gpugi/shader/traceray.glsl:
// 25-180): nodes are visited in preorder; a node whose bounds are hit with
// firstHit <= rayLength descends into firstChild (or tests the leaf block and
// then continues at escape), a missed node continues at escape, and escape 0
// ends the walk. Leaf slots are tested in order and a triangle is accepted
// when hit < rayLength (strict, so ties keep the first slot found). The
// node/leaf state machine of the shader is written here as two nested loops
// that perform the same sequence of tests.
#pragma once
#include "common.cuh"
#include "scene.cuh"

namespace gpugi {

// IntersectBox (intersectiontests.glsl:9-20). min/max are IEEE minNum/maxNum
// (fminf/fmaxf): an axis-parallel ray produces inf*0 = NaN slabs that drop out
// (a ray lying in a face plane of the box then misses it).
// ROBUST is the box test of the watertight mode (an addition): a slab of a
// ray that lies in one of its bounding planes (a NaN slab value) does not
// constrain the ray, and the exit distance is widened by 1 + 2 gamma(3),
// rounded up to 1 + 2^-21 (Ize, "Robust BVH Ray Traversal", JCGT 2(2),
// 2013), so that rounding never culls a box whose surface the ray touches:
// a ray through a vertex or edge on the box boundary still reaches the
// triangles there.
template <bool ROBUST = false>
GPUGI_D bool intersect_box(float3 o, float3 inv, float4 lo, float4 hi, float& firstHit) {
    // x and y slabs as packed pairs (add.f32x2 / mul.f32x2: per component
    // the same IEEE round-to-nearest results as the scalar operations;
    // lo - o as lo + (-o), exact for every input including signed zeros)
    const float2 no = make_float2(-o.x, -o.y), ixy = make_float2(inv.x, inv.y);
    const float2 b2 = __fmul2_rn(__fadd2_rn(make_float2(lo.x, lo.y), no), ixy);
    const float2 t2 = __fmul2_rn(__fadd2_rn(make_float2(hi.x, hi.y), no), ixy);
    float tbx = b2.x, tby = b2.y, tbz = X::mul(inv.z, X::sub(lo.z, o.z));
    float ttx = t2.x, tty = t2.y, ttz = X::mul(inv.z, X::sub(hi.z, o.z));
    float mnx = fminf(ttx, tbx), mny = fminf(tty, tby), mnz = fminf(ttz, tbz);
    float mxx = fmaxf(ttx, tbx), mxy = fmaxf(tty, tby), mxz = fmaxf(ttz, tbz);
    if (ROBUST) {
        const float inf = __int_as_float(0x7f800000);
        if (isnan(tbx) || isnan(ttx)) mnx = -inf, mxx = inf;
        if (isnan(tby) || isnan(tty)) mny = -inf, mxy = inf;
        if (isnan(tbz) || isnan(ttz)) mnz = -inf, mxz = inf;
    }
    // max(max(mnx, mny), max(mnx, mnz)) of the shader is the maximum of the
    // three (NaNs ignored either way); likewise for the minimum
    firstHit = fmaxf(0.0f, max3f(mnx, mny, mnz));
    float lastHit = min3f(mxx, mxy, mxz);
    if (ROBUST) lastHit = X::mul(lastHit, 0x1.000008p+0f);
    return firstHit <= lastHit;
}

// Ray against a stored axis-aligned ellipsoid. The node holds {center,
// ir = 1 / (radii + 1e-15)} (reciprocals taken at upload; the guard is the
// one of IntersectVirtualEllipsoid, intersectiontests.glsl:26-52). The steps
// are that function's: advance the ray to its closest approach to the centre
// for stability, scale into the unit sphere and solve the quadratic; the
// scaling multiplies by ir and the two quotients by ddotd share one
// reciprocal, so a node costs one correctly rounded reciprocal and one sqrt
// instead of eight divisions and a sqrt. The reference never walks
// ellipsoids, so this test defines the node kind; the oracle restates it
// operation for operation.
GPUGI_D bool intersect_ellipsoid(float3 ro, float3 rd, float4 c, float4 ir, float& firstHit) {
    float3 o = X::sub3(ro, xyz(c));
    const float t = fmaxf(0.0f, -X::dot(o, rd));
    o = X::add3(o, X::scale(t, rd));
    o = X::mul3(o, xyz(ir));
    const float3 d = X::mul3(rd, xyz(ir));
    const float odoto = X::dot(o, o), odotd = X::dot(o, d), ddotd = X::dot(d, d);
    const float inv = X::rcp(ddotd);
    const float phalf = X::mul(odotd, inv);
    const float q = X::mul(X::sub(odoto, 1.0f), inv);
    float rad = X::sub(X::mul(phalf, phalf), q);
    if (rad < 0.0f) return false;
    rad = __fsqrt_rn(rad);
    firstHit = fmaxf(0.0f, X::add(X::sub(-phalf, rad), t));
    return X::add(X::add(-phalf, rad), t) >= 0.0f;
}

// rotate(x, q) (intersectiontests.glsl:82-89) in the shader's operation order.
GPUGI_D float3 qrotate(float3 x, float4 q) {
    const float3 t = X::cross(make_float3(q.x, q.y, q.z), x);
    const float3 u = make_float3(X::sub(X::add(X::mul(q.w, t.x), X::mul(q.y, t.z)), X::mul(q.z, t.y)),
                                 X::sub(X::add(X::mul(q.w, t.y), X::mul(q.z, t.x)), X::mul(q.x, t.z)),
                                 X::sub(X::add(X::mul(q.w, t.z), X::mul(q.x, t.y)), X::mul(q.y, t.x)));
    return X::add3(x, X::scale(2.0f, u));
}

// FetchIntersectOBoxNode (intersectiontests.glsl:114-128) on the 48-B node
// {center | child}, {sidesHalf | escape}, rotationInv: the ray is rotated
// into the box frame (origin relative to the centre), its direction
// inverted there, and the box [-sidesHalf, sidesHalf] tested with
// IntersectBox (ROBUST: the watertight mode's box test).
template <bool ROBUST = false>
GPUGI_D bool intersect_obox(float3 ro, float3 rd, float4 a, float4 b, float4 rotationInv, float& firstHit) {
    const float3 o = qrotate(X::sub3(ro, xyz(a)), rotationInv);
    const float3 d = qrotate(rd, rotationInv);
    const float3 inv = make_float3(X::rcp(d.x), X::rcp(d.y), X::rcp(d.z));
    return intersect_box<ROBUST>(o, inv, make_float4(-b.x, -b.y, -b.z, 0.0f), b, firstHit);
}

// Node layouts: AABB and ellipsoid nodes take 2 float4, oriented boxes 3.
template <int BOUNDS>
constexpr uint32_t node_stride() {
    return BOUNDS == 2 ? 3u : 2u;
}
// The bounds test of a node kind (0 box, 1 ellipsoid, 2 oriented box); c is
// the oriented box's third texel (unused otherwise).
template <int BOUNDS, bool ROBUST>
GPUGI_D bool bounds_test(float3 o, float3 d, float3 inv, float4 a, float4 b, float4 c, float& firstHit) {
    if (BOUNDS == 0) return intersect_box<ROBUST>(o, inv, a, b, firstHit);
    if (BOUNDS == 1) return intersect_ellipsoid(o, d, a, b, firstHit);
    return intersect_obox<ROBUST>(o, d, a, b, c, firstHit);
}

// IntersectTriangle (intersectiontests.glsl:63-79) on the precomputed record
// {p0, e0, e1, n}. Returns hit distance and the two barycentrics (y, z).
GPUGI_D bool intersect_triangle_v(float3 o, float3 d, float4 a, float4 b, float4 c, float& hit, float& by,
                                  float& bz) {
    float3 p0 = make_float3(a.x, a.y, a.z);
    float3 e0 = make_float3(a.w, b.x, b.y);
    float3 e1 = make_float3(b.z, b.w, c.x);
    float3 n = make_float3(c.y, c.z, c.w);
    float3 e2 = X::scale(X::rcp(X::dot(n, d)), X::sub3(p0, o));
    float3 i = X::cross(d, e2);
    by = X::dot(i, e1);
    bz = X::dot(i, e0);
    float bx = X::sub(1.0f, X::add(bz, by));
    hit = X::dot(n, e2);
    return (hit > 0.0001f) && bx >= 0.0f && by >= 0.0f && bz >= 0.0f;
}
GPUGI_D bool intersect_triangle(float3 o, float3 d, const float4* rec, float& hit, float& by, float& bz) {
    return intersect_triangle_v(o, d, __ldg(rec), __ldg(rec + 1), __ldg(rec + 2), hit, by, bz);
}

// Watertight ray/triangle test (an addition; the reference's test above is
// not watertight): Woop, Benthin and Wald, "Watertight Ray/Triangle
// Intersection", JCGT 2(1), 2013. Per ray, the axis kz of the largest
// |direction| component becomes the ray's z axis (kx, ky follow cyclically,
// swapped when d[kz] < 0 to keep the winding) and the shear
// S = (d[kx] / d[kz], d[ky] / d[kz], 1 / d[kz]) maps the ray onto +z. Per
// triangle, the vertices relative to the origin are sheared into that frame
// and the three 2D edge functions U, V, W are evaluated; an edge function
// that comes out exactly 0 is evaluated again in double precision (products
// of two floats are exact there), so rays through shared edges and vertices
// of a closed mesh see consistent signs and never slip through. Two-sided:
// U, V, W must not have mixed signs and det = U + V + W must not be 0; then
// t = T / det with T = U Az + V Bz + W Cz. The hit rule of the reference
// test is kept: t > 1e-4 (INTERSECT_EPSILON), and the walk accepts
// t < rayLength. Barycentrics (u, v) = (V, W) / det, the weights of p1 and
// p2 as in gpugi's convention. Records hold the exact vertices
// {p0.xyz p1.x | p1.yz p2.xy | p2.z 0 0 0} (48 B, like the reference records).
struct WtRay {
    float Sx, Sy, Sz;
    uint32_t kx, ky, kz;
};
GPUGI_D float comp3(float3 v, uint32_t k) { return k == 0 ? v.x : (k == 1 ? v.y : v.z); }
GPUGI_D WtRay wt_setup(float3 d) {
    WtRay w;
    const float ax = fabsf(d.x), ay = fabsf(d.y), az = fabsf(d.z);
    w.kz = ax >= ay ? (ax >= az ? 0u : 2u) : (ay >= az ? 1u : 2u);
    w.kx = w.kz == 2u ? 0u : w.kz + 1u;
    w.ky = w.kx == 2u ? 0u : w.kx + 1u;
    const float dz = comp3(d, w.kz);
    if (dz < 0.0f) {
        const uint32_t t = w.kx;
        w.kx = w.ky;
        w.ky = t;
    }
    w.Sx = X::div(comp3(d, w.kx), dz);
    w.Sy = X::div(comp3(d, w.ky), dz);
    w.Sz = X::rcp(dz);
    return w;
}
GPUGI_D float wt_edge(float ax, float ay, float bx, float by) {  // ax * by - ay * bx
    return X::sub(X::mul(ax, by), X::mul(ay, bx));
}
GPUGI_D float wt_edge64(float ax, float ay, float bx, float by) {
    return __double2float_rn(__dsub_rn(__dmul_rn((double)ax, (double)by), __dmul_rn((double)ay, (double)bx)));
}
GPUGI_D bool intersect_triangle_wt_v(float3 o, const WtRay& w, float4 ra, float4 rb, float4 rc, float& hit,
                                     float& by, float& bz) {
    const float3 A = X::sub3(make_float3(ra.x, ra.y, ra.z), o);
    const float3 B = X::sub3(make_float3(ra.w, rb.x, rb.y), o);
    const float3 C = X::sub3(make_float3(rb.z, rb.w, rc.x), o);
    const float Akz = comp3(A, w.kz), Bkz = comp3(B, w.kz), Ckz = comp3(C, w.kz);
    const float Ax = X::sub(comp3(A, w.kx), X::mul(w.Sx, Akz)), Ay = X::sub(comp3(A, w.ky), X::mul(w.Sy, Akz));
    const float Bx = X::sub(comp3(B, w.kx), X::mul(w.Sx, Bkz)), By = X::sub(comp3(B, w.ky), X::mul(w.Sy, Bkz));
    const float Cx = X::sub(comp3(C, w.kx), X::mul(w.Sx, Ckz)), Cy = X::sub(comp3(C, w.ky), X::mul(w.Sy, Ckz));
    float U = wt_edge(Cx, Cy, Bx, By), V = wt_edge(Ax, Ay, Cx, Cy), W = wt_edge(Bx, By, Ax, Ay);
    if (U == 0.0f || V == 0.0f || W == 0.0f) {
        U = wt_edge64(Cx, Cy, Bx, By);
        V = wt_edge64(Ax, Ay, Cx, Cy);
        W = wt_edge64(Bx, By, Ax, Ay);
    }
    if ((U < 0.0f || V < 0.0f || W < 0.0f) && (U > 0.0f || V > 0.0f || W > 0.0f)) return false;
    const float det = X::add(X::add(U, V), W);
    if (det == 0.0f) return false;
    const float T = X::add(X::add(X::mul(U, X::mul(w.Sz, Akz)), X::mul(V, X::mul(w.Sz, Bkz))),
                           X::mul(W, X::mul(w.Sz, Ckz)));
    const float rcpDet = X::rcp(det);
    hit = X::mul(T, rcpDet);
    by = X::mul(V, rcpDet);
    bz = X::mul(W, rcpDet);
    return hit > 0.0001f;
}
// The triangle test of a leaf slot: TRI 0 = the reference's, 1 = watertight.
template <int TRI>
GPUGI_D bool slot_test(const DevScene& s, float3 o, float3 d, const WtRay& w, uint32_t k, float& hit, float& by,
                       float& bz) {
    if (TRI == 0) return intersect_triangle(o, d, s.tris + 3 * (size_t)k, hit, by, bz);
    const float4* rec = s.wtris + 3 * (size_t)k;
    return intersect_triangle_wt_v(o, w, __ldg(rec), __ldg(rec + 1), __ldg(rec + 2), hit, by, bz);
}

struct TraceResult {
    int32_t slot;  // -1 = miss
    float t;
    float u, v;
};

// Fetch counters of one walk, the analogue of TRACERAY_DEBUG_VARS
// (traceray.glsl:59-61,131-133): node fetches, leaf slot fetches (the shader
// also fetches the first invalid slot of a block before leaving it) and
// valid triangles tested.
struct WalkCounters {
    uint32_t nodes = 0, slots = 0, tris = 0;
};

// The walk. ANY_HIT returns at the first accepted triangle (result.slot set
// to the accepting slot). Every loop is bounded: a validated hierarchy
// strictly increases the node index, so numNodes visits always suffice; the
// cap only guards against device memory corruption and reports
// DEVERR_TRAVERSAL_CAP instead of spinning.
template <bool ANY_HIT, int BOUNDS, bool COUNT = false, int TRI = 0>
GPUGI_D TraceResult trace_ray(const DevScene& s, float3 o, float3 d, float rayLength, uint32_t* errWord,
                              WalkCounters* cnt = nullptr) {
    TraceResult r;
    r.slot = -1;
    r.u = r.v = 0.0f;
    const float3 inv = make_float3(X::rcp(d.x), X::rcp(d.y), X::rcp(d.z));
    const WtRay wt = TRI ? wt_setup(d) : WtRay{};
    uint32_t node = 0;
    uint32_t budget = s.numNodes;
    const float4* __restrict__ nodes = s.nodes;
    while (true) {
        if (budget-- == 0) {
            raise_error(errWord, DEVERR_TRAVERSAL_CAP);
            break;
        }
        if (kChecked && node >= s.numNodes) {
            raise_error(errWord, DEVERR_BOUNDS);
            break;
        }
        if (COUNT) ++cnt->nodes;
        const float4* nd = nodes + node_stride<BOUNDS>() * (size_t)node;
        const float4 a = __ldg(nd);
        const float4 b = __ldg(nd + 1);
        const float4 c = BOUNDS == 2 ? __ldg(nd + 2) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        const uint32_t child = __float_as_uint(a.w);
        const uint32_t escape = __float_as_uint(b.w);
        float firstHit;
        const bool hit = bounds_test<BOUNDS, TRI != 0>(o, d, inv, a, b, c, firstHit);
        if (hit && firstHit <= rayLength) {
            if (child & LEAF_FLAG) {
                const uint32_t count = (child >> LEAF_COUNT_SHIFT) & LEAF_COUNT_MASK;
                const uint32_t slot0 = (child & LEAF_BLOCK_MASK) * s.leafSize;
                if (kChecked && (uint64_t)slot0 + count > s.numSlots) {
                    raise_error(errWord, DEVERR_BOUNDS);
                    break;
                }
                if (COUNT) cnt->slots += count < s.leafSize ? count + 1 : count;
                for (uint32_t k = 0; k < count; ++k) {
                    if (COUNT) ++cnt->tris;
                    float h, by, bz;
                    if (slot_test<TRI>(s, o, d, wt, slot0 + k, h, by, bz) && h < rayLength) {
                        rayLength = h;
                        r.slot = (int32_t)(slot0 + k);
                        r.u = by;
                        r.v = bz;
                        if (ANY_HIT) {
                            // the shader stops fetching at the accepting slot
                            if (COUNT) cnt->slots -= (count < s.leafSize ? count + 1 : count) - (k + 1);
                            r.t = rayLength;
                            return r;
                        }
                    }
                }
                node = escape;
            } else {
                node = child;
            }
        } else {
            node = escape;
        }
        if (node == 0) break;
    }
    r.t = rayLength;
    return r;
}

// One ray's walk as a resumable state machine, advanced one test at a time.
// The sequence of node and triangle tests is the same as trace_ray's; the
// state lets a persistent warp refill a finished lane with the next ray
// instead of idling until the warp's longest walk ends. (Testing a whole
// leaf block per step, four triangles at a time, was measured 18 % slower on
// the 65,536-triangle icosphere: lanes of a warp then diverge between node
// steps and leaf loops of different lengths.)
struct WalkState {
    float3 o, d, inv;
    WtRay wt;  // used by the watertight test only
    float len;
    uint32_t node;  // next node to test, NODE_DONE when the escape chain ended
    uint32_t cur, end;  // leaf slots still to test
    uint32_t budget;
    int32_t slot;
    float u, v;
};
constexpr uint32_t NODE_DONE = 0xFFFFFFFFu;

GPUGI_D void walk_begin(WalkState& w, const DevScene& s, float3 o, float3 d, float tmax) {
    w.o = o;
    w.d = d;
    w.inv = make_float3(X::rcp(d.x), X::rcp(d.y), X::rcp(d.z));
    w.wt = wt_setup(d);  // dead code unless a watertight walker reads it
    w.len = tmax;
    w.node = 0;
    w.cur = w.end = 0;
    w.budget = s.numNodes;
    w.slot = -1;
    w.u = w.v = 0.0f;
}

// Copy the first `count` nodes (the top tree levels, see DevScene::topNodes)
// into shared memory. Called by every thread of a block before its walks.
GPUGI_D void stage_top_nodes(const DevScene& s, float4* smem, uint32_t count) {
    // oriented-box scenes stage nothing (their upload keeps the preorder layout)
    for (uint32_t i = threadIdx.x; i < 2 * count; i += blockDim.x) smem[i] = __ldg(s.nodes + i);
    __syncthreads();
}

// Perform one test. Returns true when the walk is over (for ANY_HIT also
// when a triangle was accepted). Nodes below topCount come from `top`.
// Node and triangle steps share one fetch (the record address depends on the
// step kind), so the lanes of a warp that are at different kinds of step
// wait for one memory round trip per step instead of one per kind.
template <bool ANY_HIT, int BOUNDS, int TRI = 0>
GPUGI_D bool walk_step(WalkState& w, const DevScene& s, uint32_t* errWord, const float4* top = nullptr,
                       uint32_t topCount = 0) {
    const bool isTri = w.cur < w.end;
    if (!isTri && w.budget-- == 0) {
        raise_error(errWord, DEVERR_TRAVERSAL_CAP);
        w.node = NODE_DONE;
        return true;
    }
    if (kChecked && (isTri ? w.cur >= s.numSlots : w.node >= s.numNodes)) {
        raise_error(errWord, DEVERR_BOUNDS);
        w.cur = w.end;
        w.node = NODE_DONE;
        return true;
    }
    float4 a, b, c = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    constexpr uint32_t NS = node_stride<BOUNDS>();
    if (!isTri && w.node < topCount) {
        a = top[NS * w.node];
        b = top[NS * w.node + 1];
        if (BOUNDS == 2) c = top[NS * w.node + 2];
    } else {
        const float4* src =
            isTri ? (TRI ? s.wtris : s.tris) + 3 * (size_t)w.cur : s.nodes + NS * (size_t)w.node;
        a = __ldg(src);
        b = __ldg(src + 1);
        if (isTri || BOUNDS == 2) c = __ldg(src + 2);
    }
    if (isTri) {
        float h, by, bz;
        const bool ok = TRI ? intersect_triangle_wt_v(w.o, w.wt, a, b, c, h, by, bz)
                            : intersect_triangle_v(w.o, w.d, a, b, c, h, by, bz);
        if (ok && h < w.len) {
            w.len = h;
            w.slot = (int32_t)w.cur;
            w.u = by;
            w.v = bz;
            if (ANY_HIT) return true;
        }
        ++w.cur;
    } else {
        const uint32_t child = __float_as_uint(a.w);
        const uint32_t escape = __float_as_uint(b.w);
        float firstHit;
        const bool hit = bounds_test<BOUNDS, TRI != 0>(w.o, w.d, w.inv, a, b, c, firstHit);
        if (hit && firstHit <= w.len) {
            if (child & LEAF_FLAG) {
                w.cur = (child & LEAF_BLOCK_MASK) * s.leafSize;
                w.end = w.cur + ((child >> LEAF_COUNT_SHIFT) & LEAF_COUNT_MASK);
                w.node = escape ? escape : NODE_DONE;
            } else {
                w.node = child;
            }
        } else {
            w.node = escape ? escape : NODE_DONE;
        }
    }
    return w.cur >= w.end && w.node == NODE_DONE;
}

// ---------------------------------------------------------------- group walk
// G lanes walk one ray together (G = 4, 8 or 16; every lane of the group
// holds the same state and calls group_step with it). A node round tests
// the G consecutive nodes [node, node + G) of the node array (one coalesced
// load), then resolves which of them the sequential walk visits by pointer
// jumping over the successors inside the window (log2 G shuffles): the walk
// leaves the window at a node outside it, at the end of the escape chain or
// at a hit leaf. A leaf round tests G slots of the leaf block at once and
// applies the sequential acceptance rule: a slot is accepted when
// hit < rayLength, so the result is the first slot reaching the minimum (any
// hit: the first accepted slot). Every node decision uses trace_ray's
// arithmetic with the same rayLength, so results are identical; tests of
// nodes the walk skips are discarded. Successors may point backwards (the
// breadth-first top-level layout): they simply end the round.
struct GroupWalk {
    float3 o, d, inv;
    WtRay wt;  // used by the watertight test only
    float len, u, v;
    int32_t slot;
    uint32_t node, cur, end, resume, budget;
};
constexpr uint32_t kGroupDone = 0xFFFFFFFFu, kGroupLeaf = 0x80000000u;

GPUGI_D void group_begin(GroupWalk& g, const DevScene& s, float3 o, float3 d, float tmax) {
    g.o = o;
    g.d = d;
    g.inv = make_float3(X::rcp(d.x), X::rcp(d.y), X::rcp(d.z));
    g.wt = wt_setup(d);  // dead code unless a watertight walker reads it
    g.len = tmax;
    g.u = g.v = 0.0f;
    g.slot = -1;
    g.node = 0;
    g.cur = g.end = 0;
    g.resume = kGroupDone;
    g.budget = s.numNodes;
}

// One round; returns true when the walk is over. gl = lane in the group,
// gbase = first lane of the group, gmask = the group's lanes.
template <bool ANY_HIT, int BOUNDS, int G, int TRI = 0>
GPUGI_D bool group_step(GroupWalk& g, const DevScene& s, uint32_t* err, unsigned gl, unsigned gbase,
                        unsigned gmask) {
    static_assert(G == 4 || G == 8 || G == 16, "group size");
    if (g.cur < g.end) {
        const uint32_t k = g.cur + gl;
        float h = 0.0f, by = 0.0f, bz = 0.0f;
        bool ok = false;
        if (k < g.end) ok = slot_test<TRI>(s, g.o, g.d, g.wt, k, h, by, bz) && h < g.len;
        if (ANY_HIT) {
            const uint32_t key = __reduce_min_sync(gmask, ok ? k : kGroupDone);
            if (key != kGroupDone) {
                g.slot = (int32_t)key;
                return true;
            }
        } else {
            // minimum hit distance (positive floats order like their bits),
            // then the lowest slot reaching it
            const uint32_t hb = __reduce_min_sync(gmask, ok ? __float_as_uint(h) : kGroupDone);
            const unsigned tie = __ballot_sync(gmask, ok && __float_as_uint(h) == hb);
            const unsigned src = tie ? (unsigned)(__ffs(tie) - 1) : gbase;
            const float wu = __shfl_sync(gmask, by, src), wv = __shfl_sync(gmask, bz, src);
            if (tie) {
                g.slot = (int32_t)(g.cur + (src - gbase));
                g.len = __uint_as_float(hb);
                g.u = wu;
                g.v = wv;
            }
        }
        g.cur = min(g.cur + G, g.end);
        if (g.cur >= g.end) {
            g.node = g.resume;
            if (g.node == kGroupDone) return true;
        }
        return false;
    }
    if (g.budget-- == 0) {
        raise_error(err, DEVERR_TRAVERSAL_CAP);
        return true;
    }
    if (kChecked && g.node >= s.numNodes) {
        raise_error(err, DEVERR_BOUNDS);
        return true;
    }
    const uint32_t p = g.node + gl;
    uint32_t next = kGroupDone, child = 0, escape = 0;
    if (p < s.numNodes) {
        const float4* nd = s.nodes + node_stride<BOUNDS>() * (size_t)p;
        const float4 a = __ldg(nd), b = __ldg(nd + 1);
        const float4 c = BOUNDS == 2 ? __ldg(nd + 2) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        child = __float_as_uint(a.w);
        escape = __float_as_uint(b.w);
        float firstHit;
        const bool hit = bounds_test<BOUNDS, TRI != 0>(g.o, g.d, g.inv, a, b, c, firstHit);
        if (hit && firstHit <= g.len) next = (child & LEAF_FLAG) ? (kGroupLeaf | gl) : child;
        else next = escape ? escape : kGroupDone;
    }
#pragma unroll
    for (int r = 1; r < G; r <<= 1) {
        const bool chase = next < kGroupLeaf && next - g.node < (uint32_t)G;
        const uint32_t w = __shfl_sync(gmask, next, gbase + (chase ? next - g.node : gl));
        next = chase ? w : next;
    }
    const uint32_t r0 = __shfl_sync(gmask, next, gbase);
    if (r0 == kGroupDone) return true;
    if (r0 & kGroupLeaf) {
        const unsigned src = gbase + (r0 & (kGroupLeaf - 1u));
        const uint32_t lc = __shfl_sync(gmask, child, src), le = __shfl_sync(gmask, escape, src);
        g.cur = (lc & LEAF_BLOCK_MASK) * s.leafSize;
        g.end = g.cur + ((lc >> LEAF_COUNT_SHIFT) & LEAF_COUNT_MASK);
        g.resume = le ? le : kGroupDone;
        if (kChecked && g.end > s.numSlots) {
            raise_error(err, DEVERR_BOUNDS);
            return true;
        }
        if (g.cur >= g.end) {  // empty leaf block
            g.node = g.resume;
            return g.node == kGroupDone;
        }
        return false;
    }
    g.node = r0;
    return false;
}

// Persistent loop of group walks over n work items. Group k of the grid
// takes item k first, then, whenever its walk ends, item (groups in the
// grid) + the value of one atomic increment of *work (which starts at 0).
// load(i, o, d, tmax) fills the ray of item i; finish(i, walk) runs in the
// group's first lane. With MULTI the rays belong to different scenes: load
// returns the item's scene and its bounds kind selects the node test per
// round; otherwise every ray walks `scene` with the BOUNDS test.
template <bool ANY_HIT, int BOUNDS, int G, bool MULTI, int TRI, typename Load, typename Finish>
GPUGI_D void group_walks_impl(const DevScene& scene, uint64_t n, unsigned long long* work, uint32_t* err, Load load,
                              Finish finish) {
    // The loop has no warp-wide synchronisation: all shuffles stay inside
    // the group, and a group leaves once the items are exhausted. The first
    // item needs no atomic, so a launch does not start with one increment
    // per group queued on the same counter (tens of thousands of them
    // serialise in L2 for ~10 us); small launches cost no atomics at all.
    const unsigned lane = threadIdx.x & 31u;
    const unsigned gl = lane & (G - 1), gbase = lane & ~(unsigned)(G - 1);
    const unsigned gmask = ((1u << G) - 1u) << gbase;
    const uint64_t perBlock = blockDim.x / G;
    const uint64_t groups = (uint64_t)gridDim.x * perBlock;
    GroupWalk g;
    DevScene sc;  // MULTI: the ray's scene, copied at its walk's start (fields stay in registers)
    for (uint64_t my = (uint64_t)blockIdx.x * perBlock + threadIdx.x / G; my < n;) {
        float3 o, d;
        float tmax;
        if constexpr (MULTI) {
            sc = *load(my, o, d, tmax);
            group_begin(g, sc, o, d, tmax);
        } else {
            load(my, o, d, tmax);
            group_begin(g, scene, o, d, tmax);
        }
        bool done = false;
        while (!done) {
            if constexpr (MULTI)
                done = sc.boundsKind == GPUGI_BOUNDS_ELLIPSOID ? group_step<ANY_HIT, 1, G>(g, sc, err, gl, gbase, gmask)
                       : sc.boundsKind == GPUGI_BOUNDS_OBOX    ? group_step<ANY_HIT, 2, G>(g, sc, err, gl, gbase, gmask)
                                                               : group_step<ANY_HIT, 0, G>(g, sc, err, gl, gbase, gmask);
            else
                done = group_step<ANY_HIT, BOUNDS, G, TRI>(g, scene, err, gl, gbase, gmask);
        }
        if (gl == 0) finish(my, g);
        unsigned long long next = 0;
        if (gl == 0) next = atomicAdd(work, 1ull);
        my = groups + __shfl_sync(gmask, next, gbase);
    }
}

template <bool ANY_HIT, int BOUNDS, int G, int TRI = 0, typename Load, typename Finish>
GPUGI_D void group_walks(const DevScene& scene, uint64_t n, unsigned long long* work, uint32_t* err, Load load,
                         Finish finish) {
    group_walks_impl<ANY_HIT, BOUNDS, G, false, TRI>(scene, n, work, err, load, finish);
}

template <bool ANY_HIT, int G, typename Load, typename Finish>
GPUGI_D void group_walks_multi(uint64_t n, unsigned long long* work, uint32_t* err, Load load, Finish finish) {
    group_walks_impl<ANY_HIT, 0, G, true, 0>(DevScene{}, n, work, err, load, finish);
}

// ----------------------------------------------------------------- wide walk
// Walks over the four-wide copy of an axis-aligned-box hierarchy (wide.cu):
// depth first with a stack of {reference, entry distance}, children in
// preorder, so leaves are met in exactly the order of the escape walk. The
// results are trace_ray's bit for bit although most inner levels are left
// out and four boxes are tested per fetch:
//  * The escape walk tests a leaf's triangles iff the leaf's box and all its
//    ancestors' boxes are hit with firstHit <= rayLength when they are met.
//  * Boxes are nested (checked when the wide hierarchy is made) and a slab
//    value rn(rn(plane - o) * inv) is monotone in the plane, so an
//    ancestor's firstHit is never larger and its lastHit never smaller than
//    the leaf's, and rayLength only shrinks. A leaf whose own test passes when
//    it is met has ancestors that passed when they were met: the tests of
//    the levels left out are implied. A subtree whose box fails holds no leaf
//    that would pass.
//  * A child that waits on the stack was tested with the rayLength of that
//    moment; its firstHit is compared again when it is taken, which is when
//    the escape walk would test it. So a waiting node may also be expanded
//    early; only leaves have to be tested in order.
//  * Monotonicity needs slab values that are not NaN. For finite rays that
//    leaves inv = +-inf (a zero direction component) and a plane through the
//    origin: only a box that is flat there, in a plane that also bounds an
//    ancestor, can pass where the ancestor fails. Such a box sends the ray
//    back to its start on the binary tree (`seq`), and non-finite rays walk
//    the binary tree at once. (The watertight box test drops those slabs on
//    every level, so it stays monotone.)
//
// What bounds it and why this split (98k-triangle room, second bounce of 4.2M
// camera paths, ncu): L1 wavefronts 83 % and issue slots 71 % of their peaks,
// DRAM 1 % (camera rays 58 % and 78 %): a lane reads 112 B of node per visit, 10
// visits per ray instead of 45 binary nodes. One lane per ray for nodes keeps
// an instruction useful for ~20 lanes (8-lane groups on 8-wide nodes issued 2.3x
// the instructions); leaves go to eight lanes each, four leaves at a time, because a lane that loops over a block's
// triangles waits for memory once per triangle (1.05 to 0.87 ms for 3M
// any-hit rays in the 528k-triangle terrain, then). Quantised 96-B nodes halved
// the L1 load but cost more issue slots than they freed (0.99 ms); prefetches
// of waiting children cost 2-8 %.
// Measured against the binary walkers: 3M any-hit rays in the terrain
// 2.18 to 0.80 ms, path tracing the room at 512^2 x 16 samples 15.7 to 8.8 ms,
// light tracing 9.0 to 4.6 ms, 1,000 rays (a warp each) 43.7 to 12.3 us, a
// 320 x 180 frame 1.03 to 0.62 ms (0.92 with eight lanes per ray at the end).
GPUGI_D bool finite3(float3 v) { return isfinite(v.x) && isfinite(v.y) && isfinite(v.z); }

// Lanes of a warp step through nodes together until kWideLeaves leaves wait or
// fewer than kWideNodes lanes have a node left (leaves 4 / 8 / 12: 10.09 / 9.94
// / 9.94 ms for the path-traced room; node lanes 4-12: the same), fetch new
// rays when at least kWideRefill lanes are free (1 / 8 / 12 / 16: 1.04 / 0.98 /
// 0.97 / 0.99 of the terrain's time), and hand their rays over, one after
// another, to the whole warp when no more than kWideWarpAt are left: the long
// single walks that a queue ends with then take a few rounds (at 1 / 2 / 4 / 6
// / 10 rays: 748 / 691 / 664 / 664 / 678 us for a 320 x 180 frame of one sample,
// 137 / 129 / 120 / 118 / 123 for 66k rays in the icosphere). Queues of at most
// kWideSolo rays per warp are walked that way from the start (1 / 4 / 8 / 16 /
// 32: 664 / 655 / 623 / 616 / 617 us for the frame; 119 / 127 us at 8 / 16 for
// the icosphere's 66k) or, since any-hit walks end early, kWideSoloAny
// (30,000 rays at 8 / 5: 36.3 / 29.5 us in a room of 3k triangles, 40.2 / 33.6 in
// one of 20k, the frame 608 / 615; 20,000 at 5 / 4: 34.8 / 38.4 in a terrain of
// 100k).
constexpr int kWideLeaves = 8, kWideNodes = 8, kWideRefill = 12, kWideWarpAt = 5;
constexpr uint32_t kWideSolo = 8, kWideSoloAny = 5;
// Resident blocks per SM that the wide walkers are compiled for (64
// registers; 7 / 8 / 9 blocks: 9.94 / 9.60 / 9.63 ms for the path-traced room).
#ifndef GPUGI_WIDE_MIN_BLOCKS
#define GPUGI_WIDE_MIN_BLOCKS 8
#endif

struct WideShared {
    uint2 e[kWideShared][128];  // stack entries {reference, entry distance}, a column per ray
    float4 ray[2][128];         // {origin, d.x}, {d.y, d.z, -, -}
    uint2 w[4][kWarpStack];     // stack of the ray a whole warp walks
};

// Valid slots of a leaf word (checked builds: none where they pass the end).
GPUGI_D uint32_t leaf_slots(const DevScene& s, uint32_t leaf, uint32_t* err) {
    const uint32_t c = (leaf >> LEAF_COUNT_SHIFT) & LEAF_COUNT_MASK;
    if (kChecked && (uint64_t)(leaf & LEAF_BLOCK_MASK) * s.leafSize + c > s.numSlots) {
        raise_error(err, DEVERR_BOUNDS);
        return 0u;
    }
    return c;
}

// The leaves of the lanes in `todo` (each holds a leaf word in ref), four at a
// time by eight lanes each; the rays come from shared memory (ray[.][thread]
// = {origin, d.x}, {d.y, d.z, -, -}). A leaf's result is the sequential rule's:
// the first slot reaching the minimum hit distance below the owner's len (any
// hit: slot becomes 0 when a triangle is accepted). scene_of(lane) is the
// scene of a lane's ray, own the caller's; after() runs in the owner.
template <bool ANY_HIT, int TRI, typename SceneOf, typename After>
GPUGI_D void leaf_rounds(unsigned todo, const float4 (*ray)[128], const uint32_t& ref, SceneOf scene_of,
                         const DevScene* const& own, uint32_t* err, float& len, float& u, float& v, int32_t& slot,
                         After after) {
    const unsigned lane = threadIdx.x & 31u;
    while (todo) {
        const unsigned my = lane >> 3, gl = lane & 7u;
        const unsigned m1 = todo & (todo - 1), m2 = m1 & (m1 - 1), m3 = m2 & (m2 - 1);
        const unsigned mm = my == 0 ? todo : my == 1 ? m1 : my == 2 ? m2 : m3;
        const unsigned batch = todo & ~(m3 & (m3 - 1));
        todo &= ~batch;
        const unsigned src = mm ? (unsigned)(__ffs(mm) - 1) : 0u;
        const float4 r0 = ray[0][(threadIdx.x & ~31u) + src], r1 = ray[1][(threadIdx.x & ~31u) + src];
        const float3 ro = make_float3(r0.x, r0.y, r0.z), rd = make_float3(r0.w, r1.x, r1.y);
        const uint32_t lref = __shfl_sync(0xffffffffu, ref, src);
        const DevScene* ls = scene_of(src);
        WtRay w = {};
        if (TRI) w = wt_setup(rd);
        const bool mine = (batch >> lane) & 1u;
        const unsigned owner = 8u * (unsigned)__popc(batch & ((1u << lane) - 1u));  // first lane of my leaf's group
        const uint32_t k0 = mm ? (lref & LEAF_BLOCK_MASK) * ls->leafSize : 0u;
        const uint32_t cnt = mm ? leaf_slots(*ls, lref, err) : 0u;
        for (uint32_t off = gl; __any_sync(0xffffffffu, off - gl < cnt); off += 8) {
            const float rl = __shfl_sync(0xffffffffu, len, src);
            float h = 0.0f, hu = 0.0f, hv = 0.0f;
            bool ok = false;
            if (off < cnt) {
                const float4* rec = (TRI ? ls->wtris : ls->tris) + 3 * (size_t)(k0 + off);
                const float4 a = __ldg(rec), b = __ldg(rec + 1), c = __ldg(rec + 2);
                ok = TRI ? intersect_triangle_wt_v(ro, w, a, b, c, h, hu, hv)
                         : intersect_triangle_v(ro, rd, a, b, c, h, hu, hv);
                ok = ok && h < rl;
            }
            const unsigned any = __ballot_sync(0xffffffffu, ok);
            if (ANY_HIT) {
                if (mine && (any >> (owner & 31u) & 0xffu)) slot = 0;
            } else if (any) {
                const uint32_t hb = ok ? __float_as_uint(h) : 0x7fffffffu;
                uint32_t mn = min(hb, __shfl_xor_sync(0xffffffffu, hb, 4));
                mn = min(mn, __shfl_xor_sync(0xffffffffu, mn, 2));
                mn = min(mn, __shfl_xor_sync(0xffffffffu, mn, 1));
                const unsigned tie = __ballot_sync(0xffffffffu, ok && hb == mn);
                const unsigned gm = mine ? tie >> (owner & 31u) & 0xffu : 0u;
                const unsigned wl = gm ? owner + (unsigned)__ffs(gm) - 1 : lane;
                const float wh = __shfl_sync(0xffffffffu, h, wl & 31u), wu = __shfl_sync(0xffffffffu, hu, wl & 31u),
                            wv = __shfl_sync(0xffffffffu, hv, wl & 31u);
                if (gm) {
                    len = wh;
                    u = wu;
                    v = wv;
                    slot = (int32_t)((ref & LEAF_BLOCK_MASK) * own->leafSize + (off - gl) + (wl & 7u));
                }
            }
        }
        if (mine) after();
    }
}

// Persistent loop of wide walks over n work items in blocks of 128 threads, of
// which the first `blocks` of the grid call it: their warps share the first
// items out evenly (at most 32 each), later ones come from an atomic counter
// *work, which starts at 0. load(i, o, d, tmax) fills the ray of item i (again
// when a walk restarts); finish(i, slot, t, u, v) takes its result (any hit:
// slot >= 0 when occluded). n < 2^32. work may be null where every warp gets at
// most kWideSolo items: they are then strided over the warps. MULTI: the items
// belong to several scenes, load returns the item's (a scene with a wide
// hierarchy); otherwise every ray walks `scene`.
template <bool ANY_HIT, int TRI, bool MULTI = false, typename Load, typename Finish>
GPUGI_D void wide_walks(WideShared& sh, const DevScene& scene, uint64_t n, unsigned long long* work, uint32_t* err,
                        Load load, Finish finish, unsigned blocks = gridDim.x) {
    constexpr uint32_t kNone = 0xFFFFFFFFu;  // also kWideEmpty: never a node or a leaf
    const unsigned lane = threadIdx.x & 31u;
    const DevScene* own = &scene;  // MULTI: the scene of the lane's ray
    const char* wide = reinterpret_cast<const char*>(scene.wide);
    auto shfl_scene = [&](unsigned mask, unsigned src) {
        const uint64_t p = reinterpret_cast<uint64_t>(own);
        return reinterpret_cast<const DevScene*>((uint64_t)__shfl_sync(mask, (uint32_t)(p >> 32), src) << 32 |
                                                 __shfl_sync(mask, (uint32_t)p, src));
    };
    uint2 deep[kWideStack - kWideShared];
    bool active = false;
    uint32_t item = 0;
    // -origin and 1 / direction as packed pairs
    float2 nox = {}, noy = {}, noz = {}, ivx = {}, ivy = {}, ivz = {};
    float len = 0.0f, u = 0.0f, v = 0.0f;
    int32_t slot = -1;
    uint32_t ref = kNone, sp = 0, budget = 0;
    bool axis = false, seq = false;
    unsigned col = threadIdx.x;  // the ray's column in shared memory
    auto origin = [&]() { return make_float3(-nox.x, -noy.x, -noz.x); };
    auto invdir = [&]() { return make_float3(ivx.x, ivy.x, ivz.x); };
    auto begin = [&](uint32_t i) {
        item = i;
        float3 o, d;
        if constexpr (MULTI) {
            own = load(item, o, d, len);
            wide = reinterpret_cast<const char*>(own->wide);
        } else {
            load(item, o, d, len);
        }
        slot = -1;
        u = v = 0.0f;
        const float3 inv = make_float3(X::rcp(d.x), X::rcp(d.y), X::rcp(d.z));
        sh.ray[0][col] = make_float4(o.x, o.y, o.z, d.x);
        sh.ray[1][col] = make_float4(d.y, d.z, 0.0f, 0.0f);
        nox = make_float2(-o.x, -o.x), noy = make_float2(-o.y, -o.y), noz = make_float2(-o.z, -o.z);
        ivx = make_float2(inv.x, inv.x), ivy = make_float2(inv.y, inv.y), ivz = make_float2(inv.z, inv.z);
        seq = !(finite3(o) && finite3(d));
        axis = TRI == 0 && !finite3(inv);
        ref = sp = 0;
        budget = own->numNodes;
        active = true;
    };
    auto pop = [&]() {  // the next pending child, or kNone
        ref = kNone;
        if (seq) {
            ref = sp ? sp : kNone;
            sp = 0;
            return;
        }
        while (sp > 0) {
            --sp;
            uint2 e;
            if (sp < kWideShared) e = sh.e[sp][col];
            else e = deep[sp - kWideShared];
            if (ANY_HIT || __uint_as_float(e.y) <= len) {
                ref = e.x;
                break;
            }
        }
    };
    // A node visit: every node is met once in a walk, so numNodes of them always suffice (the cap
    // only guards against device memory corruption); checked builds test the index too.
    auto guard = [&](uint32_t count) {
        const bool capped = budget-- == 0, outside = kChecked && ref >= count;
        if (capped) raise_error(err, DEVERR_TRAVERSAL_CAP);
        if (outside) raise_error(err, DEVERR_BOUNDS);
        if (capped || outside) {
            ref = kNone;
            sp = 0;
        }
        return capped || outside;
    };
    auto seq_node = [&]() {  // one node of the binary tree; sp holds the escape of a hit leaf
        const float4 a = __ldg(own->nodes + 2 * (size_t)ref), b = __ldg(own->nodes + 2 * (size_t)ref + 1);
        float f;
        const bool hit = intersect_box<TRI != 0>(origin(), invdir(), a, b, f) && f <= len;
        const uint32_t child = __float_as_uint(a.w), esc = __float_as_uint(b.w);
        if (hit && (child & LEAF_FLAG)) sp = esc;
        ref = hit ? child : (esc ? esc : kNone);
    };
    // A passing box that is flat in the plane through the origin of a ray with a zero component there.
    auto flat = [&](float3 lo, float3 hi) {
        const float3 o = origin(), inv = invdir();
        return (isinf(inv.x) && lo.x == o.x && hi.x == o.x) || (isinf(inv.y) && lo.y == o.y && hi.y == o.y) ||
               (isinf(inv.z) && lo.z == o.z && hi.z == o.z);
    };
    const unsigned warps = blocks * (blockDim.x >> 5);
    const unsigned C = n >= 32 * (uint64_t)warps ? 32u : ((uint32_t)n + warps - 1) / warps;
    const uint64_t first = (uint64_t)warps * C;
    bool more = n > first;
    const uint64_t warp = (uint64_t)(threadIdx.x >> 5) * blocks + blockIdx.x;
    const bool solo = n <= (uint64_t)warps * (ANY_HIT ? kWideSoloAny : kWideSolo);
    if (!solo) {
        const uint64_t i = warp * C + lane;
        if (lane < C && i < n) begin((uint32_t)i);
    }
    // ---- a ray per lane
    while (!solo) {
        const unsigned act = __ballot_sync(0xffffffffu, active);
        if (more && __popc(act) <= 32 - kWideRefill) {
            unsigned long long base = 0;
            if (lane == 0) base = atomicAdd(work, (unsigned long long)__popc(~act));
            base = first + __shfl_sync(0xffffffffu, base, 0);
            more = base + __popc(~act) < n;
            base += (unsigned)__popc(~act & ((1u << lane) - 1u));
            __syncwarp();  // the leaf rounds' reads of the rays that are replaced
            if (!active && base < n) begin((uint32_t)base);
        } else if (!more && __popc(act) <= kWideWarpAt) {
            break;
        }
        // nodes
        while (true) {
            if (active && !(ref & LEAF_FLAG)) {
                if (guard(seq ? own->numNodes : own->numWide)) {
                } else if (!seq) {
                    const uint32_t at = ref * 128u;
                    const uint32_t ax = at + (ivx.x < 0.0f ? 16u : 0u), ay = at + (ivy.x < 0.0f ? 48u : 32u),
                                   az = at + (ivz.x < 0.0f ? 80u : 64u);
                    auto ld = [&](uint32_t off) { return __ldg(reinterpret_cast<const float4*>(wide + off)); };
                    const float4 nx = ld(ax), fx = ld(ax ^ 16u), ny = ld(ay), fy = ld(ay ^ 16u), nz = ld(az),
                                 fz = ld(az ^ 16u);
                    const uint4 rf = __ldg(reinterpret_cast<const uint4*>(wide + (at + 96u)));
                    // slab values of two children's planes
                    auto slab = [](float p, float q, float2 no, float2 iv) {
                        return __fmul2_rn(__fadd2_rn(make_float2(p, q), no), iv);
                    };
                    const float2 nx0 = slab(nx.x, nx.y, nox, ivx), nx1 = slab(nx.z, nx.w, nox, ivx);
                    const float2 ny0 = slab(ny.x, ny.y, noy, ivy), ny1 = slab(ny.z, ny.w, noy, ivy);
                    const float2 nz0 = slab(nz.x, nz.y, noz, ivz), nz1 = slab(nz.z, nz.w, noz, ivz);
                    const float2 fx0 = slab(fx.x, fx.y, nox, ivx), fx1 = slab(fx.z, fx.w, nox, ivx);
                    const float2 fy0 = slab(fy.x, fy.y, noy, ivy), fy1 = slab(fy.z, fy.w, noy, ivy);
                    const float2 fz0 = slab(fz.x, fz.y, noz, ivz), fz1 = slab(fz.z, fz.w, noz, ivz);
                    auto widen = [](float l) { return TRI ? X::mul(l, 0x1.000008p+0f) : l; };
                    const float f0 = fmaxf(0.0f, max3f(nx0.x, ny0.x, nz0.x));
                    const float f1 = fmaxf(0.0f, max3f(nx0.y, ny0.y, nz0.y));
                    const float f2 = fmaxf(0.0f, max3f(nx1.x, ny1.x, nz1.x));
                    const float f3 = fmaxf(0.0f, max3f(nx1.y, ny1.y, nz1.y));
                    bool h0 = f0 <= widen(min3f(fx0.x, fy0.x, fz0.x)) && f0 <= len;
                    bool h1 = f1 <= widen(min3f(fx0.y, fy0.y, fz0.y)) && f1 <= len;
                    bool h2 = f2 <= widen(min3f(fx1.x, fy1.x, fz1.x)) && f2 <= len && rf.z != kWideEmpty;
                    bool h3 = f3 <= widen(min3f(fx1.y, fy1.y, fz1.y)) && f3 <= len && rf.w != kWideEmpty;
                    bool restart = false;
                    if (TRI == 0 && axis) {
                        // planes through the origin give NaN slabs: the exact test, and the binary tree
                        // where the levels left out are not implied
                        auto exact = [&](bool& h, float3 lo, float3 hi) {
                            float f;
                            h = h && intersect_box<false>(origin(), invdir(), make_float4(lo.x, lo.y, lo.z, 0.0f),
                                                          make_float4(hi.x, hi.y, hi.z, 0.0f), f) && f <= len;
                            restart = restart || (h && flat(lo, hi));
                        };
                        exact(h0, make_float3(nx.x, ny.x, nz.x), make_float3(fx.x, fy.x, fz.x));
                        exact(h1, make_float3(nx.y, ny.y, nz.y), make_float3(fx.y, fy.y, fz.y));
                        exact(h2, make_float3(nx.z, ny.z, nz.z), make_float3(fx.z, fy.z, fz.z));
                        exact(h3, make_float3(nx.w, ny.w, nz.w), make_float3(fx.w, fy.w, fz.w));
                    }
                    // the first hit child in preorder is next, the others go on the stack, last one first
                    const bool p1 = h1 && h0, p2 = h2 && (h0 || h1), p3 = h3 && (h0 || h1 || h2);
                    ref = h0 ? rf.x : h1 ? rf.y : h2 ? rf.z : h3 ? rf.w : kNone;
                    auto put = [&](bool p, uint32_t r, float f) {
                        if (p) {
                            if (sp < kWideShared) sh.e[sp][col] = make_uint2(r, __float_as_uint(f));
                            else deep[sp - kWideShared] = make_uint2(r, __float_as_uint(f));
                            ++sp;
                        }
                    };
                    if (sp + 3 <= kWideShared) {  // always, but for the deepest walks
                        uint2* e = &sh.e[sp][col];
                        if (p3) *e = make_uint2(rf.w, __float_as_uint(f3));
                        e += p3 ? 128 : 0;
                        if (p2) *e = make_uint2(rf.z, __float_as_uint(f2));
                        e += p2 ? 128 : 0;
                        if (p1) *e = make_uint2(rf.y, __float_as_uint(f1));
                        sp += (p3 ? 1u : 0u) + (p2 ? 1u : 0u) + (p1 ? 1u : 0u);
                    } else {
                        put(p3, rf.w, f3);
                        put(p2, rf.z, f2);
                        put(p1, rf.y, f1);
                    }
                    if (TRI == 0 && restart) {
                        begin(item);
                        seq = true;
                    }
                } else {
                    seq_node();
                }
                if (ref == kNone) pop();
                if (ref == kNone) {
                    finish(item, slot, len, u, v);
                    active = false;
                }
            }
            const unsigned nodes = __ballot_sync(0xffffffffu, active && !(ref & LEAF_FLAG));
            const unsigned leaves = __ballot_sync(0xffffffffu, active && (ref & LEAF_FLAG));
            if (__popc(leaves) >= kWideLeaves || __popc(nodes) < kWideNodes || !nodes) break;
        }
        // leaves: four at a time, eight lanes each
        unsigned todo = __ballot_sync(0xffffffffu, active && (ref & LEAF_FLAG));
        __syncwarp();
        leaf_rounds<ANY_HIT, TRI>(
            todo, sh.ray, ref, [&](unsigned src) { return MULTI ? shfl_scene(0xffffffffu, src) : own; }, own, err, len, u,
            v, slot, [&]() {
                if (ANY_HIT && slot >= 0) {
                    ref = kNone;
                } else {
                    pop();
                }
                if (ref == kNone) {
                    finish(item, slot, len, u, v);
                    active = false;
                }
            });
    }
    // ---- a warp per ray
    // Every lane holds the ray; the stack is the warp's. A node round expands up to eight entries from
    // the top (waiting nodes early, waiting leaves stay), a leaf round tests up to four leading leaves
    // and resolves them in order.
    uint2* const ws = sh.w[threadIdx.x >> 5];
    uint64_t next = warp;
    __syncwarp();  // a warp with few rays comes here straight from begin(), whose rays every lane reads
    while (true) {
        unsigned src = 0;
        if (solo) {
            if (next >= n) break;
            if (lane == 0) begin((uint32_t)next);
            __syncwarp();
        } else {
            const unsigned act = __ballot_sync(0xffffffffu, active);
            if (!act) break;
            src = (unsigned)(__ffs(act) - 1);
        }
        auto get = [&](float x) { return __shfl_sync(0xffffffffu, x, src); };
        auto geti = [&](uint32_t x) { return __shfl_sync(0xffffffffu, x, src); };
        const unsigned scol = (threadIdx.x & ~31u) + src;
        const float4 r0 = sh.ray[0][scol], r1 = sh.ray[1][scol];
        const float3 o = make_float3(r0.x, r0.y, r0.z), d = make_float3(r0.w, r1.x, r1.y);
        const float3 wi = make_float3(get(ivx.x), get(ivy.x), get(ivz.x));
        WtRay wt = {};
        if (TRI) wt = wt_setup(d);
        float wlen = get(len), wu = get(u), wv = get(v);
        int32_t wslot = (int32_t)geti((uint32_t)slot);
        const uint32_t witem = geti(item);
        uint32_t wref = geti(ref), wsp = geti(sp), wbudget = geti(budget);
        const bool waxis = geti(axis) != 0;
        bool wseq = geti(seq) != 0;
        const DevScene* const ws_scene = MULTI ? shfl_scene(0xffffffffu, src) : own;
        const DevScene& s = *ws_scene;
        const float4* const tris = TRI ? s.wtris : s.tris;
        const char* const wwide = reinterpret_cast<const char*>(s.wide);
        // the ray's stack, with the reference it holds on top (a sequential walk keeps its escape in wsp)
        if (!wseq) {
            for (uint32_t k = lane; k < min(wsp, kWideShared); k += 32) ws[k] = sh.e[k][scol];
            for (uint32_t k = kWideShared; k < wsp; ++k) {
                const uint2 e = deep[k - kWideShared];
                const uint2 x = make_uint2(geti(e.x), geti(e.y));
                if (lane == 0) ws[k] = x;
            }
            if (lane == 0) ws[wsp] = make_uint2(wref, 0u);  // firstHit already compared with this rayLength
            ++wsp;
            __syncwarp();
        }
        // `leaves` leading leaves, lane group g's word lref with entry distance lf; true when any hit is
        // done. Leaves that are tested together take one pass of eight lanes each.
        auto test_leaves = [&](uint32_t lref, float lf, unsigned leaves) {
            const unsigned g = lane >> 3, gl = lane & 7u;
            const uint32_t k0 = g < leaves ? (lref & LEAF_BLOCK_MASK) * s.leafSize : 0u;
            const uint32_t cnt = g < leaves ? leaf_slots(s, lref, err) : 0u;
            for (uint32_t off = gl; __any_sync(0xffffffffu, off - gl < cnt); off += 8) {
                float h = 0.0f, hu = 0.0f, hv = 0.0f;
                bool ok = false;
                if (off < cnt) {
                    const float4* rec = tris + 3 * (size_t)(k0 + off);
                    const float4 a = __ldg(rec), b = __ldg(rec + 1), c = __ldg(rec + 2);
                    ok = TRI ? intersect_triangle_wt_v(o, wt, a, b, c, h, hu, hv)
                             : intersect_triangle_v(o, d, a, b, c, h, hu, hv);
                    ok = ok && h < wlen && lf <= wlen;
                }
                if (!__any_sync(0xffffffffu, ok)) continue;
                if (ANY_HIT) {
                    wslot = 0;
                    return true;
                }
                const uint32_t hb = ok ? __float_as_uint(h) : 0x7fffffffu;
                uint32_t mn = min(hb, __shfl_xor_sync(0xffffffffu, hb, 4));
                mn = min(mn, __shfl_xor_sync(0xffffffffu, mn, 2));
                mn = min(mn, __shfl_xor_sync(0xffffffffu, mn, 1));
                const unsigned tie = __ballot_sync(0xffffffffu, ok && hb == mn);
                for (unsigned k = 0; k < leaves; ++k) {  // in order: each with the rayLength the ones before left
                    const unsigned gm = tie >> (8 * k) & 0xffu;
                    if (!gm) continue;
                    const unsigned win = 8 * k + (unsigned)__ffs(gm) - 1;
                    const float kf = __shfl_sync(0xffffffffu, lf, win), kh = __shfl_sync(0xffffffffu, h, win);
                    if (kf <= wlen && kh < wlen) {
                        wlen = kh;
                        wu = __shfl_sync(0xffffffffu, hu, win);
                        wv = __shfl_sync(0xffffffffu, hv, win);
                        wslot = (int32_t)__shfl_sync(0xffffffffu, k0 + off, win);
                    }
                }
            }
            return false;
        };
        while (true) {
            if (wseq) {  // the binary tree, one node at a time
                if (wref & LEAF_FLAG) {
                    if (test_leaves(wref, 0.0f, 1)) break;
                    if (wsp == 0) break;
                    wref = wsp;
                    wsp = 0;
                    continue;
                }
                if (wbudget-- == 0 || (kChecked && wref >= s.numNodes)) {
                    raise_error(err, kChecked && wref >= s.numNodes ? DEVERR_BOUNDS : DEVERR_TRAVERSAL_CAP);
                    break;
                }
                const float4 a = __ldg(s.nodes + 2 * (size_t)wref), b = __ldg(s.nodes + 2 * (size_t)wref + 1);
                float f;
                const bool hit = intersect_box<TRI != 0>(o, wi, a, b, f) && f <= wlen;
                const uint32_t child = __float_as_uint(a.w), esc = __float_as_uint(b.w);
                if (hit && (child & LEAF_FLAG)) wsp = esc;
                wref = hit ? child : esc;
                if (!hit && esc == 0) break;
                continue;
            }
            if (wsp == 0) break;
            if (ws[wsp - 1].x & LEAF_FLAG) {
                const unsigned g = lane >> 3;
                uint2 e = make_uint2(0, 0);
                if (g < wsp) e = ws[wsp - 1 - g];
                const bool leaf = (e.x & LEAF_FLAG) != 0, large = (e.x >> LEAF_COUNT_SHIFT & LEAF_COUNT_MASK) > 8;
                const unsigned lm = __ballot_sync(0xffffffffu, leaf);
                // leading leaves; one at a time where a block takes more than one pass of eight lanes
                const bool several = __any_sync(0xffffffffu, leaf && large);
                const unsigned lead = several ? 1u : lm == 0xffffffffu ? 4u : ((unsigned)__ffs(~lm) - 1) / 8;
                wsp -= lead;
                float lf = __uint_as_float(e.y);
                if (several) {
                    // a leaf is entered once: not compared again with the rayLength that its own earlier
                    // passes left, which rounding can put before its box
                    if (!(__shfl_sync(0xffffffffu, lf, 0) <= wlen)) continue;
                    lf = 0.0f;
                }
                if (test_leaves(e.x, lf, lead)) break;
                continue;
            }
            if (wbudget == 0) {
                raise_error(err, DEVERR_TRAVERSAL_CAP);
                break;
            }
            // several entries only while the stack keeps room for the depth first bound above them
            const uint32_t m = wsp <= 32 ? min(wsp, 8u) : 1u;
            const uint32_t k = lane >> 2;
            uint2 e = make_uint2(kNone, 0u);
            if (k < m) e = ws[wsp - 1 - k];
            bool hit = k < m && (ANY_HIT || __uint_as_float(e.y) <= wlen), restart = false;
            float f = __uint_as_float(e.y);
            uint32_t r = e.x;
            if (e.x & LEAF_FLAG) {
                hit = hit && (lane & 3u) == 0;  // a waiting leaf stays
            } else if (hit) {
                if (kChecked && e.x >= s.numWide) {
                    raise_error(err, DEVERR_BOUNDS);
                    hit = false;
                } else {
                    const float* nd = reinterpret_cast<const float*>(wwide + 128 * (size_t)e.x) + (lane & 3u);
                    const float4 lo = make_float4(__ldg(nd), __ldg(nd + 8), __ldg(nd + 16), 0.0f);
                    const float4 hi = make_float4(__ldg(nd + 4), __ldg(nd + 12), __ldg(nd + 20), 0.0f);
                    r = __float_as_uint(__ldg(nd + 24));
                    hit = intersect_box<TRI != 0>(o, wi, lo, hi, f) && f <= wlen && r != kWideEmpty;
                    if (TRI == 0 && waxis)
                        restart = hit && ((isinf(wi.x) && lo.x == o.x && hi.x == o.x) ||
                                          (isinf(wi.y) && lo.y == o.y && hi.y == o.y) ||
                                          (isinf(wi.z) && lo.z == o.z && hi.z == o.z));
                }
            }
            if (TRI == 0 && waxis && __any_sync(0xffffffffu, restart)) {
                float3 x, y;
                load(witem, x, y, wlen);
                wslot = -1;
                wu = wv = 0.0f;
                wseq = true;
                wref = wsp = 0;
                wbudget = s.numNodes;
                continue;
            }
            --wbudget;  // every round expands a node
            const unsigned hits = __ballot_sync(0xffffffffu, hit);
            __syncwarp();
            if (hit) ws[wsp - m + __popc(hits >> lane) - 1] = make_uint2(r, __float_as_uint(f));
            wsp += (uint32_t)__popc(hits) - m;
            __syncwarp();
        }
        if (lane == 0) finish(witem, wslot, wlen, wu, wv);
        __syncwarp();
        if (lane == src) active = false;
        if (solo) {
            if (!work) {
                next += warps;
                continue;
            }
            if (lane == 0) next = warps + atomicAdd(work, 1ull);
            next = __shfl_sync(0xffffffffu, next, 0);
        }
    }
}

// ----------------------------------------------------------------- lane walk
// The escape walk of the binary tree, one lane per ray, for trees that have no
// wide hierarchy (ellipsoids and oriented boxes: their bounds do not nest, so
// every ancestor has to be tested) and queues that are long enough: lanes
// step through nodes together, leaves are tested by eight lanes each as in
// wide_walks, and the last rays of a warp continue as 8-lane groups
// (group_step), whose windows shorten the long single walks that a queue
// ends with. Same items, load and finish as wide_walks.
//
// Bound by issue slots (an ellipsoid test is ~70 instructions with a
// reciprocal and a square root): 8-lane groups issued ~2,700 instructions per
// ray for windows of which a third is visited. Measured on fitted ellipsoids,
// 100k instanced triangles, rays from inside (us, 8-lane groups / this):
// 20,000 rays 143 / 158, 40,000 181 / 199, 60,000 209 / 216, 100,000 281 / 240,
// 500,000 935 / 458, 2,000,000 3,451 / 1,349; a room of 40k triangles 50,000
// rays 638 / 641, 70,000 737 / 712; an icosphere of 20k 168 / 171, 212 / 184. So
// queues of fewer rays than 48 per block of the full grid (58,000 on 152 SMs)
// stay with the groups.
// Nodes per loop 1 / 2 / 4 / 8: 496 / 489 / 458 / 473 us at 500,000; waiting
// leaves 2 / 4 / 8: 462 / 458 / 476; handed over at 2 / 3 / 4 rays: 509 / 471
// / 458.
// The node loop unrolled by 1 / 2, with the barrier before a refill: 480 / 468
// (2,000,000 rays 1,376 / 1,340; oriented boxes 344 / 336 and 948 / 926).
#ifndef GPUGI_LANE_FROM
#define GPUGI_LANE_FROM 48u
#endif
constexpr int kLaneSteps = 4, kLaneLeaves = 4, kLaneNodes = 8, kLaneRefill = 8, kLaneGroupAt = 4;
struct LaneShared {
    float4 ray[2][128];
};

template <bool ANY_HIT, int BOUNDS, int TRI, typename Load, typename Finish>
GPUGI_D void lane_walks(LaneShared& sh, const DevScene& s, uint64_t n, unsigned long long* work, uint32_t* err,
                        Load load, Finish finish) {
    constexpr uint32_t kNone = 0xFFFFFFFFu;
    const unsigned lane = threadIdx.x & 31u;
    const DevScene* const own = &s;
    bool active = false;
    uint32_t item = 0;
    float3 o = {}, d = {}, inv = {};
    float len = 0.0f, u = 0.0f, v = 0.0f;
    int32_t slot = -1;
    uint32_t ref = kNone, resume = kNone, budget = 0;  // ref: node or leaf word to take next; resume: after a leaf
    auto begin = [&](uint32_t i) {
        item = i;
        load(item, o, d, len);
        slot = -1;
        u = v = 0.0f;
        inv = make_float3(X::rcp(d.x), X::rcp(d.y), X::rcp(d.z));
        sh.ray[0][threadIdx.x] = make_float4(o.x, o.y, o.z, d.x);
        sh.ray[1][threadIdx.x] = make_float4(d.y, d.z, 0.0f, 0.0f);
        ref = 0;
        budget = s.numNodes;
        active = true;
    };
    auto step = [&]() {  // one node
        const bool capped = budget-- == 0, outside = kChecked && ref >= s.numNodes;
        if (capped || outside) {
            raise_error(err, capped ? DEVERR_TRAVERSAL_CAP : DEVERR_BOUNDS);
            ref = kNone;
            return;
        }
        const float4* nd = s.nodes + node_stride<BOUNDS>() * (size_t)ref;
        const float4 a = __ldg(nd), b = __ldg(nd + 1);
        const float4 c = BOUNDS == 2 ? __ldg(nd + 2) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        float f;
        const bool hit = bounds_test<BOUNDS, TRI != 0>(o, d, inv, a, b, c, f) && f <= len;
        const uint32_t child = __float_as_uint(a.w), esc = __float_as_uint(b.w), next = esc ? esc : kNone;
        if (hit && (child & LEAF_FLAG)) resume = next;
        ref = hit ? child : next;
    };
    const unsigned warps = gridDim.x * (blockDim.x >> 5);
    const unsigned C = n >= 32 * (uint64_t)warps ? 32u : ((uint32_t)n + warps - 1) / warps;
    const uint64_t first = (uint64_t)warps * C;
    bool more = n > first;
    {
        const uint64_t i = ((uint64_t)(threadIdx.x >> 5) * gridDim.x + blockIdx.x) * C + lane;
        if (lane < C && i < n) begin((uint32_t)i);
    }
    while (true) {
        const unsigned act = __ballot_sync(0xffffffffu, active);
        if (more && __popc(act) <= 32 - kLaneRefill) {
            unsigned long long base = 0;
            if (lane == 0) base = atomicAdd(work, (unsigned long long)__popc(~act));
            base = first + __shfl_sync(0xffffffffu, base, 0);
            more = base + __popc(~act) < n;
            base += (unsigned)__popc(~act & ((1u << lane) - 1u));
            __syncwarp();  // the leaf rounds' reads of the rays that are replaced
            if (!active && base < n) begin((uint32_t)base);
        } else if (!more && __popc(act) <= kLaneGroupAt) {
            break;
        }
        // nodes
        while (true) {
            if (active && !(ref & LEAF_FLAG)) {
#pragma unroll 2
                for (int k = 0; k < kLaneSteps && !(ref & LEAF_FLAG); ++k) step();
                if (ref == kNone) {
                    finish(item, slot, len, u, v);
                    active = false;
                }
            }
            const unsigned nodes = __ballot_sync(0xffffffffu, active && !(ref & LEAF_FLAG));
            const unsigned leaves = __ballot_sync(0xffffffffu, active && (ref & LEAF_FLAG));
            if (__popc(leaves) >= kLaneLeaves || __popc(nodes) < kLaneNodes || !nodes) break;
        }
        const unsigned todo = __ballot_sync(0xffffffffu, active && (ref & LEAF_FLAG));
        __syncwarp();
        leaf_rounds<ANY_HIT, TRI>(todo, sh.ray, ref, [&](unsigned) { return own; }, own, err, len, u, v, slot, [&]() {
            ref = ANY_HIT && slot >= 0 ? kNone : resume;
            if (ref == kNone) {
                finish(item, slot, len, u, v);
                active = false;
            }
        });
    }
    // the last rays: eight lanes each
    constexpr unsigned G = 8;
    const unsigned gl = lane & (G - 1), gbase = lane & ~(G - 1), gmask = 0xffu << gbase;
    unsigned act = __ballot_sync(0xffffffffu, active);
    for (unsigned g = 0; g < lane / G; ++g) act &= act - 1;
    const unsigned src = act ? (unsigned)(__ffs(act) - 1) : 0u;
    auto get = [&](float x) { return __shfl_sync(0xffffffffu, x, src); };
    GroupWalk g;
    g.o = make_float3(get(o.x), get(o.y), get(o.z));
    g.d = make_float3(get(d.x), get(d.y), get(d.z));
    g.inv = make_float3(get(inv.x), get(inv.y), get(inv.z));
    g.wt = wt_setup(g.d);  // dead code unless a watertight walker reads it
    g.len = get(len);
    g.u = get(u);
    g.v = get(v);
    g.slot = __shfl_sync(0xffffffffu, slot, src);
    g.budget = __shfl_sync(0xffffffffu, budget, src);
    item = __shfl_sync(0xffffffffu, item, src);
    ref = __shfl_sync(0xffffffffu, ref, src);
    resume = __shfl_sync(0xffffffffu, resume, src);
    if (!act) return;
    g.node = ref;
    g.cur = g.end = 0;
    g.resume = resume;
    bool done = false;
    if (ref & LEAF_FLAG) {
        g.cur = (ref & LEAF_BLOCK_MASK) * s.leafSize;
        g.end = g.cur + leaf_slots(s, ref, err);
        if (g.cur >= g.end) {
            g.node = resume;
            done = resume == kNone;
        }
    }
    while (!done) done = group_step<ANY_HIT, BOUNDS, (int)G, TRI>(g, s, err, gl, gbase, gmask);
    if (gl == 0) finish(item, g.slot, g.len, g.u, g.v);
}

}  // namespace gpugi
