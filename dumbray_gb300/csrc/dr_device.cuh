// dr_device.cuh - device-side scene layout and the exact octree cast for sm_103a.
//
// Layout in HBM (all read-only after upload):
//   nodes      float4[2 * node_count]  node i = {lo.xyz, w = first child (inner) or ~first ref (leaf)},
//                                               {hi.xyz, w = leaf ref count}
//              children of an inner node are 8 consecutive nodes, 8-aligned (one 256-byte group).
//   groups     float4[16 * groups]     one 256-byte record per inner node: what a cast reads to test the
//              8 children and to find the taken one (GroupRecord below)
//   leaf_tris  float4[4 * refs]        leaf reference r: the triangle's vertices and what of its test does
//              not depend on the ray (kLeafTriF4 below), duplicated in leaf order, so a leaf is one
//              contiguous stream in each of the two halves (leaf_half references apart).
//   tris       float4[3 * n]           triangles by id (shading, light sampling)
// The cast reproduces DumbRay's Octree::cast (Octree.impl.cuh:174-212) bit for bit: every
// floating-point operation of the slab test, the triangle plane test and the edge-angle
// containment predicate is issued as an explicitly rounded intrinsic (__fadd_rn, __fmul_rn,
// __fdiv_rn, __fsqrt_rn), so no FMA contraction or approximate division can change a result.
#pragma once
#include <cfloat>
#include <cstdint>
#include <cuda_runtime.h>

namespace drd {

constexpr float kEps = 0.000005f;               // VECTOR_EPSILON (Vector3.h:10)
constexpr int kMaxDepth = 24;                    // OCTREE_MAX_DEPTH (Octree.cuh:13)
constexpr int kStack = kMaxDepth + 2;

struct Material {
    int type;
    float color[3];
    float fresnel[3];
    float specular, metal, diffuse, smoothness, shininess, roughness;
    float emission[3];
    int texture[4];              // 0-based texture per channel (colour, fresnel, normal, alpha), -1 = none
    float tiling[4][2], offset[4][2];
    float normal_color[3];
    float alpha_threshold;
};

struct Light {
    int type;
    float color[3];      // spotlight: colour x luminosity
    float position[3];
    float direction[3];  // spotlight: normalised
    float radius, distance, softness;
    // spotlight (Lights::Spotlight constructor state): emitter size, cosines of the hotspot and
    // falloff half-angles, falloff power, photons per shading point, occlusion test, sphere emitter
    float emitter, inner_cos, outer_cos, falloff;
    int samples, shadows, sphere;
};

struct Scene {
    const float4 *nodes;
    // Child boxes per node group as planes of 8 floats (lo.x, lo.y, lo.z, hi.x, hi.y, hi.z; 12 float4
    // = 192 B per group), read by the group tests of the counting traversals.  gbox: refitted to the
    // non-empty leaves below each child (physical-padding scenes); gbox_ref: the reference's boxes
    // (reference-padding scenes).  Empty leaves sit at a far point in both (dr_octree_group_planes in
    // the C ABI gives both for a host-built tree).
    const float4 *gbox;
    const float4 *gbox_ref;
    const float4 *groups;       // group records (16 float4 each), read by every other traversal
    const float4 *leaf_tris;
    int64_t leaf_half;          // references in leaf_tris: where their second halves begin
    const float4 *tris;
    const float4 *nrms;
    const int *mat_id;
    const Material *mats;
    const Light *lights;
    const float4 *shade;        // physical: [n] {roughness, type bits, -, -}
    const float *albedo;        // physical: [n][3] (writable in place by an optimiser)
    const float *emission;      // physical: [n][3] (writable in place; sampling tables are not rebuilt)
    const float *light_pdf;     // physical: [n] area pdf of picking a point of this triangle by NEE
    const int *emissive;        // emissive triangle ids
    const float *emissive_cdf;  // inclusive prefix sums of power (at table build time)
    const float4 *texels;       // all textures' RGBA texels, row-major per texture
    const int4 *tex_info;       // per texture: {first texel, width, height, filtering}
    const float2 *uv;           // [n][3] corner texture coordinates (null: none set)
    float root_lo[3], root_hi[3];
    float reach;                // largest absolute coordinate of the root box
    int root_child;             // node group of the root's 8 children (0 for a standalone scene, the
                                // scene's offset in a batch arena), -1 = the root is a leaf
    int root_leaf_first, root_leaf_count;
    int n_tris, n_mats, n_lights, n_emissive;
    int shadow_photons;  // shadow records one reference-mode hit can emit (1 per light, a spotlight's samples)
    // Boxes lying entirely behind the ray origin: the reference's slab test keeps them
    // (clipBackface = false), which only costs work, since a hit at t > 0 accepted inside a leaf box
    // means that box reaches t > 0.  Every non-counting traversal skips them; the counting ones
    // (which reproduce the reference's box-test counts) skip them only when front_only = 1, i.e. for
    // scenes built with a padding scaled to the scene, whose counts are not the reference's anyway.
    int front_only;
    float emissive_total;
};

// ---- exactly rounded float3 arithmetic (reference operation order) -------------------------
struct f3 {
    float x, y, z;
};
__device__ __forceinline__ f3 mkf3(float x, float y, float z) { return f3{x, y, z}; }
__device__ __forceinline__ f3 xsub(f3 a, f3 b) { return f3{__fsub_rn(a.x, b.x), __fsub_rn(a.y, b.y), __fsub_rn(a.z, b.z)}; }
__device__ __forceinline__ f3 xadd(f3 a, f3 b) { return f3{__fadd_rn(a.x, b.x), __fadd_rn(a.y, b.y), __fadd_rn(a.z, b.z)}; }
__device__ __forceinline__ f3 xmul(f3 a, float f) { return f3{__fmul_rn(a.x, f), __fmul_rn(a.y, f), __fmul_rn(a.z, f)}; }
// Vector3 dot: (x*v.x + y*v.y) + z*v.z
__device__ __forceinline__ float xdot(f3 a, f3 b) {
    return __fadd_rn(__fadd_rn(__fmul_rn(a.x, b.x), __fmul_rn(a.y, b.y)), __fmul_rn(a.z, b.z));
}
// Vector3 cross a & v: (y*v.z - v.y*z, v.x*z - x*v.z, x*v.y - v.x*y)
__device__ __forceinline__ f3 xcross(f3 a, f3 v) {
    return f3{__fsub_rn(__fmul_rn(a.y, v.z), __fmul_rn(v.y, a.z)), __fsub_rn(__fmul_rn(v.x, a.z), __fmul_rn(a.x, v.z)),
              __fsub_rn(__fmul_rn(a.x, v.y), __fmul_rn(v.x, a.y))};
}
__device__ __forceinline__ float xmag(f3 a) { return __fsqrt_rn(xdot(a, a)); }
__device__ __forceinline__ bool xeq(f3 a, f3 b) { return a.x == b.x && a.y == b.y && a.z == b.z; }
__device__ __forceinline__ f3 f3of(float4 v) { return f3{v.x, v.y, v.z}; }

// AABB::castPreInversed + Shapes::castPreInversed<AABB>(.., clipBackface = false)
// (AABB.impl.h:116-130, Shapes.impl.cuh:143-147)
__device__ __forceinline__ bool slab_hit(float lx, float ly, float lz, float hx, float hy, float hz, f3 o, f3 inv,
                                         bool front = false) {
    float ds = __fmul_rn(__fsub_rn(lx, o.x), inv.x);
    float de = __fmul_rn(__fsub_rn(hx, o.x), inv.x);
    float mn = fminf(ds, de), mx = fmaxf(ds, de);
    ds = __fmul_rn(__fsub_rn(ly, o.y), inv.y);
    de = __fmul_rn(__fsub_rn(hy, o.y), inv.y);
    mn = fmaxf(mn, fminf(ds, de));
    mx = fminf(mx, fmaxf(ds, de));
    ds = __fmul_rn(__fsub_rn(lz, o.z), inv.z);
    de = __fmul_rn(__fsub_rn(hz, o.z), inv.z);
    mn = fmaxf(mn, fminf(ds, de));
    mx = fminf(mx, fmaxf(ds, de));
    if (mn > __fadd_rn(mx, kEps)) return false;
    if (front && mx < -kEps) return false;  // entirely behind the origin (front_only scenes)
    return mn != FLT_MAX;
}

// The slab test of a box as the reference makes it, boxes behind the origin dropped; out of line.
static __device__ __noinline__ bool exact_slab(f3 l, f3 h, f3 o, f3 d) {
    const f3 inv = mkf3(__fdiv_rn(1.0f, d.x), __fdiv_rn(1.0f, d.y), __fdiv_rn(1.0f, d.z));
    return slab_hit(l.x, l.y, l.z, h.x, h.y, h.z, o, inv, true);
}
// Bounds what rounding does to a hit point in a box of the scene (d t, then the sum: u (|o| + 2 reach),
// u = 2^-24), to the plane distances of that box (three roundings: 3 u (|o| + reach) in space) and to the
// comparison with the face (u reach): u (4 |o| + 6 reach) in all, more than twice over.
__device__ __forceinline__ float point_margin(f3 o, float reach) { return 9.5367431640625e-7f * (fabsf(o.x) + fabsf(o.y) + fabsf(o.z) + reach); }   // 2^-20

// Two floats in one register pair, and operations on both (one issue slot on sm_100 and later), each
// rounded as its scalar counterpart.
using f32x2 = unsigned long long;
__device__ __forceinline__ f32x2 pack2(float lo, float hi) {
    f32x2 v;
    asm("mov.b64 %0, {%1, %2};" : "=l"(v) : "f"(lo), "f"(hi));
    return v;
}
__device__ __forceinline__ void unpack2(f32x2 v, float &lo, float &hi) { asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v)); }
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c) {
    f32x2 d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}
__device__ __forceinline__ f32x2 mul2(f32x2 a, f32x2 b) {
    f32x2 d;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ f32x2 add2(f32x2 a, f32x2 b) {
    f32x2 d;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
// xdot of two pairs of vectors
__device__ __forceinline__ f32x2 xdot2(const f32x2 (&a)[3], const f32x2 (&b)[3]) {
    return add2(add2(mul2(a[0], b[0]), mul2(a[1], b[1])), mul2(a[2], b[2]));
}

// One edge condition of Triangle::containsVertex (Triangle.impl.h:292-302), every operation exactly
// rounded: rn(rn(X / rn(sqrt(P))) + S) >= rn(Y / rn(sqrt(Q))), X = e.px, P = px.px, Y = -(e.f), Q = f.f.
// The right side depends on the triangle alone (edge_limit).
constexpr float kEdgeSlack = 32 * kEps;
__device__ __forceinline__ float edge_limit(f3 e, f3 f) { return __fdiv_rn(-xdot(e, f), __fsqrt_rn(xdot(f, f))); }
__device__ __forceinline__ bool edge_ok(f3 e, f3 px, float limit) {
    return __fadd_rn(__fdiv_rn(xdot(e, px), __fsqrt_rn(xdot(px, px))), kEdgeSlack) >= limit;
}

// Triangle::containsVertex (Triangle.impl.h:283-302); `limit` = edge_limit at a, b, c.  Out of line:
// reached by points on a vertex or within rounding of an edge angle only.
static __device__ __noinline__ bool contains_vertex(f3 a, f3 b, f3 c, f3 p, float limit_a, float limit_b, float limit_c) {
    if (xeq(a, b) || xeq(b, c) || xeq(c, a)) return false;
    if (xeq(p, a) || xeq(p, b) || xeq(p, c)) return true;
    return edge_ok(xsub(b, a), xsub(p, a), limit_a) && edge_ok(xsub(c, b), xsub(p, b), limit_b) &&
           edge_ok(xsub(a, c), xsub(p, c), limit_c);
}

// An edge condition with rsqrtf (documented max error 2 ulp), X = e.px, P = px.px: the fast left side
// L = X rsqrt(P) + S differs from the exactly rounded one by at most ~3 ulp of |L| + S.  A difference
// D = L - limit beyond M = 2^-18 (|limit| + S), which is at least 2^-19 (|L| + |limit| + S) or about 16
// ulp there, has the sign of the exact difference.  `in` stays true while every edge is certainly inside,
// `out` becomes true at one that is certainly outside; neither for NaN and infinities, which leaves the
// decision to contains_vertex.
__device__ __forceinline__ void edge_fast(float X, float P, float limit, bool &in, bool &out) {
    const float D = __fmaf_rn(X, rsqrtf(P), kEdgeSlack) - limit;
    const float M = __fmaf_rn(fabsf(limit), 3.9e-6f, 3.9e-6f * kEdgeSlack);
    in = in && D > M;
    out = out || D < -M;
}

// Leaf reference: 64 bytes in two arrays of 32, floats a.x b.x a.y b.y a.z b.z c.x c.y | c.z, the plane
// normal (b - a) x (c - a), the right sides of the three edge conditions, the triangle id.  The normal
// and the right sides are what a test would otherwise compute again for every ray, with the same
// rounding; corners a and b lie side by side for the paired arithmetic.  Neighbouring tests of a window
// read neighbouring references, so each of the two loads is one stretch of 32-byte pieces: whole 64-byte
// references left every second piece of its lines to the other load (L1 wavefronts, 80% of their peak in
// closed rooms).  Same call: gradients 57.6 -> 55.5 ms, room 7.67 -> 7.43, incoherent casts 2.75 -> 2.68,
// batch 10.95 -> 10.74; coherent primary casts, whose tests share references, 1.15 -> 1.17.
constexpr int kLeafTriF4 = 4;
__device__ __forceinline__ int leaf_tri_id(const float4 *leaf_tris, size_t half, int pos) {
    return __float_as_int(__ldg(leaf_tris + 2 * (half + (size_t)pos) + 1).w);
}
__device__ __forceinline__ void ldg8(const void *p, f32x2 *v) {
    asm("ld.global.nc.v4.b64 {%0,%1,%2,%3}, [%4];" : "=l"(v[0]), "=l"(v[1]), "=l"(v[2]), "=l"(v[3]) : "l"(p));
}

// Triangle::cast (Triangle.impl.h:334-348) of leaf reference `pos`, with the caller's validator check
// (castInLeaf, Octree.impl.cuh:596-603) moved ahead of the containment test: the ignored triangle
// cannot change the leaf's result.  The three edges are tested together: among the 32 tests of a
// window some lane nearly always needs the last one.  Differences are taken corner - p: the signs of
// both factors of P and of X cancel or are undone exactly.
__device__ __forceinline__ bool tri_cast(const float4 *leaf_tris, size_t half, int pos, f3 o, f3 d, bool clip, int ignore, float &dist) {
    f32x2 u[4], w[4];
    ldg8(leaf_tris + 2 * (size_t)pos, u);
    ldg8(leaf_tris + 2 * (half + (size_t)pos), w);
    f3 a, b, c, n;
    float limit_a, limit_b, limit_c, id;
    unpack2(u[0], a.x, b.x);
    unpack2(u[1], a.y, b.y);
    unpack2(u[2], a.z, b.z);
    unpack2(u[3], c.x, c.y);
    unpack2(w[0], c.z, n.x);
    unpack2(w[1], n.y, n.z);
    unpack2(w[2], limit_a, limit_b);
    unpack2(w[3], limit_c, id);
    const float dp = xdot(xsub(a, o), n);
    const float dirp = xdot(d, n);
    if ((clip && dp < -kEps) || __fmul_rn(dp, dirp) <= 0.0f) return false;
    dist = __fdiv_rn(dp, dirp);
    if (!(dist < FLT_MAX) || __float_as_int(id) == ignore) return false;
    const f3 p = xadd(o, xmul(d, dist));
    const f32x2 q[3] = {add2(u[0], pack2(-p.x, -p.x)), add2(u[1], pack2(-p.y, -p.y)), add2(u[2], pack2(-p.z, -p.z))};
    const f3 qc = xsub(c, p), ab = xsub(b, a), bc = xsub(c, b), ca = xsub(a, c);
    const f32x2 e[3] = {pack2(ab.x, bc.x), pack2(ab.y, bc.y), pack2(ab.z, bc.z)};
    float Xa, Xb, Pa, Pb;
    unpack2(xdot2(e, q), Xa, Xb);
    unpack2(xdot2(q, q), Pa, Pb);
    const float Xc = xdot(ca, qc), Pc = xdot(qc, qc);
    const bool vertex = !(fminf(fminf(Pa, Pb), Pc) > 0.0f);   // on a vertex: the exact test decides
    bool in = !vertex, out = false;
    edge_fast(-Xa, Pa, limit_a, in, out);
    edge_fast(-Xb, Pb, limit_b, in, out);
    edge_fast(-Xc, Pc, limit_c, in, out);
    if (in) return true;
    if (out && !vertex) return false;
    return contains_vertex(a, b, c, p, limit_a, limit_b, limit_c);
}

struct Hit {
    int tri;     // -1 = miss
    float t;     // in units of |d|
    f3 p;        // hit point o + d * t (exactly as the reference computes it)
};

// Tests the 8 children of a group; bit k of the result = child (order ^ k) is hit.  The slab tests
// of the 8 children run plane by plane on the plane layout (x entry/exit of all children, then y,
// then z), which keeps 16 running values instead of 48 coordinates live; each child's operations are
// those of slab_hit in the same order.  Bit c of the octant-order mask then moves to c ^ order, so
// results and counts equal a test in visit order.
// Two consecutive float4 (32 bytes, 32-byte aligned) in one 256-bit read-only load (sm_100 and
// later): a node record.  Half the load instructions of two 128-bit loads, for the same bytes.
__device__ __forceinline__ void ldg2(const float4 *p, float4 &a, float4 &b) {
    asm("ld.global.nc.v8.f32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
        : "=f"(a.x), "=f"(a.y), "=f"(a.z), "=f"(a.w), "=f"(b.x), "=f"(b.y), "=f"(b.z), "=f"(b.w)
        : "l"(p));
}

__device__ __forceinline__ void slab_planes(const float4 *g, int plane, float oc, float ic, float *mn, float *mx, bool first) {
    const float4 l0 = __ldg(g + 2 * plane), l1 = __ldg(g + 2 * plane + 1);
    const float4 h0 = __ldg(g + 6 + 2 * plane), h1 = __ldg(g + 6 + 2 * plane + 1);
    const float lo[8] = {l0.x, l0.y, l0.z, l0.w, l1.x, l1.y, l1.z, l1.w};
    const float hi[8] = {h0.x, h0.y, h0.z, h0.w, h1.x, h1.y, h1.z, h1.w};
#pragma unroll
    for (int c = 0; c < 8; c++) {
        const float ds = __fmul_rn(__fsub_rn(lo[c], oc), ic);
        const float de = __fmul_rn(__fsub_rn(hi[c], oc), ic);
        if (first) {
            mn[c] = fminf(ds, de);
            mx[c] = fmaxf(ds, de);
        } else {
            mn[c] = fmaxf(mn[c], fminf(ds, de));
            mx[c] = fminf(mx[c], fmaxf(ds, de));
        }
    }
}

__device__ __forceinline__ unsigned test_group(const float4 *gbox, int group, int order, f3 o, f3 inv, bool front) {
    const float4 *g = gbox + 12 * (size_t)group;
    float mn[8], mx[8];
    slab_planes(g, 0, o.x, inv.x, mn, mx, true);
    slab_planes(g, 1, o.y, inv.y, mn, mx, false);
    slab_planes(g, 2, o.z, inv.z, mn, mx, false);
    unsigned m = 0;
#pragma unroll
    for (int c = 0; c < 8; c++) {
        const bool hit = !(mn[c] > __fadd_rn(mx[c], kEps)) && !(front && mx[c] < -kEps) && mn[c] != FLT_MAX;
        m |= (hit ? 1u : 0u) << c;
    }
    if (order & 1) m = ((m & 0x55u) << 1) | ((m >> 1) & 0x55u);
    if (order & 2) m = ((m & 0x33u) << 2) | ((m >> 2) & 0x33u);
    if (order & 4) m = ((m & 0x0Fu) << 4) | ((m >> 4) & 0x0Fu);
    return m;
}

// Traversal stack entry of a counting traversal: group << 11 | child position taken << 8 | remaining
// hit mask.  The position corrects the box-test count when a hit ends the scan of a group early; it
// leaves 21 bits of group index (2^24 nodes).
constexpr int kCountShift = 11;

// ---- group records ---------------------------------------------------------------------------
// Record of a group (256 bytes, two cache lines):
//   floats 0-47   child box planes, axis by axis: lo.x[8], hi.x[8], lo.y[8], hi.y[8], lo.z[8], hi.z[8]
//                 (the refitted boxes of gbox, widened by kRecordPad x reach on every side)
//   word   48     index of the first inner child's group << 8 | mask of the inner children
//   words  49-57  where the leaf children's references begin: child c's are [49 + c] .. [50 + c)
// Both builders number nodes breadth first, so the groups of a node's inner children are consecutive
// and so are the references of its leaf children: word 48 finds any child's group without reading
// the child's node.  A step down the tree then waits for one dependent load (the child's record)
// instead of two (node, then planes).
//
// The record's test (record_mask) only has to keep every child that the exact slab test would keep:
// a leaf whose triangles are hit has its own box tested exactly before the hit counts (leaf_accepts),
// and the exact test is monotone in the box, so a leaf that passes it passes at all its ancestors.
// That frees the group test from the reference's operation order: planes are taken near / far by the
// sign of the direction (no min / max of the pair), with one fused multiply-add each.
//   exact, per plane:  t = rn(rn(x - o) * inv), inv = rn(1 / d)
//   here:              t = rn(x' * inv - off), off = rn(o * inv) -+ slack
// Rounding separates the two by at most 7 u |x| |inv| + 8 u |o| |inv| (u = 2^-24).  Of each, 3 are the exact
// test's difference, product and reciprocal, 2 the approximate reciprocal here and 1 the fused operation; the
// last of |x| is the widened plane's rounding, the last two of |o| those of o * inv and of the offset.  The
// planes are widened by 2^-19 x reach >= 32 u |x| and the offsets by 2^-20 |o inv| = 16 u |o| |inv|, four times
// and twice that; the far offset also takes 2 kEps for the exact test's kEps on either end.
// What bounds it is instruction issue (55-69% of the issue slots at 15-17 of 32 lanes) and the wait for
// the record; against the exact test on nodes and planes, in one call: 8.4M incoherent casts on the
// 1.31M-triangle mesh 5.02 -> 4.34 ms, the 1080p 16 spp path trace 48.9 -> 44.2 ms, the room of 20k
// triangles 14.4 -> 13.2 ms, 512^2 gradients 98.2 -> 87.5 ms; two children an instruction then 1-3% on
// every case.
constexpr int kRecordF4 = 16;
constexpr float kRecordPad = 1.0f / 524288.0f;
constexpr float kRaySlack = 1.0f / 1048576.0f;

// What record_mask needs of a ray: 1 / d and the negated offsets of the near and far planes, each twice
// in a pair.
struct RaySlopes {
    f32x2 inv[3], near[3], far[3];
};
// The direction is scaled to a largest component in [1, 2) (a power of two: exact), so only origins
// beyond 1e24 could take a product out of the float range; such an axis is not tested (near = -max,
// far = +max).  A component below 2^-40 of the largest is raised to that, so that 0 * inf does not arise.
// That shears the ray along the component's axis: at parameter t by up to 2^-40 |t|, which in units of the
// axis' plane distances is |t| itself, far more than the widening when the origin is far away along another
// axis.  In any box of the scene |t| is at most reach + |o.x| + |o.y| + |o.z| (the scaled direction's largest
// component is 1 or more; 2^-22 or more if it is denormal), so both offsets of such an axis take twice that
// and the exact test's kEps (`shear`).
__device__ __forceinline__ RaySlopes ray_slopes(f3 o, f3 d, float reach) {
    RaySlopes r;
    const float oc[3] = {o.x, o.y, o.z}, dc[3] = {d.x, d.y, d.z};
    const float dmax = fmaxf(fmaxf(fabsf(d.x), fabsf(d.y)), fabsf(d.z));
    const unsigned e2 = min(__float_as_uint(dmax) >> 23, 253u);
    const float up = __uint_as_float((254u - e2) << 23), eps2 = 2.0f * kEps * __uint_as_float(e2 << 23);   // t shrinks by `up`
    constexpr float kTiny = 9.094947017729282e-13f;   // 2^-40
    const float shear = eps2 + (fabsf(o.x) + fabsf(o.y) + fabsf(o.z) + reach) * (e2 == 0u ? 8388608.0f : 2.0f);   // sum as in point_margin
#pragma unroll
    for (int k = 0; k < 3; k++) {
        const float scaled = fabsf(dc[k]) * up, a = fmaxf(scaled, kTiny);
        float inv;
        asm("rcp.approx.f32 %0, %1;" : "=f"(inv) : "f"(dc[k] < 0.0f ? -a : a));   // within an ulp: part of the slack
        const float oi = oc[k] * inv, e = fabsf(oi) * kRaySlack + (scaled < kTiny ? shear : 0.0f);
        const bool ok = fabsf(inv) * (reach + fabsf(oc[k])) < 1e37f;
        const float i = ok ? inv : 0.0f, n = ok ? -oi - e : -FLT_MAX, f = ok ? eps2 + e - oi : FLT_MAX;
        r.inv[k] = pack2(i, i);
        r.near[k] = pack2(n, n);
        r.far[k] = pack2(f, f);
    }
    return r;
}
// A ray that no triangle test accepts, whatever the triangle: zero direction (the plane test's product
// is 0 or NaN), or a component that is not finite (the distance is NaN or infinite, or the hit point NaN).
__device__ __forceinline__ bool never_hits(f3 o, f3 d) {
    const float z = (o.x - o.x) + (o.y - o.y) + (o.z - o.z) + (d.x - d.x) + (d.y - d.y) + (d.z - d.z);
    return z != 0.0f || z != z || (d.x == 0.0f && d.y == 0.0f && d.z == 0.0f);
}

// Children of group `g` that the ray may enter, bit k = child (order ^ k), and the group's word 48.
// Per child: six fused multiply-adds (two children an instruction), the interval of the three axes, and
// its sign bit shifted into the mask.
__device__ __forceinline__ unsigned record_mask(const float4 *groups, uint32_t g, int order, const RaySlopes &r, uint32_t &links) {
    const char *p = reinterpret_cast<const char *>(groups + (size_t)g * kRecordF4);
    links = __ldg(reinterpret_cast<const uint32_t *>(p + 192));
    const int sx = (order & 4) << 3, sy = (order & 2) << 4, sz = (order & 1) << 5;   // byte offset of the near plane: 0 or 32
    f32x2 n[4], f[4];
    float mn[8], mx[8];
    ldg8(p + sx, n);
    ldg8(p + (sx ^ 32), f);
#pragma unroll
    for (int c = 0; c < 4; c++) {
        unpack2(fma2(n[c], r.inv[0], r.near[0]), mn[2 * c], mn[2 * c + 1]);
        unpack2(fma2(f[c], r.inv[0], r.far[0]), mx[2 * c], mx[2 * c + 1]);
    }
    ldg8(p + 64 + sy, n);
    ldg8(p + 64 + (sy ^ 32), f);
#pragma unroll
    for (int c = 0; c < 4; c++) {
        float a, b;
        unpack2(fma2(n[c], r.inv[1], r.near[1]), a, b);
        asm("max.f32 %0, %0, %1, 0f00000000;" : "+f"(mn[2 * c]) : "f"(a));   // and not behind the origin
        asm("max.f32 %0, %0, %1, 0f00000000;" : "+f"(mn[2 * c + 1]) : "f"(b));
        unpack2(fma2(f[c], r.inv[1], r.far[1]), a, b);
        mx[2 * c] = fminf(mx[2 * c], a);
        mx[2 * c + 1] = fminf(mx[2 * c + 1], b);
    }
    ldg8(p + 128 + sz, n);
    ldg8(p + 128 + (sz ^ 32), f);
    unsigned m = 0;
#pragma unroll
    for (int c = 3; c >= 0; c--) {
        float a, b, t0, t1;
        unpack2(fma2(n[c], r.inv[2], r.near[2]), a, b);
        t0 = fmaxf(mn[2 * c], a);
        t1 = fmaxf(mn[2 * c + 1], b);
        unpack2(fma2(f[c], r.inv[2], r.far[2]), a, b);
        m = __funnelshift_l(__float_as_uint(fminf(mx[2 * c + 1], b) - t1), m, 1);
        m = __funnelshift_l(__float_as_uint(fminf(mx[2 * c], a) - t0), m, 1);
    }
    m = ~m & 0xFFu;
    if (order & 1) m = ((m & 0x55u) << 1) | ((m >> 1) & 0x55u);
    if (order & 2) m = ((m & 0x33u) << 2) | ((m >> 2) & 0x33u);
    if (order & 4) m = ((m & 0x0Fu) << 4) | ((m >> 4) & 0x0Fu);
    return m;
}

// ---- counter-based random numbers ----------------------------------------------------------
// u32 = H(H(key + 0x9E3779B9 * (bounce * 128 + dim + 1))), key = H(H(H(seed ^ 0x2545F491) ^ pixel) + sample),
// H = lowbias32 (C. Wellons' public-domain integer hash).  Float = (u >> 8) * 2^-24 in [0, 1).
__host__ __device__ __forceinline__ uint32_t hash32(uint32_t x) {
    x ^= x >> 16;
    x *= 0x7feb352dU;
    x ^= x >> 15;
    x *= 0x846ca68bU;
    x ^= x >> 16;
    return x;
}
__host__ __device__ __forceinline__ uint32_t path_key(uint32_t seed, uint32_t pixel, uint32_t sample) {
    return hash32(hash32(hash32(seed ^ 0x2545F491U) ^ pixel) + sample);
}
__device__ __forceinline__ float rnd(uint32_t key, uint32_t bounce, uint32_t dim) {
    uint32_t u = hash32(hash32(key + 0x9E3779B9U * (bounce * 128U + dim + 1U)));
    return (float)(u >> 8) * (1.0f / 16777216.0f);
}
constexpr uint32_t kLensBounce = 1023;

}  // namespace drd
