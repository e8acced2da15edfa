// dr_trace.cuh - persistent, warp-refilled octree traversal for ray batches.
//
// Each lane traces one ray at a time with exactly the visit order and leaf semantics of
// Octree::cast (Octree.impl.cuh:174-212, castInLeaf :584-612), so results are identical to a
// one-ray-at-a-time cast.  What changes is the scheduling across the 32 lanes of a warp:
//   * one unit of work per lane per loop iteration: a few traversal steps (at most one 8-child group
//     test each, or entering a leaf), then one leaf round.  A lane never waits for another lane's
//     whole descent; per-ray costs range over three orders of magnitude on displaced meshes (p99
//     ~1,700 triangle tests against a mean of ~120);
//   * leaf work is shared by the whole warp: the pending (ray, triangle) tests of all lanes that hold
//     a leaf are numbered by ballots and handed out 32 at a time, one per lane, until none is left;
//     the tester reads the owner's ray from the warp's shared slots and posts (distance, list
//     position, hit_key) to the owner's key with a 64-bit atomicMin, so the owner keeps the smallest distance
//     and, among equal distances, the earliest triangle in list order - exactly castInLeaf's
//     strict-min scan;
//   * a lane whose ray is finished takes the next ray of the warp's current chunk at once.  Chunks
//     are handed out by the caller's Source (an atomic counter for queues whose size is only known
//     on the device, a fixed range for plain batches).
// A ray's origin, direction and ignored triangle live in shared memory only: the testers need them
// from another lane and its own lane rarely does, so they cost no registers during the descent.
//
// The kernels are bound by instruction issue and by each iteration's latency, so a round is kept short:
// independent ballots number the tests instead of a chain of five shuffles, a set bit per owner and one
// shared read find a test's owner instead of a five-step search, a window of 32 is skipped when empty.
// Against 64 tests a round with prefix sum, search, ten shuffles and the triangle's constants computed
// per test (same call): 1080p primary casts on the reference tree 2.57 -> 1.59 ms, room 13.2 -> 9.5 ms,
// 1080p photon render 63.5 -> 44.2 ms, path trace 44.2 -> 38.5 ms, gradients 87.5 -> 74.8 ms.
#pragma once
#include "dr_device.cuh"

namespace drd {

constexpr int kChunk = 256;

enum : int { kIdle = 0, kTrav = 1, kLeaf = 2, kDone = 3 };

// A warp's shared slots, one per lane.
struct WarpSlots {
    float4 o[32];                    // origin, ignored triangle
    float4 d[32];                    // direction, rounding margin of hit points (point_margin)
    unsigned long long key[32];      // nearest hit of the current leaf (hit_key)
    int2 task[32];                   // round's k-th owner: its lane, its first reference - its first task
};
constexpr unsigned long long kNoHit = ~0ull;

// A hit as a key whose order is castInLeaf's: the distance (no hit has a negative one), then the list position.
// Distances are compared as floats there, so -0, which a direction whose product with the normal overflows
// gives, equals 0: the sign stands below the position.
__device__ __forceinline__ unsigned long long hit_key(float dist, int pos) {
    const unsigned b = __float_as_uint(dist);
    return (unsigned long long)(b & 0x7FFFFFFFu) << 32 | __funnelshift_l(b, (unsigned)pos, 1);
}
__device__ __forceinline__ int key_pos(unsigned long long key) { return (int)((unsigned)key >> 1); }
__device__ __forceinline__ float key_dist(unsigned long long key) { return __uint_as_float((unsigned)(key >> 32) | (unsigned)key << 31); }

struct LaneRay {
    f3 o, inv;                       // counting traversals
    RaySlopes k;                     // every other traversal
    int order;
    uint32_t cur, links;             // group << shift | remaining hit mask; the group's word 48
    int sp;
    int r, r_end;
    int node;                        // leaf node being tested, -1 = the root is the leaf
    float lx, ly, lz, hx, hy, hz;    // its box (counting traversals)
    int kleaf;
    int nb, nt;
};

// Stack entry of a traversal: the counting one packs the child position (see kCountShift), the others
// keep the group's word 48 beside its index and remaining hit mask.
template <bool COUNT>
struct StackOf {
    using type = uint2;
};
template <>
struct StackOf<true> {
    using type = uint32_t;
};

// Starts a ray: root leaf, root miss, or the root's children tested (Octree.impl.cuh:175-190).
template <bool COUNT, bool MULTI>
__device__ __forceinline__ int lane_start(const Scene &S, LaneRay &L, f3 o, f3 d) {
    L.order = (d.z < 0 ? 1 : 0) + (d.y < 0 ? 2 : 0) + (d.x < 0 ? 4 : 0);
    L.sp = 0;
    L.cur = 0;
    if (COUNT) {
        L.o = o;
        L.inv = mkf3(__fdiv_rn(1.0f, d.x), __fdiv_rn(1.0f, d.y), __fdiv_rn(1.0f, d.z));
        L.nb = 0;
        L.nt = 0;
        L.kleaf = 0;
    }
    if (S.root_child < 0) {
        L.r = S.root_leaf_first;
        L.r_end = S.root_leaf_first + S.root_leaf_count;
        L.node = -1;
        if (COUNT) {
            L.lx = S.root_lo[0]; L.ly = S.root_lo[1]; L.lz = S.root_lo[2];
            L.hx = S.root_hi[0]; L.hy = S.root_hi[1]; L.hz = S.root_hi[2];
            L.kleaf = 7;  // no group scan to correct for a root leaf
        }
        return kLeaf;
    }
    if constexpr (COUNT) {
        L.nb++;
        const bool front = S.front_only != 0;
        if (slab_hit(S.root_lo[0], S.root_lo[1], S.root_lo[2], S.root_hi[0], S.root_hi[1], S.root_hi[2], o, L.inv, front)) {
            L.cur = ((uint32_t)S.root_child << kCountShift) |
                    test_group(front ? S.gbox : S.gbox_ref, S.root_child, L.order, o, L.inv, front);
            L.nb += 8;
        }
    } else {
        // a frame whose one child left is the root's group: the first step tests it.  The root's own box is
        // tested when a hit is accepted (leaf_accepts); rays of a batch test it here, where their scene is
        // at hand.
        bool enter = !never_hits(o, d);
        if (MULTI) enter = enter && exact_slab(mkf3(S.root_lo[0], S.root_lo[1], S.root_lo[2]), mkf3(S.root_hi[0], S.root_hi[1], S.root_hi[2]), o, d);
        L.k = ray_slopes(o, d, S.reach);
        L.cur = enter ? 1u : 0u;
        L.links = ((uint32_t)S.root_child << 8) | (1u << L.order);
    }
    return kTrav;
}

// Whether the nearest hit of a leaf ends the ray (castInLeaf's acceptance): its point lies in the leaf's
// box (or `anywhere`: an occluder), and the ray passes the exact slab tests of that box and of the root,
// which the conservative group tests on the way down stand in for.  A point `margin` (point_margin) inside
// a box settles its slab test: the rounded plane distances then lie on either side of the hit's.  Hardly
// any hit is nearer to a face than that, so the divisions of the exact test stay out of the way.
__device__ __forceinline__ bool inside_by(f3 p, f3 l, f3 h, float m) {
    return p.x >= l.x + m && p.y >= l.y + m && p.z >= l.z + m && p.x <= h.x - m && p.y <= h.y - m && p.z <= h.z - m;
}
template <bool ROOT>
__device__ __forceinline__ bool leaf_accepts(const Scene &S, int node, f3 root_lo, f3 root_hi, f3 o, f3 d, f3 p, float margin, bool anywhere) {
    f3 l = root_lo, h = root_hi;
    if (node >= 0) {
        float4 lo, hi;
        ldg2(S.nodes + 2 * (size_t)node, lo, hi);
        l = f3of(lo);
        h = f3of(hi);
    }
    if (!anywhere && !inside_by(p, l, h, 0.0f)) return false;
    if (node < 0) return true;
    return (inside_by(p, l, h, margin) || exact_slab(l, h, o, d)) && (!ROOT || inside_by(p, root_lo, root_hi, margin) || exact_slab(root_lo, root_hi, o, d));
}

// Loads entry i of the source into the lane and starts its ray; kIdle when the source has nothing
// to trace for it.  Also serves a ray the source rewrote in place (a photon continuing past a
// blocker): the lane starts it at once, without going back to the warp's chunk.
template <bool COUNT, bool MULTI, class Source>
__device__ __forceinline__ int restart(const Scene &S, Source &src, int i, LaneRay &L, WarpSlots &ws, unsigned lane) {
    int ign, job;
    f3 o, d;
    if (!src.load(i, o, d, ign, job)) return kIdle;
    ws.o[lane] = make_float4(o.x, o.y, o.z, __int_as_float(ign));
    const Scene &own = MULTI ? src.scene(job) : S;
    ws.d[lane] = make_float4(d.x, d.y, d.z, point_margin(o, own.reach));
    ws.key[lane] = kNoHit;
    return lane_start<COUNT, MULTI>(own, L, o, d);
}

// Lanes per warp that take rays when `n` rays meet `warps` resident warps.  Fewer rays than lanes
// spread over every warp: a warp's iteration serves all its rays' steps one path after the other and
// waits for the slowest load among them, so a launch that cannot fill the lanes ends sooner with one
// ray in each of 32 warps than with 32 rays in one.  Same call, against 256 rays a warp: 61 casts
// 119 -> 45 us, 100,003 counted casts 302 -> 113 us, 2.07M primary casts 1.79 -> 1.18 ms (with the
// round-robin chunks of k_cast); a 161x91 preview, 14.6k rays a launch, 0.99 -> 0.74 ms.
__device__ __forceinline__ int warp_width(int n, int warps) { return max(1, min(32, (n + warps - 1) / warps)); }

// Source interface:
//   bool next(int &begin, int &end)           warp-uniform; false when no work is left
//   int entry(int k)                          the k-th ray to take
//   bool load(int i, f3 &o, f3 &d, int &ignore, int &job)   false: entry i needs no cast (done)
//   int job(int i)                            the job of entry i
//   const Scene &scene(int job)               the scene of a job (MULTI only)
//   bool clip()                               backface culling (of the first job: the same for all)
//   bool store(int i, const Hit &h, int nbox, int ntri)   true: ray i was rewritten (load() now
//                                             gives its next cast) and the lane traces it at once
//   static constexpr float kOccludeBelow      > 0: visibility-only rays (any hit nearer than this
//                                             settles them); 0: closest hit
// MULTI = false: every ray belongs to scene `S`.  MULTI = true: rays of different scenes share the
// warp; their trees live in one batch arena (S.nodes / S.leaf_tris are the arena's), so a lane only
// takes its scene's root (bounds, child group or root leaf) when it starts a ray.  Backface culling
// is uniform over a wave in both cases.
// Tests one lane may bring to a round, a bound on the ballots that number them; larger leaves (the
// unsplittable ones) take several rounds.
constexpr int kRoundBits = 5;
constexpr int kRoundCap = (1 << kRoundBits) - 1;

// steps: traversal steps a lane may take between two leaf rounds while it stays in inner nodes; more
// means fewer rounds, but lanes that reached a leaf wait longer.
// width: lanes that take rays (see warp_width); all 32 test triangles.
template <bool COUNT, bool MULTI, class Source>
__device__ __forceinline__ void trace_persistent(const Scene &S, Source &src, typename StackOf<COUNT>::type *stack, WarpSlots &ws,
                                                 int width, int steps) {
    constexpr unsigned kAll = 0xFFFFFFFFu;
    const unsigned lane = threadIdx.x & 31u;
    const unsigned lt_mask = (1u << lane) - 1u;
    int c_next = 0, c_end = 0;
    bool drained = false;
    int cur_i = -1;
    int mode = kIdle;
    const bool clip = src.clip();
    const bool front = !COUNT || S.front_only != 0;   // uniform: one scene, or one arena of a batch
    // group-test planes of a counting traversal: the reference's boxes on reference-padding scenes
    // (their counts are the reference's), the refitted ones elsewhere
    [[maybe_unused]] const float4 *G = front ? S.gbox : S.gbox_ref;
    LaneRay L;
    L.r = 0;
    L.r_end = 0;
    L.sp = 0;
    L.cur = 0;
    L.nb = 0;
    L.nt = 0;
    for (;;) {
        // ---- finished rays, then refill of idle lanes from the warp's chunk (warp-uniform control flow)
        bool start = false;
        if (mode == kDone) {
            const unsigned long long key = ws.key[lane];
            Hit h;
            h.tri = -1;
            h.t = FLT_MAX;
            if (key != kNoHit) {
                h.tri = leaf_tri_id(S.leaf_tris, S.leaf_half, key_pos(key));
                h.t = key_dist(key);
                h.p = xadd(f3of(ws.o[lane]), xmul(f3of(ws.d[lane]), h.t));
            }
            start = src.store(cur_i, h, L.nb, L.nt);
            mode = kIdle;
        }
        const bool free = mode == kIdle && !start && (int)lane < width;
        const unsigned want = __ballot_sync(kAll, free);
        if (want != 0u && !drained) {
            if (c_next >= c_end && !src.next(c_next, c_end)) drained = true;
            if (!drained) {
                const int avail = c_end - c_next;
                const int rank = __popc(want & lt_mask);
                if (free && rank < avail) {
                    cur_i = src.entry(c_next + rank);
                    start = true;
                }
                c_next += min(avail, __popc(want));
            }
        }
        if (start) mode = restart<COUNT, MULTI>(S, src, cur_i, L, ws, lane);
        if (__ballot_sync(kAll, mode != kIdle) == 0u) {
            if (drained) break;
            continue;
        }
#pragma unroll 1
        for (int step = 0; step < steps; step++) {
            if (mode != kTrav) break;
            // ---- one traversal step: pop an empty frame, then take one child
            if constexpr (COUNT) {
                while ((L.cur & 0xFFu) == 0u && L.sp > 0) L.cur = stack[--L.sp];
            } else if ((L.cur & 0xFFu) == 0u && L.sp > 0) {   // frames are stacked with children left
                const uint2 e = stack[--L.sp];
                L.cur = e.x;
                L.links = e.y;
            }
            const uint32_t m = L.cur & 0xFFu;
            if (m == 0u) {
                mode = kDone;   // a miss: the key holds no hit
            } else if constexpr (COUNT) {
                int k = __ffs(m) - 1;
                L.cur &= ~(1u << k);
                int node = (int)(L.cur >> kCountShift) * 8 + (L.order ^ k);
                float4 lo, hi;
                ldg2(S.nodes + 2 * (size_t)node, lo, hi);
                int w = __float_as_int(lo.w);
                if (w < 0) {
                    L.r = ~w;
                    L.r_end = ~w + __float_as_int(hi.w);
                    L.lx = lo.x; L.ly = lo.y; L.lz = lo.z;
                    L.hx = hi.x; L.hy = hi.y; L.hz = hi.z;
                    L.kleaf = k;
                    mode = kLeaf;
                } else if (L.sp < kStack) {
                    stack[L.sp++] = (L.cur & ~(7u << 8)) | ((uint32_t)k << 8);
                    L.cur = ((uint32_t)(w >> 3) << kCountShift) | test_group(G, w >> 3, L.order, L.o, L.inv, front);
                    L.nb += 8;
                } else {  // unreachable for depth <= 24: finish as a miss rather than overflow
                    L.cur = 0;
                    L.sp = 0;
                }
            } else {
                const uint32_t c = (uint32_t)(__ffs(m) - 1) ^ (uint32_t)L.order;
                L.cur &= L.cur - 1u;
                const uint32_t g = L.cur >> 8;
                if (((L.links >> c) & 1u) == 0u) {
                    const int *first = reinterpret_cast<const int *>(S.groups + (size_t)g * kRecordF4) + 49 + c;
                    L.r = __ldg(first);
                    L.r_end = __ldg(first + 1);
                    L.node = (int)(8u * g + c);
                    mode = kLeaf;
                } else {
                    const uint32_t child = (L.links >> 8) + __popc(L.links & ((1u << c) - 1u));
                    bool room = true;
                    if ((L.cur & 0xFFu) != 0u) {
                        room = L.sp < kStack;   // always for depth <= 24: finish as a miss rather than overflow
                        if (room) stack[L.sp++] = make_uint2(L.cur, L.links);
                    }
                    L.cur = 0;
                    if (room) L.cur = (child << 8) | record_mask(S.groups, child, L.order, L.k, L.links);
                    else L.sp = 0;
                }
            }
        }
        // ---- one leaf round (castInLeaf): up to kRoundCap tests of every lane that holds a leaf
        const unsigned owners = __ballot_sync(kAll, mode == kLeaf && L.r < L.r_end);
        if (owners != 0u) {
            const bool mine = (owners >> lane) & 1u;
            const int count = mine ? min(L.r_end - L.r, kRoundCap) : 0;
            int before = 0, total = 0;   // tests of the lanes below; of all
#pragma unroll
            for (int j = 0; j < kRoundBits; j++) {
                const unsigned b = __ballot_sync(kAll, (count >> j) & 1);
                before += __popc(b & lt_mask) << j;
                total += __popc(b) << j;
            }
            if (mine) ws.task[__popc(owners & lt_mask)] = make_int2((int)lane, L.r - before);
            __syncwarp();
            int owned = 0;   // owners whose tests began in an earlier window
            for (int base = 0; base < total; base += 32) {
                const int at = before - base;
                const unsigned begins = __reduce_or_sync(kAll, mine && at >= 0 && at < 32 ? 1u << at : 0u);
                const int t = base + (int)lane;
                if (t < total) {
                    const int2 task = ws.task[owned + __popc(begins & (lt_mask << 1 | 1u)) - 1];
                    const int pos = task.y + t;
                    const float4 o = ws.o[task.x], d = ws.d[task.x];
                    float dist;
                    if (tri_cast(S.leaf_tris, S.leaf_half, pos, f3of(o), f3of(d), clip, __float_as_int(o.w), dist))
                        atomicMin(&ws.key[task.x], hit_key(dist, pos));
                }
                owned += __popc(begins);
            }
            __syncwarp();
            if (COUNT) L.nt += count;
            L.r += count;
        }
        if (mode == kLeaf && L.r >= L.r_end) {
            // occlusion sources end a ray at the first leaf holding a hit nearer than their limit, even
            // one whose point lies in a later leaf: that hit's own leaf would end the ray there anyway
            mode = kTrav;
            const unsigned long long key = ws.key[lane];
            if (key != kNoHit) {
                const float t = key_dist(key);
                const bool occluded = Source::kOccludeBelow > 0.0f && t < Source::kOccludeBelow;
                const float4 dm = ws.d[lane];
                const f3 o = f3of(ws.o[lane]), d = f3of(dm), p = xadd(o, xmul(d, t));
                if constexpr (COUNT) {
                    if (occluded || (p.x >= L.lx && p.y >= L.ly && p.z >= L.lz && p.x <= L.hx && p.y <= L.hy && p.z <= L.hz)) {
                        L.nb -= 7 - L.kleaf;
                        for (int s = 0; s < L.sp; s++) L.nb -= 7 - (int)((stack[s] >> 8) & 7u);
                        mode = kDone;
                    }
                } else {
                    const Scene &own = MULTI && L.node < 0 ? src.scene(src.job(cur_i)) : S;
                    if (leaf_accepts<!MULTI>(S, L.node, mkf3(own.root_lo[0], own.root_lo[1], own.root_lo[2]),
                                             mkf3(own.root_hi[0], own.root_hi[1], own.root_hi[2]), o, d, p, dm.w, occluded))
                        mode = kDone;
                }
                if (mode != kDone) ws.key[lane] = kNoHit;
            }
        }
    }
}

}  // namespace drd
