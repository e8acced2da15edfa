// octree_gpu.cu - the octree build on the GPU, bit-identical to the host builder (and so to the
// reference's Octree::build, Octree.impl.cuh:114-129, 339-533).
//
// Level by level, like the host builder; per level the GPU runs
//   (1) owner of every reference (binary search over the level's reference ranges),
//   (2) the clipped centre of every reference of a splittable node (parallel over references),
//   (3) the split point of every splittable node: the float sum of its references' centres in list
//       order (a warp per node loads, a lane per axis adds: the order of a float sum is part of the
//       result) and its octants,
//   (4) the octant overlap mask of every reference (parallel),
//   (5) per node the octant occupancy and the split decision (a warp per node; integer sums),
//   (6) the clipped bounds of every reference of a leaf (parallel) and each leaf's box: min / max in
//       list order from the node box, then the padded shrink (a warp per leaf),
//   (7) prefix sums over the level's nodes of their split flags, leaf references and child references:
//       where each split node's children and each leaf's list go (breadth-first order),
//   (8) the next level's nodes and, for every split node, its references copied to the lists of the
//       octants they overlap, in list order (a warp per node, the block for large ones).
// Staging the sums of (3), a thread per octant in (4) and the block's part in (8) took a scene of 82k triangles
// (displaced icosphere, physical padding, split 4) from 22.2 to 18.6 ms and one of 1.31M from 352 to 297 ms; what
// the later steps gave stands at their kernels.
// After the last level inner boxes shrink to their children's, level by level from the deepest.  The
// host reads three totals a level (sizes of the next level's arrays) and the finished tree.  All geometry
// comes from octree_geom.h; nvcc compiles it with -fmad=false and IEEE division / square root, the host
// builder with -ffp-contract=off, so both perform the same single-precision operations.
#include <cuda_runtime.h>

#include <algorithm>
#include <memory>
#include <string>
#include <vector>

#include "octree_device.h"
#include "octree_geom.h"

namespace drb {
namespace {

using namespace geom;

const float kBoxEpsGpu = 0.000005f * 256.0f;   // OCTREE_AABB_EPSILON (Octree.impl.cuh:3-5)

__device__ __forceinline__ T3 load_tri(const float *xyz, int id) {
    const float *p = xyz + 9 * (size_t)id;
    return T3{mk(p[0], p[1], p[2]), mk(p[3], p[4], p[5]), mk(p[6], p[7], p[8])};
}
__device__ __forceinline__ Bx load_box(const float *b, int k) {
    const float *p = b + 6 * (size_t)k;
    return Bx{mk(p[0], p[1], p[2]), mk(p[3], p[4], p[5])};
}
__device__ __forceinline__ void store_box(float *b, int k, const Bx &x) {
    float *p = b + 6 * (size_t)k;
    p[0] = x.lo.x; p[1] = x.lo.y; p[2] = x.lo.z;
    p[3] = x.hi.x; p[4] = x.hi.y; p[5] = x.hi.z;
}
__device__ __forceinline__ bool splittable(const int *off, int k, int depth, int max_depth, int split_n) {
    return depth < max_depth && (off[k + 1] - off[k]) >= split_n;
}

__global__ void k_iota(int *v, int n) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) v[i] = i;
}

__global__ void k_owner(const int *off, int nl, int nr, int *owner) {
    const int r = blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= nr) return;
    int lo = 0, hi = nl - 1;   // last node with off[k] <= r (empty nodes share offsets; take the last)
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (off[mid] <= r) lo = mid;
        else hi = mid - 1;
    }
    owner[r] = lo;
}

__global__ void k_centres(const float *xyz, const int *refs, const int *owner, const int *off, const float *box, int nr,
                          int depth, int max_depth, int split_n, float *centre) {
    const int r = blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= nr) return;
    const int k = owner[r];
    if (!splittable(off, k, depth, max_depth, split_n)) return;
    Pieces l, x, y;
    const P3 c = clipped_centre(load_box(box, k), load_tri(xyz, refs[r]), l, x, y);
    centre[3 * (size_t)r] = c.x;
    centre[3 * (size_t)r + 1] = c.y;
    centre[3 * (size_t)r + 2] = c.z;
}

// One warp per node: the lanes stage kStage centres at a time in shared memory, axis by axis, and lanes
// 0-2 add one axis each in list order, so the float sum has the host builder's order.  The chain of
// dependent additions is what a large node costs (4 cycles each, three shuffles and 58 cycles a
// reference when every lane added broadcast values); the next stage's loads are issued before it.
constexpr int kStage = 128, kStageWarps = 4;
__global__ void __launch_bounds__(32 * kStageWarps) k_split_points(const float *centre, const int *off, const float *box, int nl, int depth,
                                                                   int max_depth, int split_n, float E, float *sub) {
    __shared__ __align__(16) float stage[kStageWarps][3][kStage];
    const int k = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (k >= nl || !splittable(off, k, depth, max_depth, split_n)) return;
    float (&st)[3][kStage] = stage[threadIdx.x >> 5];
    const int rb = off[k], re = off[k + 1];
    constexpr int kLoads = 3 * kStage / 32;
    float v[kLoads];
    auto load = [&](int base) {
        const int m = 3 * min(kStage, re - base);
        const float *c = centre + 3 * (size_t)base;
#pragma unroll
        for (int j = 0; j < kLoads; j++) v[j] = 32 * j + lane < m ? c[32 * j + lane] : 0.0f;
    };
    load(rb);
    float sum = 0.0f;
    for (int base = rb; base < re; base += kStage) {
#pragma unroll
        for (int j = 0; j < kLoads; j++) st[(32 * j + lane) % 3][(32 * j + lane) / 3] = v[j];
        __syncwarp();
        if (base + kStage < re) load(base + kStage);
        if (lane < 3) {
            const int m = min(kStage, re - base);
            int j = 0;
            for (; j + 4 <= m; j += 4) {
                const float4 q = *reinterpret_cast<const float4 *>(&st[lane][j]);
                sum = (((sum + q.x) + q.y) + q.z) + q.w;
            }
            for (; j < m; j++) sum += st[lane][j];
        }
        __syncwarp();
    }
    const P3 c = divs(mk(__shfl_sync(0xFFFFFFFFu, sum, 0), __shfl_sync(0xFFFFFFFFu, sum, 1), __shfl_sync(0xFFFFFFFFu, sum, 2)),
                      (float)(re - rb));
    if (lane != 0) return;
    Bx o[8];
    octants(load_box(box, k), c, o, E);
    for (int i = 0; i < 8; i++) store_box(sub, 8 * k + i, o[i]);
}

// Octant overlap of every reference: a thread per (reference, octant), the mask byte from a ballot.
// (One thread per reference took its eight tests one after another, each as long as the longest of the
// warp's.  Gathering a block's clipped pairs before clipping them was slower than both.)
__global__ void k_masks(const float *xyz, const int *refs, const int *owner, const int *off, const float *sub, int nr, int depth,
                        int max_depth, int split_n, unsigned char *mask) {
    const long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    const int r = (int)(t >> 3), i = (int)(t & 7);
    bool hit = false;
    if (r < nr) {
        const int k = owner[r];
        if (splittable(off, k, depth, max_depth, split_n)) hit = overlaps(load_box(sub, 8 * k + i), load_tri(xyz, refs[r]));
    }
    const unsigned bal = __ballot_sync(0xFFFFFFFFu, hit);
    if (r < nr && i == 0) mask[r] = (unsigned char)(bal >> (threadIdx.x & 24));
}

// What a node adds to the level's prefix sums.  (Splits, lists and boxes of a level used to go to the host
// for this bookkeeping: 82k triangles 17.3 -> 12.6 ms, 1.31M triangles 291 -> 169 ms a scene, same call.)
struct Sums {
    int splits, leaf_refs;
    long long child_refs;
};
__host__ __device__ __forceinline__ Sums operator+(Sums a, Sums b) {
    return Sums{a.splits + b.splits, a.leaf_refs + b.leaf_refs, a.child_refs + b.child_refs};
}

// splittingMakesSence (Octree.impl.cuh:437-475): one warp per node.
constexpr int kDecideLoads = 8;
__global__ void k_decide(const unsigned char *mask, const int *off, int nl, int depth, int max_depth, int split_n, int *occ,
                         int *does_split, Sums *sums) {
    const int k = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (k >= nl) return;
    const bool can = splittable(off, k, depth, max_depth, split_n);
    int c[8] = {0, 0, 0, 0, 0, 0, 0, 0};
    if (can)
        for (int base = off[k] + lane; base < off[k + 1]; base += 32 * kDecideLoads) {   // several loads in flight
            unsigned m[kDecideLoads];
#pragma unroll
            for (int q = 0; q < kDecideLoads; q++) m[q] = base + 32 * q < off[k + 1] ? mask[base + 32 * q] : 0u;
            // bits to byte counters: 4 octants a word
            unsigned lo = 0, hi = 0;
#pragma unroll
            for (int q = 0; q < kDecideLoads; q++) {
                lo += ((m[q] & 0xFu) * 0x00204081u) & 0x01010101u;
                hi += ((m[q] >> 4) * 0x00204081u) & 0x01010101u;
            }
            for (int i = 0; i < 4; i++) {
                c[i] += (lo >> (8 * i)) & 0xFF;
                c[4 + i] += (hi >> (8 * i)) & 0xFF;
            }
        }
    for (int i = 0; i < 8; i++)
        for (int s = 16; s > 0; s >>= 1) c[i] += __shfl_xor_sync(0xFFFFFFFFu, c[i], s);
    if (lane != 0) return;
    bool ok = false;
    if (can) {
        const int cnt = off[k + 1] - off[k];
        int full = 0;
        float load = 0.0f;
        for (int i = 0; i < 8; i++) {
            if (c[i] >= cnt) full++;
            load += ((float)c[i]) / ((float)cnt);
        }
        ok = (full < 1) && (load < fminf(((float)cnt) / ((float)split_n), 6.0f));
    }
    does_split[k] = ok ? 1 : 0;
    long long all = 0;
    for (int i = 0; i < 8; i++) {
        occ[8 * k + i] = c[i];
        all += c[i];
    }
    sums[k] = ok ? Sums{1, 0, all} : Sums{0, off[k + 1] - off[k], 0};
}

// Exclusive prefix sums in place: chunks of kScan nodes a block, the chunk totals by one block (the grand
// total after the last).  The sum before node k is sums[k] + totals[k / kScan].
constexpr int kScanThreads = 256, kScan = 4 * kScanThreads;
__device__ __forceinline__ Sums block_scan(Sums v, Sums &total) {   // exclusive, over the block's threads
    __shared__ Sums warps[kScanThreads / 32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    Sums x = v;
    for (int s = 1; s < 32; s <<= 1) {
        const Sums y{__shfl_up_sync(0xFFFFFFFFu, x.splits, s), __shfl_up_sync(0xFFFFFFFFu, x.leaf_refs, s),
                     __shfl_up_sync(0xFFFFFFFFu, x.child_refs, s)};
        if (lane >= s) x = x + y;
    }
    __syncthreads();   // a caller's previous scan is read
    if (lane == 31) warps[warp] = x;
    __syncthreads();
    Sums before{0, 0, 0};
    total = before;
    for (int w = 0; w < kScanThreads / 32; w++) {
        if (w == warp) before = total;
        total = total + warps[w];
    }
    return Sums{before.splits + x.splits - v.splits, before.leaf_refs + x.leaf_refs - v.leaf_refs,
                before.child_refs + x.child_refs - v.child_refs};
}
__global__ void __launch_bounds__(kScanThreads) k_scan_chunks(Sums *sums, int n, Sums *totals) {
    const long long first = (long long)blockIdx.x * kScan + 4 * threadIdx.x;
    Sums v[4], all{0, 0, 0}, total;
    for (int q = 0; q < 4; q++) {
        v[q] = first + q < n ? sums[first + q] : Sums{0, 0, 0};
        all = all + v[q];
    }
    Sums at = block_scan(all, total);
    for (int q = 0; q < 4; q++) {
        if (first + q < n) sums[first + q] = at;
        at = at + v[q];
    }
    if (threadIdx.x == 0) totals[blockIdx.x] = total;
}
__global__ void __launch_bounds__(kScanThreads) k_scan_totals(Sums *totals, int m) {
    Sums carry{0, 0, 0};
    for (int base = 0; base < m; base += kScanThreads) {
        const int i = base + (int)threadIdx.x;
        Sums total;
        const Sums at = block_scan(i < m ? totals[i] : Sums{0, 0, 0}, total);
        if (i < m) totals[i] = carry + at;
        carry = carry + total;
    }
    if (threadIdx.x == 0) totals[m] = carry;
}
__device__ __forceinline__ Sums sums_before(const Sums *sums, const Sums *totals, int k) { return sums[k] + totals[k / kScan]; }

// The level's finished nodes and the next level's: one thread per node.  A split node's children start at
// 8 x the split nodes before it, in the next level and (plus next_base) in the tree; a leaf takes its
// shrunk box and its place in the tree's reference list.
__global__ void k_emit(const Sums *sums, const Sums *totals, const int *off, const int *does_split, const int *occ, const float *sub,
                       const float *lbox, int nl, long long leaf_base, int next_base, float *box, int *child, int *first_child,
                       long long *leaf_first, int *leaf_count, int *next_off, float *next_box) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= nl) return;
    const Sums at = sums_before(sums, totals, k);
    if (!does_split[k]) {
        store_box(box, k, load_box(lbox, k));
        child[k] = -1;
        first_child[k] = -1;
        leaf_first[k] = leaf_base + at.leaf_refs;
        leaf_count[k] = off[k + 1] - off[k];
        return;
    }
    child[k] = next_base + 8 * at.splits;
    first_child[k] = 8 * at.splits;
    leaf_first[k] = 0;
    leaf_count[k] = 0;
    int r = (int)at.child_refs;
    for (int i = 0; i < 8; i++) {
        next_off[8 * at.splits + i] = r;
        r += occ[8 * k + i];
        store_box(next_box, 8 * at.splits + i, load_box(sub, 8 * k + i));
    }
    if (8LL * (at.splits + 1) == 8LL * totals[(nl + kScan - 1) / kScan].splits) next_off[8 * at.splits + 8] = r;   // the last one
}

// The leaves' references into the tree's list.
__global__ void k_leaf_refs(const Sums *sums, const Sums *totals, const int *refs, const int *owner, const int *off, const int *does_split,
                            int nr, int *out) {
    const int r = blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= nr) return;
    const int k = owner[r];
    if (!does_split[k]) out[sums_before(sums, totals, k).leaf_refs + r - off[k]] = refs[r];
}

// reduceNode(0, false) after the build: inner boxes shrink to the union of their children's; `child` less
// `next_base` is the first child's place in the next level.
__global__ void k_reduce(float *box, const int *child, int nl, int next_base, const float *next_box, float E) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= nl || child[k] < 0) return;
    const Bx b = load_box(box, k);
    P3 lo = b.hi, hi = b.lo;
    for (int c = 0; c < 8; c++) {
        const Bx cb = load_box(next_box, child[k] - next_base + c);
        lo = mk(fmin_(lo.x, cb.lo.x), fmin_(lo.y, cb.lo.y), fmin_(lo.z, cb.lo.z));
        hi = mk(fmax_(hi.x, cb.hi.x), fmax_(hi.y, cb.hi.y), fmax_(hi.z, cb.hi.z));
    }
    store_box(box, k, shrink(b, lo, hi, E));
}

// A level's nodes into the finished arrays.
__global__ void k_finish(const float *box, int nl, float *lo, float *hi) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= 3 * nl) return;
    const int k = i / 3, a = i - 3 * k;
    lo[i] = box[6 * (size_t)k + a];
    hi[i] = box[6 * (size_t)k + 3 + a];
}

__global__ void k_leaf_bounds(const float *xyz, const int *refs, const int *owner, const float *box, const int *does_split,
                              int nr, float *bounds) {
    const int r = blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= nr) return;
    const int k = owner[r];
    if (does_split[k]) return;
    Pieces l, x, y;
    store_box(bounds, r, clipped_bounds(load_box(box, k), load_tri(xyz, refs[r]), l, x, y));
}

// reduceNode(index, true) of a leaf: min / max over the clipped bounds in list order (broadcast
// from the warp's loads), then shrink.  One warp per leaf.
__global__ void k_leaf_boxes(const float *bounds, const int *off, const float *box, const int *does_split, int nl, float E,
                             float *lbox) {
    const int k = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (k >= nl || does_split[k]) return;
    const Bx b = load_box(box, k);
    P3 lo = b.hi, hi = b.lo;
    const int rb = off[k], re = off[k + 1];
    for (int base = rb; base < re; base += 32) {
        Bx ob = b;
        if (base + lane < re) ob = load_box(bounds, base + lane);
        const int m = min(32, re - base);
        for (int j = 0; j < m; j++) {
            const float l0 = __shfl_sync(0xFFFFFFFFu, ob.lo.x, j), l1 = __shfl_sync(0xFFFFFFFFu, ob.lo.y, j),
                        l2 = __shfl_sync(0xFFFFFFFFu, ob.lo.z, j);
            const float h0 = __shfl_sync(0xFFFFFFFFu, ob.hi.x, j), h1 = __shfl_sync(0xFFFFFFFFu, ob.hi.y, j),
                        h2 = __shfl_sync(0xFFFFFFFFu, ob.hi.z, j);
            lo = mk(fmin_(lo.x, l0), fmin_(lo.y, l1), fmin_(lo.z, l2));
            hi = mk(fmax_(hi.x, h0), fmax_(hi.y, h1), fmax_(hi.z, h2));
        }
    }
    if (lane == 0) store_box(lbox, k, shrink(b, lo, hi, E));
}

// Children's reference lists (Octree.impl.cuh:392-404), in list order: a reference's position in an
// octant's list is the count of earlier references that also overlap it.  A warp per split node, 32
// references at a time by ballots; nodes of more than kBlockRefs references go to the whole block
// afterwards, 4 references a thread: counts per octant as bytes of a 64-bit word, scanned over the warp
// by shuffles and over the block in shared memory.
constexpr int kScatterWarps = 8, kBlockRefs = 2048, kPerThread = 4;
__global__ void __launch_bounds__(32 * kScatterWarps) k_scatter(const int *refs, const unsigned char *mask, const int *off, const int *first_child,
                                                                const int *next_off, int nl, int *next_refs) {
    __shared__ int totals[kScatterWarps][8];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const unsigned lt = (1u << lane) - 1u;
    const int k0 = blockIdx.x * kScatterWarps;
    const int k = k0 + warp;
    if (k < nl && first_child[k] >= 0 && off[k + 1] - off[k] <= kBlockRefs) {
        int w[8];
        for (int i = 0; i < 8; i++) w[i] = next_off[first_child[k] + i];
        for (int base = off[k]; base < off[k + 1]; base += 32) {
            const int r = base + lane;
            const bool in = r < off[k + 1];
            const unsigned m = in ? mask[r] : 0u;
            const int id = in ? refs[r] : 0;
            for (int i = 0; i < 8; i++) {
                const unsigned bal = __ballot_sync(0xFFFFFFFFu, (m >> i) & 1u);
                if ((m >> i) & 1u) next_refs[w[i] + __popc(bal & lt)] = id;
                w[i] += __popc(bal);
            }
        }
    }
    for (int j = k0; j < min(k0 + kScatterWarps, nl); j++) {
        const int rb = off[j], re = off[j + 1];
        if (first_child[j] < 0 || re - rb <= kBlockRefs) continue;   // the same for the whole block
        int w[8];
        for (int i = 0; i < 8; i++) w[i] = next_off[first_child[j] + i];
        unsigned char m[kPerThread];
        int id[kPerThread];
        auto load = [&](int base) {
            for (int q = 0; q < kPerThread; q++) {
                const int r = base + kPerThread * (int)threadIdx.x + q;
                m[q] = r < re ? mask[r] : 0;
                id[q] = r < re ? refs[r] : 0;
            }
        };
        load(rb);
        for (int base = rb; base < re; base += 32 * kScatterWarps * kPerThread) {
            // bit i of a mask -> byte i of a word: at most 4 a thread, 128 a warp
            unsigned long long mine = 0;
            for (int q = 0; q < kPerThread; q++)
                for (int i = 0; i < 8; i++) mine += (unsigned long long)((m[q] >> i) & 1u) << (8 * i);
            unsigned long long incl = mine;
            for (int s = 1; s < 32; s <<= 1) {
                const unsigned long long v = __shfl_up_sync(0xFFFFFFFFu, incl, s);
                if (lane >= s) incl += v;
            }
            if (lane == 31)
                for (int i = 0; i < 8; i++) totals[warp][i] = (int)((incl >> (8 * i)) & 0xFF);
            __syncthreads();
            const unsigned long long excl = incl - mine;
            int at[8];
            for (int i = 0; i < 8; i++) {
                int before = 0, all = 0;
                for (int v = 0; v < kScatterWarps; v++) {
                    if (v < warp) before += totals[v][i];
                    all += totals[v][i];
                }
                at[i] = w[i] + before + (int)((excl >> (8 * i)) & 0xFF);
                w[i] += all;
            }
            for (int q = 0; q < kPerThread; q++)
                for (int i = 0; i < 8; i++)
                    if ((m[q] >> i) & 1u) next_refs[at[i]++] = id[q];
            load(base + 32 * kScatterWarps * kPerThread);
            __syncthreads();
        }
    }
}

inline unsigned blocks(long long n, int t) { return (unsigned)((n + t - 1) / t); }

// One allocation that a build's buffers start out from: the levels of a tree would otherwise allocate and
// free some hundred times (82k triangles, same call: 9.66 -> 7.49 ms a scene, with the decide kernel's
// loads in flight; 1.31M triangles 109 -> 104 ms).
struct Slab {
    char *p = nullptr;
    size_t bytes = 0, used = 0;
    const bool tight;   // no more memory than needed: buffers that grow take no reserve either
    Slab(size_t want, bool tight_) : tight(tight_) {
        if (want == 0 || tight) return;
        if (cudaMalloc((void **)&p, want) == cudaSuccess) bytes = want;
        else {
            p = nullptr;
            (void)cudaGetLastError();   // the buffers then allocate by themselves
        }
    }
    Slab(const Slab &) = delete;
    Slab &operator=(const Slab &) = delete;
    ~Slab() { cudaFree(p); }
    void *take(size_t want) {
        want = (want + 255) & ~size_t(255);
        if (want > bytes - used) return nullptr;
        void *q = p + used;
        used += want;
        return q;
    }
};

struct DevBuf {
    void *p = nullptr;
    size_t bytes = 0;
    bool owned = false;
    DevBuf() = default;
    DevBuf(const DevBuf &) = delete;
    DevBuf &operator=(const DevBuf &) = delete;
    ~DevBuf() {
        if (owned) cudaFree(p);
    }
    // At least `count` elements, contents undefined.  With a slab the first allocation comes from it, of
    // `guess` elements if that is more; growing takes half as much again as needed.
    template <class T>
    T *get(size_t count, Slab *slab = nullptr, size_t guess = 0) {
        const size_t need = std::max<size_t>(count, 1) * sizeof(T);
        if (need > bytes) {
            const size_t take = bytes && !(slab && slab->tight) ? need + need / 2 : need;
            if (owned) cudaFree(p);
            p = nullptr;
            owned = false;
            if (!bytes && slab) {
                const size_t want = std::max(need, guess * sizeof(T));
                p = slab->take(want);
                bytes = p ? want : 0;
            }
            if (!p) {
                bytes = 0;
                if (cudaMalloc(&p, take) != cudaSuccess) {
                    p = nullptr;
                    return nullptr;
                }
                owned = true;
                bytes = take;
            }
        }
        return (T *)p;
    }
    void *release() {
        void *q = p;
        p = nullptr;
        bytes = 0;
        owned = false;
        return q;
    }
    void swap(DevBuf &o) {
        std::swap(p, o.p);
        std::swap(bytes, o.bytes);
        std::swap(owned, o.owned);
    }
};

const char kNoMemory[] = "device allocation failed";

bool build(const float *xyz, int64_t n, const BuildOptions &opt, FlatOctree &out, DeviceTree *keep, std::string &err, bool tight) {
    out = FlatOctree();
    if (n <= 0) return true;
    if (n >= (int64_t(1) << 31)) {
        err = "too many triangles for the device build";
        return false;
    }
    const int max_depth = opt.max_depth > 0 ? opt.max_depth : 24;
    const int split_n = opt.split_threshold > 0 ? opt.split_threshold : 8;
    float E = opt.box_eps > 0.0f ? opt.box_eps : kBoxEpsGpu;
    if (opt.box_eps < 0.0f) {
        float m = 0.0f;
        for (int64_t i = 0; i < 9 * n; i++) m = std::fmax(m, std::fabs(xyz[i]));
        E = std::fmax(m, 1e-30f) * (1.0f / 262144.0f);
    }
    // root box (push, Octree.impl.cuh:97-111): host, serial like the host builder
    Bx root;
    for (int64_t i = 0; i < n; i++) {
        const float *p = xyz + 9 * i;
        Bx b = tri_box(T3{mk(p[0], p[1], p[2]), mk(p[3], p[4], p[5]), mk(p[6], p[7], p[8])});
        if (i == 0) root = b;
        else {
            P3 bl = sub(b.lo, mk(E, E, E)), bh = add(b.hi, mk(E, E, E));
            root = fixed_box(mk(std::fmin(root.lo.x, bl.x), std::fmin(root.lo.y, bl.y), std::fmin(root.lo.z, bl.z)),
                             mk(std::fmax(root.hi.x, bh.x), std::fmax(root.hi.y, bh.y), std::fmax(root.hi.z, bh.z)));
        }
    }

    // references of a level: 4 a triangle with the physical padding, up to 10 with the reference's; nodes:
    // about one a triangle.  What a level needs beyond that it allocates; past 4M triangles (2.6 GB here)
    // the allocations no longer show and the guesses would only hold memory.
    const size_t few = (size_t)n + 64, many = 4 * (size_t)n + 1024;
    Slab slab(n <= (4 << 20) ? many * 49 + few * 284 + 160 * few : 0, tight);
    DevBuf b_xyz, b_refs, b_next, b_owner, b_centre, b_bounds, b_mask, b_off, b_noff, b_sub, b_occ, b_split, b_lbox, b_fc, b_sums, b_tot;
    float *d_xyz = b_xyz.get<float>(9 * (size_t)n);
    int *d_refs = b_refs.get<int>((size_t)n, &slab, many);
    if (!d_xyz || !d_refs) { err = kNoMemory; return false; }
    cudaMemcpy(d_xyz, xyz, 36 * (size_t)n, cudaMemcpyHostToDevice);
    k_iota<<<blocks(n, 256), 256>>>(d_refs, (int)n);

    // what the tree keeps of every level
    struct Level {
        DevBuf box, child, first, count, leaf;
        int nodes = 0, base = 0;     // base: the level's first node in the tree (the root has none)
        long long leaf_base = 0;
        int leaf_refs = 0;
    };
    std::vector<std::unique_ptr<Level>> levels;
    levels.push_back(std::make_unique<Level>());
    levels[0]->nodes = 1;
    {
        const float b[6] = {root.lo.x, root.lo.y, root.lo.z, root.hi.x, root.hi.y, root.hi.z};
        const int off[2] = {0, (int)n};
        float *d_box = levels[0]->box.get<float>(6, &slab);
        int *d_off = b_off.get<int>(2, &slab, few);
        if (!d_box || !d_off) { err = kNoMemory; return false; }
        cudaMemcpy(d_box, b, sizeof(b), cudaMemcpyHostToDevice);
        cudaMemcpy(d_off, off, sizeof(off), cudaMemcpyHostToDevice);
    }
    int nr = (int)n, next_base = 0;
    long long leaf_total = 0;
    for (int depth = 0;; depth++) {
        Level &lv = *levels[depth];
        const int nl = lv.nodes;
        const int chunks = (nl + kScan - 1) / kScan;
        const int *d_off = (const int *)b_off.p;
        float *d_box = (float *)lv.box.p;
        int *d_owner = b_owner.get<int>(nr, &slab, many);
        float *d_centre = b_centre.get<float>(3 * (size_t)nr, &slab, 3 * many);
        float *d_sub = b_sub.get<float>(48 * (size_t)nl, &slab, 48 * few);
        unsigned char *d_mask = b_mask.get<unsigned char>(nr, &slab, many);
        int *d_occ = b_occ.get<int>(8 * (size_t)nl, &slab, 8 * few);
        int *d_split = b_split.get<int>(nl, &slab, few);
        float *d_bounds = b_bounds.get<float>(6 * (size_t)nr, &slab, 6 * many);
        float *d_lbox = b_lbox.get<float>(6 * (size_t)nl, &slab, 6 * few);
        Sums *d_sums = b_sums.get<Sums>(nl, &slab, few), *d_tot = b_tot.get<Sums>(chunks + 1, &slab, few / kScan + 2);
        int *d_fc = b_fc.get<int>(nl, &slab, few);
        int *d_child = lv.child.get<int>(nl, &slab), *d_count = lv.count.get<int>(nl, &slab);
        long long *d_first = lv.first.get<long long>(nl, &slab);
        if (!d_owner || !d_centre || !d_sub || !d_mask || !d_occ || !d_split || !d_bounds || !d_lbox || !d_sums || !d_tot || !d_fc ||
            !d_child || !d_count || !d_first) {
            err = kNoMemory;
            return false;
        }
        if (nr > 0) {
            k_owner<<<blocks(nr, 256), 256>>>(d_off, nl, nr, d_owner);
            k_centres<<<blocks(nr, 128), 128>>>(d_xyz, d_refs, d_owner, d_off, d_box, nr, depth, max_depth, split_n, d_centre);
        }
        k_split_points<<<blocks(nl, kStageWarps), 32 * kStageWarps>>>(d_centre, d_off, d_box, nl, depth, max_depth, split_n, E, d_sub);
        if (nr > 0) k_masks<<<blocks(8LL * nr, 256), 256>>>(d_xyz, d_refs, d_owner, d_off, d_sub, nr, depth, max_depth, split_n, d_mask);
        k_decide<<<blocks(32LL * nl, 256), 256>>>(d_mask, d_off, nl, depth, max_depth, split_n, d_occ, d_split, d_sums);
        if (nr > 0) k_leaf_bounds<<<blocks(nr, 128), 128>>>(d_xyz, d_refs, d_owner, d_box, d_split, nr, d_bounds);
        k_leaf_boxes<<<blocks(32LL * nl, 256), 256>>>(d_bounds, d_off, d_box, d_split, nl, E, d_lbox);
        k_scan_chunks<<<chunks, kScanThreads>>>(d_sums, nl, d_tot);
        k_scan_totals<<<1, kScanThreads>>>(d_tot, chunks);
        Sums total;
        cudaError_t e = cudaGetLastError();
        if (e == cudaSuccess) e = cudaMemcpy(&total, d_tot + chunks, sizeof(Sums), cudaMemcpyDeviceToHost);
        if (e != cudaSuccess) {
            err = std::string("device build: ") + cudaGetErrorString(e);
            return false;
        }
        if (total.child_refs >= (int64_t(1) << 31)) {
            err = "too many references in one level for the device build";
            return false;
        }
        if (next_base + 8LL * total.splits >= (int64_t(1) << 31)) {
            err = "too many nodes for the device build";
            return false;
        }
        auto next = std::make_unique<Level>();
        next->nodes = 8 * total.splits;
        next->base = next_base;
        lv.leaf_base = leaf_total;
        lv.leaf_refs = total.leaf_refs;
        float *d_nbox = next->box.get<float>(6 * (size_t)next->nodes, &slab);
        int *d_noff = b_noff.get<int>((size_t)next->nodes + 1, &slab, few);
        int *d_next = b_next.get<int>((size_t)total.child_refs, &slab, many);
        int *d_leaf = lv.leaf.get<int>((size_t)total.leaf_refs, &slab);
        if (!d_nbox || !d_noff || !d_next || !d_leaf) { err = kNoMemory; return false; }
        k_emit<<<blocks(nl, 128), 128>>>(d_sums, d_tot, d_off, d_split, d_occ, d_sub, d_lbox, nl, leaf_total, next_base, d_box, d_child,
                                         d_fc, d_first, d_count, d_noff, d_nbox);
        if (nr > 0) k_leaf_refs<<<blocks(nr, 256), 256>>>(d_sums, d_tot, d_refs, d_owner, d_off, d_split, nr, d_leaf);
        if (next->nodes > 0)
            k_scatter<<<blocks(nl, kScatterWarps), 32 * kScatterWarps>>>(d_refs, d_mask, d_off, d_fc, d_noff, nl, d_next);
        leaf_total += total.leaf_refs;
        next_base += next->nodes;
        nr = (int)total.child_refs;
        b_refs.swap(b_next);
        d_refs = (int *)b_refs.p;
        b_off.swap(b_noff);
        if (next->nodes == 0) {
            out.depth = depth;
            break;
        }
        levels.push_back(std::move(next));
    }

    for (int depth = out.depth - 1; depth >= 0; depth--) {
        Level &lv = *levels[depth], &nx = *levels[depth + 1];
        k_reduce<<<blocks(lv.nodes, 128), 128>>>((float *)lv.box.p, (const int *)lv.child.p, lv.nodes, nx.base, (const float *)nx.box.p, E);
    }

    // the finished tree
    const int64_t nn = next_base;
    out.node_count = nn;
    out.node_lo.resize(3 * nn);
    out.node_hi.resize(3 * nn);
    out.node_child.resize(nn);
    out.node_leaf_first.resize(nn);
    out.node_leaf_count.resize(nn);
    out.leaf_refs.resize((size_t)leaf_total);
    DevBuf b_lo, b_hi, b_child, b_first, b_count, b_leaf;
    float *d_lo = b_lo.get<float>(3 * (size_t)nn), *d_hi = b_hi.get<float>(3 * (size_t)nn);
    int *d_child = b_child.get<int>((size_t)nn), *d_count = b_count.get<int>((size_t)nn);
    long long *d_first = b_first.get<long long>((size_t)nn);
    int *d_leaf = b_leaf.get<int>((size_t)leaf_total);
    if (!d_lo || !d_hi || !d_child || !d_count || !d_first || !d_leaf) { err = kNoMemory; return false; }
    cudaError_t e = cudaGetLastError();
    auto copy = [&](void *dst, const void *src, size_t bytes, cudaMemcpyKind kind) {
        if (e == cudaSuccess && bytes) e = cudaMemcpy(dst, src, bytes, kind);
    };
    for (size_t d = 0; d < levels.size(); d++) {
        const Level &lv = *levels[d];
        copy(d_leaf + lv.leaf_base, lv.leaf.p, 4 * (size_t)lv.leaf_refs, cudaMemcpyDeviceToDevice);
        if (d == 0) {
            float b[6];
            copy(b, lv.box.p, sizeof(b), cudaMemcpyDeviceToHost);
            copy(&out.root_child, lv.child.p, 4, cudaMemcpyDeviceToHost);
            copy(&out.root_leaf_count, lv.count.p, 4, cudaMemcpyDeviceToHost);
            for (int k = 0; k < 3; k++) { out.root_lo[k] = b[k]; out.root_hi[k] = b[3 + k]; }
            out.root_leaf_first = 0;
            continue;
        }
        k_finish<<<blocks(3LL * lv.nodes, 256), 256>>>((const float *)lv.box.p, lv.nodes, d_lo + 3 * (size_t)lv.base, d_hi + 3 * (size_t)lv.base);
        copy(d_child + lv.base, lv.child.p, 4 * (size_t)lv.nodes, cudaMemcpyDeviceToDevice);
        copy(d_first + lv.base, lv.first.p, 8 * (size_t)lv.nodes, cudaMemcpyDeviceToDevice);
        copy(d_count + lv.base, lv.count.p, 4 * (size_t)lv.nodes, cudaMemcpyDeviceToDevice);
    }
    if (e == cudaSuccess) e = cudaGetLastError();
    static_assert(sizeof(long long) == sizeof(int64_t), "leaf_first is copied as it is");
    copy(out.node_lo.data(), d_lo, 12 * (size_t)nn, cudaMemcpyDeviceToHost);
    copy(out.node_hi.data(), d_hi, 12 * (size_t)nn, cudaMemcpyDeviceToHost);
    copy(out.node_child.data(), d_child, 4 * (size_t)nn, cudaMemcpyDeviceToHost);
    copy(out.node_leaf_first.data(), d_first, 8 * (size_t)nn, cudaMemcpyDeviceToHost);
    copy(out.node_leaf_count.data(), d_count, 4 * (size_t)nn, cudaMemcpyDeviceToHost);
    copy(out.leaf_refs.data(), d_leaf, 4 * (size_t)leaf_total, cudaMemcpyDeviceToHost);
    if (e != cudaSuccess) {
        err = std::string("device build: ") + cudaGetErrorString(e);
        return false;
    }
    if (keep) {
        keep->xyz = (float *)b_xyz.release();
        keep->lo = (float *)b_lo.release();
        keep->hi = (float *)b_hi.release();
        keep->child = (int32_t *)b_child.release();
        keep->leaf_first = (long long *)b_first.release();
        keep->leaf_count = (int32_t *)b_count.release();
        keep->refs = (int32_t *)b_leaf.release();
    }
    return true;
}

}  // namespace

bool build_octree_gpu(const float *xyz, int64_t n, const BuildOptions &opt, FlatOctree &out, DeviceTree *keep, std::string &err) {
    if (build(xyz, n, opt, out, keep, err, false)) return true;
    if (err != kNoMemory) return false;
    // the slab and the buffers' reserves may be what there was no memory for
    (void)cudaGetLastError();
    err.clear();
    return build(xyz, n, opt, out, keep, err, true);
}

}  // namespace drb
