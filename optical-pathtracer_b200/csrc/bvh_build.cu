// Device construction of the 8-wide quantised BVH.
//
//  1. 63-bit Morton codes of the primitives' box centres (21 bits per axis in the centres' bounds),
//     the 64th bit set for a primitive larger than an eighth of the scene;
//  2. a radix sort of (code, primitive) pairs (CUB);
//  3. the binary radix tree over the sorted codes, one thread per inner node (Karras 2012), every
//     node covering a contiguous range of sorted primitives;
//  4. boxes and primitive counts bottom-up, the second child to finish computing its parent;
//  5. a top-down collapse into 8-wide nodes, level by level: each wide node opens the binary
//     subtree below it greedily by surface area until it has eight children; a child with at most
//     kLeafMax (two) primitives becomes a leaf slot, the others new wide nodes; children boxes are stored
//     as 8-bit offsets against the node's origin and per-axis power-of-two scales, rounded outward.
//     Children take the node's eight slots by direction: slot s (bit k set: negative along axis k)
//     goes to the child whose centre lies farthest along that octant's diagonal from the node's
//     centre (a greedy auction), so that a ray of octant o meets the children roughly in the order
//     of slot ^ o ^ 7, and the traversal orders its hits without a sort (Ylitie, Karras and Laine,
//     "Efficient incoherent ray traversal on GPUs through compressed wide BVHs", HPG 2017).
//
// This replaces the reference's host-side binned SAH builds (src/owe/scene/bvh.cpp:100-337) of the
// world hierarchy and of every mesh's own hierarchy with one hierarchy over all primitives.
#include <cub/device/device_radix_sort.cuh>

#include <algorithm>
#include <vector>

#include "bvh_build.hpp"

namespace owec {

namespace {

// Primitives a leaf slot may hold (at most 3: eight slots of three fill the traversal's 24-bit mask).
// Two: a ray tests fewer primitives per leaf it enters (2.98 instead of 5.43 per query on the
// 2^20-triangle room, with 3.94 node visits instead of 4.09), and the pass runs 8 % faster.
#ifndef OWEC_LEAF_MAX
#define OWEC_LEAF_MAX 2
#endif
constexpr uint32_t kLeafMax = OWEC_LEAF_MAX;
static_assert(kLeafMax >= 1 && kLeafMax <= 3, "a leaf slot holds one to three primitives");
// The size, against the scene's, from which a primitive counts as large (sorted after the others).
#ifndef OWEC_LARGE_PRIMITIVE
#define OWEC_LARGE_PRIMITIVE 0.125f
#endif
constexpr uint32_t kNoParent = 0xFFFFFFFFu;

__device__ __forceinline__ uint64_t spread21(uint64_t v) {
    v &= 0x1FFFFFull;
    v = (v | v << 32) & 0x1F00000000FFFFull;
    v = (v | v << 16) & 0x1F0000FF0000FFull;
    v = (v | v << 8) & 0x100F00F00F00F00Full;
    v = (v | v << 4) & 0x10C30C30C30C30C3ull;
    v = (v | v << 2) & 0x1249249249249249ull;
    return v;
}

// Order-preserving integer image of a float (and back), so integer atomics give float min / max.
__device__ __forceinline__ int floatToOrdered(float f) {
    const int i = __float_as_int(f);
    return i >= 0 ? i : i ^ 0x7FFFFFFF;
}

__global__ void kCentroidBounds(const float4* lo, const float4* hi, uint32_t n, int* bounds) {
    float mn[3] = {INFINITY, INFINITY, INFINITY}, mx[3] = {-INFINITY, -INFINITY, -INFINITY};
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const float4 a = lo[i], b = hi[i];
        const float c[3] = {0.5f * (a.x + b.x), 0.5f * (a.y + b.y), 0.5f * (a.z + b.z)};
        for (int k = 0; k < 3; ++k) { mn[k] = fminf(mn[k], c[k]); mx[k] = fmaxf(mx[k], c[k]); }
    }
    // one set of atomics per block: with one per warp the six addresses took most of the kernel's time
    __shared__ int part[6][8];
    for (int k = 0; k < 3; ++k) {
        const int l = __reduce_min_sync(0xFFFFFFFFu, floatToOrdered(mn[k]));
        const int h = __reduce_max_sync(0xFFFFFFFFu, floatToOrdered(mx[k]));
        if ((threadIdx.x & 31) == 0) {
            part[k][threadIdx.x >> 5] = l;
            part[3 + k][threadIdx.x >> 5] = h;
        }
    }
    __syncthreads();
    if (threadIdx.x < 6) {
        const int k = threadIdx.x, warps = int(blockDim.x >> 5);
        int v = part[k][0];
        for (int w = 1; w < warps; ++w) v = k < 3 ? min(v, part[k][w]) : max(v, part[k][w]);
        if (k < 3) atomicMin(bounds + k, v);
        else atomicMax(bounds + k, v);
    }
}

__device__ __forceinline__ float orderedToFloat(int v) { return __int_as_float(v >= 0 ? v : v ^ 0x7FFFFFFF); }

__global__ void kMorton(const float4* lo, const float4* hi, uint32_t n, const int* bounds, uint64_t* keys,
                        uint32_t* vals) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const int* bi = bounds;
    const float mn[3] = {orderedToFloat(bi[0]), orderedToFloat(bi[1]), orderedToFloat(bi[2])};
    const float mx[3] = {orderedToFloat(bi[3]), orderedToFloat(bi[4]), orderedToFloat(bi[5])};
    const float4 a = lo[i], b = hi[i];
    const float c[3] = {0.5f * (a.x + b.x), 0.5f * (a.y + b.y), 0.5f * (a.z + b.z)};
    const float size[3] = {b.x - a.x, b.y - a.y, b.z - a.z};
    uint64_t code = 0;
    float sceneExt = 0.f, primExt = 0.f;
    for (int k = 0; k < 3; ++k) {
        const float ext = mx[k] - mn[k];
        float u = ext > 0.f ? (c[k] - mn[k]) / ext : 0.5f;
        u = fminf(fmaxf(u, 0.f), 1.f);
        const uint64_t q = uint64_t(fminf(u * 2097152.0f, 2097151.0f));
        code |= spread21(q) << (2 - k);
        sceneExt = fmaxf(sceneExt, ext);
        primExt = fmaxf(primExt, size[k]);
    }
    // A primitive larger than an eighth of the scene (a wall, a floor, a lamp beside a finely
    // tessellated body) sorts after all the others: the tree's root split separates the two sets,
    // so no subtree of small primitives takes a wall's box.
    if (primExt > OWEC_LARGE_PRIMITIVE * sceneExt) code |= 1ull << 63;
    keys[i] = code;
    vals[i] = i;
}

__device__ __forceinline__ int commonPrefix(const uint64_t* k, int n, int i, int j) {
    if (j < 0 || j >= n) return -1;
    const uint64_t a = k[i], b = k[j];
    if (a == b) return 64 + __clz(uint32_t(i ^ j));
    return __clzll(a ^ b);
}

// Inner node i of the radix tree: children (combined index: inner 0..n-2, leaf k at n-1+k) and range.
__global__ void kRadixTree(const uint64_t* keys, int n, int2* children, int2* ranges, uint32_t* parents) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n - 1) return;
    const int d = commonPrefix(keys, n, i, i + 1) - commonPrefix(keys, n, i, i - 1) >= 0 ? 1 : -1;
    const int dmin = commonPrefix(keys, n, i, i - d);
    int lmax = 2;
    while (commonPrefix(keys, n, i, i + lmax * d) > dmin) lmax *= 2;
    int l = 0;
    for (int t = lmax / 2; t >= 1; t /= 2)
        if (commonPrefix(keys, n, i, i + (l + t) * d) > dmin) l += t;
    const int j = i + l * d;
    const int dnode = commonPrefix(keys, n, i, j);
    int s = 0;
    for (int div = 2;; div *= 2) {
        const int t = (l + div - 1) / div;
        if (commonPrefix(keys, n, i, i + (s + t) * d) > dnode) s += t;
        if (t <= 1) break;
    }
    const int gamma = i + s * d + min(d, 0);
    const int lo = min(i, j), hi = max(i, j);
    const int left = lo == gamma ? (n - 1 + gamma) : gamma;
    const int right = hi == gamma + 1 ? (n - 1 + gamma + 1) : gamma + 1;
    children[i] = make_int2(left, right);
    ranges[i] = make_int2(lo, hi);
    parents[left] = uint32_t(i);
    parents[right] = uint32_t(i);
}

__global__ void kBottomUp(const float4* primLo, const float4* primHi, const uint32_t* vals, int n,
                          const int2* children, const uint32_t* parents, float4* boxLo, float4* boxHi,
                          uint32_t* counts, uint32_t* flags) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= n) return;
    const int leaf = n - 1 + k;
    boxLo[leaf] = primLo[vals[k]];
    boxHi[leaf] = primHi[vals[k]];
    counts[leaf] = 1;
    __threadfence();
    uint32_t p = parents[leaf];
    for (int level = 0; p != kNoParent; ++level) {
        if (level > 4096 || p >= uint32_t(n - 1)) {  // a malformed tree: stop and report
            atomicAdd(&flags[n - 1 > 0 ? n - 1 : 0], 0x10000u);
            return;
        }
        if (atomicAdd(&flags[p], 1u) == 0) return;  // the sibling finishes this parent
        __threadfence();
        const int2 c = children[p];
        const float4 la = __ldcg(boxLo + c.x), lb = __ldcg(boxLo + c.y);
        const float4 ha = __ldcg(boxHi + c.x), hb = __ldcg(boxHi + c.y);
        boxLo[p] = make_float4(fminf(la.x, lb.x), fminf(la.y, lb.y), fminf(la.z, lb.z), 0.f);
        boxHi[p] = make_float4(fmaxf(ha.x, hb.x), fmaxf(ha.y, hb.y), fmaxf(ha.z, hb.z), 0.f);
        counts[p] = __ldcg(counts + c.x) + __ldcg(counts + c.y);
        __threadfence();
        p = parents[p];
    }
}

__device__ __forceinline__ float halfArea(float4 lo, float4 hi) {
    const float x = hi.x - lo.x, y = hi.y - lo.y, z = hi.z - lo.z;
    return x * y + y * z + z * x;
}

// Smallest power-of-two scale (as a biased exponent byte) whose 254 steps cover ext (one step of
// slack for the rounding of ext / 254).
__device__ __forceinline__ uint32_t scaleExponent(float ext) {
    const float s = ext / 254.0f;
    if (!(s > 0.f)) return 1u;
    int e;
    const float m = frexpf(s, &e);  // s = m * 2^e, m in [0.5, 1)
    int biased = (m == 0.5f ? e - 1 : e) + 127;
    if (biased < 1) biased = 1;
    if (biased > 254) biased = 254;
    return uint32_t(biased);
}

// The build's counters: [0] wide nodes allocated, [1] primitives placed, [2 + level] the wide nodes of
// a level still to be made from their binary nodes.
constexpr uint32_t kMaxLevels = 4096;
constexpr uint32_t kCounters = 2 + kMaxLevels + 2;

struct CollapseArgs {
    const int2* children;
    const int2* ranges;
    const float4* boxLo;
    const float4* boxHi;
    const uint32_t* counts;
    const uint32_t* vals;
    const uint32_t* errors;  // kBottomUp's report: nothing is collapsed from a malformed tree
    int n;
    WideNode* nodes;
    uint32_t* leafOrder;
    uint32_t* counters;
};

// Sets what the build's kernels start from: the empty bounds, the counters and the root's work item.
__global__ void kBeginBuild(int* bounds, uint32_t* counters, uint2* work) {
    for (uint32_t i = threadIdx.x; i < kCounters; i += blockDim.x) counters[i] = i == 0 || i == 2 ? 1u : 0u;
    if (threadIdx.x < 6) bounds[threadIdx.x] = threadIdx.x < 3 ? 0x7F800000 : int(0x807FFFFFu);  // +inf, -inf
    // the binary root: inner node 0, or with one primitive its leaf (combined index n - 1 = 0)
    if (threadIdx.x == 0) work[0] = make_uint2(0u, 0u);
}

// One level of wide nodes, eight lanes to a node, a lane to a child. The widest levels hold n / 8 nodes
// and the first ones 1, 8, 64: with one thread per node a level lasted as long as its node's chain of
// dependent loads, eight openings and the 8 x 8 auction from local memory (about 50 us), whatever its
// width. The level's node count is read on the device, so the host queues levels without waiting.
// owec_set_heightfield of a 256 x 256 heightfield (262,141 primitives in the scene): 9.80 -> 0.56 ms with
// kDeformHeightfield; the seven levels alone were 0.40 ms of kernel time and a host round trip each.
__global__ void __launch_bounds__(128) kCollapse(CollapseArgs a, int level, const uint2* work, uint2* next) {
    // work: the (binary node, wide node) pairs of this level, next: those of the one below
    const uint32_t nWork = *a.errors >= 0x10000u ? 0u : a.counters[2 + level];
    const int n = a.n;
    const uint32_t lane = threadIdx.x & 7u;
    const uint32_t group = 0xFFu << (threadIdx.x & 24u);  // the node's eight lanes
    const int lead = int(threadIdx.x & 24u);              // their first lane
    for (uint32_t w = (blockIdx.x * blockDim.x + threadIdx.x) >> 3; w < nWork; w += (gridDim.x * blockDim.x) >> 3) {
        const uint2 item = work[w];
        int c = -1;  // this lane's child
        int nc;
        if (int(item.x) >= n - 1) {  // a single-leaf root
            if (lane == 0) c = int(item.x);
            nc = 1;
        } else {
            const int2 ch = a.children[item.x];
            if (lane < 2) c = lane == 0 ? ch.x : ch.y;
            nc = 2;
        }
        float4 l = make_float4(INFINITY, INFINITY, INFINITY, 0.f), h = make_float4(-INFINITY, -INFINITY, -INFINITY, 0.f);
        uint32_t cnt = 0;
        if (c >= 0) { l = a.boxLo[c]; h = a.boxHi[c]; cnt = a.counts[c]; }
        // open the largest openable child (the first of equals) until there are eight
        while (nc < 8) {
            float area = c >= 0 && c < n - 1 && cnt > kLeafMax ? halfArea(l, h) : -1.f;
            if (!(area > -1.f)) area = -1.f;
            float best = area;
            for (int off = 4; off > 0; off >>= 1) best = fmaxf(best, __shfl_xor_sync(group, best, off));
            if (!(best > -1.f)) break;
            const int src = __ffs(__ballot_sync(group, area == best) & group) - 1;
            const int2 ch = a.children[__shfl_sync(group, c, src)];
            if (int(threadIdx.x & 31u) == src) c = ch.x;
            else if (int(lane) == nc) c = ch.y;
            if (int(threadIdx.x & 31u) == src || int(lane) == nc) { l = a.boxLo[c]; h = a.boxHi[c]; cnt = a.counts[c]; }
            ++nc;
        }
        float4 lo = l, hi = h;
        for (int off = 4; off > 0; off >>= 1) {
            lo.x = fminf(lo.x, __shfl_xor_sync(group, lo.x, off));
            lo.y = fminf(lo.y, __shfl_xor_sync(group, lo.y, off));
            lo.z = fminf(lo.z, __shfl_xor_sync(group, lo.z, off));
            hi.x = fmaxf(hi.x, __shfl_xor_sync(group, hi.x, off));
            hi.y = fmaxf(hi.y, __shfl_xor_sync(group, hi.y, off));
            hi.z = fmaxf(hi.z, __shfl_xor_sync(group, hi.z, off));
        }
        // slot auction: repeatedly give the free slot and unplaced child with the largest projection of
        // the child's centre (relative to the node's) on the slot's octant diagonal to each other; of
        // equals the first child, then the first slot
        const float px = 0.5f * (lo.x + hi.x), py = 0.5f * (lo.y + hi.y), pz = 0.5f * (lo.z + hi.z);
        const float cx = 0.5f * (l.x + h.x) - px, cy = 0.5f * (l.y + h.y) - py, cz = 0.5f * (l.z + h.z) - pz;
        int slot = -1;
        uint32_t taken = 0;
        for (int round = 0; round < nc; ++round) {
            int bk = -1;
            float bc = -INFINITY;
            if (c >= 0 && slot < 0) {
#pragma unroll
                for (int k = 0; k < 8; ++k) {
                    const float cost = ((k & 1) ? -cx : cx) + ((k & 2) ? -cy : cy) + ((k & 4) ? -cz : cz);
                    if (!(taken >> k & 1u) && (bk < 0 || cost > bc)) { bc = cost; bk = k; }
                }
                if (!(bc > -INFINITY)) bc = -INFINITY;
            }
            float best = bc;
            for (int off = 4; off > 0; off >>= 1) best = fmaxf(best, __shfl_xor_sync(group, best, off));
            const int src = __ffs(__ballot_sync(group, bk >= 0 && bc == best) & group) - 1;
            const int k = __shfl_sync(group, bk, src);
            if (int(threadIdx.x & 31u) == src) slot = k;
            taken |= 1u << k;
        }
        // the lanes without a child take the empty slots in order: a lane to a slot from here on
        if (c < 0) {
            uint32_t empty = ~taken & 0xFFu;
            for (int k = nc; k < int(lane); ++k) empty &= empty - 1u;
            slot = __ffs(empty) - 1;
        }
        const bool inner = c >= 0 && cnt > kLeafMax;
        const uint32_t leafCnt = c >= 0 && !inner ? cnt : 0u;
        const uint32_t imask = __reduce_or_sync(group, inner ? 1u << slot : 0u);
        const uint32_t leafCounts = __reduce_or_sync(group, leafCnt << (4 * slot));  // by slot
        const uint32_t nInner = uint32_t(__popc(imask)), nLeafPrims = __reduce_add_sync(group, leafCnt);
        // inner children are stored in slot order, so that the k-th inner slot's node is child_base + k
        const uint32_t innerK = uint32_t(__popc(imask & ((1u << slot) - 1u)));
        uint32_t leafOff = 0;
        for (int k = 0; k < slot; ++k) leafOff += (leafCounts >> (4 * k)) & 15u;
        uint32_t childBase = 0, primBase = 0, nextBase = 0;
        if (lane == 0) {
            if (nInner) {
                childBase = atomicAdd(&a.counters[0], nInner);
                nextBase = atomicAdd(&a.counters[2 + level + 1], nInner);
            }
            if (nLeafPrims) primBase = atomicAdd(&a.counters[1], nLeafPrims);
        }
        childBase = __shfl_sync(group, childBase, lead);
        primBase = __shfl_sync(group, primBase, lead);
        nextBase = __shfl_sync(group, nextBase, lead);
        const uint32_t ex = scaleExponent(hi.x - lo.x), ey = scaleExponent(hi.y - lo.y), ez = scaleExponent(hi.z - lo.z);
        const float sx = __uint_as_float(ex << 23), sy = __uint_as_float(ey << 23), sz = __uint_as_float(ez << 23);
        auto qlo = [](float v, float o, float s) {
            return uint8_t(fminf(fmaxf(floorf(__fsub_rd(v, o) / s), 0.f), 255.f));
        };
        auto qhi = [](float v, float o, float s) {
            return uint8_t(fminf(fmaxf(ceilf(__fsub_ru(v, o) / s), 0.f), 255.f));
        };
        WideNode& nd = a.nodes[item.y];
        if (lane == 0) {
            nd.ox = lo.x;
            nd.oy = lo.y;
            nd.oz = lo.z;
            nd.ex = uint8_t(ex);
            nd.ey = uint8_t(ey);
            nd.ez = uint8_t(ez);
            nd.imask = uint8_t(imask);
            nd.child_base = childBase;
            nd.prim_base = primBase;
        }
        if (c < 0) {  // an empty slot's box is inverted: no ray passes it
            nd.meta[slot] = 0;
            nd.qlox[slot] = nd.qloy[slot] = nd.qloz[slot] = 255;
            nd.qhix[slot] = nd.qhiy[slot] = nd.qhiz[slot] = 0;
        } else {
            nd.qlox[slot] = qlo(l.x, lo.x, sx);
            nd.qloy[slot] = qlo(l.y, lo.y, sy);
            nd.qloz[slot] = qlo(l.z, lo.z, sz);
            nd.qhix[slot] = qhi(h.x, lo.x, sx);
            nd.qhiy[slot] = qhi(h.y, lo.y, sy);
            nd.qhiz[slot] = qhi(h.z, lo.z, sz);
            if (inner) {
                nd.meta[slot] = uint8_t(8u | innerK);
                next[nextBase + innerK] = make_uint2(uint32_t(c), childBase + innerK);
            } else {
                nd.meta[slot] = uint8_t((cnt << 5) | leafOff);
                const int first = c >= n - 1 ? c - (n - 1) : a.ranges[c].x;
                for (uint32_t k = 0; k < cnt; ++k) a.leafOrder[primBase + leafOff + k] = a.vals[first + k];
            }
        }
    }
}

// ------------------------------------------------------------------ deformed heightfields
// One triangle of a heightfield whose vertices moved to z = baseZ + height: its FP64 and FP32 vertices
// and its padded box, as the scene upload computes them on the host, operation by operation (no
// contraction), so that a heightfield set on the device is the mesh uploaded with those heights.
__device__ __forceinline__ double frameRow(const double* m, double x, double y, double z) {
    return __dadd_rn(__dadd_rn(__dadd_rn(__dmul_rn(m[0], x), __dmul_rn(m[1], y)), __dmul_rn(m[2], z)), m[3]);
}
// Bound by its 152 bytes written a triangle; the host's loop over them and four copies, with every
// triangle of the scene uploaded again in FP64, were most of owec_set_heightfield's 9.80 ms (kCollapse).
__global__ void __launch_bounds__(128) kDeformHeightfield(HeightfieldMesh m, const double* heights, float4* tri,
                                                          double* tri64, float4* primLo, float4* primHi) {
    const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= m.nTriangles) return;
    double w[3][3];
    float f[3][3];
    for (int k = 0; k < 3; ++k) {
        const uint32_t v = m.tris[3 * size_t(t) + k];
        const double x = m.verts[3 * size_t(v)], y = m.verts[3 * size_t(v) + 1], z = __dadd_rn(m.baseZ, heights[v]);
        for (int a = 0; a < 3; ++a) {
            w[k][a] = frameRow(m.toWorld.m + 4 * a, x, y, z);
            f[k][a] = float(w[k][a]);
        }
    }
    const size_t p = size_t(m.firstPrim) + t;
    const uint32_t ids[3] = {m.boundary, t, kPrimTriangle};
    double lo[3], hi[3], ext = 0, mag = 0;
    for (int k = 0; k < 3; ++k) {
        tri[3 * p + k] = make_float4(f[k][0], f[k][1], f[k][2], __uint_as_float(ids[k]));
        for (int a = 0; a < 3; ++a) tri64[9 * p + 3 * k + a] = w[k][a];
    }
    for (int a = 0; a < 3; ++a) {
        const double v[6] = {f[0][a], f[1][a], f[2][a], w[0][a], w[1][a], w[2][a]};
        lo[a] = hi[a] = v[0];
        for (int k = 1; k < 6; ++k) {
            if (v[k] < lo[a]) lo[a] = v[k];
            if (hi[a] < v[k]) hi[a] = v[k];
        }
        const double e = __dadd_rn(hi[a], -lo[a]);
        if (ext < e) ext = e;
        if (mag < fabs(lo[a])) mag = fabs(lo[a]);
        if (mag < fabs(hi[a])) mag = fabs(hi[a]);
    }
    const double pad = __dadd_rn(__dmul_rn(1e-6, __dadd_rn(mag, ext)), 1e-9);
    float bl[3], bh[3];
    for (int a = 0; a < 3; ++a) {
        bl[a] = nextafterf(float(__dadd_rn(lo[a], -pad)), -INFINITY);
        bh[a] = nextafterf(float(__dadd_rn(hi[a], pad)), INFINITY);
    }
    primLo[p] = make_float4(bl[0], bl[1], bl[2], 0.f);
    primHi[p] = make_float4(bh[0], bh[1], bh[2], 0.f);
}

}  // namespace

void launchDeformHeightfield(const HeightfieldMesh& m, const double* heights, float4* tri, double* tri64, float4* primLo,
                             float4* primHi, cudaStream_t s) {
    if (m.nTriangles == 0) return;
    kDeformHeightfield<<<(m.nTriangles + 127) / 128, 128, 0, s>>>(m, heights, tri, tri64, primLo, primHi);
}

uint32_t buildWideBvh(const float4* primLo, const float4* primHi, uint32_t n, BvhScratch& s, DBuf<WideNode>& nodes,
                      DBuf<uint32_t>& leafOrder, cudaStream_t stream) {
    if (n == 0) return 0;
    const uint32_t nAll = 2 * n - 1;
    s.keys.reserve(n);
    s.keysAlt.reserve(n);
    s.vals.reserve(n);
    s.valsAlt.reserve(n);
    s.children.reserve(n);
    s.ranges.reserve(n);
    s.parents.reserve(nAll);
    s.boxLo.reserve(nAll);
    s.boxHi.reserve(nAll);
    s.counts.reserve(nAll);
    s.flags.reserve(n);
    s.work.reserve(n);
    s.next.reserve(n);
    s.counters.reserve(kCounters);
    s.bounds.reserve(8);
    nodes.reserve(std::max<uint32_t>(1, n));
    leafOrder.reserve(n);

    kBeginBuild<<<1, 256, 0, stream>>>(s.bounds.get(), s.counters.get(), s.work.get());
    const int T = 256;
    kCentroidBounds<<<std::min<uint32_t>((n + T - 1) / T, 1184), T, 0, stream>>>(primLo, primHi, n, s.bounds.get());
    kMorton<<<(n + T - 1) / T, T, 0, stream>>>(primLo, primHi, n, s.bounds.get(), s.keys.get(), s.vals.get());
    size_t tempBytes = 0;
    cub::DoubleBuffer<uint64_t> dk(s.keys.get(), s.keysAlt.get());
    cub::DoubleBuffer<uint32_t> dv(s.vals.get(), s.valsAlt.get());
    OWEC_CUDA(cub::DeviceRadixSort::SortPairs(nullptr, tempBytes, dk, dv, int(n), 0, 64, stream));
    s.cubTemp.reserve(tempBytes);
    OWEC_CUDA(cub::DeviceRadixSort::SortPairs(s.cubTemp.get(), tempBytes, dk, dv, int(n), 0, 64, stream));
    const uint64_t* keys = dk.Current();
    const uint32_t* vals = dv.Current();

    OWEC_CUDA(cudaMemsetAsync(s.parents.get(), 0xFF, nAll * sizeof(uint32_t), stream));
    OWEC_CUDA(cudaMemsetAsync(s.flags.get(), 0, n * sizeof(uint32_t), stream));
    if (n > 1)
        kRadixTree<<<(n - 1 + T - 1) / T, T, 0, stream>>>(keys, int(n), s.children.get(), s.ranges.get(),
                                                           s.parents.get());
    kBottomUp<<<(n + T - 1) / T, T, 0, stream>>>(primLo, primHi, vals, int(n), s.children.get(), s.parents.get(),
                                                  s.boxLo.get(), s.boxHi.get(), s.counts.get(), s.flags.get());

    CollapseArgs a{s.children.get(), s.ranges.get(), s.boxLo.get(), s.boxHi.get(), s.counts.get(), vals,
                   s.flags.get() + (n - 1),  // no inner node's: it collects malformed-tree reports
                   int(n), nodes.get(), leafOrder.get(), s.counters.get()};
    uint2 *work = s.work.get(), *next = s.next.get();
    // Levels are queued a batch at a time, a tree of full nodes' depth and a few more first, and the host
    // looks at the counters once per batch: a level past the last one finds no work.
    int batch = 4;
    for (uint64_t full = 1; full < n; full *= 8) ++batch;
    uint64_t width = 1;  // nodes the level can hold
    for (int level = 0;;) {
        for (int k = 0; k < batch; ++k, ++level) {
            const uint64_t items = std::min<uint64_t>(width, n);
            kCollapse<<<int(std::min<uint64_t>((items * 8 + 127) / 128, 2368)), 128, 0, stream>>>(a, level, work, next);
            std::swap(work, next);
            width = std::min<uint64_t>(width * 8, n);
        }
        std::vector<uint32_t> h(3 + level);
        uint32_t err = 0;
        OWEC_CUDA(cudaMemcpyAsync(h.data(), s.counters.get(), h.size() * sizeof(uint32_t), cudaMemcpyDeviceToHost, stream));
        OWEC_CUDA(cudaMemcpyAsync(&err, s.flags.get() + (n - 1), sizeof(err), cudaMemcpyDeviceToHost, stream));
        OWEC_CUDA(cudaStreamSynchronize(stream));
        if (err >= 0x10000u) throw std::runtime_error("BVH build: malformed radix tree");
        s.nodeCount = h[0];
        s.placedPrims = h[1];
        if (h[2 + level] == 0) {
            s.levels = uint32_t(std::find(h.begin() + 2, h.end(), 0u) - (h.begin() + 2));
            break;
        }
        if (level + batch > int(kMaxLevels)) throw std::runtime_error("BVH collapse did not terminate");
    }
    if (s.placedPrims != n) throw std::runtime_error("BVH collapse placed " + std::to_string(s.placedPrims) +
                                                     " of " + std::to_string(n) + " primitives");
    return s.nodeCount;
}

}  // namespace owec
