// bvh.cu -- device build of the compressed 8-wide BVH.
//
// Replaces the reference's serial binary SAH build (accelerators/bvh.cc:150-237,
// BVHAccel::constructRec) with a data-parallel one on the GPU:
//   1. per-triangle bounds and centroid bounds              (k_prim_bounds)
//   2. 63-bit Morton codes of the centroids under a large-triangle bit, radix sort
//                                                            (k_morton + cub)
//   3. binary tree by parallel locally-ordered clustering   (k_leaf_bounds, k_ploc_*)
//      -- Meister and Bittner, "Parallel Locally-Ordered Clustering for Bounding
//         Volume Hierarchy Construction" (IEEE TVCG 2018): clusters start as the
//         triangles in code order; each round every cluster finds the neighbour
//         within kPlocRadius positions whose merged box has the least surface area,
//         mutual nearest neighbours merge into a new node, and the clusters are
//         compacted in order, until one is left
//   4. SAH-optimal choice of the wide tree, bottom-up over the clustering rounds
//      (dpNode, with each round's new nodes) -- the dynamic programme of Ylitie, Karras and Laine,
//      "Efficient Incoherent Ray Traversal on GPUs Through Compressed Wide BVHs"
//      (HPG 2017): for every binary node, the least SAH cost of spreading 1..8
//      child slots over its subtree, where a node is a leaf (at most 3 triangles),
//      a wide node, or passes slots on to its two children
//   5. top-down collapse into 8-wide nodes, level by level  (k_collapse),
//      following those decisions
//      Children are placed in slots by a greedy octant assignment so that the
//      traversal's slot order s ^ (7 - octant) runs roughly front to back, their
//      boxes are quantised conservatively to 8 bits on the node's grid, and leaf
//      triangles are copied into leaf order as (v0, v1, v2) records.
// The triangle set, and so the closest hit of every ray, is the reference's; only
// the tree differs.  Its build is deterministic (no atomics decide structure).
//
// A build was bound by what surrounds its kernels: some 75 clustering rounds of eight launches
// and a host round trip each, 30 allocations, and one thread per wide node in the collapse.  With
// rounds that run ahead of the host, the last rounds in one block, one scratch allocation and
// eight threads per wide node, 2.03M triangles take 11.4 -> 2.9 ms, 256 triangles 1.96 -> 0.28.
#include <cub/device/device_radix_sort.cuh>

#include <algorithm>
#include <cstdio>

#include "bvh.cuh"

namespace spgpu {

namespace {

constexpr int kLeafMax = 3;   // triangles a wide-node leaf may hold

__device__ __forceinline__ void atomicMinFloat(float *a, float v) {
    if (v >= 0.0f) atomicMin(reinterpret_cast<int *>(a), __float_as_int(v));
    else atomicMax(reinterpret_cast<unsigned int *>(a), __float_as_uint(v));
}
__device__ __forceinline__ void atomicMaxFloat(float *a, float v) {
    if (v >= 0.0f) atomicMax(reinterpret_cast<int *>(a), __float_as_int(v));
    else atomicMin(reinterpret_cast<unsigned int *>(a), __float_as_uint(v));
}

// scene bounds [0..5] and centroid bounds [6..11]
constexpr int kBoundsBlock = 256;
__global__ void __launch_bounds__(kBoundsBlock) k_prim_bounds(const float *__restrict__ verts, int n, float *__restrict__ bounds) {
    float lo[6], hi[6];
    for (int k = 0; k < 6; k++) {
        lo[k] = 3.0e38f;
        hi[k] = -3.0e38f;
    }
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const float *v = verts + 9 * static_cast<int64_t>(i);
        for (int a = 0; a < 3; a++) {
            const float mn = fminf(v[a], fminf(v[3 + a], v[6 + a]));
            const float mx = fmaxf(v[a], fmaxf(v[3 + a], v[6 + a]));
            lo[a] = fminf(lo[a], mn);
            hi[a] = fmaxf(hi[a], mx);
            const float c = 0.5f * (mn + mx);
            lo[3 + a] = fminf(lo[3 + a], c);
            hi[3 + a] = fmaxf(hi[3 + a], c);
        }
    }
    for (int k = 0; k < 6; k++) {
        for (int off = 16; off > 0; off >>= 1) {
            lo[k] = fminf(lo[k], __shfl_xor_sync(0xffffffffu, lo[k], off));
            hi[k] = fmaxf(hi[k], __shfl_xor_sync(0xffffffffu, hi[k], off));
        }
    }
    // one update of the twelve bounds per block: all warps' updates of the same words would queue
    __shared__ float part[kBoundsBlock / 32][12];
    const int warp = threadIdx.x >> 5;
    if ((threadIdx.x & 31) == 0)
        for (int k = 0; k < 6; k++) {
            part[warp][k] = lo[k];
            part[warp][6 + k] = hi[k];
        }
    __syncthreads();
    if (threadIdx.x < 12) {
        const int k = threadIdx.x;
        float v = part[0][k];
        for (int w = 1; w < kBoundsBlock / 32; w++) v = k < 6 ? fminf(v, part[w][k]) : fmaxf(v, part[w][k]);
        // lo[0..2], lo[3..5] (centroids), hi[0..2], hi[3..5] go to 0..2, 6..8, 3..5, 9..11
        const int at = (k % 6) % 3 + 3 * (k / 6) + 6 * ((k % 6) / 3);
        if (k < 6) atomicMinFloat(&bounds[at], v);
        else atomicMaxFloat(&bounds[at], v);
    }
}

__device__ __forceinline__ uint64_t spread21(uint32_t x) {
    uint64_t v = x & 0x1FFFFFu;
    v = (v | (v << 32)) & 0x1F00000000FFFFull;
    v = (v | (v << 16)) & 0x1F0000FF0000FFull;
    v = (v | (v << 8)) & 0x100F00F00F00F00Full;
    v = (v | (v << 4)) & 0x10C30C30C30C30C3ull;
    v = (v | (v << 2)) & 0x1249249249249249ull;
    return v;
}

// Sort key: bit 63 marks a large triangle (box diagonal above 1/8 of the scene's), bits
// 0-62 are the 63-bit Morton code of its box centre.  The size bit is the extended
// Morton code idea of Vinkler, Bittner and Havran ("Extended Morton codes for high
// performance bounding volume hierarchy construction", HPG 2017) reduced to one class:
// large triangles (a floor quad, room walls) sort after all others, so the clustering,
// which merges only within a window of this order, joins them with each other first and
// with the rest near the root, instead of leaving them deep among small ones where every
// ancestor's box would span them.
constexpr float kLargeTriangle = 1.0f / 8.0f;

__global__ void k_morton(const float *__restrict__ verts, int n, const float *__restrict__ bounds,
                         uint64_t *__restrict__ keys, uint32_t *__restrict__ vals) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float *v = verts + 9 * static_cast<int64_t>(i);
    uint32_t q[3];
    float d2 = 0.0f, s2 = 0.0f;
    for (int a = 0; a < 3; a++) {
        const float mn = fminf(v[a], fminf(v[3 + a], v[6 + a])), mx = fmaxf(v[a], fmaxf(v[3 + a], v[6 + a]));
        const float c = 0.5f * (mn + mx);
        const float lo = bounds[6 + a], ext = bounds[9 + a] - bounds[6 + a];
        const float u = ext > 0.0f ? (c - lo) / ext : 0.5f;
        q[a] = static_cast<uint32_t>(fminf(fmaxf(u * 2097152.0f, 0.0f), 2097151.0f));
        d2 += (mx - mn) * (mx - mn);
        s2 += (bounds[3 + a] - bounds[a]) * (bounds[3 + a] - bounds[a]);
    }
    const uint64_t large = d2 > kLargeTriangle * kLargeTriangle * s2 ? 1ull << 63 : 0ull;
    keys[i] = large | (spread21(q[0]) << 2) | (spread21(q[1]) << 1) | spread21(q[2]);
    vals[i] = static_cast<uint32_t>(i);
}

__device__ __forceinline__ float areaOf(float4 lo, float4 hi) {
    const float dx = hi.x - lo.x, dy = hi.y - lo.y, dz = hi.z - lo.z;
    return 2.0f * (dx * dy + dy * dz + dz * dx);
}

// ---------------------------------------------------------------- clustering
constexpr int kPlocRadius = 32;   // neighbours searched on each side, in code order
constexpr int kPlocBlock = 256;   // clusters of a block of k_ploc_nn

// leaves: node n-1+j is the j-th triangle in code order
// SAH weights of the wide tree: a wide-node visit, a triangle test.  Equal weights were
// measured best for this traversal (triangle weight 0.3 / 0.6 / 1.0 / 1.5: 884 / 892 /
// 900 / 887 M path samples/s on the 1080p render; the 1M-triangle microbench also peaks
// at 1.0)
constexpr float kCostNode = 1.0f, kCostTri = 1.0f;

// per inner binary node (ids 0..n-2): cost[8 * node + j - 1] = least SAH cost of its subtree
// over j child slots; split[8 * node + j - 1] = slots given to the left child (0: the node
// itself takes one slot); split of j = 8 before that choice is the node's own split as a wide
// node (wideSplit); leaf[node]: the node itself is cheaper as a leaf than as a wide node.  A
// triangle (ids n-1..) costs the same over any number of slots, which its box gives.
struct DpArgs {
    float *cost;
    uint8_t *split;
    uint8_t *wideSplit;
    uint8_t *leaf;
};

__global__ void k_leaf_bounds(const float *__restrict__ verts, const uint32_t *__restrict__ order, int n,
                              float4 *bmin, float4 *bmax, int *count, int *clusters) {
    const int j = blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= n) return;
    const float *v = verts + 9 * static_cast<int64_t>(order[j]);
    const int node = n - 1 + j;
    bmin[node] = make_float4(fminf(v[0], fminf(v[3], v[6])), fminf(v[1], fminf(v[4], v[7])),
                             fminf(v[2], fminf(v[5], v[8])), 0.0f);
    bmax[node] = make_float4(fmaxf(v[0], fmaxf(v[3], v[6])), fmaxf(v[1], fmaxf(v[4], v[7])),
                             fmaxf(v[2], fmaxf(v[5], v[8])), 0.0f);
    count[node] = 1;
    clusters[j] = node;
}

// The clustering runs ahead of the host: round r reads its cluster count m and the next free
// node id top from rounds[r] and leaves the next round's in rounds[r + 1], so the host launches
// kRoundsAhead rounds, sized by the last count it knows, between two looks.  From kTailClusters
// clusters on, one block does the rest (k_ploc_tail): with 4096 / 2048 / 1024 / 512 of them the
// 2M-triangle build takes 3.50 / 3.48 / 3.47 / 3.60 ms, 16k triangles 1.12 / 1.08 / 1.10 / 1.16.
// A round is three kernels of a few microseconds, so they are dependent launches: each is set up
// while the one before it runs, and waits for it before its first access.  A round's SAH
// programme runs beside the next round's counting (and the last round's in k_ploc_tail).  Both
// together, and the collapse's levels as dependent launches: 2M triangles 3.53 -> 3.16 ms, 16k
// 1.09 -> 0.98 ms.
struct RoundState {
    int m, top;
};
constexpr int kRoundsAhead = 8;   // 4 / 6 / 8: 2M triangles 3.18 / 3.12 / 3.08 ms, 16k 0.98 / 0.95 / 0.97
constexpr int kMaxRounds = 1024;
constexpr int kTailClusters = 2048;
constexpr int kMergeBlock = 1024;

// nearest neighbour of each cluster: least surface area of the merged box among the
// clusters within kPlocRadius positions (ties: the lower position); the window's boxes
// are staged in shared memory, and reading them from there is what bounds this.  So a thread
// takes two neighbouring clusters, whose windows share all but their ends, and each box read
// serves both; even and odd positions have their own arrays, so that the threads' reads, two
// positions apart, fall on different banks.  Beyond the first and last cluster the arrays hold
// boxes of infinite area.  2M triangles 3.05 -> 2.91 ms (2.95 / 3.00 / 3.02 unrolled by 11 / 3 /
// not at all), 256k 1.54 -> 1.49; blocks of 512 clusters 3.02.
__global__ void __launch_bounds__(kPlocBlock / 2) k_ploc_nn(const int *__restrict__ clusters,
                                                            const RoundState *__restrict__ round,
                                                            const float4 *__restrict__ bmin,
                                                            const float4 *__restrict__ bmax, int *nn) {
    constexpr int kSpan = kPlocBlock + 2 * kPlocRadius, kHalf = kPlocRadius / 2;
    static_assert(kPlocRadius % 2 == 0 && kPlocBlock % 2 == 0, "a thread's first cluster is at an even position");
    __shared__ float4 slo[2][kSpan / 2], shi[2][kSpan / 2];
    cudaGridDependencySynchronize();
    cudaTriggerProgrammaticLaunchCompletion();
    const int m = round->m;
    if (m <= kTailClusters || static_cast<int>(blockIdx.x) * kPlocBlock >= m) return;
    const int base = blockIdx.x * kPlocBlock - kPlocRadius;
    for (int k = threadIdx.x; k < kSpan; k += kPlocBlock / 2) {
        const int p = base + k;
        float4 lo = make_float4(-1e30f, -1e30f, -1e30f, 0.0f), hi = make_float4(1e30f, 1e30f, 1e30f, 0.0f);
        if (p >= 0 && p < m) {
            const int c = clusters[p];
            lo = bmin[c];
            hi = bmax[c];
        }
        slo[k & 1][k >> 1] = lo;
        shi[k & 1][k >> 1] = hi;
    }
    __syncthreads();
    const int i = blockIdx.x * kPlocBlock + 2 * static_cast<int>(threadIdx.x);   // and i + 1
    if (i >= m) return;
    const int own = threadIdx.x + kHalf;
    const float4 lo0 = slo[0][own], hi0 = shi[0][own], lo1 = slo[1][own], hi1 = shi[1][own];
    float best0 = 3.0e38f, best1 = 3.0e38f;
    int at0 = -1, at1 = -1;
    auto closer = [](const float4 &lo, const float4 &hi, const float4 &a, const float4 &b, int j, float *best, int *at) {
        const float area = areaOf(make_float4(fminf(lo.x, a.x), fminf(lo.y, a.y), fminf(lo.z, a.z), 0.0f),
                                  make_float4(fmaxf(hi.x, b.x), fmaxf(hi.y, b.y), fmaxf(hi.z, b.z), 0.0f));
        if (area < *best) {
            *best = area;
            *at = j;
        }
    };
#pragma unroll
    for (int e = -kHalf; e <= kHalf; e++) {   // positions i + 2 e and i + 2 e + 1
        const int j = i + 2 * e;
        const float4 a0 = slo[0][own + e], b0 = shi[0][own + e];
        if (e != 0) closer(lo0, hi0, a0, b0, j, &best0, &at0);
        if (e != -kHalf) closer(lo1, hi1, a0, b0, j, &best1, &at1);
        const float4 a1 = slo[1][own + e], b1 = shi[1][own + e];
        if (e != kHalf) closer(lo0, hi0, a1, b1, j + 1, &best0, &at0);
        if (e != 0) closer(lo1, hi1, a1, b1, j + 1, &best1, &at1);
    }
    nn[i] = at0;
    if (i + 1 < m) nn[i + 1] = at1;
}

// A cluster leads a merge when it and its neighbour chose each other and it comes first; it
// survives the round unless it is the second of such a pair.
__device__ __forceinline__ void mergeFlags(const int *nn, int i, int m, bool *lead, bool *keep) {
    const int j = i < m ? nn[i] : -1;
    const bool mutual = j >= 0 && nn[j] == i;
    *lead = mutual && i < j;
    *keep = i < m && !(mutual && i > j);
}
// exclusive counts of the block's flags before this thread (lead | keep << 16), and the block's
// totals; called by all threads of a block of kMergeBlock
__device__ __forceinline__ uint32_t countBefore(bool lead, bool keep, uint32_t *warpSum, uint32_t *total) {
    const unsigned lb = __ballot_sync(0xffffffffu, lead), kb = __ballot_sync(0xffffffffu, keep);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const unsigned below = (1u << lane) - 1u;
    if (lane == 0) warpSum[warp] = static_cast<uint32_t>(__popc(lb)) | static_cast<uint32_t>(__popc(kb)) << 16;
    __syncthreads();
    // every warp scans the warps' sums for itself
    const uint32_t mine = warpSum[lane];
    uint32_t sum = mine;
    for (int off = 1; off < 32; off <<= 1) {
        const uint32_t v = __shfl_up_sync(0xffffffffu, sum, off);
        if (lane >= off) sum += v;
    }
    *total = __shfl_sync(0xffffffffu, sum, 31);
    const uint32_t before = __shfl_sync(0xffffffffu, sum - mine, warp);
    return before + (static_cast<uint32_t>(__popc(lb & below)) | static_cast<uint32_t>(__popc(kb & below)) << 16);
}
static_assert(kMergeBlock == 1024, "32 warps, a lane for each in countBefore; counts of 16 bits");

// merged nodes take ids top - (leads before) (descending, so the last merge, the root, is node
// 0); survivors are compacted in order.  Each block adds up the counts of the blocks before it.
__global__ void __launch_bounds__(kMergeBlock) k_ploc_merge(const int *__restrict__ clusters, RoundState *round,
                                                            const int *__restrict__ nn,
                                                            const uint32_t *__restrict__ sums, int2 *child,
                                                            float4 *bmin, float4 *bmax, int *count, int *next) {
    __shared__ uint32_t warpSum[32];
    __shared__ int base[2];
    cudaGridDependencySynchronize();
    cudaTriggerProgrammaticLaunchCompletion();
    const int m = round->m, top = round->top;
    if (static_cast<int>(blockIdx.x) * kMergeBlock >= m) return;
    if (m <= kTailClusters) {   // nothing left for the rounds: clusters and state go on to the tail
        const int i = blockIdx.x * kMergeBlock + threadIdx.x;
        if (i < m) next[i] = clusters[i];
        if (i == 0) round[1] = round[0];
        return;
    }
    if (threadIdx.x < 2) base[threadIdx.x] = 0;
    __syncthreads();
    int lsum = 0, ksum = 0;
    for (int b = threadIdx.x; b < static_cast<int>(blockIdx.x); b += kMergeBlock) {
        lsum += sums[b] & 0xFFFFu;
        ksum += sums[b] >> 16;
    }
    for (int off = 16; off > 0; off >>= 1) {
        lsum += __shfl_xor_sync(0xffffffffu, lsum, off);
        ksum += __shfl_xor_sync(0xffffffffu, ksum, off);
    }
    if ((threadIdx.x & 31) == 0 && (lsum | ksum)) {
        atomicAdd(&base[0], lsum);
        atomicAdd(&base[1], ksum);
    }
    const int i = blockIdx.x * kMergeBlock + threadIdx.x;
    bool lead, keep;
    mergeFlags(nn, i, m, &lead, &keep);
    uint32_t total;
    const uint32_t before = countBefore(lead, keep, warpSum, &total);   // synchronises: base is complete
    if (threadIdx.x == 0 && (blockIdx.x + 1) * kMergeBlock >= static_cast<unsigned>(m)) {
        round[1].m = base[1] + static_cast<int>(total >> 16);
        round[1].top = top - base[0] - static_cast<int>(total & 0xFFFFu);
    }
    if (!keep) return;
    int node = clusters[i];
    if (lead) {
        const int a = node, b = clusters[nn[i]];
        const int id = top - base[0] - static_cast<int>(before & 0xFFFFu);
        child[id] = make_int2(a, b);
        const float4 a0 = bmin[a], a1 = bmax[a], b0 = bmin[b], b1 = bmax[b];
        bmin[id] = make_float4(fminf(a0.x, b0.x), fminf(a0.y, b0.y), fminf(a0.z, b0.z), 0.0f);
        bmax[id] = make_float4(fmaxf(a1.x, b1.x), fmaxf(a1.y, b1.y), fmaxf(a1.z, b1.z), 0.0f);
        count[id] = count[a] + count[b];
        node = id;
    }
    next[base[1] + static_cast<int>(before >> 16)] = node;
}

// the SAH programme of one node, from its children's (n: triangles of the scene)
__device__ __forceinline__ void dpNode(const DpArgs &D, int n, int id, int2 c, int triangles, float4 lo, float4 hi,
                                       const float4 *bmin, const float4 *bmax) {
    float CL[7], CR[7];
    auto load = [&](int x, float *C) {
        if (x >= n - 1) {
            const float4 l = bmin[x], h = bmax[x];
            const float2 dx = make_float2(h.x - l.x, h.y - l.y);
            const float v = kCostTri * 2.0f * (dx.x * dx.y + dx.y * (h.z - l.z) + (h.z - l.z) * dx.x);
#pragma unroll
            for (int k = 0; k < 7; k++) C[k] = v;
        } else {
            const float4 *p = reinterpret_cast<const float4 *>(D.cost + 8 * static_cast<int64_t>(x));
            const float4 a = p[0], b = p[1];
            C[0] = a.x;
            C[1] = a.y;
            C[2] = a.z;
            C[3] = a.w;
            C[4] = b.x;
            C[5] = b.y;
            C[6] = b.z;
        }
    };
    load(c.x, CL);
    load(c.y, CR);
    float S[9];
    uint8_t K[9];
    S[1] = 3.0e38f;
    K[1] = 0;
#pragma unroll
    for (int j = 2; j <= 8; j++) {
        float best = 3.0e38f;
        uint8_t bk = 1;
#pragma unroll
        for (int k = 1; k < j; k++) {
            const float v = CL[k - 1] + CR[j - k - 1];
            if (v < best) {
                best = v;
                bk = static_cast<uint8_t>(k);
            }
        }
        S[j] = best;
        K[j] = bk;
        if (j > 2 && S[j - 1] <= S[j]) {   // fewer slots may be cheaper: keep that split
            S[j] = S[j - 1];
            K[j] = K[j - 1];
        }
    }
    const float A = areaOf(lo, hi);
    const float cInternal = kCostNode * A + S[8];
    const float cLeaf = triangles <= kLeafMax ? kCostTri * A * static_cast<float>(triangles) : 3.0e38f;
    const bool asLeaf = cLeaf <= cInternal;
    const float C = asLeaf ? cLeaf : cInternal;
    float out[8];
    uint32_t sp[2] = {0u, 0u};
    out[0] = C;
#pragma unroll
    for (int j = 2; j <= 8; j++) {
        const bool self = C <= S[j];
        out[j - 1] = self ? C : S[j];
        if (!self) sp[(j - 1) >> 2] |= static_cast<uint32_t>(K[j]) << (8 * ((j - 1) & 3));
    }
    float4 *o = reinterpret_cast<float4 *>(D.cost + 8 * static_cast<int64_t>(id));
    o[0] = make_float4(out[0], out[1], out[2], out[3]);
    o[1] = make_float4(out[4], out[5], out[6], out[7]);
    reinterpret_cast<uint2 *>(D.split)[id] = make_uint2(sp[0], sp[1]);
    D.wideSplit[id] = K[8];
    D.leaf[id] = asLeaf ? 1 : 0;
}

// the SAH programme of the nodes that the round before this one merged (round[0].top < id <=
// round[-1].top; their children are from earlier rounds), thread by thread of stride threads
__device__ __forceinline__ void dpLastRound(const DpArgs &D, int n, const RoundState *round, int thread, int stride,
                                            const int2 *child, const int *count, const float4 *bmin,
                                            const float4 *bmax) {
    const int last = round[-1].top;
    for (int id = round[0].top + 1 + thread; id <= last; id += stride)
        dpNode(D, n, id, child[id], count[id], bmin[id], bmax[id], bmin, bmax);
}

// Leads and survivors of each block of kMergeBlock clusters, and beside them, in the launch's
// first dpBlocks blocks, the last round's SAH programme: both wait on memory most of the time,
// and apart they were 4 and 6 us a round of a 2M-triangle build, with a launch each.
__global__ void __launch_bounds__(kMergeBlock) k_ploc_count(const int *__restrict__ nn,
                                                            const RoundState *__restrict__ round, uint32_t *sums,
                                                            int dpBlocks, const int2 *__restrict__ child,
                                                            const int *__restrict__ count,
                                                            const float4 *__restrict__ bmin,
                                                            const float4 *__restrict__ bmax, int n, DpArgs D) {
    __shared__ uint32_t warpSum[32];
    cudaGridDependencySynchronize();
    cudaTriggerProgrammaticLaunchCompletion();
    const int block = static_cast<int>(blockIdx.x) - dpBlocks;
    if (block < 0) {
        dpLastRound(D, n, round, blockIdx.x * kMergeBlock + threadIdx.x, dpBlocks * kMergeBlock, child, count, bmin, bmax);
        return;
    }
    const int m = round->m;
    if (m <= kTailClusters || block * kMergeBlock >= m) return;
    bool lead, keep;
    mergeFlags(nn, block * kMergeBlock + threadIdx.x, m, &lead, &keep);
    uint32_t total;
    countBefore(lead, keep, warpSum, &total);
    if (threadIdx.x == 0) sums[block] = total;
}

// The clustering's last rounds, with their SAH programme, in one block: at most kTailClusters
// clusters, whose boxes stay in shared memory.  A round of a few thousand clusters is too little
// for the chip and its launches cost more than its work; there are some forty of them.
// state: in, the clusters and next free id; out, what is left (one cluster, top -1).  After
// rounds of their own kernels (rounds true) the last one's SAH programme comes first.
constexpr int kTailSmem = kTailClusters * (2 * static_cast<int>(sizeof(float4)) + static_cast<int>(sizeof(int)));
__global__ void __launch_bounds__(kMergeBlock) k_ploc_tail(const int *__restrict__ clusters, RoundState *state,
                                                           int2 *child, float4 *bmin, float4 *bmax, int *count, int n,
                                                           bool rounds, DpArgs D) {
    extern __shared__ float4 box[];   // per cluster: lo (w: node id), hi (w: triangles)
    __shared__ uint32_t warpSum[32];
    float4 *slo = box, *shi = box + kTailClusters;
    int *nn = reinterpret_cast<int *>(shi + kTailClusters);
    int m = state->m, top = state->top;
    if (m > kTailClusters) return;
    const int t = threadIdx.x;
    if (rounds) dpLastRound(D, n, state, t, kMergeBlock, child, count, bmin, bmax);   // complete at the barrier below
    for (int i = t; i < m; i += kMergeBlock) {
        const int c = clusters[i];
        float4 lo = bmin[c], hi = bmax[c];
        lo.w = __int_as_float(c);
        hi.w = __int_as_float(count[c]);
        slo[i] = lo;
        shi[i] = hi;
    }
    __syncthreads();
    while (m > 1) {
        // nearest neighbours as in k_ploc_nn; few clusters share the block's threads, P to a
        // cluster, each over every P-th position of the window
        int P = 1;
        while (P < 32 && 2 * P * m <= kMergeBlock) P *= 2;
        for (int w = t; w < (m * P + 31) / 32 * 32; w += kMergeBlock) {   // whole warps
            const int i = min(w / P, m - 1);
            const float4 lo = slo[i], hi = shi[i];
            float best = 3.0e38f;
            int bestJ = -1;
            const int j1 = min(i + kPlocRadius, m - 1);
            for (int j = max(i - kPlocRadius, 0) + w % P; j <= j1; j += P) {
                if (j == i) continue;
                const float4 a = slo[j], b = shi[j];
                const float area = areaOf(make_float4(fminf(lo.x, a.x), fminf(lo.y, a.y), fminf(lo.z, a.z), 0.0f),
                                          make_float4(fmaxf(hi.x, b.x), fmaxf(hi.y, b.y), fmaxf(hi.z, b.z), 0.0f));
                if (area < best) {
                    best = area;
                    bestJ = j;
                }
            }
            for (int off = 1; off < P; off <<= 1) {   // the least area, the lowest position of equals
                const float a2 = __shfl_xor_sync(0xffffffffu, best, off);
                const int j2 = __shfl_xor_sync(0xffffffffu, bestJ, off);
                if (j2 >= 0 && (bestJ < 0 || a2 < best || (a2 == best && j2 < bestJ))) {
                    best = a2;
                    bestJ = j2;
                }
            }
            if (w < m * P && w % P == 0) nn[i] = bestJ;
        }
        __syncthreads();
        // merge and compact, a block's width of clusters at a time; a tile writes only positions
        // at or before its own clusters, once all of them are read
        int merges = 0, kept = 0;
        for (int base = 0; base < m; base += kMergeBlock) {
            const int i = base + t;
            bool lead, keep;
            mergeFlags(nn, i, m, &lead, &keep);
            uint32_t total;
            const uint32_t before = countBefore(lead, keep, warpSum, &total);
            float4 lo = make_float4(0, 0, 0, 0), hi = lo;
            if (keep) {
                lo = slo[i];
                hi = shi[i];
                if (lead) {
                    const float4 l2 = slo[nn[i]], h2 = shi[nn[i]];
                    const int a = __float_as_int(lo.w), b = __float_as_int(l2.w);
                    const int triangles = __float_as_int(hi.w) + __float_as_int(h2.w);
                    const int id = top - merges - static_cast<int>(before & 0xFFFFu);
                    lo = make_float4(fminf(lo.x, l2.x), fminf(lo.y, l2.y), fminf(lo.z, l2.z), 0.0f);
                    hi = make_float4(fmaxf(hi.x, h2.x), fmaxf(hi.y, h2.y), fmaxf(hi.z, h2.z), 0.0f);
                    child[id] = make_int2(a, b);
                    bmin[id] = lo;
                    bmax[id] = hi;
                    count[id] = triangles;
                    dpNode(D, n, id, make_int2(a, b), triangles, lo, hi, bmin, bmax);
                    lo.w = __int_as_float(id);
                    hi.w = __int_as_float(triangles);
                }
            }
            __syncthreads();
            if (keep) {
                const int at = kept + static_cast<int>(before >> 16);
                slo[at] = lo;
                shi[at] = hi;
            }
            merges += static_cast<int>(total & 0xFFFFu);
            kept += static_cast<int>(total >> 16);
            __syncthreads();
        }
        if (merges == 0) break;   // reported by the host: clusters are left
        top -= merges;
        m = kept;
    }
    if (t == 0) {
        state[1].m = m;
        state[1].top = top;
    }
}

struct CollapseArgs {
    const float *verts;
    const uint32_t *order;
    const int *tri_mat;
    const int *tri_light;
    int n;
    const int2 *child;
    const int *count;   // triangles under each binary node
    DpArgs dp;
    const float4 *bmin;
    const float4 *bmax;
    WideNode *nodes;
    TriRecord *tris;
    int2 *slot_shade;
    unsigned long long *level;   // per level: wide nodes (low half) and triangles (high half) it allocated
};

__device__ __forceinline__ float groupMin(float v) {
    for (int off = 1; off < 8; off <<= 1) v = fminf(v, __shfl_xor_sync(0xffffffffu, v, off));
    return v;
}
__device__ __forceinline__ float groupMax(float v) {
    for (int off = 1; off < 8; off <<= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, off));
    return v;
}
__device__ __forceinline__ uint32_t groupOr(uint32_t v) {
    for (int off = 1; off < 8; off <<= 1) v |= __shfl_xor_sync(0xffffffffu, v, off);
    return v;
}

// One level of the wide tree, eight threads per wide node (a thread per child, then per slot);
// items are (binary node, wide node), a level's items in the order its parents allocated them.
// Its levels are few and the upper ones small, so a level costs the latency of one node: with
// a thread per node that was the greedy assignment over a local 8 x 8 table and 48 FP64
// divisions (73 us for the 5 nodes of the box room); here each thread keeps its child's eight
// costs in registers, planes are quantised exactly in float32 with directed rounding, and the
// allocations of a block's 16 nodes take one atomic instead of 48.
constexpr int kCollapseBlock = 128, kCollapseNodes = kCollapseBlock / 8;
__global__ void __launch_bounds__(kCollapseBlock) k_collapse(CollapseArgs A, int levelIdx,
                                                             const int2 *__restrict__ items, int2 *__restrict__ next) {
    __shared__ unsigned long long alloc[kCollapseNodes];
    cudaGridDependencySynchronize();
    cudaTriggerProgrammaticLaunchCompletion();
    // nodes and triangles placed by the levels before this one; this level's items
    int nodeBase = 1, triBase0 = 0;
    for (int l = 0; l < levelIdx; l++) {
        nodeBase += static_cast<int>(A.level[l] & 0xFFFFFFFFull);
        triBase0 += static_cast<int>(A.level[l] >> 32);
    }
    const int nitems = levelIdx == 0 ? 1 : static_cast<int>(A.level[levelIdx - 1] & 0xFFFFFFFFull);
    const int lane = threadIdx.x & 31, sub = lane & 7, group = threadIdx.x >> 3;
    const unsigned groupShift = static_cast<unsigned>(lane & 24);
    for (int tile = blockIdx.x * kCollapseNodes; tile < nitems; tile += gridDim.x * kCollapseNodes) {
        const bool live = tile + group < nitems;
        const int2 item = live ? items[tile + group] : make_int2(A.n - 1, 0);
        // the eight slots of the wide node spread over its subtree as the SAH programme decided:
        // thread s follows the part that slot s belongs to, [start, start + slots)
        int x = item.x, start = 0, slots = 8;
        {
            int k = x < A.n - 1 ? A.dp.wideSplit[x] : 0;   // 0: a single-triangle scene's root
            while (__any_sync(0xffffffffu, k != 0)) {
                if (k != 0) {
                    const int2 c = A.child[x];
                    if (sub - start < k) {
                        x = c.x;
                        slots = k;
                    } else {
                        x = c.y;
                        start += k;
                        slots -= k;
                    }
                    k = x < A.n - 1 && slots > 1 ? A.dp.split[8 * static_cast<int64_t>(x) + slots - 1] : 0;
                }
            }
        }
        const bool isChild = live && sub == start;   // children in the order of their slots, left first
        const unsigned childMask = (__ballot_sync(0xffffffffu, isChild) >> groupShift) & 0xFFu;
        const int nc = __popc(childMask);
        const float4 cl = isChild ? A.bmin[x] : make_float4(3.0e38f, 3.0e38f, 3.0e38f, 0.0f);
        const float4 ch = isChild ? A.bmax[x] : make_float4(-3.0e38f, -3.0e38f, -3.0e38f, 0.0f);
        const float3 lo = mk(groupMin(cl.x), groupMin(cl.y), groupMin(cl.z));
        const float3 hi = mk(groupMax(ch.x), groupMax(ch.y), groupMax(ch.z));
        const float3 ctr = (lo + hi) * 0.5f;
        const float3 c = (xyz(cl) + xyz(ch)) * 0.5f - ctr;
        // greedy slot assignment: child whose centroid offset lies in octant o prefers slot o;
        // the cheapest pair of an unplaced child and a free slot first (ties: the first child,
        // then the first slot)
        float cost[8];
#pragma unroll
        for (int s = 0; s < 8; s++)
            cost[s] = -(((s & 1) ? -c.x : c.x) + ((s & 2) ? -c.y : c.y) + ((s & 4) ? -c.z : c.z));
        uint32_t used = 0u;
        int slot = -1;
        const int rounds = __reduce_max_sync(0xffffffffu, nc);
        for (int r = 0; r < rounds; r++) {
            float bc = 3.0e38f;
            int bs = -1;
#pragma unroll
            for (int s = 0; s < 8; s++)
                if (!((used >> s) & 1u) && (cost[s] < bc || bs < 0)) {
                    bc = cost[s];
                    bs = s;
                }
            const bool open = isChild && slot < 0 && r < nc;
            float v = open ? bc : INFINITY;
            int who = open ? sub : 8 + sub;
            for (int off = 1; off < 8; off <<= 1) {
                const float v2 = __shfl_xor_sync(0xffffffffu, v, off);
                const int who2 = __shfl_xor_sync(0xffffffffu, who, off);
                if ((who2 < 8 && who >= 8) || ((who2 < 8) == (who < 8) && (v2 < v || (!(v < v2) && who2 < who)))) {
                    v = v2;
                    who = who2;
                }
            }
            const int taken = __shfl_sync(0xffffffffu, bs, static_cast<int>(groupShift) + (who & 7));
            if (who < 8) {
                used |= 1u << taken;
                if (sub == who) slot = taken;
            }
        }
        // the threads without a child take the free slots, which stay empty
        if (slot < 0) slot = static_cast<int>(__fns(~used & 0xFFu, 0, __popc(~childMask & ((1u << sub) - 1u) & 0xFFu) + 1)) & 7;
        // children: internal (wide node) or leaf (<= 3 triangles)
        const int triangles = isChild ? A.count[x] : 0;
        const bool inner = isChild && x < A.n - 1 && (triangles > kLeafMax || !A.dp.leaf[x]);
        const int leafTris = isChild && !inner ? triangles : 0;
        const uint32_t imask = groupOr(inner ? 1u << slot : 0u);
        const uint32_t tri2 = groupOr(static_cast<uint32_t>(leafTris) << (2 * slot));   // 2 bits per slot
        const int nInt = __popc(imask), nTri = __popc(tri2 & 0x5555u) + 2 * __popc(tri2 & 0xAAAAu);
        const uint32_t triBelow = tri2 & ((1u << (2 * slot)) - 1u);
        const int triOff = __popc(triBelow & 0x5555u) + 2 * __popc(triBelow & 0xAAAAu);
        const int rank = __popc(imask & ((1u << slot) - 1u));
        if (sub == 0) alloc[group] = static_cast<unsigned long long>(nInt) | static_cast<unsigned long long>(nTri) << 32;
        __syncthreads();
        if (threadIdx.x == 0) {
            unsigned long long sum = 0;
            for (int g = 0; g < kCollapseNodes; g++) {
                const unsigned long long v = alloc[g];
                alloc[g] = sum;
                sum += v;
            }
            const unsigned long long at = sum ? atomicAdd(&A.level[levelIdx], sum) : 0ull;
            for (int g = 0; g < kCollapseNodes; g++) alloc[g] += at;
        }
        __syncthreads();
        const int levelOff = static_cast<int>(alloc[group] & 0xFFFFFFFFull);   // among this level's new nodes
        const int childBase = nInt ? nodeBase + levelOff : 0;
        const int triBase = nTri ? triBase0 + static_cast<int>(alloc[group] >> 32) : 0;
        __syncthreads();   // alloc is read: the next tile may overwrite it

        int e[3];
        const float ext[3] = {hi.x - lo.x, hi.y - lo.y, hi.z - lo.z};
#pragma unroll
        for (int a = 0; a < 3; a++) {
            int ex = -126;
            if (ext[a] > 0.0f) {
                frexpf(ext[a] / 255.0f, &ex);   // ext/255 = m 2^ex, m in [0.5, 1)
                ex = max(ex, -126);
                for (int g = 0; g < 4 && ldexpf(255.0f, ex) < ext[a]; g++) ex++;
            }
            e[a] = ex;
        }
        if (!live) continue;
        WideNode &node = A.nodes[item.y];
        if (sub == 0) {
            node.px = lo.x;
            node.py = lo.y;
            node.pz = lo.z;
            *reinterpret_cast<uint32_t *>(&node.ex) =
                static_cast<uint32_t>(static_cast<uint8_t>(e[0] + 127)) |
                static_cast<uint32_t>(static_cast<uint8_t>(e[1] + 127)) << 8 |
                static_cast<uint32_t>(static_cast<uint8_t>(e[2] + 127)) << 16 | imask << 24;
            node.child_base = static_cast<uint32_t>(childBase);
            node.tri_base = static_cast<uint32_t>(triBase);
        }
        // floor and ceiling of (bound - origin) / 2^e in real arithmetic: every k 2^e with k <=
        // 255 is a float, so rounding the difference towards it does not pass an integer, and
        // the scaling is exact (an underflow to 0 keeps a ceiling of 1)
        uint8_t ql[3] = {0, 0, 0}, qh[3] = {0, 0, 0};
        uint8_t meta = 0;
        if (isChild) {
            const float p[3] = {lo.x, lo.y, lo.z}, b0[3] = {cl.x, cl.y, cl.z}, b1[3] = {ch.x, ch.y, ch.z};
#pragma unroll
            for (int a = 0; a < 3; a++) {
                const float down = __fsub_rd(b0[a], p[a]), up = __fsub_ru(b1[a], p[a]);
                const float l = floorf(ldexpf(down, -e[a]));
                float h = ceilf(ldexpf(up, -e[a]));
                if (up > 0.0f && h < 1.0f) h = 1.0f;
                ql[a] = static_cast<uint8_t>(fminf(fmaxf(l, 0.0f), 255.0f));
                qh[a] = static_cast<uint8_t>(fminf(fmaxf(h, 0.0f), 255.0f));
            }
            meta = inner ? static_cast<uint8_t>(0x20 | (24 + slot))
                         : static_cast<uint8_t>((((1u << leafTris) - 1u) << 5) | static_cast<uint32_t>(triOff));
        }
        node.meta[slot] = meta;
        node.qlo_x[slot] = ql[0];
        node.qlo_y[slot] = ql[1];
        node.qlo_z[slot] = ql[2];
        node.qhi_x[slot] = qh[0];
        node.qhi_y[slot] = qh[1];
        node.qhi_z[slot] = qh[2];
        if (inner) {
            next[levelOff + rank] = make_int2(x, childBase + rank);
        } else if (isChild) {
            // the leaf's triangles (code-order positions), left subtree first
            int prim[kLeafMax] = {x, x, x};
            if (leafTris > 1) {
                const int2 cc = A.child[x];
                if (leafTris == 2) {
                    prim[0] = cc.x;
                    prim[1] = cc.y;
                } else if (cc.x >= A.n - 1) {
                    const int2 c2 = A.child[cc.y];
                    prim[0] = cc.x;
                    prim[1] = c2.x;
                    prim[2] = c2.y;
                } else {
                    const int2 c2 = A.child[cc.x];
                    prim[0] = c2.x;
                    prim[1] = c2.y;
                    prim[2] = cc.y;
                }
            }
#pragma unroll
            for (int q = 0; q < kLeafMax; q++) {
                if (q >= leafTris) break;
                const uint32_t id = A.order[prim[q] - (A.n - 1)];
                const float *v = A.verts + 9 * static_cast<int64_t>(id);
                TriRecord r;
                r.v0 = make_float4(v[0], v[1], v[2], __int_as_float(static_cast<int>(id)));
                r.v1 = make_float4(v[3], v[4], v[5], 0.0f);
                r.v2 = make_float4(v[6], v[7], v[8], 0.0f);
                A.tris[triBase + triOff + q] = r;
                A.slot_shade[triBase + triOff + q] =
                    make_int2(A.tri_mat ? A.tri_mat[id] : 0, A.tri_light ? A.tri_light[id] : -1);
            }
        }
    }
}

template <class T>
T *dalloc(size_t n) {
    T *p = nullptr;
    if (cudaMalloc(&p, sizeof(T) * std::max<size_t>(n, 1)) != cudaSuccess) return nullptr;
    return p;
}

// hands out 256-byte aligned pieces of one allocation; with base null it only adds them up
struct Scratch {
    unsigned char *base = nullptr;
    size_t used = 0;
    template <class T>
    T *take(size_t n) {
        const size_t at = used;
        used = (used + sizeof(T) * std::max<size_t>(n, 1) + 255) & ~size_t(255);
        return base ? reinterpret_cast<T *>(base + at) : nullptr;
    }
};

}  // namespace

void freeWideBVH(DeviceBVH *b) {
    cudaFree(b->nodes);
    cudaFree(b->tris);
    cudaFree(b->slot_shade);
    *b = DeviceBVH{};
}

int buildWideBVH(const float *d_verts, int n, const int *d_tri_mat, const int *d_tri_light, DeviceBVH *out,
                 cudaStream_t stream, char *err, size_t errlen) {
    freeWideBVH(out);
    if (n <= 0) {
        snprintf(err, errlen, "buildWideBVH: empty scene");
        return -2;
    }
    int rc = 0;
    auto fail = [&](const char *what, cudaError_t e) {
        snprintf(err, errlen, "buildWideBVH: %s: %s", what, cudaGetErrorString(e));
        rc = -3;
    };
    const size_t N = static_cast<size_t>(n), nNodes = 2 * N - 1;
    constexpr int kMaxLevels = 4096 / 64;   // more than the traversal accepts (kStackDepth)
    static_assert(kMaxLevels > kStackDepth, "the depth check needs the levels past the limit");
    float *d_bounds = nullptr;
    uint64_t *keys[2] = {};
    uint32_t *vals[2] = {};
    int2 *child = nullptr, *items[2] = {};
    int *count = nullptr, *clusters[2] = {}, *nn = nullptr;
    uint32_t *sums = nullptr;
    float4 *bmin = nullptr, *bmax = nullptr;
    DpArgs dp{};
    RoundState *rounds = nullptr;
    unsigned long long *level = nullptr;
    void *tmp = nullptr;
    size_t tmpBytes = 0;
    {
        cub::DoubleBuffer<uint64_t> kb(keys[0], keys[1]);
        cub::DoubleBuffer<uint32_t> vb(vals[0], vals[1]);
        cub::DeviceRadixSort::SortPairs(nullptr, tmpBytes, kb, vb, n, 0, 64, stream);
    }
    // all scratch in one allocation: sized, then handed out
    Scratch sc;
    for (int pass = 0; pass < 2; pass++) {
        sc.used = 0;
        d_bounds = sc.take<float>(12);
        for (int k = 0; k < 2; k++) {
            keys[k] = sc.take<uint64_t>(N);
            vals[k] = sc.take<uint32_t>(N);
            clusters[k] = sc.take<int>(N);
            items[k] = sc.take<int2>(N);
        }
        child = sc.take<int2>(N);
        count = sc.take<int>(nNodes);
        nn = sc.take<int>(N);
        sums = sc.take<uint32_t>(N / kMergeBlock + 1);
        bmin = sc.take<float4>(nNodes);
        bmax = sc.take<float4>(nNodes);
        dp = DpArgs{sc.take<float>(8 * N), sc.take<uint8_t>(8 * N), sc.take<uint8_t>(N), sc.take<uint8_t>(N)};
        rounds = sc.take<RoundState>(kMaxRounds + 2);
        level = sc.take<unsigned long long>(kMaxLevels + 1);
        tmp = sc.take<unsigned char>(tmpBytes);
        if (pass == 0 && cudaMalloc(&sc.base, sc.used) != cudaSuccess) break;
    }
    out->nodes = dalloc<WideNode>(n);
    out->tris = dalloc<TriRecord>(n);
    out->slot_shade = dalloc<int2>(n);
    if (!sc.base || !out->nodes || !out->tris || !out->slot_shade) {
        cudaGetLastError();
        snprintf(err, errlen, "buildWideBVH: device allocation failed for %d triangles", n);
        rc = -4;
    }
    if (rc == 0) {
        const float init[12] = {3e38f, 3e38f, 3e38f, -3e38f, -3e38f, -3e38f,
                                3e38f, 3e38f, 3e38f, -3e38f, -3e38f, -3e38f};
        cudaMemcpyAsync(d_bounds, init, sizeof(init), cudaMemcpyHostToDevice, stream);
        cudaMemsetAsync(level, 0, sizeof(unsigned long long) * (kMaxLevels + 1), stream);
        const int T = 256;
        k_prim_bounds<<<std::min((n + kBoundsBlock - 1) / kBoundsBlock, 1216), kBoundsBlock, 0, stream>>>(d_verts, n,
                                                                                                      d_bounds);
        k_morton<<<(n + T - 1) / T, T, 0, stream>>>(d_verts, n, d_bounds, keys[0], vals[0]);
        cub::DoubleBuffer<uint64_t> kb(keys[0], keys[1]);
        cub::DoubleBuffer<uint32_t> vb(vals[0], vals[1]);
        cub::DeviceRadixSort::SortPairs(tmp, tmpBytes, kb, vb, n, 0, 64, stream);
        const uint32_t *order = vb.Current();
        k_leaf_bounds<<<(n + T - 1) / T, T, 0, stream>>>(d_verts, order, n, bmin, bmax, count, clusters[0]);
        // clustering rounds (merged nodes numbered downwards), then the rest in one block
        RoundState st{n, n - 2};
        cudaError_t e = cudaMemcpyAsync(rounds, &st, sizeof(st), cudaMemcpyHostToDevice, stream);
        int r = 0;
        while (st.m > kTailClusters && e == cudaSuccess) {
            if (r + kRoundsAhead > kMaxRounds) {
                snprintf(err, errlen, "buildWideBVH: clustering made no progress");
                rc = -5;
                break;
            }
            for (int k = 0; k < kRoundsAhead; k++, r++) {
                const int *in = clusters[r & 1];
                // at most half of the last round's clusters merged; a few blocks run over more
                const int dpBlocks = r == 0 ? 0 : std::min((st.m / 2 + kMergeBlock - 1) / kMergeBlock, 152);
                const int blocks = (st.m + kMergeBlock - 1) / kMergeBlock;
                if (e == cudaSuccess)
                    e = launchDependent(k_ploc_nn, dim3((st.m + kPlocBlock - 1) / kPlocBlock), dim3(kPlocBlock / 2), 0,
                                        stream, k > 0, in, rounds + r, bmin, bmax, nn);
                if (e == cudaSuccess)
                    e = launchDependent(k_ploc_count, dim3(dpBlocks + blocks), dim3(kMergeBlock), 0, stream, true, nn,
                                        rounds + r, sums, dpBlocks, child, count, bmin, bmax, n, dp);
                if (e == cudaSuccess)
                    e = launchDependent(k_ploc_merge, dim3(blocks), dim3(kMergeBlock), 0, stream, true, in, rounds + r, nn,
                                        sums, child, bmin, bmax, count, clusters[(r & 1) ^ 1]);
            }
            const int before = st.m;
            if (e == cudaSuccess) e = cudaMemcpyAsync(&st, rounds + r, sizeof(st), cudaMemcpyDeviceToHost, stream);
            if (e == cudaSuccess) e = cudaStreamSynchronize(stream);
            if (e == cudaSuccess && st.m >= before) {
                snprintf(err, errlen, "buildWideBVH: clustering made no progress");
                rc = -5;
                break;
            }
        }
        if (e == cudaSuccess && rc == 0) {
            e = cudaFuncSetAttribute(k_ploc_tail, cudaFuncAttributeMaxDynamicSharedMemorySize, kTailSmem);
            if (e == cudaSuccess)
                k_ploc_tail<<<1, kMergeBlock, kTailSmem, stream>>>(clusters[r & 1], rounds + r, child, bmin, bmax,
                                                                   count, n, r > 0, dp);
        }
        // the wide tree, kRoundsAhead levels between two looks at what they allocated
        const int2 root = make_int2(n > 1 ? 0 : n - 1, 0);
        cudaMemcpyAsync(items[0], &root, sizeof(int2), cudaMemcpyHostToDevice, stream);
        CollapseArgs A{d_verts, order, d_tri_mat, d_tri_light, n, child, count, dp, bmin, bmax,
                       out->nodes, out->tris, out->slot_shade, level};
        unsigned long long got[kMaxLevels + 1] = {};
        RoundState left{0, 0};
        float hb[12] = {};
        int depth = 0;
        bool open = rc == 0;
        while (open && e == cudaSuccess) {
            long long most = 1;   // nodes of the first level launched now, at most eight times that in the next
            if (depth > 0) most = static_cast<long long>(got[depth - 1] & 0xFFFFFFFFull);
            for (int k = 0; k < kRoundsAhead && depth + k < kMaxLevels; k++) {
                const long long blocks = (std::min<long long>(most, n) + kCollapseNodes - 1) / kCollapseNodes;
                if (e == cudaSuccess)
                    e = launchDependent(k_collapse, dim3(static_cast<unsigned>(std::min<long long>(blocks, 152 * 16))),
                                        dim3(kCollapseBlock), 0, stream, k > 0, A, depth + k, items[(depth + k) & 1],
                                        items[((depth + k) & 1) ^ 1]);
                most = std::min<long long>(8 * most, n);
            }
            if (e == cudaSuccess) e = cudaMemcpyAsync(got, level, sizeof(got), cudaMemcpyDeviceToHost, stream);
            if (e == cudaSuccess && depth == 0)
                e = cudaMemcpyAsync(&left, rounds + r + 1, sizeof(left), cudaMemcpyDeviceToHost, stream);
            if (e == cudaSuccess && depth == 0) e = cudaMemcpyAsync(hb, d_bounds, sizeof(hb), cudaMemcpyDeviceToHost, stream);
            if (e == cudaSuccess) e = cudaStreamSynchronize(stream);
            if (e != cudaSuccess) break;
            if (n > 1 && (left.m != 1 || left.top != -1)) {
                snprintf(err, errlen, "buildWideBVH: clustering left %d clusters and %d node ids", left.m, left.top + 1);
                rc = -5;
                break;
            }
            for (int k = 0; k < kRoundsAhead && open && depth < kMaxLevels; k++) {
                depth++;   // a level of at least one item has run
                open = (got[depth - 1] & 0xFFFFFFFFull) != 0;
            }
            if (depth >= kMaxLevels) open = false;
        }
        if (e != cudaSuccess && rc == 0) fail("build", e);
        if (rc == 0) {
            long long nodes = 1, tris = 0;
            for (int k = 0; k < depth; k++) {
                nodes += static_cast<long long>(got[k] & 0xFFFFFFFFull);
                tris += static_cast<long long>(got[k] >> 32);
            }
            out->lo = mk(hb[0], hb[1], hb[2]);
            out->hi = mk(hb[3], hb[4], hb[5]);
            out->n_nodes = static_cast<int>(nodes);
            out->ntri = n;
            out->depth = depth;
            if (depth > kStackDepth) {
                snprintf(err, errlen, "buildWideBVH: tree depth %d exceeds the traversal stack (%d)", depth, kStackDepth);
                rc = -7;
            } else if (tris != n) {
                snprintf(err, errlen, "buildWideBVH: placed %lld of %d triangles", tris, n);
                rc = -6;
            }
        }
    }
    cudaFree(sc.base);
    if (rc != 0) freeWideBVH(out);
    return rc;
}

}  // namespace spgpu
