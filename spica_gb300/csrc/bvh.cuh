// bvh.cuh -- the device-built compressed 8-wide BVH: its host-side handle and the
// traversal routine shared by the ray-batch kernels and the wavefront renderer.
#pragma once

#include <type_traits>

#include <cstdint>
#include <cuda_runtime.h>

#include "common.cuh"

namespace spgpu {

// Largest wide-tree depth the traversal kernels accept.  The per-thread stack holds
// one node group per level of the current path: its first kStackShared entries live
// in shared memory, deeper ones spill to a per-thread local array.
constexpr int kStackDepth = 48;
#ifndef SPGPU_STACK_SHARED
#define SPGPU_STACK_SHARED 8
#endif
constexpr int kStackShared = SPGPU_STACK_SHARED;
constexpr int kTraceBlock = 128;

struct DeviceBVH {
    WideNode *nodes = nullptr;     // [n_nodes]
    TriRecord *tris = nullptr;     // [ntri], leaf order
    int2 *slot_shade = nullptr;    // [ntri]: (material, light index or -1) per leaf slot
    int n_nodes = 0;
    int ntri = 0;
    int depth = 0;                 // levels of wide nodes
    float3 lo{0, 0, 0}, hi{0, 0, 0};
};

struct TraceStats {   // per-ray visit counters, for the roofline's algorithmic bytes
    unsigned long long rays;
    unsigned long long nodes;
    unsigned long long tris;
};

// ---------------------------------------------------------------------------
// Traversal of the compressed wide BVH (after Ylitie, Karras and Laine, "Efficient
// Incoherent Ray Traversal on GPUs Through Compressed Wide BVHs", HPG 2017):
// node groups (child base, pending-child bits in visit order, internal mask) on a
// per-thread stack in shared memory, triangle groups tested as soon as a node is
// opened.  Closest hit keeps the reference's acceptance rule t in (eps, tmax]
// (core/triangle.cc:117), so on an exact tie the later-tested triangle wins.
// Any hit returns on the first triangle with t in (eps, tmax].
// Returns false and sets *overflow if the tree is deeper than the stack.
// ---------------------------------------------------------------------------
// two floats in one 64-bit register: the packed FP32 instructions work on both halves in
// one issue slot, each half rounded as the scalar instruction rounds it
__device__ __forceinline__ uint64_t pack2(float lo, float hi) {
    uint64_t r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ float2 unpack2(uint64_t v) {
    float2 r;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
    return r;
}
__device__ __forceinline__ uint64_t fma2(uint64_t a, uint64_t b, uint64_t c) {
    uint64_t r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
__device__ __forceinline__ uint64_t add2(uint64_t a, uint64_t b) {
    uint64_t r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ uint64_t mul2(uint64_t a, uint64_t b) {
    uint64_t r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
// bytes k and k + 1 of w as exact floats: PRMT assembles 0x4B0000bb (= 2^23 + b) for each,
// one packed add takes 2^23 off both
__device__ __forceinline__ uint64_t bytesToFloat2(uint32_t w, int k) {
    const float lo = __uint_as_float(__byte_perm(w, 0x4B000000u, 0x7650u | static_cast<uint32_t>(k)));
    const float hi = __uint_as_float(__byte_perm(w, 0x4B000000u, 0x7650u | static_cast<uint32_t>(k + 1)));
    return add2(pack2(lo, hi), pack2(-8388608.0f, -8388608.0f));
}
__device__ __forceinline__ float fmax3f(float a, float b, float c) {
    float d;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
    return d;
}
__device__ __forceinline__ float fmin3f(float a, float b, float c) {
    float d;
    asm("min.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
    return d;
}
// bit s of an 8-bit slot mask moved to bit s ^ x (x in 0..7): the visit order of the slots
__device__ __forceinline__ uint32_t xorBits8(uint32_t m, uint32_t x) {
    m = (x & 1u) ? ((m << 1) & 0xAAu) | ((m >> 1) & 0x55u) : m;
    m = (x & 2u) ? ((m << 2) & 0xCCu) | ((m >> 2) & 0x33u) : m;
    return (x & 4u) ? ((m << 4) & 0xF0u) | (m >> 4) : m;
}

// Every node and triangle index is checked against the tree's sizes and the loop is
// bounded (kMaxVisits), so a malformed tree ends the ray with *overflow set instead of
// reading out of bounds or spinning.
constexpr uint32_t kMaxVisits = 1u << 22;

// Traversal state of one ray, kept in registers between steps so that a warp can
// retire finished rays and start new ones in the middle of a traversal.
struct TraceLane {
    float3 o, d, idir;
    float tmin, tmax;
    uint32_t octInv;  // bit a: the direction is not negative along axis a (7 - its sign octant)
    uint2 G;          // node group: child base, pending-child bits (visit order) | internal mask
    int sp;
    uint32_t visits;
    int hitSlot;
    float hu, hv;
    bool found;
    // split form (splitOpen): triangles still to be tested, as bits relative to pbase, and
    // whether a second such group waits on top of the stack
    uint32_t pbase, pbits;
    bool pmore;
};

__device__ __forceinline__ void laneInit(TraceLane &L, float3 o, float3 d, float tmin, float tmax,
                                         uint32_t root = 0) {
    L.o = o;
    L.d = d;
    L.idir = mk(d.x == 0.0f ? kInfT : 1.0f / d.x, d.y == 0.0f ? kInfT : 1.0f / d.y, d.z == 0.0f ? kInfT : 1.0f / d.z);
    L.octInv = (d.x < 0.0f ? 0u : 1u) | (d.y < 0.0f ? 0u : 2u) | (d.z < 0.0f ? 0u : 4u);
    L.tmin = tmin;
    L.tmax = tmax;
    L.G = make_uint2(root, (1u << (24 + L.octInv)) | 1u);   // the root as slot 0 of a virtual parent
    L.sp = 0;
    L.visits = 0;
    L.hitSlot = -1;
    L.hu = L.hv = 0.0f;
    L.found = false;
    L.pbase = L.pbits = 0u;
    L.pmore = false;
}

// Open the next pending child of the current node group (popping a group from the stack
// first when the current one is exhausted; the caller has checked that one is left).  The
// triangles of the leaves it hits come back as bits relative to *tbase, in test order.
// Returns true on a malformed tree, with *overflow set.
//
// Bound by instruction issue on divergent lanes (half to two thirds of the issue slots, L1
// and L2 serve the nodes), so it is the instructions per node that count.  The 48 planes are
// decoded and scaled two at a time with the packed FP32 instructions, and the children's
// hits are collected in slot order and brought into visit order by one bit permutation,
// where eight variable shifts did that before: 16M closest-hit rays on 1M triangles 3.67 ->
// 3.37 ms (4.58 -> 4.98 G rays/s), the 1080p mid-scale render 27.8 -> 26.5 ms; with scalar
// decoding in the same form the first gains a quarter less, the second half as much.
template <bool STATS>
__device__ __forceinline__ bool openChild(TraceLane &L, const WideNode *__restrict__ nodes, uint32_t nNodes,
                                          uint2 *__restrict__ stack, int stride, uint2 *spill, uint32_t *nodeCount,
                                          uint32_t *tbase, uint32_t *tbits, bool *overflow) {
    if (++L.visits > kMaxVisits) {
        *overflow = true;
        return true;
    }
    if (!(L.G.y & 0xFF000000u)) {
        L.sp--;
        L.G = L.sp < kStackShared ? stack[L.sp * stride] : spill[L.sp - kStackShared];
    }
    const uint32_t key = __ffs(L.G.y >> 24) - 1;
    L.G.y &= ~(1u << (24 + key));
    const uint32_t slot = key ^ L.octInv;
    const uint32_t child = L.G.x + __popc((L.G.y & 0xFFu) & ((1u << slot) - 1u));
    if (child >= nNodes) {
        *overflow = true;
        return true;
    }
    if (L.G.y & 0xFF000000u) {
        if (L.sp >= kStackDepth) {
            *overflow = true;
            return true;
        }
        if (L.sp < kStackShared) stack[L.sp * stride] = L.G;
        else spill[L.sp - kStackShared] = L.G;
        L.sp++;
    }
    if (STATS) (*nodeCount)++;
    const float4 *nodes4 = reinterpret_cast<const float4 *>(nodes);
    const float4 n0 = __ldg(nodes4 + 5 * child + 0);
    const float4 n1 = __ldg(nodes4 + 5 * child + 1);
    const float4 n2 = __ldg(nodes4 + 5 * child + 2);
    const float4 n3 = __ldg(nodes4 + 5 * child + 3);
    const float4 n4 = __ldg(nodes4 + 5 * child + 4);
    const uint32_t ew = __float_as_uint(n0.w);
    const float sx = __uint_as_float((ew & 0xFFu) << 23);
    const float sy = __uint_as_float(((ew >> 8) & 0xFFu) << 23);
    const float sz = __uint_as_float(((ew >> 16) & 0xFFu) << 23);
    const float ax = sx * L.idir.x, ay = sy * L.idir.y, az = sz * L.idir.z;
    const float bx = (n0.x - L.o.x) * L.idir.x, by = (n0.y - L.o.y) * L.idir.y, bz = (n0.z - L.o.z) * L.idir.z;
    // near / far quantised planes per axis, swapped for negative directions
    const uint2 qlx = make_uint2(__float_as_uint(n2.x), __float_as_uint(n2.y));
    const uint2 qly = make_uint2(__float_as_uint(n2.z), __float_as_uint(n2.w));
    const uint2 qlz = make_uint2(__float_as_uint(n3.x), __float_as_uint(n3.y));
    const uint2 qhx = make_uint2(__float_as_uint(n3.z), __float_as_uint(n3.w));
    const uint2 qhy = make_uint2(__float_as_uint(n4.x), __float_as_uint(n4.y));
    const uint2 qhz = make_uint2(__float_as_uint(n4.z), __float_as_uint(n4.w));
    const uint2 nx = (L.octInv & 1u) ? qlx : qhx, fx = (L.octInv & 1u) ? qhx : qlx;
    const uint2 ny = (L.octInv & 2u) ? qly : qhy, fy = (L.octInv & 2u) ? qhy : qly;
    const uint2 nz = (L.octInv & 4u) ? qlz : qhz, fz = (L.octInv & 4u) ? qhz : qlz;
    const uint64_t ax2 = pack2(ax, ax), ay2 = pack2(ay, ay), az2 = pack2(az, az);
    const uint64_t bx2 = pack2(bx, bx), by2 = pack2(by, by), bz2 = pack2(bz, bz);
    uint32_t hits = 0u;   // bit s: the box of slot s is hit
#pragma unroll
    for (int k = 0; k < 8; k += 2) {
        const int h = k >> 2, b = k & 3;
        const float2 tnx = unpack2(fma2(bytesToFloat2(h ? nx.y : nx.x, b), ax2, bx2));
        const float2 tny = unpack2(fma2(bytesToFloat2(h ? ny.y : ny.x, b), ay2, by2));
        const float2 tnz = unpack2(fma2(bytesToFloat2(h ? nz.y : nz.x, b), az2, bz2));
        const float2 tfx = unpack2(fma2(bytesToFloat2(h ? fx.y : fx.x, b), ax2, bx2));
        const float2 tfy = unpack2(fma2(bytesToFloat2(h ? fy.y : fy.x, b), ay2, by2));
        const float2 tfz = unpack2(fma2(bytesToFloat2(h ? fz.y : fz.x, b), az2, bz2));
        const float2 t1 = unpack2(mul2(pack2(fminf(fmin3f(tfx.x, tfy.x, tfz.x), L.tmax),
                                             fminf(fmin3f(tfx.y, tfy.y, tfz.y), L.tmax)),
                                       pack2(1.0000010f, 1.0000010f)));
        if (fmaxf(fmax3f(tnx.x, tny.x, tnz.x), L.tmin) <= t1.x) hits |= 1u << k;
        if (fmaxf(fmax3f(tnx.y, tny.y, tnz.y), L.tmin) <= t1.y) hits |= 2u << k;
    }
    const uint32_t imask = ew >> 24;
    L.G = make_uint2(__float_as_uint(n1.x), (xorBits8(hits & imask, L.octInv) << 24) | imask);
    // the hit leaves' triangles, in slot order (an empty slot's meta byte names none)
    uint32_t bits = 0u;
    for (uint32_t leaf = hits & ~imask; leaf; leaf &= leaf - 1u) {
        const uint32_t meta = __byte_perm(__float_as_uint(n1.z), __float_as_uint(n1.w), __ffs(leaf) - 1) & 0xFFu;
        bits |= (meta >> 5) << (meta & 31u);
    }
    *tbits = bits;
    *tbase = __float_as_uint(n1.y);
    return false;
}

// Whether the ray has nodes left to open.
__device__ __forceinline__ bool nodesLeft(const TraceLane &L) { return (L.G.y & 0xFF000000u) || L.sp > 0; }

// Moller-Trumbore of triangle ti; an accepted hit shortens the ray.  Returns true when the
// ray is finished (any hit found, or *overflow set by an index out of range).
template <bool ANY, bool STATS>
__device__ __forceinline__ bool testTriangle(TraceLane &L, const TriRecord *__restrict__ tris, uint32_t nTris,
                                             uint32_t ti, uint32_t *triCount, bool *overflow) {
    if (ti >= nTris) {
        *overflow = true;
        return true;
    }
    if (STATS) (*triCount)++;
    const float4 v0 = __ldg(&tris[ti].v0);
    const float4 v1 = __ldg(&tris[ti].v1);
    const float4 v2 = __ldg(&tris[ti].v2);
    const float3 E1 = xyz(v1) - xyz(v0), E2 = xyz(v2) - xyz(v0);
    const float3 pv = cross(L.d, E2);
    const float det = dot(E1, pv);
    if (det > -kEpsT && det < kEpsT) return false;
    const float inv = 1.0f / det;
    const float3 tv = L.o - xyz(v0);
    const float u = dot(tv, pv) * inv;
    if (u < 0.0f || u > 1.0f) return false;
    const float3 qv = cross(tv, E1);
    const float v = dot(L.d, qv) * inv;
    if (v < 0.0f || u + v > 1.0f) return false;
    const float t = dot(E2, qv) * inv;
    if (t <= fmaxf(L.tmin, kEpsT) || t > L.tmax) return false;
    L.found = true;
    if (ANY) return true;
    L.tmax = t;
    L.hitSlot = static_cast<int>(ti);
    L.hu = u;
    L.hv = v;
    return false;
}

// One step of the traversal: open the next child and test all the triangles it leaves.
// Returns true when the ray is finished.
template <bool ANY, bool STATS>
__device__ __forceinline__ bool laneStep(TraceLane &L, const WideNode *__restrict__ nodes,
                                         const TriRecord *__restrict__ tris, uint32_t nNodes, uint32_t nTris,
                                         uint2 *__restrict__ stack, int stride, uint2 *spill, uint32_t *nodeCount,
                                         uint32_t *triCount, bool *overflow) {
    if (!nodesLeft(L)) return true;
    uint32_t tbase = 0u, tbits = 0u;
    if (openChild<STATS>(L, nodes, nNodes, stack, stride, spill, nodeCount, &tbase, &tbits, overflow)) return true;
    while (tbits) {
        const uint32_t ti = tbase + static_cast<uint32_t>(__ffs(tbits) - 1);
        tbits &= tbits - 1u;
        if (testTriangle<ANY, STATS>(L, tris, nTris, ti, triCount, overflow)) return true;
    }
    return !nodesLeft(L);
}

// The split form of a traversal step: splitOpen, then splitTest on the lanes that have a
// pending triangle.  A lane whose node left several triangles does not hold up the warp while
// it tests them all; it goes on to its next node with them pending, and waits only when that
// node leaves a second group.  Triangles are tested in the same order as in laneStep, with
// some more of them and of the nodes visited before a hit shortens the ray, so the result is
// the same.  The stack needs one entry more than the tree's depth for the second group.
template <bool STATS>
__device__ __forceinline__ bool splitOpen(TraceLane &L, const WideNode *__restrict__ nodes,
                                          uint32_t nNodes, uint2 *__restrict__ stack, int stride, uint2 *spill,
                                          uint32_t *nodeCount, bool *overflow) {
    uint32_t tbase, tbits;
    if (openChild<STATS>(L, nodes, nNodes, stack, stride, spill, nodeCount, &tbase, &tbits, overflow)) return true;
    if (tbits) {
        if (!L.pbits) {
            L.pbase = tbase;
            L.pbits = tbits;
        } else {
            if (L.sp < kStackShared) stack[L.sp * stride] = make_uint2(tbase, tbits);
            else spill[L.sp - kStackShared] = make_uint2(tbase, tbits);
            L.sp++;
            L.pmore = true;
        }
    }
    return false;
}
template <bool ANY, bool STATS>
__device__ __forceinline__ bool splitTest(TraceLane &L, const TriRecord *__restrict__ tris,
                                          uint32_t nTris, uint2 *__restrict__ stack, int stride, uint2 *spill,
                                          uint32_t *triCount, bool *overflow) {
    const uint32_t ti = L.pbase + static_cast<uint32_t>(__ffs(L.pbits) - 1);
    L.pbits &= L.pbits - 1u;
    if (ti >= nTris) {
        *overflow = true;
        return true;
    }
    if (!L.pbits && L.pmore) {
        L.sp--;
        const uint2 g = L.sp < kStackShared ? stack[L.sp * stride] : spill[L.sp - kStackShared];
        L.pbase = g.x;
        L.pbits = g.y;
        L.pmore = false;
    }
    return testTriangle<ANY, STATS>(L, tris, nTris, ti, triCount, overflow);
}

// The split form is taken for trees of at least kSplitMinNodes wide nodes and queues of at
// least kSplitMinRays rays.  A larger tree's rays test few triangles per node (0.35 on the
// 2M-triangle scene), a few lanes of a warp at a time; a few dozen triangles in a handful of
// nodes are tested by most lanes at once, and one at a time they only wait.  Below some
// millions of rays a launch waits for its slowest rays, whose own chain the split form
// lengthens.  Measured, whole steps / split: spheres of 256, 1024, 4096 and 16k triangles (36
// nodes and up), 4M closest-hit rays 0.460 / 0.475, 0.487 / 0.472, 0.601 / 0.569, 0.653 /
// 0.615 ms; 1M triangles, 1k, 300k, 1.2M, 2.5M and 16M rays 0.084 / 0.101, 0.179 / 0.182,
// 0.375 / 0.382, 0.616 / 0.600, 3.37 / 3.20 ms; the mid-scale render 26.5 / 25.6 ms; the
// guided room's 2,418 triangles 4.02 / 4.12 ms, the box room's 36 in a batch 148 / 173 ms.
// Any-hit batches end at their first hit and gain nothing (2.5M on 1M triangles 0.404 /
// 0.425 ms); shadow rays of a full pool do (the mid-scale render 25.8 / 25.6 ms).
constexpr uint32_t kSplitMinNodes = 512;
constexpr int kSplitMinRays = 1 << 21;

template <bool ANY, bool STATS>
__device__ __forceinline__ bool traceWide(const WideNode *__restrict__ nodes, const TriRecord *__restrict__ tris,
                                          uint32_t nNodes, uint32_t nTris, float3 o, float3 d, float tmin,
                                          float &tmax, int &hitSlot, float &hu, float &hv, uint2 *__restrict__ stack,
                                          int stride, uint32_t *nodeCount, uint32_t *triCount, bool *overflow,
                                          uint32_t root = 0) {
    uint2 spill[kStackDepth - kStackShared];
    TraceLane L;
    laneInit(L, o, d, tmin, tmax, root);
    while (!laneStep<ANY, STATS>(L, nodes, tris, nNodes, nTris, stack, stride, spill, nodeCount, triCount,
                                 overflow)) {
    }
    tmax = L.tmax;
    hitSlot = L.hitSlot;
    hu = L.hu;
    hv = L.hv;
    return L.found;
}

// Persistent driver: a warp keeps up to 32 rays in flight and refills the lanes whose
// rays have finished, kRefill or more at a time, from a global ray counter (one
// atomicAdd per refill; the grid is one-dimensional), so lanes do not idle while the slowest ray of a batch finishes
// (after Aila and Laine, "Understanding the Efficiency of Ray Traversal on GPUs", HPG
// 2009).  fetch(i, &o, &d, &tmin, &tmax) loads ray i; done(i, L) consumes its result.
// All 32 lanes of each warp execute every iteration of the loop (warp-uniform control),
// so done() may use warp-collective operations.  SPLIT: steps in
// the split form.  OWN: where a launch with no more rays than lanes takes them from: the counter
// (kFromCounter), or each warp its own 32 without touching the counter, counted from the first
// block or, for the second of two queues in one launch, from the last.
enum : int { kFromCounter = 0, kOwnFromFirst, kOwnFromLast };
#ifndef SPGPU_REFILL
#define SPGPU_REFILL 12
#endif
constexpr int kRefill = SPGPU_REFILL;
// a finished ray's result waits for the warp's next refill, so that the finished lanes
// consume their results together (done() runs on up to 32 lanes instead of one or two)
#ifndef SPGPU_DEFER_DONE
#define SPGPU_DEFER_DONE 1
#endif
constexpr bool kDeferDone = SPGPU_DEFER_DONE != 0;
// traversal steps between two looks at the warp's idle lanes
#ifndef SPGPU_STEPS_PER_CHECK
#define SPGPU_STEPS_PER_CHECK 2
#endif
constexpr int kStepsPerCheck = SPGPU_STEPS_PER_CHECK;

template <bool ANY, bool STATS, bool SPLIT, int OWN = kFromCounter, class Fetch, class Done>
__device__ __forceinline__ void tracePersistent(const WideNode *__restrict__ nodes,
                                                const TriRecord *__restrict__ tris, uint32_t nNodes,
                                                uint32_t nTris, int n, int *rayCounter, uint2 *__restrict__ stack,
                                                int stride, uint32_t *nodeCount, uint32_t *triCount,
                                                bool *overflow, Fetch fetch, Done done) {
    uint2 spill[kStackDepth - kStackShared + (SPLIT ? 1 : 0)];
    TraceLane L;
    int ray = -1;            // >= 0 in flight (or finished), -1 idle, -2 no work left
    bool finished = false;   // the ray has finished, its result not yet consumed
    const int lane = threadIdx.x & 31;
    [[maybe_unused]] const int lanes = gridDim.x * blockDim.x;
    [[maybe_unused]] bool first = true;
    while (true) {
        if (!kDeferDone) {
            done(finished ? ray : -1, L);
            if (finished) {
                ray = -1;
                finished = false;
            }
        }
        const unsigned idle = __ballot_sync(0xffffffffu, ray == -1 || finished);
        const unsigned busy = __ballot_sync(0xffffffffu, ray >= 0 && !finished);
        if (idle && (__popc(idle) >= kRefill || busy == 0)) {
            if (kDeferDone) {
                // the results of the rays finished since the last refill, consumed together
                done(finished ? ray : -1, L);
                if (finished) {
                    ray = -1;
                    finished = false;
                }
            }
            int base = 0;
            if (OWN == kFromCounter || n > lanes) {
                if (lane == __ffs(idle) - 1) base = atomicAdd(rayCounter, __popc(idle));
                base = __shfl_sync(0xffffffffu, base, __ffs(idle) - 1);
            } else if (first) {
                base = (OWN == kOwnFromFirst ? blockIdx.x : gridDim.x - 1 - blockIdx.x) * blockDim.x + (threadIdx.x & ~31);
                first = false;
            } else {
                base = n;
            }
            if (ray == -1) {
                const int r = base + __popc(idle & ((1u << lane) - 1u));
                if (r < n) {
                    float3 o, d;
                    float t0, t1;
                    uint32_t root = 0;   // a fetch that takes a sixth argument names the ray's tree root
                    if constexpr (std::is_invocable_v<Fetch &, int, float3 *, float3 *, float *, float *, uint32_t *>)
                        fetch(r, &o, &d, &t0, &t1, &root);
                    else
                        fetch(r, &o, &d, &t0, &t1);
                    laneInit(L, o, d, t0, t1, root);
                    ray = r;
                } else {
                    ray = -2;
                }
            }
        }
        if (__all_sync(0xffffffffu, ray == -2)) break;
#pragma unroll 1
        for (int k = 0; k < kStepsPerCheck; k++) {
            if constexpr (SPLIT) {
                bool act = ray >= 0 && !finished;
                const bool more = act && nodesLeft(L);
                if (more && !L.pmore)
                    finished = splitOpen<STATS>(L, nodes, nNodes, stack, stride, spill, nodeCount, overflow);
                act = act && !finished;
                if (act && L.pbits)
                    finished = splitTest<ANY, STATS>(L, tris, nTris, stack, stride, spill, triCount, overflow);
                if (act && !finished) finished = !L.pbits && !nodesLeft(L);
            } else {
                if (ray >= 0 && !finished)
                    finished = laneStep<ANY, STATS>(L, nodes, tris, nNodes, nTris, stack, stride, spill, nodeCount,
                                                    triCount, overflow);
            }
        }
    }
}

// host entry points (bvh.cu)
int buildWideBVH(const float *d_verts, int ntri, const int *d_tri_mat, const int *d_tri_light, DeviceBVH *out,
                 cudaStream_t stream, char *err, size_t errlen);
void freeWideBVH(DeviceBVH *b);

}  // namespace spgpu
