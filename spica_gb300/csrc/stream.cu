// stream.cu -- the path integrator as a streaming wavefront: a fixed pool of path slots
// in HBM that is refilled with new camera paths as paths end, so every launch works on a
// full pool and the latency-bound tail of a sample pass occurs once per render instead of
// once per pass.
//
// One iteration (all slots advance one vertex):
//   regen            new camera rays (PerspectiveCamera::spawnRay) into the free slots,
//                    taken in order from the render's path sequence: path g is sample
//                    sampleOffset + g / npix of pixel g % npix
//   extend           closest hit of every ray in the pool; a miss adds the environment
//                    (first vertex or after a specular bounce) and ends the path; a hit
//                    copies the whole path record (ray, throughput, pixel, sample, depth,
//                    hit) into the queue of its material class, in coalesced 64-byte rows
//   shade<class>     emission, next-event estimation with MIS, BSDF sampling and Russian
//                    roulette (shadeHit, the reference's PathIntegrator::Li,
//                    integrators/path/path.cc:42-125); continuing paths are written back
//                    into the pool, shadow rays into the shadow queue
//   shadow           any-hit for the shadow rays; unoccluded ones add to the film
//   advance          counters for the next iteration, the render's done flag
// A guided render (learned guiding proposal) shades the Lambert queue with the network
// instead (k_sshade_guided: tensor-core tiles of 128 queue rows).
// A path's random numbers are keyed by (seed, film pixel) and counted by (sample, depth,
// stream), exactly as in the pass-by-pass wavefront (wavefront.cu), so a render draws the
// same samples whichever slot or iteration a path runs in; only the order of the film's
// floating-point additions differs.
//
// The iterations are captured into one CUDA graph of kIterPerGraph iterations, replayed
// until the device reports that every path of the render has ended.  The host reads the
// done flag of the replay kReplayLag launches back, so the GPU always has work queued;
// replays past the end find empty queues and return at once.  A render whose paths fit the
// pools at once runs without the graph, one vertex depth per iteration (renderOnePass).
// Scenes of one material class are shaded from the pool itself, without class queues.
#include <algorithm>
#include <cstring>
#include <type_traits>
#include <vector>

#include "../../include/spica_gpu.h"
#include "ctx.cuh"
#include "guided_shade.cuh"
#include "shade.cuh"

namespace spgpu {

namespace {

constexpr int kShadeBlockS = 128;
#ifndef SPGPU_TRACE_MIN_BLOCKS
#define SPGPU_TRACE_MIN_BLOCKS 8
#endif
constexpr int kTraceMinBlocks = SPGPU_TRACE_MIN_BLOCKS;   // resident traversal blocks per SM (register budget)
// resident shading blocks per SM (register budget) by class: Lambert, the other two
#ifndef SPGPU_SHADE_MIN_BLOCKS_L
#define SPGPU_SHADE_MIN_BLOCKS_L 8
#endif
#ifndef SPGPU_SHADE_MIN_BLOCKS_G
#define SPGPU_SHADE_MIN_BLOCKS_G 6
#endif
constexpr int shadeMinBlocks(int cls) { return cls == 0 ? SPGPU_SHADE_MIN_BLOCKS_L : SPGPU_SHADE_MIN_BLOCKS_G; }
#ifndef SPGPU_GUIDED_MIN_BLOCKS
#define SPGPU_GUIDED_MIN_BLOCKS 4
#endif
constexpr int kGuidedMinBlocks = SPGPU_GUIDED_MIN_BLOCKS;   // resident guided shading blocks per SM
#ifndef SPGPU_ITER_PER_GRAPH
#define SPGPU_ITER_PER_GRAPH 8
#endif
#ifndef SPGPU_REPLAY_LAG
#define SPGPU_REPLAY_LAG 1
#endif
constexpr int kIterPerGraph = SPGPU_ITER_PER_GRAPH;   // iterations captured in one graph
constexpr int kReplayLag = SPGPU_REPLAY_LAG;          // replays in flight before the host reads a done flag
constexpr int kDoneRing = StreamQueues::kEvents;
// counters (ints): [0] rays in the pool, [1] continuations written, [2..4] class
// counts, [5] shadow rays, [6] extend ray fetch, [7] shadow ray fetch, [8] done, [9]
// iterations, [10] error flags
enum : int { kCtrRays = 0, kCtrCont, kCtrClass0, kCtrShadow = 5, kCtrFetchE, kCtrFetchS, kCtrDone, kCtrIter, kCtrErr };
constexpr int kNumCtr = 16;
constexpr int kMaxIters = 66;   // iterations of a one-pass render: depths 0..64, and the counters after the last
// 64-bit counters: [0] paths started, [1] paths, [2] closest rays, [3] shadow rays,
// [4..7] visits (extend nodes, triangles, shadow nodes, triangles); then the call's own
// parameters, written by the host per render so that one captured graph serves every
// call: [8] paths of the render (spp * npix), [9] sample offset (batches: the lane's
// first path of the batch's sequence), [10] film address; [11] iterations run (batches)
enum : int { kBigStarted = 0, kBigPaths, kBigClosest, kBigShadow, kBigVisit, kBigTotal = 8, kBigOffset, kBigFilm,
             kBigIters };
constexpr int kNumBig = 12;

// a path's depth (bits 0..7), specular flag (bit 8) and, in batches, its render (bits
// 9..), carried in the w of its direction
__device__ __forceinline__ float packMeta(int depth, bool spec, int render = 0) {
    return __int_as_float(depth | (spec ? 256 : 0) | (render << 9));
}
__device__ __forceinline__ int metaRender(int meta) { return static_cast<int>(static_cast<unsigned>(meta) >> 9); }

// First statement of the kernels that one-pass renders launch back to back as dependent
// launches: the next kernel may be set up now, this one's work begins once the last kernel's
// is complete and visible.  (No effect where a kernel is launched without that attribute.)
__device__ __forceinline__ void awaitLastKernel() {
    cudaTriggerProgrammaticLaunchCompletion();
    cudaGridDependencySynchronize();
}

struct StreamArgs {
    SceneView sv;
    CameraView cam;
    int W, H, npix;
    int maxDepth;
    uint32_t seed;
    int direct;
    int cap;           // path slots
    // the pool: (origin, pixel), (direction, depth | specular << 8), (throughput, sample)
    float4 *rO, *rD, *rB;
    // class queues, cap rows per class: the pool record and the hit (t, slot, u, v)
    float4 *qO, *qD, *qB, *qH;
    // Where continuations go: the pool itself, or, in scenes of one shading class (singleClass,
    // else -1), the other of two pools, rays and continuations changing places every iteration.
    // There the class queue would only copy the pool: extend leaves the hit of pool ray i in
    // qH[i] (slot -1: none) and the class's shading reads the pool.  The second pool is the
    // space of the class queues, which such scenes do not use.  A vertex then moves 96 bytes
    // less and its extend appends to no queue: a batch of 16 box rooms 150.1 -> 146.4 ms, the
    // guided room at 640 x 360 3.30 -> 3.16.
    float4 *nO, *nD, *nB;
    int singleClass;
    float4 *shO, *shD, *shL;   // shadow queue, 2 * cap rows: (origin, film index), (dir, tmax), contribution
    int *ctr;
    int *cont;         // continuations written
    unsigned long long *big;
    // one-pass renders (renderOnePass): every path starts in the first iteration, ctr is the
    // iteration's own set of counters, cont the next one's ray count; shadowCtr: the counters
    // of the iteration whose shadow rays k_strace traces (null: none)
    int onePass;
    int *shadowCtr;
    int besideLast, besideNext;   // k_sshade: runs beside the last / next kernel (launchShading)
    // guided renders: the network's packed weights and biases (null: plain BSDF
    // sampling), the proposal's BSDF share, the depths that sample it (0: all but the
    // last), and the scene box that normalises the network's position input
    const uint8_t *packFwd;
    const float *biasPad;
    float guideAlpha;
    int guidedBounces;
    float3 guideLo, guideInvExt;
    // batches: the renders, the first path of each in the batch's path sequence
    // (nRenders + 1 entries), paths ended per render, the start and completion times
    // (globaltimer ns: [0] start, [1 + r] render r), the device loop's condition and its
    // iteration limit
    const RenderMeta *renders;
    const long long *pathStart;
    int nRenders;
    unsigned long long *ended;
    unsigned long long *times;
    cudaGraphConditionalHandle cond;
    int devLoop;        // the iterations run in a device loop on cond (else the host drives them)
    long long iterLimit;
};

// The path records (pool, class queues, hits, shadow queue) are written once and read once, by
// another kernel and far apart, so they are loaded and stored as streaming data (evict first):
// L1 and L2 keep the tree, the triangles and the materials.  Default policy against loads / both
// as streaming: a batch of 16 box rooms 145.1 / 145.0 / 142.3 ms, the mid-scale scene at 1080p
// with 16 samples 25.6 / 25.4 / 25.1, the material room at 333 x 217 1.31 / 1.30 / 1.28, the
// guided room 3.17 / 3.13 / 3.12.  (Rays that the end of a traversal reads again come from DRAM
// again, 262 instead of 202 MB an average extend launch of that frame; keeping those in the
// caches costs the tree 0.6-1 %.)

__device__ __forceinline__ int filmIndexS(const StreamArgs &p, int pix) {
    const int y = pix / p.W, x = pix - y * p.W;
    return y * p.W + (p.W - 1 - x);   // film pixel (W-1-x, y), core/integrator.cc:88
}

// slots refilled this iteration (every kernel of the iteration derives the same number
// from the counters, which only k_sadvance changes); not of one-pass renders
__device__ __forceinline__ long long totalPaths(const StreamArgs &p) { return static_cast<long long>(p.big[kBigTotal]); }
__device__ __forceinline__ float4 *filmOf(const StreamArgs &p) { return reinterpret_cast<float4 *>(p.big[kBigFilm]); }
__device__ __forceinline__ int newPaths(const StreamArgs &p) {
    const long long left = totalPaths(p) - static_cast<long long>(p.big[kBigStarted]);
    const long long freeSlots = p.cap - p.ctr[kCtrRays];
    return static_cast<int>(max(0LL, min(freeSlots, left)));
}

__device__ __forceinline__ int warpAppendS(bool want, int *counter) {
    const unsigned active = __activemask();
    const unsigned mask = __ballot_sync(active, want);
    if (!mask) return -1;
    const int lane = threadIdx.x & 31;
    const int leader = __ffs(mask) - 1;
    int base = 0;
    if (lane == leader) base = atomicAdd(counter, __popc(mask));
    base = __shfl_sync(active, base, leader);
    return want ? base + __popc(mask & ((1u << lane) - 1u)) : -1;
}

// batches: the render of path g of the batch's sequence (binary search of pathStart)
__device__ __forceinline__ int renderOfPath(const StreamArgs &p, long long g) {
    int lo = 0, hi = p.nRenders;   // pathStart[lo] <= g < pathStart[hi]
    while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        if (__ldg(&p.pathStart[mid]) <= g) lo = mid;
        else hi = mid;
    }
    return lo;
}

// batches: add the warp's ended paths to their renders' counts (whole warps call this)
__device__ __forceinline__ void countEnded(const StreamArgs &p, bool ended, int render) {
    const unsigned mask = __ballot_sync(__activemask(), ended);
    if (!ended) return;
    const unsigned same = __match_any_sync(mask, render);
    if ((threadIdx.x & 31) == __ffs(same) - 1)
        atomicAdd(&p.ended[render], static_cast<unsigned long long>(__popc(same)));
}

// film pixel of raster pixel pix in a film of width W (x mirrored, core/integrator.cc:88)
__device__ __forceinline__ int mirrored(int pix, int W) {
    const int y = pix / W, x = pix - y * W;
    return y * W + (W - 1 - x);
}

template <bool BATCH>
__global__ void k_sregen(StreamArgs p) {
    awaitLastKernel();
    const int have = p.onePass ? 0 : p.ctr[kCtrRays];
    const int nNew = p.onePass ? static_cast<int>(totalPaths(p)) : newPaths(p);
    if (p.onePass && blockIdx.x == 0 && threadIdx.x == 0) p.ctr[kCtrRays] = nNew;
    const long long started = static_cast<long long>(p.big[kBigStarted]);
    // one render: the first sample of the call; batches: the lane's first path in the
    // batch's sequence
    const long long offset = static_cast<long long>(p.big[kBigOffset]);
    float4 *film = filmOf(p);
    for (int j = blockIdx.x * blockDim.x + threadIdx.x; j < nNew; j += gridDim.x * blockDim.x) {
        const long long g = started + j;
        int render = 0, sample, pix, fi;
        long long filmBase = 0;
        float3 o, d;
        if constexpr (BATCH) {
            const long long gb = offset + g;
            render = renderOfPath(p, gb);
            const RenderMeta &M = p.renders[render];
            const long long local = gb - __ldg(&p.pathStart[render]);
            const int npix = M.W * M.H;
            sample = static_cast<int>(local / npix);
            pix = static_cast<int>(local % npix);
            const int y = pix / M.W, x = pix - y * M.W;
            fi = y * M.W + (M.W - 1 - x);
            const Rand4 r = rand4(M.seed, static_cast<uint32_t>(fi), static_cast<uint32_t>(sample), 0xFFFFu, 0u);
            spawnCameraRay(M.cam, x, y, r.a, r.b, &o, &d);
            filmBase = M.filmOffset;
        } else {
            sample = static_cast<int>(offset) + static_cast<int>(g / p.npix);
            pix = static_cast<int>(g % p.npix);
            const int y = pix / p.W, x = pix - y * p.W;
            fi = y * p.W + (p.W - 1 - x);
            const Rand4 r = rand4(p.seed, static_cast<uint32_t>(fi), static_cast<uint32_t>(sample), 0xFFFFu, 0u);
            spawnCameraRay(p.cam, x, y, r.a, r.b, &o, &d);
        }
        const int k = have + j;
        __stcs(&p.rO[k], make_float4(o.x, o.y, o.z, __int_as_float(pix)));
        __stcs(&p.rD[k], make_float4(d.x, d.y, d.z, packMeta(0, false, render)));
        __stcs(&p.rB[k], make_float4(1.0f, 1.0f, 1.0f, __int_as_float(sample)));
        atomicAdd(&film[filmBase + fi].w, 1.0f);
    }
}

// closest hit of the pool's rays into the class queues (every thread of the block)
// (OWN other than kFromCounter: a one-pass render, whose counter holds all its rays)
template <bool STATS, bool BATCH, bool SPLIT, bool SINGLE, int OWN = kFromCounter>
__device__ __forceinline__ void extendQueue(const StreamArgs &p, uint2 *stack) {
    uint32_t nodeCount = 0, triCount = 0;
    const int n = p.ctr[kCtrRays] + (OWN != kFromCounter ? 0 : newPaths(p));
    float4 *film = filmOf(p);
    bool overflow = false;
    auto done = [&](int i, const TraceLane &L) {
        if (!__any_sync(0xffffffffu, i >= 0)) return;
        if constexpr (SINGLE) {
            int render = 0;
            if (i >= 0) {
                __stcs(&p.qH[i], make_float4(L.tmax, __int_as_float(L.found ? L.hitSlot : -1), L.hu, L.hv));
                if (!L.found && (BATCH || p.sv.hasEnv)) {
                    const int meta = __float_as_int(__ldcs(&p.rD[i]).w);
                    if (BATCH) render = metaRender(meta);
                    else if ((meta & 255) == 0 || (meta & 256)) {
                        const float3 c = xyz(__ldcs(&p.rB[i])) * envLe(p.sv.env, L.d);
                        const int pix = __float_as_int(__ldcs(&p.rO[i]).w);
                        atomicAdd(&film[filmIndexS(p, pix)], make_float4(c.x, c.y, c.z, 0.0f));
                    }
                }
            }
            if constexpr (BATCH) countEnded(p, i >= 0 && !L.found, render);   // no environment
            return;
        }
        int cls = -1;
        float4 o4 = make_float4(0, 0, 0, 0), d4 = o4, b4 = o4;
        if (i >= 0) {
            o4 = __ldcs(&p.rO[i]);
            d4 = __ldcs(&p.rD[i]);
            b4 = __ldcs(&p.rB[i]);
            if (L.found) {
                cls = shadeClass(__ldg(&p.sv.mats[__ldg(&p.sv.slotShade[L.hitSlot]).x].type));
            } else if (!BATCH && p.sv.hasEnv) {
                // escaped: the environment at the first vertex or after a specular bounce
                const int meta = __float_as_int(d4.w);
                if ((meta & 255) == 0 || (meta & 256)) {
                    const float3 c = xyz(b4) * envLe(p.sv.env, L.d);
                    atomicAdd(&film[filmIndexS(p, __float_as_int(o4.w))], make_float4(c.x, c.y, c.z, 0.0f));
                }
            }
        }
        if constexpr (BATCH) countEnded(p, i >= 0 && !L.found, metaRender(__float_as_int(d4.w)));   // no environment
#pragma unroll
        for (int c = 0; c < 3; c++) {
            const int k = warpAppendS(cls == c, &p.ctr[kCtrClass0 + c]);
            if (k >= 0) {
                const int64_t row = static_cast<int64_t>(c) * p.cap + k;
                __stcs(&p.qO[row], o4);
                __stcs(&p.qD[row], d4);
                __stcs(&p.qB[row], b4);
                __stcs(&p.qH[row], make_float4(L.tmax, __int_as_float(L.hitSlot), L.hu, L.hv));
            }
        }
    };
    if constexpr (BATCH) {
        // each render's rays start at its own tree's root
        auto fetch = [&](int i, float3 *o, float3 *d, float *t0, float *t1, uint32_t *root) {
            const float4 d4 = __ldcs(&p.rD[i]);
            *o = xyz(__ldcs(&p.rO[i]));
            *d = xyz(d4);
            *t0 = 0.0f;
            *t1 = kInfT;
            *root = p.renders[metaRender(__float_as_int(d4.w))].root;
        };
        tracePersistent<false, STATS, SPLIT, OWN>(p.sv.nodes, p.sv.tris, p.sv.nNodes, p.sv.nTris, n, &p.ctr[kCtrFetchE],
                                      stack + threadIdx.x, kTraceBlock, &nodeCount, &triCount, &overflow, fetch,
                                      done);
    } else {
        auto fetch = [&](int i, float3 *o, float3 *d, float *t0, float *t1) {
            *o = xyz(__ldcs(&p.rO[i]));
            *d = xyz(__ldcs(&p.rD[i]));
            *t0 = 0.0f;
            *t1 = kInfT;
        };
        tracePersistent<false, STATS, SPLIT, OWN>(p.sv.nodes, p.sv.tris, p.sv.nNodes, p.sv.nTris, n, &p.ctr[kCtrFetchE],
                                      stack + threadIdx.x, kTraceBlock, &nodeCount, &triCount, &overflow, fetch,
                                      done);
    }
    if (overflow) atomicOr(&p.ctr[kCtrErr], 1);
    if (STATS) {
        atomicAdd(&p.big[kBigVisit + 0], static_cast<unsigned long long>(nodeCount));
        atomicAdd(&p.big[kBigVisit + 1], static_cast<unsigned long long>(triCount));
    }
}

template <bool STATS, bool BATCH, bool SPLIT, bool SINGLE>
__global__ void __launch_bounds__(kTraceBlock, kTraceMinBlocks) k_sextend(StreamArgs p) {
    __shared__ uint2 stack[kStackShared * kTraceBlock];
    extendQueue<STATS, BATCH, SPLIT, SINGLE>(p, stack);
}

// one shadow ray into the shadow queue; the lanes that have one at the same point of the
// shading append together
__device__ __forceinline__ void appendShadow(const StreamArgs &p, float4 so, float4 sd, float4 sl) {
    const int k = warpAppendS(true, &p.ctr[kCtrShadow]);
    __stcs(&p.shO[k], so);
    __stcs(&p.shD[k], sd);
    __stcs(&p.shL[k], sl);
}

// a shaded hit's emission (at film pixel filmIdx) and continuation (back into the pool);
// whole warps call this.  Batches count the paths that end here.
template <bool BATCH = false>
__device__ __forceinline__ void emitShadeResultS(const StreamArgs &p, const ShadeOut &R, bool live, long long filmIdx,
                                                 int pix, int meta, int sample) {
    if (live && !isBlack(R.emit))
        atomicAdd(&filmOf(p)[filmIdx], make_float4(R.emit.x, R.emit.y, R.emit.z, 0.0f));
    if constexpr (BATCH) countEnded(p, live && !R.cont, metaRender(meta));
    const int k = warpAppendS(R.cont && !p.direct, p.cont);
    if (k >= 0) {
        __stcs(&p.nO[k], make_float4(R.cO.x, R.cO.y, R.cO.z, __int_as_float(pix)));
        __stcs(&p.nD[k], make_float4(R.cD.x, R.cD.y, R.cD.z, packMeta((meta & 255) + 1, R.spec, metaRender(meta))));
        __stcs(&p.nB[k], make_float4(R.beta.x, R.beta.y, R.beta.z, __int_as_float(sample)));
    }
}

// First statement of the shading kernels (launchShading): a class that runs beside the last
// kernel does not wait for it, and one that lets the next run beside it does so only once what
// both depend on is complete.
__device__ __forceinline__ void beginShading(const StreamArgs &p) {
    if (p.besideLast) {
        cudaTriggerProgrammaticLaunchCompletion();
    } else if (p.besideNext) {
        cudaGridDependencySynchronize();
        cudaTriggerProgrammaticLaunchCompletion();
    } else {
        awaitLastKernel();
    }
}

// the rows that class cls shades in this iteration: its queue, or the pool's rays where the
// scene has that class alone
struct ShadeRows {
    const float4 *o, *d, *b, *h;
    int n;
};
__device__ __forceinline__ ShadeRows shadeRows(const StreamArgs &p, int cls) {
    if (p.singleClass >= 0) {
        const int rays = p.ctr[kCtrRays] + (p.onePass ? 0 : newPaths(p));
        return {p.rO, p.rD, p.rB, p.qH, p.singleClass == cls ? rays : 0};
    }
    const int64_t base = static_cast<int64_t>(cls) * p.cap;
    return {p.qO + base, p.qD + base, p.qB + base, p.qH + base, p.ctr[kCtrClass0 + cls]};
}

__device__ __forceinline__ HitRecord hitOfRow(float4 h4) {
    HitRecord h;
    h.t = h4.x;
    h.prim = __float_as_int(h4.y);
    h.u = h4.z;
    h.v = h4.w;
    return h;
}

// One class's queue, a row per thread.  Bound by latency (loads of the hit's triangle,
// material and light) and by instruction fetch, so the kernel holds its class's BSDFs only
// (narrowType), shadow rays leave the registers as soon as they are known (shadeHitTo), and
// the Lambert class, which then needs few registers, keeps 8 CTAs of 128 threads per SM
// (5 / 6 / 7 / 8: 154.3 / 153.1 / 153.1 / 151.6 ms for a batch of 16 box rooms).  Against
// every BSDF in each class's kernel and both shadow rays held to the end: that batch 185.3
// -> 151.6 ms, the 1080p mid-scale render (16 samples) 29.2 -> 27.7 ms, the material room
// at 333 x 217 (24 samples) 1.94 -> 1.81 ms.
template <int CLS, bool BATCH>
__global__ void __launch_bounds__(kShadeBlockS, shadeMinBlocks(CLS)) k_sshade(StreamArgs p) {
    beginShading(p);
    const ShadeRows rows = shadeRows(p, CLS);
    const int n = rows.n;
    const int stride = gridDim.x * blockDim.x;
    const int nIter = (n + stride - 1) / stride;   // uniform trip count keeps warps whole for the ballots
    for (int it = 0; it < nIter; it++) {
        const int j = it * stride + blockIdx.x * blockDim.x + threadIdx.x;
        ShadeOut R;
        R.cont = false;
        int pix = 0, meta = 0, sample = 0;
        long long filmIdx = 0;
        bool live = false;
        float4 h4 = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        if (j < n) {
            h4 = __ldcs(rows.h + j);
            live = p.singleClass < 0 || __float_as_int(h4.y) >= 0;   // a class queue holds hits only
        }
        if (live) {
            const float4 o4 = __ldcs(rows.o + j), d4 = __ldcs(rows.d + j), b4 = __ldcs(rows.b + j);
            pix = __float_as_int(o4.w);
            meta = __float_as_int(d4.w);
            sample = __float_as_int(b4.w);
            if constexpr (BATCH) {
                // the render's own lights, film, depth and random streams
                const int render = metaRender(meta);
                const RenderMeta &M = p.renders[render];
                SceneView S = p.sv;
                S.lightBase = M.lightBase;
                S.nArea = M.nArea;
                S.nLights = M.nArea;
                const int fi = mirrored(pix, M.W);
                filmIdx = M.filmOffset + fi;
                shadeHitTo<CLS>(S, hitOfRow(h4), xyz(o4), xyz(d4), xyz(b4), (meta & 256) != 0, meta & 255, M.maxDepth,
                                M.seed, static_cast<uint32_t>(fi), static_cast<uint32_t>(sample),
                                static_cast<int>(filmIdx), R, false, [&](int, float4 so, float4 sd, float4 sl) {
                                    sl.w = __int_as_float(render);   // the shadow ray's tree
                                    appendShadow(p, so, sd, sl);
                                });
            } else {
                const int fi = filmIndexS(p, pix);
                filmIdx = fi;
                shadeHitTo<CLS>(p.sv, hitOfRow(h4), xyz(o4), xyz(d4), xyz(b4), (meta & 256) != 0, meta & 255,
                                p.maxDepth, p.seed, static_cast<uint32_t>(fi), static_cast<uint32_t>(sample), fi, R,
                                p.direct != 0, [&](int, float4 so, float4 sd, float4 sl) { appendShadow(p, so, sd, sl); });
            }
        }
        emitShadeResultS<BATCH>(p, R, live, filmIdx, pix, meta, sample);
    }
    if (p.besideLast) cudaGridDependencySynchronize();
}

// Lambert hits of a guided render.  Each CTA takes 128-row tiles of the Lambert queue:
// every thread forms its row's network inputs, the tile runs through the four layers on
// the tensor cores (tcgen05, accumulator in TMEM), and each row is shaded with its
// mixture (shadeGuidedLambert), kept in shared memory.  Rows at the last depth, or past
// the guided depths, are shaded with plain BSDF sampling as in k_sshade.  The queue
// mixes depths, so one launch covers what the pass-by-pass wavefront does in one guided
// launch per bounce.
__global__ void __launch_bounds__(kGTile, kGuidedMinBlocks) k_sshade_guided(StreamArgs p) {
    beginShading(p);
    const ShadeRows rows = shadeRows(p, kMatLambert);
    const int n = rows.n;
    if (static_cast<int>(blockIdx.x) * kGTile >= n) return;   // no tile for this CTA
    extern __shared__ __align__(128) uint8_t sm[];
    bool ok = true;
    const uint32_t tmem = tileKernelSetup(sm, p.packFwd, p.biasPad, &ok, kGsOffBar);
    const float *bias = reinterpret_cast<const float *>(sm + kTileSmOffBias);
    uint8_t *xh = sm + kGsOffXH;
    MixRow &mix = reinterpret_cast<MixRow *>(sm + kGsOffXH)[threadIdx.x];
    uint64_t *bar = reinterpret_cast<uint64_t *>(sm + kGsOffBar);
    uint32_t phase = 0;
    for (int tile = blockIdx.x; ok && tile * kGTile < n; tile += gridDim.x) {
        const int j = tile * kGTile + static_cast<int>(threadIdx.x);
        float4 o4 = make_float4(0, 0, 0, 0), d4 = make_float4(0, 0, 1, 0), b4 = o4;
        float4 h4 = make_float4(0.0f, __int_as_float(-1), 0.0f, 0.0f);
        if (j < n) {
            o4 = __ldcs(rows.o + j);
            d4 = __ldcs(rows.d + j);
            b4 = __ldcs(rows.b + j);
            h4 = __ldcs(rows.h + j);
        }
        const bool live = __float_as_int(h4.y) >= 0;
        float3 ps = mk(0, 0, 0), nn = mk(0, 0, 1);
        float xf[16];
        for (int k = 0; k < 16; k++) xf[k] = 0.0f;
        if (live) {
            ps = hitPoint(xyz(o4), xyz(d4), h4.x);
            nn = triNormal(p.sv.tris[__float_as_int(h4.y)]);
            guideFeatures(ps, nn, -xyz(d4), p.guideLo, p.guideInvExt, xf);
        }
        __syncthreads();   // every row of the last tile is shaded: its mixtures may go
        storeRow8(xh, threadIdx.x, 0, kGK0, xf);
        storeRow8(xh, threadIdx.x, 8, kGK0, xf + 8);
        {
            float raw[kGOut];
            ok = mlpForwardRow(tmem, sm, bias, xh, bar, phase, raw);   // CTA-uniform
            // the last layer's MMA has read the tile, so each row's mixture may take its place
            if (ok) mixtureFromRaw(raw, mix.m);
        }
        if (!ok) break;
        ShadeOut R;
        R.cont = false;
        auto shadow = [&](int, float4 so, float4 sd, float4 sl) { appendShadow(p, so, sd, sl); };
        const int pix = __float_as_int(o4.w), meta = __float_as_int(d4.w), sample = __float_as_int(b4.w);
        if (live) {
            const int fi = filmIndexS(p, pix);
            const int depth = meta & 255;
            const bool spec = (meta & 256) != 0;
            if (depth < p.maxDepth && (p.guidedBounces <= 0 || depth < p.guidedBounces)) {
                const int2 sh = __ldg(&p.sv.slotShade[__float_as_int(h4.y)]);
                MaterialRecord m = p.sv.mats[sh.x];
                narrowType<kMatLambert>(m);
                float3 fc;
                float pdf;
                shadeGuidedLambertTo(p.sv, ps, nn, m, sh.y, xyz(d4), xyz(b4), spec, depth, mix.m, p.guideAlpha, p.seed,
                                     static_cast<uint32_t>(fi), static_cast<uint32_t>(sample), R, &fc, &pdf, shadow);
            } else {
                shadeHitTo<kMatLambert>(p.sv, hitOfRow(h4), xyz(o4), xyz(d4), xyz(b4), spec, depth, p.maxDepth, p.seed,
                                        static_cast<uint32_t>(fi), static_cast<uint32_t>(sample), fi, R, false, shadow);
            }
        }
        emitShadeResultS(p, R, live, live ? filmIndexS(p, pix) : 0, pix, meta, sample);
    }
    tileKernelTeardown(sm, tmem, ok, phase, kGsOffBar);
    if (!ok && threadIdx.x == 0) atomicOr(&p.ctr[kCtrErr], 2);
}

// any hit of the shadow rays counted in ctr, unoccluded ones to the film (every thread of the
// block)
template <bool STATS, bool BATCH, bool SPLIT, int OWN = kFromCounter>
__device__ __forceinline__ void shadowQueue(const StreamArgs &p, int *ctr, uint2 *stack) {
    const int n = ctr[kCtrShadow];
    float4 *film = filmOf(p);
    bool overflow = false;
    uint32_t nodeCount = 0, triCount = 0;
    auto done = [&](int i, const TraceLane &L) {
        if (i >= 0 && !L.found) {
            const float3 c = xyz(__ldcs(&p.shL[i]));
            atomicAdd(&film[__float_as_int(__ldcs(&p.shO[i]).w)], make_float4(c.x, c.y, c.z, 0.0f));
        }
    };
    if constexpr (BATCH) {
        auto fetch = [&](int i, float3 *o, float3 *d, float *t0, float *t1, uint32_t *root) {
            const float4 d4 = __ldcs(&p.shD[i]);
            *o = xyz(__ldcs(&p.shO[i]));
            *d = xyz(d4);
            *t0 = 0.0f;
            *t1 = d4.w;
            *root = p.renders[__float_as_int(p.shL[i].w)].root;
        };
        tracePersistent<true, STATS, SPLIT, OWN>(p.sv.nodes, p.sv.tris, p.sv.nNodes, p.sv.nTris, n, &ctr[kCtrFetchS],
                                     stack + threadIdx.x, kTraceBlock, &nodeCount, &triCount, &overflow, fetch, done);
    } else {
        auto fetch = [&](int i, float3 *o, float3 *d, float *t0, float *t1) {
            const float4 d4 = __ldcs(&p.shD[i]);
            *o = xyz(__ldcs(&p.shO[i]));
            *d = xyz(d4);
            *t0 = 0.0f;
            *t1 = d4.w;
        };
        tracePersistent<true, STATS, SPLIT, OWN>(p.sv.nodes, p.sv.tris, p.sv.nNodes, p.sv.nTris, n, &ctr[kCtrFetchS],
                                     stack + threadIdx.x, kTraceBlock, &nodeCount, &triCount, &overflow, fetch, done);
    }
    if (overflow) atomicOr(&ctr[kCtrErr], 1);
    if (STATS) {
        atomicAdd(&p.big[kBigVisit + 2], static_cast<unsigned long long>(nodeCount));
        atomicAdd(&p.big[kBigVisit + 3], static_cast<unsigned long long>(triCount));
    }
}

template <bool STATS, bool BATCH, bool SPLIT>
__global__ void __launch_bounds__(kTraceBlock, kTraceMinBlocks) k_sshadow(StreamArgs p) {
    __shared__ uint2 stack[kStackShared * kTraceBlock];
    shadowQueue<STATS, BATCH, SPLIT>(p, p.ctr, stack);
}

// One-pass renders: an iteration's closest hits (EXTEND) and the last iteration's shadow rays,
// which do not depend on each other, in one launch; a warp that finds no more of the first
// goes on with the second.
template <bool EXTEND, bool SPLIT, bool SINGLE>
__global__ void __launch_bounds__(kTraceBlock, kTraceMinBlocks) k_strace(StreamArgs p) {
    __shared__ uint2 stack[kStackShared * kTraceBlock];
    awaitLastKernel();
    if constexpr (EXTEND) extendQueue<false, false, SPLIT, SINGLE, kOwnFromFirst>(p, stack);
    if (p.shadowCtr) shadowQueue<false, false, SPLIT, kOwnFromLast>(p, p.shadowCtr, stack);
}

// one thread: account the iteration, hand the continuations to the next one, reset the
// per-iteration counters, raise the done flag once no path is left.  Batches also stamp
// the completion time of every render whose paths have all ended (all the block's
// threads, renders strided over them), and set the device loop's condition: another
// round while paths remain and the iteration limit is not reached.
template <bool BATCH>
__global__ void k_sadvance(StreamArgs p) {
    if (blockIdx.x != 0) return;
    if constexpr (BATCH) {
        // completion stamps, the renders strided over the block's threads
        unsigned long long now;
        asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(now));
        for (int r = threadIdx.x; r < p.nRenders; r += blockDim.x) {
            const unsigned long long paths = static_cast<unsigned long long>(p.pathStart[r + 1] - p.pathStart[r]);
            if (p.times[1 + r] == 0 && atomicAdd(&p.ended[r], 0ull) == paths) atomicCAS(&p.times[1 + r], 0ull, now);
        }
    }
    if (threadIdx.x != 0) return;
    const int nNew = newPaths(p);
    const int n = p.ctr[kCtrRays] + nNew;
    p.big[kBigStarted] += static_cast<unsigned long long>(nNew);
    p.big[kBigPaths] += static_cast<unsigned long long>(nNew);
    p.big[kBigClosest] += static_cast<unsigned long long>(n);
    p.big[kBigShadow] += static_cast<unsigned long long>(p.ctr[kCtrShadow]);
    p.ctr[kCtrRays] = p.ctr[kCtrCont];
    for (int k = kCtrCont; k <= kCtrFetchS; k++) p.ctr[k] = 0;
    if (n > 0) p.ctr[kCtrIter] += 1;
    const bool done = p.ctr[kCtrRays] == 0 && static_cast<long long>(p.big[kBigStarted]) >= totalPaths(p);
    p.ctr[kCtrDone] = done ? 1 : 0;
    if constexpr (BATCH) {
        const long long iters = static_cast<long long>(++p.big[kBigIters]);
        if (!done && iters >= p.iterLimit) p.ctr[kCtrErr] |= 4;   // the pool did not drain in time
        if (p.devLoop) cudaGraphSetConditional(p.cond, !done && iters < p.iterLimit ? 1u : 0u);
    }
}

enum KernelClassS { kSRegen = 0, kSExtend, kSShadeL, kSShadeC, kSShadeD, kSShadow, kSAdvance, kSNumClasses };

struct GridsS {
    int trace, shade, regen, guided;
};

// The traversal kernels' eight blocks per SM use 64 KB of shared memory.  A carveout of a third
// (72 of 228 KB) leaves the rest to L1, which serves half of their node loads: 30 / 40 / 60 % and
// the driver's choice, a batch of 16 box rooms 145.2 / 145.1 / 148.1 / 146.3 ms, the mid-scale
// render 25.51 / 25.53 / 25.72 / 25.62.  (Not for k_strace, whose launches alternate with small
// shading launches.)
bool preferL1() {
    for (const void *k : {reinterpret_cast<const void *>(k_sextend<false, false, false, false>),
                          reinterpret_cast<const void *>(k_sextend<false, false, false, true>),
                          reinterpret_cast<const void *>(k_sextend<false, false, true, false>),
                          reinterpret_cast<const void *>(k_sextend<false, false, true, true>),
                          reinterpret_cast<const void *>(k_sextend<false, true, false, false>),
                          reinterpret_cast<const void *>(k_sextend<false, true, false, true>),
                          reinterpret_cast<const void *>(k_sshadow<false, false, false>),
                          reinterpret_cast<const void *>(k_sshadow<false, false, true>),
                          reinterpret_cast<const void *>(k_sshadow<false, true, false>)})
        cudaFuncSetAttribute(k, cudaFuncAttributePreferredSharedMemoryCarveout, 32);
    cudaGetLastError();   // a preference
    return true;
}

GridsS streamGrids(int device, int cap, bool guided) {
    int sms = 0;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
    // resident blocks per SM: properties of the compiled kernels
    static const int occT = [] {
        int o = 0;
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&o, k_sextend<false, false, true, false>, kTraceBlock, 0);
        return o;
    }();
    static const int occS = [] {
        int o = 0;
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&o, k_sshade<0, false>, kShadeBlockS, 0);
        return o;
    }();
    static const bool carved = preferL1();
    (void)carved;
    GridsS g;
    g.trace = sms * std::max(occT, 1);
    g.shade = sms * std::max(occS, 1);
    g.regen = std::max(1, std::min((cap + 255) / 256, sms * 8));
    g.guided = guided ? guideTileKernelGrid(reinterpret_cast<const void *>(k_sshade_guided), device, kGsSmem) : 0;
    return g;
}

// a kernel of an iteration; one-pass renders launch it as dependent on the stream's last kernel
// (awaitLastKernel), so that its set-up overlaps that kernel's end
template <class K>
cudaError_t launchStreamKernel(K kernel, int grid, int block, size_t smem, cudaStream_t s, const StreamArgs &a) {
    cudaLaunchAttribute dependent;
    dependent.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    dependent.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(static_cast<unsigned>(grid));
    cfg.blockDim = dim3(static_cast<unsigned>(block));
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cfg.attrs = &dependent;
    cfg.numAttrs = a.onePass ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, kernel, a);
}

// Pools and class of a render's iterations: two pools where the scene has one shading class (its
// mask has one bit), the pool and the class queues otherwise.
void setPools(StreamArgs &a, int classMask) {
    a.singleClass = classMask == 1 ? 0 : classMask == 2 ? 1 : classMask == 4 ? 2 : -1;
    a.nO = a.singleClass >= 0 ? a.qO : a.rO;
    a.nD = a.singleClass >= 0 ? a.qD : a.rD;
    a.nB = a.singleClass >= 0 ? a.qB : a.rB;
}
// every other iteration's arguments
StreamArgs poolsSwapped(StreamArgs a) {
    if (a.singleClass >= 0) {
        std::swap(a.rO, a.nO);
        std::swap(a.rD, a.nD);
        std::swap(a.rB, a.nB);
    }
    return a;
}

// The shading kernels of the classes in mask; returns how many.  In one-pass renders they run
// beside each other: they depend on the extend before them, not on one another.  The first waits
// for it and then lets the second begin, which lets the third begin at once; each of these ends
// only after the one before it, so whatever follows the last follows all.  Small queues' rows
// take long (a rough dielectric's five evaluations and its iterated slope inversion), so the
// glossy class goes first: the conductor room at 281 x 159 (15 samples) 0.77 -> 0.70 ms, the
// material room at 100 x 80 (4) 0.52 -> 0.49, the mid-scale scene at 1080p (8) 13.4 -> 13.1.
template <bool BATCH>
int launchShading(const StreamArgs &a, const GridsS &g, cudaStream_t s, int mask) {
    const int total = (mask & 1) + (mask >> 1 & 1) + (mask >> 2 & 1);
    int n = 0;
    StreamArgs p = a;
    auto launch = [&](auto kernel, int grid, int block, size_t smem) {
        p.besideLast = a.onePass && n > 0;
        p.besideNext = a.onePass && n + 1 < total;
        launchStreamKernel(kernel, grid, block, smem, s, p);
        n++;
    };
    if ((mask & 1) && a.packFwd) launch(k_sshade_guided, g.guided, kGTile, kGsSmem);
    if (mask & 2) launch(k_sshade<1, BATCH>, g.shade, kShadeBlockS, 0);
    if (mask & 4) launch(k_sshade<2, BATCH>, g.shade, kShadeBlockS, 0);
    if ((mask & 1) && !a.packFwd) launch(k_sshade<0, BATCH>, g.shade, kShadeBlockS, 0);
    return n;
}

// one iteration on stream s with the shading classes in mask; with ev, every kernel is bracketed
// by a pair of events
template <bool STATS, bool BATCH = false>
void launchIteration(const StreamArgs &a, const GridsS &g, cudaStream_t s, cudaEvent_t *ev, int *evClass, int *nev,
                     int mask = 7) {
    auto mark = [&](int cls) {
        if (ev) {
            evClass[*nev / 2] = cls;
            cudaEventRecord(ev[(*nev)++], s);
        }
    };
    auto done = [&]() {
        if (ev) cudaEventRecord(ev[(*nev)++], s);
    };
    // batches are of many small trees
    const bool split = !BATCH && a.sv.nNodes >= kSplitMinNodes && a.cap >= kSplitMinRays;
    mark(kSRegen);
    k_sregen<BATCH><<<g.regen, 256, 0, s>>>(a);
    done();
    mark(kSExtend);
    const bool single = !STATS && a.singleClass >= 0;
    if (split && single) k_sextend<STATS, BATCH, !BATCH, !STATS><<<g.trace, kTraceBlock, 0, s>>>(a);
    else if (split) k_sextend<STATS, BATCH, !BATCH, false><<<g.trace, kTraceBlock, 0, s>>>(a);
    else if (single) k_sextend<STATS, BATCH, false, !STATS><<<g.trace, kTraceBlock, 0, s>>>(a);
    else k_sextend<STATS, BATCH, false, false><<<g.trace, kTraceBlock, 0, s>>>(a);
    done();
    for (int c = 0; c < 3; c++) {
        if (!((mask >> c) & 1)) continue;
        mark(kSShadeL + c);
        launchShading<BATCH>(a, g, s, 1 << c);
        done();
    }
    mark(kSShadow);
    if (split) k_sshadow<STATS, BATCH, !BATCH><<<g.trace, kTraceBlock, 0, s>>>(a);
    else k_sshadow<STATS, BATCH, false><<<g.trace, kTraceBlock, 0, s>>>(a);
    done();
    mark(kSAdvance);
    k_sadvance<BATCH><<<1, BATCH ? 256 : 32, 0, s>>>(a);
    done();
}

uint64_t hashBytesS(const void *d, size_t n, uint64_t h = 1469598103934665603ull) {
    const unsigned char *c = static_cast<const unsigned char *>(d);
    for (size_t i = 0; i < n; i++) h = (h ^ c[i]) * 1099511628211ull;
    return h;
}

int ensureStreamQueues(StreamQueues &q, int cap) {
    if (q.capacity >= cap && q.rO) return 0;
    freeStreamQueues(&q);
    auto alloc = [&](auto **ptr, size_t count) {
        using T = std::remove_pointer_t<std::remove_reference_t<decltype(*ptr)>>;
        return cudaMalloc(reinterpret_cast<void **>(ptr), sizeof(T) * std::max<size_t>(count, 1)) == cudaSuccess;
    };
    const size_t c = static_cast<size_t>(cap);
    bool ok = alloc(&q.rO, c) && alloc(&q.rD, c) && alloc(&q.rB, c) && alloc(&q.qO, 3 * c) && alloc(&q.qD, 3 * c) &&
              alloc(&q.qB, 3 * c) && alloc(&q.qH, 3 * c) && alloc(&q.shO, 2 * c) && alloc(&q.shD, 2 * c) &&
              alloc(&q.shL, 2 * c) && alloc(&q.ctr, kNumCtr * kMaxIters) && alloc(&q.big, kNumBig);
    if (ok) ok = cudaMallocHost(reinterpret_cast<void **>(&q.doneHost), sizeof(int) * kDoneRing) == cudaSuccess;
    if (ok) ok = cudaMallocHost(reinterpret_cast<void **>(&q.ctrHost), sizeof(int) * kNumCtr * kMaxIters) == cudaSuccess;
    if (ok) {
        for (int k = 0; k < kDoneRing && ok; k++) ok = cudaEventCreateWithFlags(&q.doneEv[k], cudaEventDisableTiming) == cudaSuccess;
    }
    if (!ok) {
        cudaGetLastError();
        freeStreamQueues(&q);
        setError("spgpu_render: device allocation of the streaming path pool failed");
        return SPGPU_ENOMEM;
    }
    q.capacity = cap;
    return 0;
}

// the render's own parameters for the device (kBigTotal.. kBigFilm), the other counters zero
struct StreamInit {
    unsigned long long big[kNumBig];
};
StreamInit streamInit(long long total, int sampleOffset, float4 *film) {
    StreamInit s;
    std::memset(&s, 0, sizeof(s));
    s.big[kBigTotal] = static_cast<unsigned long long>(total);
    s.big[kBigOffset] = static_cast<unsigned long long>(static_cast<long long>(sampleOffset));
    s.big[kBigFilm] = reinterpret_cast<unsigned long long>(film);
    return s;
}

int setupStream(Ctx &C, StreamQueues &q, const float *camera, int W, int H, int spp, int maxDepth, uint32_t seed,
                int integrator, const GuideView *gv, StreamArgs *out) {
    const long long npix = static_cast<long long>(W) * H;
    const long long total = npix * spp;
    const int cap = static_cast<int>(std::min<long long>(std::max<long long>(total, 1), Ctx::kStreamSlots));
    if (int rc = ensureStreamQueues(q, cap)) return rc;
    StreamArgs &a = *out;
    std::memset(&a, 0, sizeof(a));
    a.sv = C.view();
    a.cam = makeCamera(camera, W, H);
    a.W = W;
    a.H = H;
    a.npix = static_cast<int>(npix);
    a.maxDepth = integrator == SPGPU_INTEGRATOR_DIRECT ? 1 : maxDepth;
    a.seed = seed;
    a.direct = integrator == SPGPU_INTEGRATOR_DIRECT ? 1 : 0;
    a.cap = q.capacity;
    a.rO = q.rO;
    a.rD = q.rD;
    a.rB = q.rB;
    a.qO = q.qO;
    a.qD = q.qD;
    a.qB = q.qB;
    a.qH = q.qH;
    a.shO = q.shO;
    a.shD = q.shD;
    a.shL = q.shL;
    a.ctr = q.ctr;
    a.cont = q.ctr + kCtrCont;
    a.big = q.big;
    setPools(a, C.classMask);
    if (gv) {
        a.packFwd = gv->packFwd;
        a.biasPad = gv->biasPad;
        a.guideAlpha = gv->alpha;
        a.guidedBounces = gv->guidedBounces;
        a.guideLo = C.bvh.lo;
        const float3 ext = C.bvh.hi - C.bvh.lo;
        a.guideInvExt = mk(ext.x > 0 ? 1.0f / ext.x : 0.0f, ext.y > 0 ? 1.0f / ext.y : 0.0f,
                           ext.z > 0 ? 1.0f / ext.z : 0.0f);
    }
    return 0;
}

// (re)capture the graph of kIterPerGraph iterations when anything baked into it changes
int ensureStreamGraph(Ctx &C, StreamQueues &q, const StreamArgs &a, cudaStream_t s) {
    const uint64_t key = hashBytesS(&a, sizeof(a));
    if (q.graph && q.graphKey == key) return 0;
    if (q.graph) cudaGraphExecDestroy(q.graph);
    q.graph = nullptr;
    const GridsS g = streamGrids(C.device, a.cap, a.packFwd != nullptr);
    cudaGraph_t graph = nullptr;
    cudaError_t e = cudaStreamBeginCapture(s, cudaStreamCaptureModeThreadLocal);
    if (e != cudaSuccess) return cudaFail("cudaStreamBeginCapture", e);
    static_assert(kIterPerGraph % 2 == 0, "the two pools of a one-class scene end up in their places");
    for (int it = 0; it < kIterPerGraph; it++)
        launchIteration<false>(it % 2 ? poolsSwapped(a) : a, g, s, nullptr, nullptr, nullptr);
    e = cudaStreamEndCapture(s, &graph);
    if (e != cudaSuccess) return cudaFail("cudaStreamEndCapture", e);
    e = cudaGraphInstantiate(&q.graph, graph, 0);
    cudaGraphDestroy(graph);
    if (e != cudaSuccess) return cudaFail("cudaGraphInstantiate", e);
    q.graphKey = key;
    return 0;
}

// a generous bound on the iterations of a render: a path ends within maxDepth + 1
// iterations of its start, and a full pool is refilled at least once in that time
long long iterationBound(const StreamArgs &a, long long total) {
    return 2 * (static_cast<long long>(a.maxDepth) + 2) * (total / std::max(a.cap, 1) + 2) + 16;
}

// the start of a batch run: every lane's counters and parameters (its share of the
// batch's path sequence, the film), the per-render counts and times.  One kernel, so
// that the reset is part of the batch's graph.
struct BatchReset {
    int *ctr[Ctx::kPoolLanes];
    unsigned long long *big[Ctx::kPoolLanes];
    long long first[Ctx::kPoolLanes], count[Ctx::kPoolLanes];
    int lanes;
    int nRenders;
    unsigned long long film;
    unsigned long long *ended, *times;
};

__global__ void k_sbatch_reset(BatchReset in) {
    const int t = threadIdx.x;
    for (int k = 0; k < in.lanes; k++) {
        for (int i = t; i < kNumCtr; i += blockDim.x) in.ctr[k][i] = 0;
        for (int i = t; i < kNumBig; i += blockDim.x)
            in.big[k][i] = i == kBigTotal    ? static_cast<unsigned long long>(in.count[k])
                           : i == kBigOffset ? static_cast<unsigned long long>(in.first[k])
                           : i == kBigFilm   ? in.film
                                             : 0ull;
    }
    for (int r = t; r < in.nRenders; r += blockDim.x) {
        in.ended[r] = 0;
        in.times[1 + r] = 0;
    }
    if (t == 0) {
        unsigned long long now;
        asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(now));
        in.times[0] = now;
    }
}

}  // namespace

inline int popcount3(int mask) { return (mask & 1) + (mask >> 1 & 1) + (mask >> 2 & 1); }

struct StreamBatch {
    int lanes = 1, iterations = 0;
    StreamQueues q[Ctx::kPoolLanes];   // the batch's own pools (the context's serve spgpu_render)
    SceneView sv{};                    // the merged scenes
    RenderMeta *renders = nullptr;     // device
    long long *pathStart = nullptr;    // device, nRenders + 1
    unsigned long long *ended = nullptr, *times = nullptr;
    int nRenders = 0, maxDepth = 0, classMask = 7;
    std::vector<long long> hostStart;
    cudaGraphExec_t exec = nullptr;
    float4 *execFilm = nullptr;
};

void freeStreamBatch(StreamBatch *SB) {
    if (!SB) return;
    if (SB->exec) cudaGraphExecDestroy(SB->exec);
    for (auto &q : SB->q) freeStreamQueues(&q);
    cudaFree(SB->renders);
    cudaFree(SB->pathStart);
    cudaFree(SB->ended);
    cudaFree(SB->times);
    delete SB;
}

int streamBatchCreate(Ctx &C, StreamBatch **slot, const SceneView &merged, const std::vector<RenderMeta> &renders,
                      int classMask, int poolSlots, int lanes, int iterations) {
    freeStreamBatch(*slot);
    *slot = nullptr;
    // a path carries its render in bits 9..30 of its meta word
    if (renders.empty() || renders.size() >= (1u << 22) || poolSlots <= 0 || lanes < 1 || lanes > Ctx::kPoolLanes ||
        iterations < 1) {
        setError("spgpu_batch_prepare: invalid streaming batch shape (at most 2^22 - 1 renders)");
        return SPGPU_EINVAL;
    }
    auto *SB = new StreamBatch();
    SB->lanes = lanes;
    SB->iterations = iterations;
    SB->classMask = classMask;
    SB->sv = merged;
    SB->nRenders = static_cast<int>(renders.size());
    SB->hostStart.assign(renders.size() + 1, 0);
    for (size_t r = 0; r < renders.size(); r++) {
        const RenderMeta &M = renders[r];
        SB->hostStart[r + 1] = SB->hostStart[r] + static_cast<long long>(M.W) * M.H * M.spp;
        SB->maxDepth = std::max(SB->maxDepth, M.maxDepth);
    }
    const long long total = SB->hostStart.back();
    const int cap = static_cast<int>(std::min<long long>(poolSlots, std::max<long long>(1, (total + lanes - 1) / lanes)));
    int rc = 0;
    for (int k = 0; k < lanes && rc == 0; k++) rc = ensureStreamQueues(SB->q[k], cap);
    cudaError_t e = cudaSuccess;
    if (rc == 0) e = cudaMalloc(&SB->renders, sizeof(RenderMeta) * renders.size());
    if (rc == 0 && e == cudaSuccess) e = cudaMalloc(&SB->pathStart, sizeof(long long) * SB->hostStart.size());
    if (rc == 0 && e == cudaSuccess) e = cudaMalloc(&SB->ended, sizeof(unsigned long long) * renders.size());
    if (rc == 0 && e == cudaSuccess) e = cudaMalloc(&SB->times, sizeof(unsigned long long) * (renders.size() + 1));
    if (rc == 0 && e == cudaSuccess)
        e = cudaMemcpy(SB->renders, renders.data(), sizeof(RenderMeta) * renders.size(), cudaMemcpyHostToDevice);
    if (rc == 0 && e == cudaSuccess)
        e = cudaMemcpy(SB->pathStart, SB->hostStart.data(), sizeof(long long) * SB->hostStart.size(),
                       cudaMemcpyHostToDevice);
    if (rc == 0 && e != cudaSuccess) rc = cudaFail("spgpu_batch_prepare", e);
    if (rc) {
        freeStreamBatch(SB);
        return rc;
    }
    *slot = SB;
    return 0;
}

namespace {

// the lane's kernel arguments: the merged scenes, the lane's pool, the batch tables
StreamArgs batchLaneArgs(const StreamBatch &SB, int k, cudaGraphConditionalHandle cond) {
    StreamArgs a;
    std::memset(&a, 0, sizeof(a));
    const StreamQueues &q = SB.q[k];
    a.sv = SB.sv;
    a.maxDepth = SB.maxDepth;
    a.cap = q.capacity;
    a.rO = q.rO;
    a.rD = q.rD;
    a.rB = q.rB;
    a.qO = q.qO;
    a.qD = q.qD;
    a.qB = q.qB;
    a.qH = q.qH;
    a.shO = q.shO;
    a.shD = q.shD;
    a.shL = q.shL;
    a.ctr = q.ctr;
    a.cont = q.ctr + kCtrCont;
    a.big = q.big;
    // an odd number of iterations would leave the rays in the other pool
    setPools(a, SB.iterations % 2 == 0 ? SB.classMask : 0);
    a.renders = SB.renders;
    a.pathStart = SB.pathStart;
    a.nRenders = SB.nRenders;
    a.ended = SB.ended;
    a.times = SB.times;
    a.cond = cond;
    return a;
}

// The batch's graph: the reset kernel, then per lane a conditional while node whose
// body is `iterations` wavefront iterations; the body's last k_sadvance decides
// whether the loop goes round again.  Film address baked in (recaptured per film).
int buildBatchGraph(Ctx &C, StreamBatch &SB, float4 *film) {
    if (SB.exec) cudaGraphExecDestroy(SB.exec);
    SB.exec = nullptr;
    const long long total = SB.hostStart.back();
    BatchReset init;
    std::memset(&init, 0, sizeof(init));
    init.lanes = SB.lanes;
    init.nRenders = SB.nRenders;
    init.film = reinterpret_cast<unsigned long long>(film);
    init.ended = SB.ended;
    init.times = SB.times;
    for (int k = 0; k < SB.lanes; k++) {
        init.ctr[k] = SB.q[k].ctr;
        init.big[k] = SB.q[k].big;
        init.first[k] = total * k / SB.lanes;
        init.count[k] = total * (k + 1) / SB.lanes - init.first[k];
    }
    cudaStream_t cs = C.stream;
    cudaGraph_t G = nullptr;
    cudaError_t e = cudaGraphCreate(&G, 0);
    if (e == cudaSuccess) e = cudaStreamBeginCaptureToGraph(cs, G, nullptr, nullptr, 0, cudaStreamCaptureModeThreadLocal);
    if (e == cudaSuccess) {
        k_sbatch_reset<<<1, 256, 0, cs>>>(init);
        e = cudaStreamEndCapture(cs, &G);
    }
    cudaGraphNode_t resetNode = nullptr;
    size_t nNodes = 1;
    if (e == cudaSuccess) e = cudaGraphGetNodes(G, &resetNode, &nNodes);
    const GridsS g = streamGrids(C.device, SB.q[0].capacity, false);
    for (int k = 0; k < SB.lanes && e == cudaSuccess; k++) {
        cudaGraphConditionalHandle h = 0;
        e = cudaGraphConditionalHandleCreate(&h, G, 1, cudaGraphCondAssignDefault);
        cudaGraphNodeParams cp = {};
        cp.type = cudaGraphNodeTypeConditional;
        cp.conditional.handle = h;
        cp.conditional.type = cudaGraphCondTypeWhile;
        cp.conditional.size = 1;
        cudaGraphNode_t node = nullptr;
        if (e == cudaSuccess) e = cudaGraphAddNode(&node, G, &resetNode, nullptr, 1, &cp);
        if (e != cudaSuccess) break;
        cudaGraph_t body = cp.conditional.phGraph_out[0];
        StreamArgs a = batchLaneArgs(SB, k, h);
        a.devLoop = 1;
        a.iterLimit = iterationBound(a, init.count[k]);
        e = cudaStreamBeginCaptureToGraph(cs, body, nullptr, nullptr, 0, cudaStreamCaptureModeThreadLocal);
        if (e != cudaSuccess) break;
        for (int it = 0; it < SB.iterations; it++)
            launchIteration<false, true>(it % 2 ? poolsSwapped(a) : a, g, cs, nullptr, nullptr, nullptr, SB.classMask);
        e = cudaStreamEndCapture(cs, &body);
    }
    if (e == cudaSuccess) e = cudaGraphInstantiate(&SB.exec, G, 0);
    if (G) cudaGraphDestroy(G);
    if (e != cudaSuccess) {
        SB.exec = nullptr;
        return cudaFail("spgpu_batch_run (graph)", e);
    }
    SB.execFilm = film;
    return 0;
}

}  // namespace

int streamBatchRun(Ctx &C, StreamBatch &SB, float4 *film, double *renderMs, unsigned long long *statsOut,
                   float *msOut, cudaStream_t stream) {
    if (!SB.exec || SB.execFilm != film) {
        if (int rc = buildBatchGraph(C, SB, film)) return rc;
    }
    cudaEvent_t e0, e1;
    cudaEventCreate(&e0);
    cudaEventCreate(&e1);
    cudaError_t e = cudaEventRecord(e0, stream);
    if (e == cudaSuccess) e = cudaGraphLaunch(SB.exec, stream);
    if (e == cudaSuccess) e = cudaEventRecord(e1, stream);
    std::vector<unsigned long long> times(SB.nRenders + 1);
    unsigned long long big[Ctx::kPoolLanes][kNumBig] = {};
    int ctr[Ctx::kPoolLanes][kNumCtr] = {};
    if (e == cudaSuccess)
        e = cudaMemcpyAsync(times.data(), SB.times, sizeof(unsigned long long) * times.size(), cudaMemcpyDeviceToHost,
                            stream);
    for (int k = 0; k < SB.lanes && e == cudaSuccess; k++) {
        e = cudaMemcpyAsync(big[k], SB.q[k].big, sizeof(big[k]), cudaMemcpyDeviceToHost, stream);
        if (e == cudaSuccess) e = cudaMemcpyAsync(ctr[k], SB.q[k].ctr, sizeof(ctr[k]), cudaMemcpyDeviceToHost, stream);
    }
    if (e == cudaSuccess) e = cudaStreamSynchronize(stream);
    float ms = 0.0f;
    if (e == cudaSuccess) cudaEventElapsedTime(&ms, e0, e1);
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    if (e != cudaSuccess) return cudaFail("spgpu_batch_run", e);
    int err = 0;
    bool drained = true;
    for (int k = 0; k < 4; k++) statsOut[k] = 0;
    for (int k = 0; k < SB.lanes; k++) {
        statsOut[0] += big[k][kBigPaths];
        statsOut[1] += big[k][kBigClosest];
        statsOut[2] += big[k][kBigShadow];
        // an iteration: regen, extend, the batch's shading classes, shadow, advance; and the reset
        statsOut[3] += big[k][kBigIters] * (4 + popcount3(SB.classMask)) + 1;
        err |= ctr[k][kCtrErr];
        drained = drained && ctr[k][kCtrDone];
    }
    for (int r = 0; r < SB.nRenders; r++)
        renderMs[r] = times[1 + r] >= times[0] && times[1 + r] ? (times[1 + r] - times[0]) * 1.0e-6 : -1.0;
    *msOut = ms;
    if (err & 1) {
        setError("spgpu_batch_run: traversal stack overflow");
        return SPGPU_EKERNEL;
    }
    if ((err & 4) || !drained) {
        setError("spgpu_batch_run: the path pools did not drain within their iteration bound");
        return SPGPU_EKERNEL;
    }
    return 0;
}

void freeStreamQueues(StreamQueues *q) {
    if (q->graph) cudaGraphExecDestroy(q->graph);
    cudaFree(q->rO);
    cudaFree(q->rD);
    cudaFree(q->rB);
    cudaFree(q->qO);
    cudaFree(q->qD);
    cudaFree(q->qB);
    cudaFree(q->qH);
    cudaFree(q->shO);
    cudaFree(q->shD);
    cudaFree(q->shL);
    cudaFree(q->ctr);
    cudaFree(q->big);
    if (q->doneHost) cudaFreeHost(q->doneHost);
    if (q->ctrHost) cudaFreeHost(q->ctrHost);
    for (int k = 0; k < StreamQueues::kEvents; k++)
        if (q->doneEv[k]) cudaEventDestroy(q->doneEv[k]);
    *q = StreamQueues{};
}

namespace {

// Paths up to which a one-pass render takes a single lane.  Two lanes' kernels overlap, but each
// has its own launches, and they take turns on the chip; several classes, which run beside each
// other, and guided shading fill it alone for longer.  One lane / two: box room, 393k paths 0.419
// / 0.427 ms, 720k 0.500 / 0.490, 1M 0.620 / 0.601; mid-scale scene, 518k 1.95 / 2.74; conductor
// room, 670k 0.70 / 0.76; material room, 1.7M 1.39 / 1.31; guided room, 460k 1.37 / 1.47, 922k
// 1.95 / 2.01, 1.8M 3.31 / 3.32.
long long oneLanePaths(const StreamArgs &a) {
    return a.singleClass >= 0 && !a.packFwd ? 1 << 19 : 1 << 20;
}

// A render whose paths all fit the pools' slots at once.  Every path starts in the first
// iteration and iteration b handles depth b, so the iterations are known beforehand: no refill,
// no done flag, no replays past the end, and no graph to capture for a new camera.  Each
// iteration has its own counters (nothing resets them), its shadow rays are traced in the next
// iteration's launch, and the classes that the scene has no material of are not launched: two
// kernels for an iteration of a one-class scene instead of seven.  Bound by the launches' own
// latency at the small end.  Against the refilling loop's replays: box room, 64 x 64, 16
// samples (host film) 1.00 -> 0.43 ms (0.26 with the context's kept host film); material room,
// 333 x 217, 24 samples 1.82 -> 1.32; guided room, 640 x 360, 8 samples 4.04 -> 3.23.
int renderOnePass(Ctx &C, const float *camera, int W, int H, int spp, int sampleOffset, int maxDepth, uint32_t seed,
                  int integrator, float4 *film, unsigned long long *statsOut, float *msOut, cudaStream_t stream,
                  const GuideView *gv) {
    const long long total = static_cast<long long>(W) * H * spp;
    StreamArgs a[Ctx::kPoolLanes] = {};
    setPools(a[0], C.classMask);
    a[0].packFwd = gv ? gv->packFwd : nullptr;
    const int lanes = total <= oneLanePaths(a[0]) ? 1 : std::max(1, std::min(spp, Ctx::kPoolLanes));
    StreamInit init[Ctx::kPoolLanes];
    cudaStream_t ls[Ctx::kPoolLanes];
    int first = sampleOffset;
    for (int k = 0; k < lanes; k++) {
        const int sppK = spp / lanes + (k < spp % lanes ? 1 : 0);
        if (int rc = setupStream(C, C.sq[k], camera, W, H, sppK, maxDepth, seed, integrator, gv, &a[k])) return rc;
        a[k].onePass = 1;
        init[k] = streamInit(static_cast<long long>(W) * H * sppK, first, film);
        first += sppK;
        ls[k] = k == 0 ? stream : C.laneStream[k - 1];
    }
    // a path's last vertex (depth maxDepth) is shaded in the last iteration and has no shadow
    // rays; direct lighting has one vertex, whose shadow rays take a launch of their own
    const bool direct = integrator == SPGPU_INTEGRATOR_DIRECT;
    const int iters = direct ? 1 : maxDepth + 1;
    const GridsS g = streamGrids(C.device, a[0].cap, a[0].packFwd != nullptr);
    const bool split = a[0].sv.nNodes >= kSplitMinNodes && a[0].cap >= kSplitMinRays;
    long long launches = 0;
    cudaEvent_t e0, e1;
    cudaEventCreate(&e0);
    cudaEventCreate(&e1);
    cudaError_t e = cudaEventRecord(e0, stream);
    if (e == cudaSuccess && lanes > 1) e = cudaEventRecord(C.laneFork, stream);
    for (int k = 0; k < lanes && e == cudaSuccess; k++) {
        if (k > 0) e = cudaStreamWaitEvent(ls[k], C.laneFork, 0);
        if (e == cudaSuccess) e = cudaMemsetAsync(C.sq[k].ctr, 0, sizeof(int) * kNumCtr * (iters + 1), ls[k]);
        if (e == cudaSuccess)
            e = cudaMemcpyAsync(C.sq[k].big, init[k].big, sizeof(init[k].big), cudaMemcpyHostToDevice, ls[k]);
        if (e != cudaSuccess) break;
        k_sregen<false><<<g.regen, 256, 0, ls[k]>>>(a[k]);
        launches++;
    }
    constexpr int kLookAhead = 16;   // deep renders: iterations launched between two looks at the paths left
    int done = iters;                // iterations launched
    for (int it = 0; it < iters && e == cudaSuccess; it++) {
        if (it > 0 && it % kLookAhead == 0) {
            int left = 0;
            for (int k = 0; k < lanes && e == cudaSuccess; k++) {
                e = cudaMemcpyAsync(C.sq[k].ctrHost, a[k].cont, sizeof(int), cudaMemcpyDeviceToHost, ls[k]);
                if (e == cudaSuccess) e = cudaStreamSynchronize(ls[k]);
                if (e == cudaSuccess) left += C.sq[k].ctrHost[0];
            }
            if (e == cudaSuccess && left == 0) {
                done = it;
                break;
            }
        }
        for (int k = 0; k < lanes && e == cudaSuccess; k++) {
            StreamArgs &p = a[k];
            p.ctr = C.sq[k].ctr + kNumCtr * it;
            p.cont = p.ctr + kNumCtr + kCtrRays;
            p.shadowCtr = it > 0 ? p.ctr - kNumCtr : nullptr;
            if (it > 0) p = poolsSwapped(p);
            const bool single = p.singleClass >= 0;
            launchStreamKernel(split ? (single ? k_strace<true, true, true> : k_strace<true, true, false>)
                                     : (single ? k_strace<true, false, true> : k_strace<true, false, false>),
                               g.trace, kTraceBlock, 0, ls[k], p);
            launches++;
            launches += launchShading<false>(p, g, ls[k], C.classMask);
            e = cudaGetLastError();
        }
    }
    if (direct || done < iters) {   // the shadow rays of the last iteration launched
        for (int k = 0; k < lanes && e == cudaSuccess; k++) {
            a[k].shadowCtr = C.sq[k].ctr + kNumCtr * (done - 1);
            launchStreamKernel(split ? k_strace<false, true, false> : k_strace<false, false, false>, g.trace, kTraceBlock, 0,
                               ls[k], a[k]);
            launches++;
            e = cudaGetLastError();
        }
    }
    for (int k = 0; k < lanes && e == cudaSuccess; k++)
        e = cudaMemcpyAsync(C.sq[k].ctrHost, C.sq[k].ctr, sizeof(int) * kNumCtr * (done + 1), cudaMemcpyDeviceToHost, ls[k]);
    for (int k = 1; k < lanes && e == cudaSuccess; k++) {
        e = cudaEventRecord(C.laneJoin[k - 1], ls[k]);
        if (e == cudaSuccess) e = cudaStreamWaitEvent(stream, C.laneJoin[k - 1], 0);
    }
    if (e == cudaSuccess) e = cudaEventRecord(e1, stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(stream);
    float ms = 0.0f;
    if (e == cudaSuccess) cudaEventElapsedTime(&ms, e0, e1);
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    if (e != cudaSuccess) return cudaFail("spgpu_render", e);
    int err = 0;
    for (int k = 0; k < lanes; k++) {
        const int *c = C.sq[k].ctrHost;
        statsOut[0] += init[k].big[kBigTotal];
        for (int it = 0; it < done; it++, c += kNumCtr) {
            statsOut[1] += static_cast<unsigned long long>(c[kCtrRays]);
            statsOut[2] += static_cast<unsigned long long>(c[kCtrShadow]);
            err |= c[kCtrErr];
        }
    }
    statsOut[3] = static_cast<unsigned long long>(launches);
    *msOut = ms;
    if (err) {
        setError(err & 1 ? "spgpu_render: traversal stack overflow"
                         : "spgpu_render: tensor-core wait of the guided shading timed out");
        return SPGPU_EKERNEL;
    }
    return 0;
}

}  // namespace

int renderStream(Ctx *ctx, const float *camera, int W, int H, int spp, int sampleOffset, int maxDepth, uint32_t seed,
                 int integrator, float4 *film, unsigned long long *statsOut, float *msOut, cudaStream_t stream,
                 const GuideView *gv) {
    Ctx &C = *ctx;
    for (int j = 0; j < 4; j++) statsOut[j] = 0;
    *msOut = 0.0f;
    if (spp <= 0 || W <= 0 || H <= 0) return 0;
    // one pass where each lane's samples fit its pool's slots
    const int perLane = (spp + Ctx::kPoolLanes - 1) / Ctx::kPoolLanes;
    if (static_cast<long long>(W) * H * perLane <= Ctx::kStreamSlots)
        return renderOnePass(C, camera, W, H, spp, sampleOffset, maxDepth, seed, integrator, film, statsOut, msOut,
                             stream, gv);
    // pool lanes: lane k renders a contiguous share of the samples, lane 0 on the caller's
    // stream, lane k > 0 on the context's lane stream k - 1
    const int lanes = std::max(1, std::min(spp, Ctx::kPoolLanes));
    StreamArgs a[Ctx::kPoolLanes];
    StreamInit init[Ctx::kPoolLanes];
    cudaStream_t ls[Ctx::kPoolLanes];
    long long maxReplays[Ctx::kPoolLanes], replays[Ctx::kPoolLanes];
    bool finished[Ctx::kPoolLanes];
    int first = sampleOffset;
    for (int k = 0; k < lanes; k++) {
        const int sppK = spp / lanes + (k < spp % lanes ? 1 : 0);
        if (int rc = setupStream(C, C.sq[k], camera, W, H, sppK, maxDepth, seed, integrator, gv, &a[k])) return rc;
        // captured on the context's own stream (the caller's may be the legacy default
        // stream, which cannot be captured), replayed on the lane's
        if (int rc = ensureStreamGraph(C, C.sq[k], a[k], C.stream)) return rc;
        const long long total = static_cast<long long>(W) * H * sppK;
        init[k] = streamInit(total, first, film);
        first += sppK;
        ls[k] = k == 0 ? stream : C.laneStream[k - 1];
        maxReplays[k] = iterationBound(a[k], total) / kIterPerGraph + kReplayLag + 2;
        replays[k] = 0;
        finished[k] = false;
    }
    cudaEvent_t e0, e1;
    cudaEventCreate(&e0);
    cudaEventCreate(&e1);
    cudaError_t e = cudaEventRecord(e0, stream);
    if (e == cudaSuccess && lanes > 1) e = cudaEventRecord(C.laneFork, stream);
    for (int k = 0; k < lanes && e == cudaSuccess; k++) {
        StreamQueues &q = C.sq[k];
        if (k > 0) e = cudaStreamWaitEvent(ls[k], C.laneFork, 0);
        if (e == cudaSuccess) e = cudaMemsetAsync(q.ctr, 0, sizeof(int) * kNumCtr, ls[k]);
        if (e == cudaSuccess)
            e = cudaMemcpyAsync(q.big, init[k].big, sizeof(init[k].big), cudaMemcpyHostToDevice, ls[k]);
    }
    // replay each lane's graph until its pool drains, reading each lane's done flag
    // kReplayLag replays back
    int open = lanes;
    while (e == cudaSuccess && open > 0) {
        for (int k = 0; k < lanes && e == cudaSuccess; k++) {
            if (finished[k]) continue;
            StreamQueues &q = C.sq[k];
            if (replays[k] >= maxReplays[k]) {
                finished[k] = true;   // reported below: the done flag stays unset
                open--;
                continue;
            }
            const int slot = static_cast<int>(replays[k] % kDoneRing);
            e = cudaGraphLaunch(q.graph, ls[k]);
            if (e == cudaSuccess)
                e = cudaMemcpyAsync(&q.doneHost[slot], q.ctr + kCtrDone, sizeof(int), cudaMemcpyDeviceToHost, ls[k]);
            if (e == cudaSuccess) e = cudaEventRecord(q.doneEv[slot], ls[k]);
            replays[k]++;
            if (e == cudaSuccess && replays[k] > kReplayLag) {
                const int back = static_cast<int>((replays[k] - 1 - kReplayLag) % kDoneRing);
                e = cudaEventSynchronize(q.doneEv[back]);
                if (e == cudaSuccess && q.doneHost[back]) {
                    finished[k] = true;
                    open--;
                }
            }
        }
    }
    for (int k = 1; k < lanes && e == cudaSuccess; k++) {
        e = cudaEventRecord(C.laneJoin[k - 1], ls[k]);
        if (e == cudaSuccess) e = cudaStreamWaitEvent(stream, C.laneJoin[k - 1], 0);
    }
    if (e == cudaSuccess) e = cudaEventRecord(e1, stream);
    unsigned long long big[Ctx::kPoolLanes][kNumBig] = {};
    int ctr[Ctx::kPoolLanes][kNumCtr] = {};
    for (int k = 0; k < lanes && e == cudaSuccess; k++) {
        e = cudaMemcpyAsync(big[k], C.sq[k].big, sizeof(big[k]), cudaMemcpyDeviceToHost, stream);
        if (e == cudaSuccess) e = cudaMemcpyAsync(ctr[k], C.sq[k].ctr, sizeof(ctr[k]), cudaMemcpyDeviceToHost, stream);
    }
    if (e == cudaSuccess) e = cudaStreamSynchronize(stream);
    float ms = 0.0f;
    if (e == cudaSuccess) cudaEventElapsedTime(&ms, e0, e1);
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    if (e != cudaSuccess) return cudaFail("spgpu_render", e);
    int err = 0;
    bool drained = true;
    for (int k = 0; k < lanes; k++) {
        statsOut[0] += big[k][kBigPaths];
        statsOut[1] += big[k][kBigClosest];
        statsOut[2] += big[k][kBigShadow];
        statsOut[3] += static_cast<unsigned long long>(replays[k]) * kIterPerGraph * kSNumClasses;
        err |= ctr[k][kCtrErr];
        drained = drained && ctr[k][kCtrDone];
    }
    *msOut = ms;
    if (err) {
        setError(err & 1 ? "spgpu_render: traversal stack overflow"
                         : "spgpu_render: tensor-core wait of the guided shading timed out");
        return SPGPU_EKERNEL;
    }
    if (!drained) {
        setError("spgpu_render: the path pool did not drain within its iteration bound");
        return SPGPU_EKERNEL;
    }
    return 0;
}

int renderStreamProfile(Ctx *ctx, const float *camera, int W, int H, int spp, int sampleOffset, int maxDepth,
                        uint32_t seed, int integrator, float4 *film, double *kernelMs, long long *launches,
                        unsigned long long *statsOut, unsigned long long *visitOut, cudaStream_t stream,
                        const GuideView *gv) {
    Ctx &C = *ctx;
    for (int k = 0; k < kSNumClasses; k++) {
        kernelMs[k] = 0.0;
        launches[k] = 0;
    }
    for (int k = 0; k < 4; k++) statsOut[k] = visitOut[k] = 0;
    if (spp <= 0 || W <= 0 || H <= 0) return 0;
    StreamArgs a;
    StreamQueues &q = C.sq[0];
    if (int rc = setupStream(C, q, camera, W, H, spp, maxDepth, seed, integrator, gv, &a)) return rc;
    setPools(a, 7);   // through the class queues, whose kernels the profile times
    const GridsS g = streamGrids(C.device, a.cap, a.packFwd != nullptr);
    const long long total = static_cast<long long>(W) * H * spp;
    const StreamInit init = streamInit(total, sampleOffset, film);
    const long long bound = iterationBound(a, total);
    std::vector<cudaEvent_t> ev(2 * 7);
    std::vector<int> cls(8);
    for (auto &x : ev) cudaEventCreate(&x);
    unsigned long long big[kNumBig] = {};
    int ctr[kNumCtr] = {};
    cudaError_t e = cudaSuccess;
    // pass 0: every kernel timed by events, one iteration at a time; pass 1: the same
    // paths again with the visit counters on
    for (int pass = 0; pass < 2 && e == cudaSuccess; pass++) {
        e = cudaMemsetAsync(q.ctr, 0, sizeof(int) * kNumCtr, stream);
        if (e == cudaSuccess) e = cudaMemcpyAsync(q.big, init.big, sizeof(init.big), cudaMemcpyHostToDevice, stream);
        for (long long it = 0; it < bound && e == cudaSuccess; it++) {
            int nev = 0;
            if (pass == 0) launchIteration<false>(a, g, stream, ev.data(), cls.data(), &nev);
            else launchIteration<true>(a, g, stream, nullptr, nullptr, nullptr);
            e = cudaGetLastError();
            if (e == cudaSuccess) e = cudaMemcpyAsync(ctr, q.ctr, sizeof(ctr), cudaMemcpyDeviceToHost, stream);
            if (e == cudaSuccess) e = cudaStreamSynchronize(stream);
            for (int i = 0; i + 1 < nev && e == cudaSuccess; i += 2) {
                float ms = 0.0f;
                cudaEventElapsedTime(&ms, ev[i], ev[i + 1]);
                kernelMs[cls[i / 2]] += ms;
                launches[cls[i / 2]] += 1;
            }
            if (ctr[kCtrDone]) break;
        }
        if (e == cudaSuccess) e = cudaMemcpy(big, q.big, sizeof(big), cudaMemcpyDeviceToHost);
        if (pass == 0)
            for (int k = 0; k < 3; k++) statsOut[k] = big[kBigPaths + k];
        else
            for (int k = 0; k < 4; k++) visitOut[k] = big[kBigVisit + k];
    }
    for (auto &x : ev) cudaEventDestroy(x);
    if (e != cudaSuccess) return cudaFail("spgpu_render_profile", e);
    if (ctr[kCtrErr]) {
        setError(ctr[kCtrErr] & 1 ? "spgpu_render_profile: traversal stack overflow"
                                  : "spgpu_render_profile: tensor-core wait of the guided shading timed out");
        return SPGPU_EKERNEL;
    }
    return 0;
}

}  // namespace spgpu

namespace spgpu {

// The batch's streaming wavefront launched kernel by kernel from the host (no graph),
// lane 0's pool taking the whole path sequence: pass 0 times every kernel with events,
// pass 1 renders the same paths again with the BVH visit counters on (the film receives
// both passes).  kernelMs/launches per kernel class.
int streamBatchProfile(Ctx &C, StreamBatch &SB, float4 *film, double *kernelMs, long long *launches,
                       unsigned long long *statsOut, unsigned long long *visitOut, cudaStream_t stream) {
    for (int k = 0; k < kSNumClasses; k++) {
        kernelMs[k] = 0.0;
        launches[k] = 0;
    }
    for (int k = 0; k < 4; k++) statsOut[k] = visitOut[k] = 0;
    StreamArgs a = batchLaneArgs(SB, 0, 0);
    setPools(a, 7);   // through the class queues, whose kernels the profile times
    const long long total = SB.hostStart.back();
    a.iterLimit = iterationBound(a, total);
    BatchReset init;
    std::memset(&init, 0, sizeof(init));
    init.lanes = 1;
    init.nRenders = SB.nRenders;
    init.film = reinterpret_cast<unsigned long long>(film);
    init.ended = SB.ended;
    init.times = SB.times;
    init.ctr[0] = SB.q[0].ctr;
    init.big[0] = SB.q[0].big;
    init.first[0] = 0;
    init.count[0] = total;
    const GridsS g = streamGrids(C.device, a.cap, false);
    std::vector<cudaEvent_t> ev(2 * kSNumClasses);
    std::vector<int> cls(kSNumClasses + 1);
    for (auto &x : ev) cudaEventCreate(&x);
    unsigned long long big[kNumBig] = {};
    int ctr[kNumCtr] = {};
    cudaError_t e = cudaSuccess;
    for (int pass = 0; pass < 2 && e == cudaSuccess; pass++) {
        k_sbatch_reset<<<1, 256, 0, stream>>>(init);
        e = cudaGetLastError();
        for (long long it = 0; it < a.iterLimit && e == cudaSuccess; it++) {
            int nev = 0;
            if (pass == 0) launchIteration<false, true>(a, g, stream, ev.data(), cls.data(), &nev);
            else launchIteration<true, true>(a, g, stream, nullptr, nullptr, nullptr);
            e = cudaGetLastError();
            if (e == cudaSuccess) e = cudaMemcpyAsync(ctr, SB.q[0].ctr, sizeof(ctr), cudaMemcpyDeviceToHost, stream);
            if (e == cudaSuccess) e = cudaStreamSynchronize(stream);
            for (int i = 0; i + 1 < nev && e == cudaSuccess; i += 2) {
                float ms = 0.0f;
                cudaEventElapsedTime(&ms, ev[i], ev[i + 1]);
                kernelMs[cls[i / 2]] += ms;
                launches[cls[i / 2]] += 1;
            }
            if (ctr[kCtrDone]) break;
        }
        if (e == cudaSuccess) e = cudaMemcpy(big, SB.q[0].big, sizeof(big), cudaMemcpyDeviceToHost);
        if (pass == 0)
            for (int k = 0; k < 3; k++) statsOut[k] = big[kBigPaths + k];
        else
            for (int k = 0; k < 4; k++) visitOut[k] = big[kBigVisit + k];
    }
    for (auto &x : ev) cudaEventDestroy(x);
    if (e != cudaSuccess) return cudaFail("spgpu_batch_profile", e);
    if (ctr[kCtrErr] & 1) {
        setError("spgpu_batch_profile: traversal stack overflow");
        return SPGPU_EKERNEL;
    }
    if (!ctr[kCtrDone]) {
        setError("spgpu_batch_profile: the path pool did not drain within its iteration bound");
        return SPGPU_EKERNEL;
    }
    return 0;
}

}  // namespace spgpu
