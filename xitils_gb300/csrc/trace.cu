// Extension (closest-hit) and shadow (any-hit) kernels of the wavefront.
//
// Both are persistent: a grid of (SMs x resident blocks) whose warps claim queue entries
// with one atomicAdd for all their lanes that want one -- 32 at a time in the general
// kernels, as many as are free in the per-lane ones (RayClaims) -- so the grid drains queues
// of any length without a relaunch per batch.
#include <map>
#include <mutex>

#include "trace.cuh"
#include "xgb_kernels.h"

#include <type_traits>

namespace xgb {

__device__ __forceinline__ void filmAdd(const RenderParams& rp, int pix, V3 c) {
    if (rp.dropNonFinite && !(isfinite(c.x) && isfinite(c.y) && isfinite(c.z))) return;
    if (rp.filmFp64) {
        double* f = (double*)rp.film + 4 * (size_t)pix;
        atomicAdd(f, (double)c.x);
        atomicAdd(f + 1, (double)c.y);
        atomicAdd(f + 2, (double)c.z);
    } else {
        float4* f = (float4*)rp.film + pix;
        atomicAdd(f, make_float4(c.x, c.y, c.z, 0.0f));
    }
}

// Guide training: a visible light's contribution also goes to its path's accumulator.
__device__ __forceinline__ void creditPath(const RenderParams& rp, unsigned int pid, float4 c) {
    float4 a = rp.pathAcc[pid];
    rp.pathAcc[pid] = make_float4(a.x + c.x, a.y + c.y, a.z + c.z, a.w);
}

constexpr int kTraceBlock = 128;

template <bool COUNT>
__global__ void __launch_bounds__(kTraceBlock) k_extend(SceneDev sc, PathQueue q, HitQueue h, Ctrl* ctrl) {
    const unsigned int n = ctrl->nActive;
    const int lane = threadIdx.x & 31;
    WorkCount wc;
    for (;;) {
        unsigned int base = 0;
        if (lane == 0) base = atomicAdd(&ctrl->extendHead, 32u);
        base = __shfl_sync(0xFFFFFFFFu, base, 0);
        if (base >= n) break;
        unsigned int i = base + lane;
        if (i < n) {
            float4 o = q.o[i], d = q.d[i];
            TraceHit hit;
            traceScene<false, COUNT>(sc, V3(o.x, o.y, o.z), V3(d.x, d.y, d.z), __int_as_float(0x7f800000), hit,
                                     &ctrl->errors, wc);
            h.h[i] = make_float4(hit.t, hit.b0, hit.b1, __int_as_float(hit.prim));
            h.inst[i] = hit.inst;
        }
    }
    if (COUNT) {
        unsigned long long nv = wc.nodes, nt = wc.tris;
        for (int off = 16; off > 0; off >>= 1) {
            nv += __shfl_down_sync(0xFFFFFFFFu, nv, off);
            nt += __shfl_down_sync(0xFFFFFFFFu, nt, off);
        }
        if (lane == 0) {
            atomicAdd(&ctrl->nodeVisits, nv);
            atomicAdd(&ctrl->triTests, nt);
        }
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) atomicAdd(&ctrl->extensionRays, (unsigned long long)n);
}

__global__ void __launch_bounds__(kTraceBlock) k_shadow(SceneDev sc, RenderParams rp, ShadowQueue s, PathQueue out,
                                                        Ctrl* ctrl) {
    const unsigned int n = ctrl->nShadowDue;
    const int lane = threadIdx.x & 31;
    for (;;) {
        unsigned int base = 0;
        if (lane == 0) base = atomicAdd(&ctrl->shadowHead, 32u);
        base = __shfl_sync(0xFFFFFFFFu, base, 0);
        if (base >= n) break;
        unsigned int i = base + lane;
        if (i < n) {
            float4 o = s.o[i], d = s.d[i];
            TraceHit hit;
            WorkCount wc;
            bool occluded = traceScene<true>(sc, V3(o.x, o.y, o.z), V3(d.x, d.y, d.z), o.w, hit, &ctrl->errors, wc);
            if (!occluded) {
                float4 c = s.c[i];
                filmAdd(rp, __float_as_int(d.w), V3(c.x, c.y, c.z));
                int target = __float_as_int(c.w);
                // A stochastic bsdfCos (MicrofacetNormalMapping) drew from the path's
                // stream only because the light was visible (PathTracer.h:209-227):
                // commit the stream position it left.
                if (target >= 0) out.rng[target] = s.rng[i];
                if (rp.train) creditPath(rp, s.pid[i], c);
            }
        }
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) atomicAdd(&ctrl->shadowRays, (unsigned long long)n);
}

// Scene lookup of the flat kernels: one scene (the kernel argument) or one per
// job of a batch (the job in the high byte of the ray's pixel field).
struct OneScene {
    SceneDev sc;
    RenderParams rp;
    __device__ __forceinline__ int jobOf(unsigned int) const { return 0; }
    __device__ __forceinline__ int pixelOf(unsigned int packed) const { return (int)packed; }
    __device__ __forceinline__ bool teams() const { return sc.teams != 0; }
    __device__ __forceinline__ bool counted() const { return sc.maxSteps != kDefaultMaxSteps; }
    __device__ __forceinline__ const SceneDev& scene(int) const { return sc; }
    __device__ __forceinline__ const RenderParams& params(int) const { return rp; }
};
struct BatchScenes {
    BatchView b;
    __device__ __forceinline__ int jobOf(unsigned int packed) const { return (int)(packed >> 24); }
    __device__ __forceinline__ int pixelOf(unsigned int packed) const { return (int)(packed & 0xFFFFFFu); }
    __device__ __forceinline__ bool teams() const { return b.teams != 0; }
    __device__ __forceinline__ bool counted() const { return b.counted != 0; }
    __device__ __forceinline__ const SceneDev& scene(int j) const { return b.scenes[j]; }
    __device__ __forceinline__ const RenderParams& params(int j) const { return b.params[j]; }
};
// What an unoccluded shadow ray does.
template <class S>
__device__ __forceinline__ void shadowLit(const S& scenes, int job, ShadowQueue s, PathQueue out, unsigned int ray) {
    const float4 cc = s.c[ray];
    const RenderParams& rp = scenes.params(job);
    filmAdd(rp, scenes.pixelOf(__float_as_uint(s.d[ray].w)), V3(cc.x, cc.y, cc.z));
    const int target = __float_as_int(cc.w);
    if (target >= 0) out.rng[target] = s.rng[ray];
    if (rp.train) creditPath(rp, s.pid[ray], cc);
}
// Ray queries on a scene of one instance (xgb_scene_intersect / xgb_scene_occluded): the rays
// and results are the caller's rows, 7 floats (o, d, tMax) and 5 (t, instance, triangle, b0,
// b1; -1 for none) or a flag.
struct QueryRays {
    SceneDev sc;
    const float* rays;
    float* hits;
    int* occluded;
    __device__ __forceinline__ int jobOf(unsigned int) const { return 0; }
    __device__ __forceinline__ bool teams() const { return false; }
    __device__ __forceinline__ bool counted() const { return false; }
    __device__ __forceinline__ const SceneDev& scene(int) const { return sc; }
};

// ---- scenes of a few instances: 8-wide mesh BVHs ------------------------------
// With at most kFlatInstances instances the top level is a short list: a lane
// walks the instances in order (those whose world box the ray still reaches
// within tMax) and traverses each mesh's 8-wide BVH as a persistent per-lane
// state machine in the style of Aila & Laine ("Understanding the Efficiency of
// Ray Traversal on GPUs", HPG 2009): the lanes of a warp test nodes together
// until each holds a leaf child (postponing it) or has no nodes left, then test
// their leaves' triangles together; a lane whose ray is finished fetches the
// next one at once (one atomicAdd per group of lanes), so the warp never waits
// for its slowest ray. Results are those of traceScene: the same watertight
// tests and the same closest-hit acceptance (tMax shrinks across instances).

template <bool ANY, bool COUNT>
__global__ void __launch_bounds__(kTraceBlock) k_trace_wide(SceneDev sc, RenderParams rp, PathQueue q, HitQueue h,
                                                            ShadowQueue s, PathQueue out, Ctrl* ctrl) {
    const unsigned int n = ANY ? ctrl->nShadowDue : ctrl->nActive;
    unsigned int* head = ANY ? &ctrl->shadowHead : &ctrl->extendHead;
    const int nInst = sc.nInstances;
    const int lane = threadIdx.x & 31;
    const unsigned int ltMask = (1u << lane) - 1u;
    unsigned int stack[kWideStack];
    int sp = 0;
    int inst = nInst;  // instance being traversed
    unsigned int ray = 0;
    V3 wo(0.f, 0.f, 0.f), wd(0.f, 0.f, 1.f);
    BoxRay br{0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    WRay r;
    int oct = 0;
    const WNode* nodes = nullptr;
    const TriV* tris = nullptr;
    WideHdr hd;
    hd.imask = 0; hd.childBase = 0; hd.triBase = 0; hd.meta0 = 0; hd.meta1 = 0;
    int node = 0;
    unsigned int mask = 0;
    bool inMesh = false;  // a mesh traversal is under way
    int leafFirst = 0, leafCnt = 0;  // postponed leaf child
    float tMax = 0.0f;
    TraceHit hit;
    hit.prim = -1;
    hit.inst = -1;
    hit.t = 0.0f;
    hit.b0 = hit.b1 = 0.0f;
    bool occluded = false;
    bool fetch = true;
    int steps = 0;  // traversal steps of the current ray
    WorkCount wc;
    for (;;) {
        if (fetch) {
            // lanes without a ray fetch the next ones together
            const unsigned int act = __activemask();
            const int leader = __ffs(act) - 1;
            unsigned int base = 0;
            if (lane == leader) base = atomicAdd(head, (unsigned int)__popc(act));
            base = __shfl_sync(act, base, leader);
            ray = base + __popc(act & ltMask);
            if (ray >= n) break;
            float4 o4, d4;
            // queue records: streaming loads / stores, as in k_shade
            if (ANY) { o4 = __ldcs(&s.o[ray]); d4 = __ldcs(&s.d[ray]); tMax = o4.w; }
            else { o4 = __ldcs(&q.o[ray]); d4 = __ldcs(&q.d[ray]); tMax = __int_as_float(0x7f800000); }
            wo = V3(o4.x, o4.y, o4.z);
            wd = V3(d4.x, d4.y, d4.z);
            br = BoxRay{wo.x, wo.y, wo.z, 1.0f / wd.x, 1.0f / wd.y, 1.0f / wd.z};
            hit.prim = -1;
            hit.inst = -1;
            hit.t = tMax;
            occluded = false;
            inst = -1;
            inMesh = false;
            leafCnt = 0;
            steps = 0;
            fetch = false;
        }
        if (!inMesh) {
            // next instance whose world box the ray still reaches, or the end of the ray
            if (!(ANY && occluded))
                for (++inst; inst < nInst; ++inst)
                    if (instBoxHit(br, sc.instBox, inst, tMax)) break;
            if ((ANY && occluded) || inst >= nInst) {
                if (ANY) {
                    if (!occluded) {
                        float4 cc = s.c[ray];
                        filmAdd(rp, __float_as_int(s.d[ray].w), V3(cc.x, cc.y, cc.z));
                        int target = __float_as_int(cc.w);
                        if (target >= 0) out.rng[target] = s.rng[ray];
                        if (rp.train) creditPath(rp, s.pid[ray], cc);
                    }
                } else {
                    __stcs(&h.h[ray], make_float4(hit.prim >= 0 ? hit.t : tMax, hit.b0, hit.b1, __int_as_float(hit.prim)));
                    __stcs(&h.inst[ray], hit.inst);
                }
                fetch = true;
            } else {
                const Instance& in = sc.instances[inst];
                const MeshDev& m = sc.meshes[in.mesh];
                nodes = m.nodes;
                tris = m.tris;
                if (in.identity) r = makeWRay(wo, wd);
                else r = makeWRay(xformPointRn(in.matInv, wo), xformVectorRn(in.matInv, wd));
                if (m.rootIsLeaf) {  // the whole mesh is one leaf: test it below, then the next instance
                    leafFirst = 0;
                    leafCnt = m.nTris;
                } else {
                    oct = rayOctant(r);
                    sp = 0;
                    node = 0;
                    mask = wideEval(nodes, r, oct, tMax, hd);
                    if (COUNT) wc.nodes++;
                    inMesh = true;
                }
            }
        }
        // node phase: the warp steps through nodes until every lane holds a leaf child or has none left
        for (;;) {
            const bool active = inMesh && leafCnt == 0;
            if (!__any_sync(__activemask(), active)) break;
            if (!active) continue;
            if (++steps > sc.maxSteps) {
                atomicOr(&ctrl->errors, 4u);
                inMesh = false;
                inst = nInst;
                continue;
            }
            if (mask == 0u) {
                if (sp == 0) {
                    inMesh = false;  // this mesh is done
                } else {
                    const unsigned int e = stack[--sp];
                    node = (int)(e >> 8);
                    mask = e & 0xFFu;
                    wideHeader(nodes + node, hd);
                }
                continue;
            }
            const int slot = (__ffs(mask) - 1) ^ oct;
            mask &= mask - 1u;
            const unsigned int mb = byteOf(slot >> 2 ? hd.meta1 : hd.meta0, slot);
            if ((hd.imask >> slot) & 1u) {
                if (mask) {
                    if (sp >= kWideStack || sp >= sc.stackLimit) {
                        atomicOr(&ctrl->errors, 1u);
                        inMesh = false;
                        inst = nInst;
                        continue;
                    }
                    stack[sp++] = ((unsigned int)node << 8) | mask;
                }
                node = hd.childBase + (int)mb;
                mask = wideEval(nodes + node, r, oct, tMax, hd);
                if (COUNT) wc.nodes++;
            } else {
                leafFirst = hd.triBase + (int)(mb & 31u);
                leafCnt = (int)(mb >> 5);
            }
        }
        // leaf phase: the postponed leaf children's triangles, together
        if (leafCnt) {
            if (COUNT) wc.tris += leafCnt;
            if (testTris(tris, leafFirst, leafCnt, r, tMax, hit, inst, ANY) && ANY) {
                occluded = true;
                inMesh = false;
            }
            leafCnt = 0;
        }
    }
    if (COUNT) {
        __syncwarp();  // every lane of the warp has left the loop
        unsigned long long nv = wc.nodes, nt = wc.tris;
        for (int off = 16; off > 0; off >>= 1) {
            nv += __shfl_down_sync(0xFFFFFFFFu, nv, off);
            nt += __shfl_down_sync(0xFFFFFFFFu, nt, off);
        }
        if (lane == 0) {
            atomicAdd(&ctrl->nodeVisits, nv);
            atomicAdd(&ctrl->triTests, nt);
        }
    }
    if (blockIdx.x == 0 && threadIdx.x == 0)
        atomicAdd(ANY ? &ctrl->shadowRays : &ctrl->extensionRays, (unsigned long long)n);
}

// The warp goes on to test triangles when fewer lanes than this are still looking for a
// leaf. Measured in the flat kernel with 1 / 4 / 8 / 16 lanes: occluded room 47.1 / 42.7 /
// 42.2 / 44.1 ms per call, Cornell box 4.57 / 4.50 / 4.58 / 4.82, batch 11.8 / 11.5 / 11.7 /
// 12.8; with discarded hits (shell-mapped cloth) 21.4 / 22.2 / 22.8 / 24.3.
template <bool SHELL>
constexpr int kLookingLanes = SHELL ? 1 : 4;

// ---- ray fetch of the persistent per-lane kernels ---------------------------------
constexpr unsigned int kWarp = 0xFFFFFFFFu;
// A warp takes new rays when this many of its lanes are without one (or all are). Taking
// each as soon as a lane is free stalls the other lanes for an atomic and two loads from
// DRAM each time, and mixes rays that started together: with 1 / 8 lanes the terrain's
// render took 38.7 / 37.5 ms, the Cornell box's 4.51 / 4.48. Rays that are alike (closest hits on one
// BVH) or short (scenes of few triangles) wait for more lanes, 16 / 20 / 24 / 28: terrain
// 30.9 / 30.6 / 30.5 / 30.8 ms, Cornell box 3.59 / 3.52 / 3.43 / 3.41. Elsewhere 8 / 16 / 22: occluded room
// 37.4 / 37.8 / 38.8, shell-mapped cloth 19.3 / 19.2 / 19.2, batch 10.04 / 10.04 / 10.06.
constexpr unsigned int kFetchLanes = 16, kFetchLanesMore = 24;
// Rays of the queue for the lanes of a warp, in order, one atomicAdd for all that want one.
// Every lane of the warp makes the same calls. (Claiming chunks of 32 / 64 / 128 rays ahead,
// to save atomics, left some warps with work when the others had none: the batch took
// 12.1 / 13.2 / 16.6 ms instead of 11.3.)
// counted: the caller has set a bound on the steps of a ray (xgb_scene_set_traversal_limits).
// A step of the loop takes a ray as far as the warp's lanes go on together, so that full
// warps, filled up at once, that test triangles when no lane is looking any more need the
// fewest steps: they keep a ray inside a bound that it met on such a warp.
constexpr unsigned int kCountedLanes = 64;  // all, and none waits for another
struct RayClaims {
    unsigned int* head;
    unsigned int n, lanes, next, enough;
    // few rays: a warp works with its share of lanes only, so that they wait for fewer others
    __device__ __forceinline__ RayClaims(unsigned int* h, unsigned int count, unsigned int fetchLanes, bool counted)
        : head(h), n(count), next(0) {
        const unsigned int warps = gridDim.x * (kTraceBlock / 32);
        lanes = counted ? kCountedLanes : min(32u, (n + warps - 1u) / warps);
        enough = counted ? 1u : min(fetchLanes, lanes);
    }
    // The lanes that want a ray (0: none, or not yet worth the trip).
    __device__ __forceinline__ unsigned int wanted(bool idle) const {
        const unsigned int m = __ballot_sync(kWarp, idle && (threadIdx.x & 31) < lanes && next < n);
        return (unsigned int)__popc(m) >= enough ? m : 0u;
    }
    // The next rays for the lanes of `want`; returns whether this lane got one.
    __device__ __forceinline__ bool take(unsigned int want, unsigned int* ray) {
        const unsigned int lane = threadIdx.x & 31;
        const unsigned int rank = __popc(want & ((1u << lane) - 1u)), count = __popc(want);
        unsigned int base = 0;
        if (lane == 0) base = atomicAdd(head, count);
        base = __shfl_sync(kWarp, base, 0);
        const unsigned int i = base + rank;
        next = base + count;
        if (((want >> lane) & 1u) && i < n) {
            *ray = i;
            return true;
        }
        return false;
    }
};

// ---- scenes of a few instances: binary mesh BVHs ------------------------------------------------
// With at most kFlatInstances instances the top level is a short list: a lane
// walks the instances in order (those whose world box the ray still reaches
// within tMax) and traverses each mesh BVH as a persistent per-lane state machine
// in the style of Aila & Laine ("Understanding the Efficiency of Ray Traversal
// on GPUs", HPG 2009): lanes whose rays are finished fetch the next ones together
// (RayClaims), inner nodes and leaves are processed in separate inner loops, and
// the first leaf a lane reaches is postponed until few lanes of the warp are
// still looking for one, so that the warp tests triangles together.
// Results are those of traceScene: the same slab and watertight tests and the
// same closest-hit acceptance (tMax shrinks across instances).
constexpr int kSentinel = 0x7FFFFFFF;

// The instance boxes are tested when the warp fetches, by all lanes that take a ray
// together; afterwards a lane goes from one reached instance to the next, and tests a box again only
// where a hit has come closer. Against a search by each lane at its own time: Cornell box
// (8 instances) 3.43 -> 3.34 ms per call, 3.28 held to eight blocks per SM (64 registers; seven
// with shell mapping); scenes of two to seven instances the same within 0.3 %.
//
// SHELL: the scene has shell-mapped meshes, whose accepted hits go through the
// discard test (shellDiscard, trace.cuh) before tMax shrinks.
template <bool ANY, bool COUNT, class S, bool SHELL = false>
__global__ void __launch_bounds__(kTraceBlock, SHELL ? 7 : 8) k_trace_flat2(S scenes, PathQueue q, HitQueue h, ShadowQueue s,
                                                            PathQueue out, Ctrl* ctrl) {
    const unsigned int n = ANY ? ctrl->nShadowDue : ctrl->nActive;
    if (n <= kTeamQueue && scenes.teams()) return;  // k_trace_team's
    unsigned int* head = ANY ? &ctrl->shadowHead : &ctrl->extendHead;
    constexpr bool kBatch = !std::is_same<S, OneScene>::value;
    int rayMaxSteps = 0, rayStack = 0;  // a batch: the current ray's job's bounds
    int job = 0;
    const int lane = threadIdx.x & 31;
    RayClaims claims(head, n, kBatch || scenes.scene(0).large ? kFetchLanes : kFetchLanesMore, scenes.counted());
    const int looking = claims.lanes == 32u ? kLookingLanes<SHELL> : 1;
    int stack[kStackDepth];
    int sp = 0;
    int nodeAddr = kSentinel, leafAddr = 0;
    int inst = 0;               // instance being traversed
    unsigned int reached = 0;  // instances after it whose world box the ray reaches
    unsigned int ray = 0;
    V3 wo(0.f, 0.f, 0.f), wd(0.f, 0.f, 1.f);
    BoxRay br{0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    WRay r;
    const Node2* nodes = nullptr;
    const TriV* tris = nullptr;
    const MeshDev* mesh = nullptr;
    float tMax = 0.0f;
    TraceHit hit;
    hit.prim = -1;
    hit.inst = -1;
    hit.t = 0.0f;
    hit.b0 = hit.b1 = 0.0f;
    bool occluded = false;
    bool fetch = true;
    WorkCount wc;
    for (int guard = 0;; ++guard) {
        // every lane of the warp comes here; those without a ray take the next ones together
        const unsigned int want = claims.wanted(fetch);
        if (want && claims.take(want, &ray)) {
            float4 o4, d4;
            if (ANY) { o4 = __ldcs(&s.o[ray]); d4 = __ldcs(&s.d[ray]); tMax = o4.w; }
            else { o4 = __ldcs(&q.o[ray]); d4 = __ldcs(&q.d[ray]); tMax = __int_as_float(0x7f800000); }
            wo = V3(o4.x, o4.y, o4.z);
            wd = V3(d4.x, d4.y, d4.z);
            br = BoxRay{wo.x, wo.y, wo.z, 1.0f / wd.x, 1.0f / wd.y, 1.0f / wd.z};
            job = scenes.jobOf(ANY ? __float_as_uint(d4.w) : __float_as_uint(q.thr[ray].w));
            if (kBatch) {  // the job's traversal bounds, read once per ray
                rayMaxSteps = scenes.scene(job).maxSteps;
                rayStack = min(kStackDepth, scenes.scene(job).stackLimit);
            }
            hit.prim = -1;
            hit.inst = -1;
            hit.t = tMax;
            occluded = false;
            guard = 0;
            {
                const SceneDev& sc = scenes.scene(job);
                reached = 0;
                for (int k = 0; k < sc.nInstances; ++k)
                    if (instBoxHit(br, sc.instBox, k, tMax)) reached |= 1u << k;
            }
            nodeAddr = kSentinel;
            leafAddr = 0;
            fetch = false;
        }
        if (!__any_sync(kWarp, !fetch)) break;
        if (fetch) continue;
        if (nodeAddr == kSentinel && leafAddr >= 0) {
            // next instance whose world box the ray still reaches
            bool more = false;
            while (reached && !(ANY && occluded) && !more) {
                inst = __ffs(reached) - 1;
                reached &= reached - 1;
                more = ANY || hit.prim < 0 || instBoxHit(br, scenes.scene(job).instBox, inst, tMax);
            }
            if (!more) {  // ray finished
                if (ANY) {
                    if (!occluded) shadowLit(scenes, job, s, out, ray);
                } else {
                    __stcs(&h.h[ray], make_float4(hit.prim >= 0 ? hit.t : tMax, hit.b0, hit.b1, __int_as_float(hit.prim)));
                    __stcs(&h.inst[ray], hit.inst);
                }
                fetch = true;
                continue;
            }
            const SceneDev& sc = scenes.scene(job);
            const Instance& in = sc.instances[inst];
            const MeshDev& m = sc.meshes[in.mesh];
            nodes = m.nodes2;
            tris = m.tris;
            mesh = &m;
            if (in.identity) r = makeWRay(wo, wd);
            else r = makeWRay(xformPointRn(in.matInv, wo), xformVectorRn(in.matInv, wd));
            sp = 0;
            if (m.rootIsLeaf) { leafAddr = m.rootLeaf; nodeAddr = kSentinel; }
            else { leafAddr = 0; nodeAddr = 0; }
        }
        if (guard > (kBatch ? rayMaxSteps : scenes.scene(0).maxSteps)) {
            atomicOr(&ctrl->errors, 4u);
            nodeAddr = kSentinel;
            leafAddr = 0;
            reached = 0;
        }
        bool searching = true;
        while ((unsigned int)nodeAddr < (unsigned int)kSentinel) {
            if (COUNT) wc.nodes++;
            const Node2* nd = nodes + nodeAddr;
            const NodeHits hit2 = slabs(nd, r, tMax);
            const int2 dd = hit2.child;
            const bool h0 = hit2.h0, h1 = hit2.h1;
            const float t0 = hit2.t0, t1 = hit2.t1;
            if (h0 && h1) {
                int near = dd.x, far = dd.y;
                if (t1 < t0) { near = dd.y; far = dd.x; }
                if (sp >= (kBatch ? rayStack : min(kStackDepth, scenes.scene(0).stackLimit))) {
                    atomicOr(&ctrl->errors, 1u);
                    sp = 0;
                    nodeAddr = kSentinel;
                    break;
                }
                stack[sp++] = far;
                nodeAddr = near;
            } else if (h0) {
                nodeAddr = dd.x;
            } else if (h1) {
                nodeAddr = dd.y;
            } else {
                nodeAddr = sp > 0 ? stack[--sp] : kSentinel;
            }
            if (nodeAddr < 0 && leafAddr >= 0) {  // first leaf: postpone it, keep descending
                searching = false;
                leafAddr = nodeAddr;
                nodeAddr = sp > 0 ? stack[--sp] : kSentinel;
            }
            if (__popc(__ballot_sync(__activemask(), searching)) < looking) break;
        }
        while (leafAddr < 0) {
            int first = leafFirst(leafAddr), cnt = leafCount(leafAddr);
            if (COUNT) wc.tris += cnt;
            for (int k = 0; k < cnt; ++k) {
                const TriV* tv = tris + first + k;
                float4 p0 = __ldg(&tv->p0), p1 = __ldg(&tv->p1), p2 = __ldg(&tv->p2);
                float t, b0, b1;
                if (watertight(r, p0, p1, p2, tMax, t, b0, b1)) {
                    if (SHELL && mesh->shellLayers && shellDiscard(*mesh, __float_as_int(p0.w), b0, b1)) continue;
                    tMax = t;
                    if (ANY) { occluded = true; break; }
                    hit.t = t; hit.b0 = b0; hit.b1 = b1;
                    hit.prim = __float_as_int(p0.w);
                    hit.inst = inst;
                }
            }
            if (ANY && occluded) { leafAddr = 0; nodeAddr = kSentinel; sp = 0; break; }
            leafAddr = nodeAddr;  // another leaf was postponed: take it next
            if (nodeAddr < 0) nodeAddr = sp > 0 ? stack[--sp] : kSentinel;
        }
    }
    if (COUNT) {
        unsigned long long nv = wc.nodes, nt = wc.tris;
        for (int off = 16; off > 0; off >>= 1) {
            nv += __shfl_down_sync(0xFFFFFFFFu, nv, off);
            nt += __shfl_down_sync(0xFFFFFFFFu, nt, off);
        }
        if (lane == 0) {
            atomicAdd(&ctrl->nodeVisits, nv);
            atomicAdd(&ctrl->triTests, nt);
        }
    }
    if (blockIdx.x == 0 && threadIdx.x == 0)
        atomicAdd(ANY ? &ctrl->shadowRays : &ctrl->extensionRays, (unsigned long long)n);
}

// ---- one BVH per scene -------------------------------------------------------------
// The traversal of every scene with binary meshes: the scene's world BVH (WorldDev) as a
// persistent per-lane state machine in the style of Aila & Laine ("Understanding the
// Efficiency of Ray Traversal on GPUs", HPG 2009): lanes whose rays are finished fetch
// the next ones together (RayClaims), inner nodes and leaves are
// processed in separate inner loops, and the first leaf a lane reaches is postponed until
// few lanes of the warp are still looking for one, so that the warp tests triangles
// together.
//
// ENTER: some leaves are instances with a transform. A lane that takes one pushes what it
// has left, then kReturn, moves its ray into object space and goes on in that mesh; when
// kReturn comes back it reads its ray again from the queue.
//
// The order of the instances: the flat and general kernels visit instances in the scene's
// order (or top-level order) and a hit is accepted while t <= tMax, so where two
// instances are hit at distances within rounding of each other, the order decides. Here
// the nearer box goes first, whatever its instance. So boxes and triangles are visited
// up to a little beyond the best hit (cullMul, cullAbs), a triangle of another instance
// accepted or refused within that margin marks the ray, and a marked ray is traced again in the
// instance order (k_retrace).
//
// Ten blocks per SM (48 registers, 28 bytes of spills outside the node loop) rather than the
// nine that 55 registers allow: the terrain's traversal ran 2.5 % faster; twelve (40
// registers) spill more and ran 7 % slower. A batch (S = BatchScenes) reads its ray's BVH when it fetches the ray.
constexpr int kReturn = kSentinel - 1;
constexpr int kWorldDepth = kStackDepth + kTlasStack;  // a mesh's entries and the top level's
constexpr int kWorldStack = kWorldDepth + 2;           // and a return
constexpr int kMarked = 0x40000000;  // in the hit triangle's index: traced again in instance order
// A scene of one instance keeps the mesh's own bound (xgb_scene_set_traversal_limits).
__device__ __forceinline__ int worldStackCap(const SceneDev& sc) {
    return sc.nInstances == 1 ? sc.stackLimit : kWorldDepth;
}

template <class S, bool ENTER>
struct WorldTraits {
    static constexpr int kMinBlocks = !std::is_same<S, BatchScenes>::value && !ENTER ? 10 : 8;
};

template <bool ANY, bool COUNT, class S, bool ENTER, bool SHELL>
__global__ void __launch_bounds__(kTraceBlock, (WorldTraits<S, ENTER>::kMinBlocks))
    k_trace_world(S scenes, PathQueue q, HitQueue h, unsigned int* retrace, ShadowQueue s, PathQueue out, Ctrl* ctrl) {
    constexpr bool kBatch = std::is_same<S, BatchScenes>::value, kQuery = std::is_same<S, QueryRays>::value;
    const unsigned int n = ANY ? ctrl->nShadowDue : ctrl->nActive;
    if (n <= kTeamQueue && scenes.teams()) return;  // k_trace_team's
    unsigned int* head = ANY ? &ctrl->shadowHead : &ctrl->extendHead;
    RayClaims claims(head, n, ANY ? kFetchLanes : kFetchLanesMore, scenes.counted());
    const int looking = claims.lanes == 32u ? kLookingLanes<SHELL> : 1;
    bool holds = false;  // the lane has a ray
    // one scene: its BVH for every ray; a batch: the current ray's
    const Node2* nodes = kBatch ? nullptr : scenes.scene(0).world.nodes;
    const TriV* tris = kBatch ? nullptr : scenes.scene(0).world.tris;
    int job = 0;
    int rayStack = 0;   // a batch: the current ray's job's bound
    int inst = -1;      // ENTER: the instance the ray is in (-1: world space)
    int hitInst = -1;   // ENTER: the instance of a hit found inside one
    int stack[kWorldStack + 1];
    int sp = 0;
    int nodeAddr = kSentinel, leafAddr = 0;
    unsigned int ray = 0;
    WRay r;
    float tMax = 0.0f, tCull = 0.0f, b0 = 0.0f, b1 = 0.0f;
    int hitTri = -1;  // index in the triangle array, ENTER: the original triangle index
    bool occluded = false;
    WorkCount wc;
    for (int guard = 0;; ++guard) {
        // every lane of the warp comes here; those without a ray take the next ones together
        const unsigned int want = claims.wanted(!holds);
        if (want && claims.take(want, &ray)) {
            holds = true;
            float4 o4, d4;
            if constexpr (kQuery) {
                const float* in = scenes.rays + 7 * (size_t)ray;
                o4 = make_float4(in[0], in[1], in[2], in[6]);
                d4 = make_float4(in[3], in[4], in[5], 0.0f);
                tMax = o4.w;
            } else if (ANY) {
                o4 = __ldcs(&s.o[ray]);
                d4 = __ldcs(&s.d[ray]);
                tMax = o4.w;
            } else {
                o4 = __ldcs(&q.o[ray]);
                d4 = __ldcs(&q.d[ray]);
                tMax = __int_as_float(0x7f800000);
            }
            V3 o(o4.x, o4.y, o4.z), d(d4.x, d4.y, d4.z);
            if (kBatch) job = scenes.jobOf(ANY ? __float_as_uint(d4.w) : __float_as_uint(__ldg(&q.thr[ray].w)));
            const SceneDev& sc = scenes.scene(job);
            if (kBatch || ENTER) {  // a shadow ray may have ended inside an instance
                nodes = sc.world.nodes;
                tris = sc.world.tris;
            }
            if (kBatch) rayStack = worldStackCap(sc);
            if (sc.nInstances == 1) {  // the mesh's own arrays: its transform applies to every ray
                const Instance& in = sc.instances[0];
                if (!in.identity) {
                    o = xformPointRn(in.matInv, o);
                    d = xformVectorRn(in.matInv, d);
                }
            }
            r = makeWRay(o, d);
            hitTri = -1;
            tCull = tMax;
            occluded = false;
            sp = 0;
            guard = 0;
            if (ENTER) inst = hitInst = -1;
            const int root = sc.world.root;
            if (root < 0) { leafAddr = root; nodeAddr = kSentinel; }
            else { leafAddr = 0; nodeAddr = root; }
        }
        if (!__any_sync(kWarp, holds)) break;
        if (!holds) continue;
        if (guard > scenes.scene(job).maxSteps) {
            atomicOr(&ctrl->errors, 4u);
            nodeAddr = kSentinel;
            leafAddr = 0;
        }
        bool searching = true;
        while ((unsigned int)nodeAddr < (unsigned int)kReturn) {
            if (COUNT) wc.nodes++;
            const Node2* nd = nodes + nodeAddr;
            const NodeHits hit2 = slabs(nd, r, tCull);
            const int2 dd = hit2.child;
            const bool h0 = hit2.h0, h1 = hit2.h1;
            const float t0 = hit2.t0, t1 = hit2.t1;
            // one branch for a hit or a pop, selects within: 31.8 -> 31.5 ms for the terrain
            // against a branch per combination, 32.4 with the bound checked before the push
            if (h0 || h1) {
                const bool second = !h0 || (h1 && t1 < t0);
                nodeAddr = second ? dd.y : dd.x;
                if (h0 && h1) stack[sp++] = second ? dd.x : dd.y;
            } else {
                nodeAddr = sp > 0 ? stack[--sp] : kSentinel;
            }
            if (sp > (kBatch ? rayStack : worldStackCap(scenes.scene(0)))) {
                atomicOr(&ctrl->errors, 1u);
                sp = 0;
                nodeAddr = kSentinel;
                break;
            }
            if (nodeAddr < 0 && leafAddr >= 0) {  // first leaf: postpone it, keep descending
                searching = false;
                leafAddr = nodeAddr;
                nodeAddr = sp > 0 ? stack[--sp] : kSentinel;
            }
            if (__popc(__ballot_sync(__activemask(), searching)) < looking) break;
        }
        if (ENTER && nodeAddr < 0 && leafAddr >= 0) {  // a leaf waited below kReturn
            leafAddr = nodeAddr;
            nodeAddr = sp > 0 ? stack[--sp] : kSentinel;
        }
        while (leafAddr < 0) {
            const int first = leafFirst(leafAddr), cnt = leafCount(leafAddr);
            if (ENTER && cnt == kEnterCount) {
                // into the instance: what is left of the world waits below kReturn
                if (nodeAddr != kSentinel) stack[sp++] = nodeAddr;
                stack[sp++] = kReturn;
                const SceneDev& sc = scenes.scene(job);
                const Instance& in = sc.instances[first];
                const MeshDev& m = sc.meshes[in.mesh];
                const float4 o4 = ANY ? s.o[ray] : q.o[ray], d4 = ANY ? s.d[ray] : q.d[ray];
                r = makeWRay(xformPointRn(in.matInv, V3(o4.x, o4.y, o4.z)), xformVectorRn(in.matInv, V3(d4.x, d4.y, d4.z)));
                inst = first;
                nodes = m.nodes2;
                tris = m.tris;
                leafAddr = m.rootIsLeaf ? m.rootLeaf : 0;
                nodeAddr = m.rootIsLeaf ? stack[--sp] : 0;
                if (!m.rootIsLeaf) break;
                continue;
            }
            if (COUNT) wc.tris += cnt;
            for (int k = 0; k < cnt; ++k) {
                const TriV* tv = tris + first + k;
                const float4 p0 = __ldg(&tv->p0), p1 = __ldg(&tv->p1), p2 = __ldg(&tv->p2);
                float t, c0, c1;
                if (watertight(r, p0, p1, p2, ANY ? tMax : tCull, t, c0, c1)) {
                    if (SHELL) {
                        const int of = ENTER && inst >= 0 ? inst : __float_as_int(p1.w);
                        const SceneDev& sc = scenes.scene(job);
                        const MeshDev& m = sc.meshes[sc.instances[of].mesh];
                        if (m.shellLayers && shellDiscard(m, __float_as_int(p0.w), c0, c1)) continue;
                    }
                    if (ANY) { occluded = true; break; }
                    const WorldDev& w = scenes.scene(job).world;
                    const float beyond = fmaf(t, w.cullMul, w.cullAbs);
                    int marked = hitTri >= 0 ? hitTri & kMarked : 0;
                    if (hitTri >= 0 && !(beyond < tMax)) {  // refused, or hardly nearer
                        const int now = ENTER && inst >= 0 ? inst : __float_as_int(p1.w);
                        const int before = ENTER ? hitInst : __float_as_int(__ldg(&tris[hitTri & ~kMarked].p1.w));
                        if (now != before) {
                            marked = kMarked;
                            hitTri |= kMarked;
                            if (!(t <= tMax)) continue;
                        } else if (!watertight(r, p0, p1, p2, tMax, t, c0, c1)) {
                            continue;  // within a mesh the order is its own, and so is the rule
                        }
                    }
                    tMax = t;
                    tCull = beyond;
                    b0 = c0;
                    b1 = c1;
                    hitTri = marked | (ENTER ? __float_as_int(p0.w) : first + k);
                    if (ENTER) hitInst = inst >= 0 ? inst : __float_as_int(p1.w);
                }
            }
            if (ANY && occluded) { leafAddr = 0; nodeAddr = kSentinel; break; }
            leafAddr = nodeAddr;  // another leaf was postponed: take it next
            if (nodeAddr < 0) nodeAddr = sp > 0 ? stack[--sp] : kSentinel;
        }
        if (ENTER && nodeAddr == kReturn && leafAddr >= 0) {  // back to world space
            const SceneDev& sc = scenes.scene(job);
            const float4 o4 = ANY ? s.o[ray] : q.o[ray], d4 = ANY ? s.d[ray] : q.d[ray];
            r = makeWRay(V3(o4.x, o4.y, o4.z), V3(d4.x, d4.y, d4.z));
            inst = -1;
            nodes = sc.world.nodes;
            tris = sc.world.tris;
            nodeAddr = sp > 0 ? stack[--sp] : kSentinel;
            leafAddr = 0;
        }
        if (nodeAddr == kSentinel && leafAddr >= 0) {  // ray finished
            holds = false;
            const SceneDev& sc = scenes.scene(job);
            if constexpr (kQuery && ANY) {
                scenes.occluded[ray] = occluded ? 1 : 0;
            } else if constexpr (ANY) {
                if (!occluded) shadowLit(scenes, job, s, out, ray);
            } else {
                int prim = -1, of = -1;
                if (hitTri >= 0) {
                    if ((hitTri & kMarked) && sc.nInstances > 1) retrace[atomicAdd(&ctrl->nRetrace, 1u)] = ray;
                    if (ENTER) {
                        prim = hitTri & ~kMarked;
                        of = hitInst;
                    } else {
                        const TriV* tv = tris + (hitTri & ~kMarked);
                        prim = __float_as_int(__ldg(&tv->p0.w));
                        of = __float_as_int(__ldg(&tv->p1.w));
                    }
                }
                if constexpr (kQuery) {
                    float* out5 = scenes.hits + 5 * (size_t)ray;
                    out5[0] = tMax;
                    out5[1] = (float)of;
                    out5[2] = (float)prim;
                    out5[3] = prim >= 0 ? b0 : 0.0f;
                    out5[4] = prim >= 0 ? b1 : 0.0f;
                } else {
                    __stcs(&h.h[ray], make_float4(tMax, b0, b1, __int_as_float(prim)));
                    __stcs(&h.inst[ray], of);
                }
            }
        }
    }
    if (COUNT) {
        unsigned long long nv = wc.nodes, nt = wc.tris;
        for (int off = 16; off > 0; off >>= 1) {
            nv += __shfl_down_sync(0xFFFFFFFFu, nv, off);
            nt += __shfl_down_sync(0xFFFFFFFFu, nt, off);
        }
        if ((threadIdx.x & 31) == 0) {
            atomicAdd(&ctrl->nodeVisits, nv);
            atomicAdd(&ctrl->triTests, nt);
        }
    }
    if (blockIdx.x == 0 && threadIdx.x == 0)
        atomicAdd(ANY ? &ctrl->shadowRays : &ctrl->extensionRays, (unsigned long long)n);
}

// The marked rays of a k_trace_world launch, in the instance order. The hit that was found
// bounds them: what is no more than the margin of cullMul and cullAbs beyond it has been
// seen to be hit, so boxes further off need no visit, and where several hits within the
// margin follow one another the order alone decides, as from an unbounded start. Usually few
// rays are marked, so each warp takes one: together in a warp they would wait for one
// another (microfacet normal mapping 400^2 x 4: 5.31 -> 5.18 ms per call). Where surfaces of
// many instances lie upon one another most rays are: then the warps of a full grid take 32 at a
// time (a terrain with 2,000 boxes whose tops are level, 4.2 million paths: 35.3 ms per
// call with 152 blocks and fixed shares, 15.9 with a full grid, 12.7 so; 11.9 without
// a world BVH, 6.6 with it where the boxes are not level).
template <class S>
__global__ void __launch_bounds__(kTraceBlock) k_retrace(S scenes, PathQueue q, HitQueue h, const unsigned int* retrace,
                                                         Ctrl* ctrl) {
    const unsigned int n = ctrl->nRetrace;
    const unsigned int warps = gridDim.x * (kTraceBlock / 32), lane = threadIdx.x & 31;
    const unsigned int lanes = min(32u, (n + warps - 1u) / warps);
    while (n) {
        unsigned int k = 0;
        if (lane == 0) k = atomicAdd(&ctrl->retraceHead, lanes);
        k = __shfl_sync(kWarp, k, 0);
        if (k >= n) break;
        k += lane;
        if (lane >= lanes || k >= n) continue;
        const unsigned int ray = retrace[k];
        const float4 o = q.o[ray], d = q.d[ray];
        const SceneDev& sc = scenes.scene(scenes.jobOf(__float_as_uint(q.thr[ray].w)));
        TraceHit hit;
        traceCall(sc, V3(o.x, o.y, o.z), V3(d.x, d.y, d.z), fmaf(h.h[ray].x, sc.world.cullMul, sc.world.cullAbs), false,
                  hit, &ctrl->errors);
        h.h[ray] = make_float4(hit.t, hit.b0, hit.b1, __int_as_float(hit.prim));
        h.inst[ray] = hit.inst;
    }
}

// Launches of at most kTeamQueue rays: a ray for each team of lanes, up to kTeamRays per warp.
// Such a launch is bound by the chain of node fetches of its longest ray, which 32 lanes
// shorten: the occluded room with the proposal (256^2 x 8, whose last thirty iterations are such
// launches) 10.9 -> 9.15 ms per call, a batch of 8 9.93 -> 9.87.
template <bool ANY, class S>
__global__ void __launch_bounds__(kTraceBlock, 6) k_trace_team(const __grid_constant__ S scenes, PathQueue q, HitQueue h,
                                                               ShadowQueue s, PathQueue out, Ctrl* ctrl) {
    __shared__ uint2 sStacks[kTraceBlock / 32][kTeamEntries];
    const unsigned int n = ANY ? ctrl->nShadowDue : ctrl->nActive;
    if (n == 0 || n > kTeamQueue || !scenes.teams()) return;
    const unsigned int warps = gridDim.x * (kTraceBlock / 32), lane = threadIdx.x & 31;
    const unsigned int teams = n <= warps ? 1u : n <= 2u * warps ? 2u : kTeamRays;
    for (;;) {
        unsigned int base = 0;
        if (lane == 0) base = atomicAdd(ANY ? &ctrl->shadowHead : &ctrl->extendHead, teams);
        base = __shfl_sync(kWarp, base, 0);
        if (base >= n) break;
        const unsigned int k = base + lane / (32u / teams);
        const bool has = k < n;
        const unsigned int ray = has ? k : base;
        const float4 o = ANY ? s.o[ray] : q.o[ray], d = ANY ? s.d[ray] : q.d[ray];
        const int job = scenes.jobOf(ANY ? __float_as_uint(d.w) : __float_as_uint(q.thr[ray].w));
        TraceHit hit;
        const bool mine = traceTeam(scenes.scene(job), has, V3(o.x, o.y, o.z), V3(d.x, d.y, d.z),
                                    ANY ? o.w : __int_as_float(0x7f800000), ANY, 32u / teams, sStacks[threadIdx.x >> 5], hit,
                                    &ctrl->errors);
        if (mine) {
            if constexpr (ANY) {
                if (hit.prim < 0) shadowLit(scenes, job, s, out, ray);
            } else {
                h.h[ray] = make_float4(hit.t, hit.b0, hit.b1, __int_as_float(hit.prim));
                h.inst[ray] = hit.inst;
            }
        }
        __syncwarp();
    }
    if (blockIdx.x == 0 && threadIdx.x == 0)
        atomicAdd(ANY ? &ctrl->shadowRays : &ctrl->extensionRays, (unsigned long long)n);
}

// ---- batches of scenes (xgb_render_batch) -----------------------------------------
// Each ray finds its job (and so its scene) in the high bits of its pixel field
// and is traced by the general two-level traversal.
__global__ void __launch_bounds__(kTraceBlock) k_extend_batch(BatchView b, PathQueue q, HitQueue h, Ctrl* ctrl) {
    const unsigned int n = ctrl->nActive;
    const int lane = threadIdx.x & 31;
    WorkCount wc;
    for (;;) {
        unsigned int base = 0;
        if (lane == 0) base = atomicAdd(&ctrl->extendHead, 32u);
        base = __shfl_sync(0xFFFFFFFFu, base, 0);
        if (base >= n) break;
        const unsigned int i = base + lane;
        if (i < n) {
            const float4 o = q.o[i], d = q.d[i];
            const int job = (int)(__float_as_uint(q.thr[i].w) >> 24);
            TraceHit hit;
            traceScene<false>(b.scenes[job], V3(o.x, o.y, o.z), V3(d.x, d.y, d.z), __int_as_float(0x7f800000), hit,
                              &ctrl->errors, wc);
            h.h[i] = make_float4(hit.t, hit.b0, hit.b1, __int_as_float(hit.prim));
            h.inst[i] = hit.inst;
        }
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) atomicAdd(&ctrl->extensionRays, (unsigned long long)n);
}

__global__ void __launch_bounds__(kTraceBlock) k_shadow_batch(BatchView b, ShadowQueue s, PathQueue out, Ctrl* ctrl) {
    const unsigned int n = ctrl->nShadowDue;
    const int lane = threadIdx.x & 31;
    WorkCount wc;
    for (;;) {
        unsigned int base = 0;
        if (lane == 0) base = atomicAdd(&ctrl->shadowHead, 32u);
        base = __shfl_sync(0xFFFFFFFFu, base, 0);
        if (base >= n) break;
        const unsigned int i = base + lane;
        if (i < n) {
            const float4 o = s.o[i], d = s.d[i];
            const unsigned int packed = __float_as_uint(d.w);
            const int job = (int)(packed >> 24), pix = (int)(packed & 0xFFFFFFu);
            TraceHit hit;
            if (!traceScene<true>(b.scenes[job], V3(o.x, o.y, o.z), V3(d.x, d.y, d.z), o.w, hit, &ctrl->errors, wc)) {
                const float4 c = s.c[i];
                filmAdd(b.params[job], pix, V3(c.x, c.y, c.z));
                const int target = __float_as_int(c.w);
                if (target >= 0) out.rng[target] = s.rng[i];
            }
        }
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) atomicAdd(&ctrl->shadowRays, (unsigned long long)n);
}

// ---- ray queries (xgb_scene_intersect / xgb_scene_occluded) -------------------
// Scenes of several instances (and wide or shell-mapped meshes): a warp takes 32 rays at a
// time; traceScene's top-level order is the instance order of queries.
template <bool ANY>
__global__ void __launch_bounds__(kTraceBlock) k_query(SceneDev sc, const float* __restrict__ rays, int n, float* hits,
                                                       int* occluded, Ctrl* ctrl) {
    const int lane = threadIdx.x & 31;
    for (;;) {
        unsigned int base = 0;
        if (lane == 0) base = atomicAdd(&ctrl->extendHead, 32u);
        base = __shfl_sync(0xFFFFFFFFu, base, 0);
        if (base >= (unsigned int)n) break;
        const unsigned int i = base + lane;
        if (i < (unsigned int)n) {
            const float* r = rays + 7 * (size_t)i;
            TraceHit hit;
            hit.b0 = hit.b1 = 0.0f;
            WorkCount wc;
            const bool found = traceScene<ANY>(sc, V3(r[0], r[1], r[2]), V3(r[3], r[4], r[5]), r[6], hit, &ctrl->errors, wc);
            if (ANY) {
                occluded[i] = found ? 1 : 0;
            } else {
                float* h = hits + 5 * (size_t)i;
                h[0] = hit.t;
                h[1] = (float)hit.inst;
                h[2] = (float)hit.prim;
                h[3] = hit.b0;
                h[4] = hit.b1;
            }
        }
    }
}

// Persistent grids: SMs x resident blocks of the kernel actually launched
// (looked up once per kernel; all kernels here use kTraceBlock threads).
template <class K>
static int persistentGrid(K kernel, int numSMs) {
    static std::mutex mu;
    static std::map<const void*, int> blocks;
    std::lock_guard<std::mutex> lock(mu);
    auto it = blocks.find((const void*)kernel);
    if (it == blocks.end()) {
        int b = 0;
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, kernel, kTraceBlock, 0);
        it = blocks.emplace((const void*)kernel, b > 0 ? b : 1).first;
    }
    return numSMs * it->second;
}

// The world BVH's kernel takes scenes of one instance, scenes of more than kFlatInstances,
// and the shadow rays of those between that have a world BVH (large ones, see
// xgb_scene_build), unless several instances come with traversal limits other than the
// defaults, which count the steps of the kernels that walk the instances. Against the
// flat kernel on scenes of few instances: any hit 17.0 -> 13.9 ms per call in the occluded
// room (200,000 triangles and a light), 3.5 -> 2.9 with the proposal, 0.73 -> 0.79 in the
// Cornell box (36 triangles, ten instances), the shell-mapped cloth 7.6 -> 7.8; closest hit
// 42.6 -> 44.6, 8.1 -> 8.7, 1.85 -> 2.14, 21.6 -> 22.1. Against the generic pair (67 instances,
// normal mapping): 3.15 -> 2.34 and 1.40 -> 1.03. 8-wide meshes keep the wide kernel (at most
// kFlatInstances instances) and the generic pair (any other, and shell-mapped ones).
static bool useWorld(const SceneDev& sc, bool any) {
    if (!sc.world.tris) return false;
    if (sc.nInstances == 1) return true;
    return (any || sc.nInstances > kFlatInstances) && sc.maxSteps == kDefaultMaxSteps && sc.stackLimit == kMaxStackLimit;
}
#define XGB_LAUNCH(K) K<<<persistentGrid(K, numSMs), kTraceBlock, 0, s>>>
// Traversal limits other than the defaults count the steps of the kernels below.
static SceneDev withTeams(const SceneDev& sc, bool any, bool teams) {
    SceneDev r = sc;
    r.teams = sc.teams && teams && sc.maxSteps == kDefaultMaxSteps && sc.stackLimit == kMaxStackLimit &&
              (sc.nInstances <= kFlatInstances || useWorld(sc, any));
    return r;
}
int batchCounted(const SceneDev* scenes, int n) {
    for (int j = 0; j < n; ++j)
        if (scenes[j].maxSteps != kDefaultMaxSteps) return 1;
    return 0;
}
int batchTeams(const SceneDev* scenes, int n) {
    bool teams = true;
    for (int j = 0; j < n; ++j) teams = teams && withTeams(scenes[j], false, true).teams;
    return teams && batchKernels(scenes, n) != kBatchGeneral;
}
template <bool ANY, bool COUNT>
static int launchWorld(const SceneDev& sc, const RenderParams& rp, PathQueue q, HitQueue h, unsigned int* retrace,
                        ShadowQueue sq, PathQueue out, Ctrl* ctrl, int numSMs, cudaStream_t s) {
    const OneScene one{sc, rp};
    if (sc.shell) {
        if (sc.world.enters) XGB_LAUNCH((k_trace_world<ANY, COUNT, OneScene, true, true>))(one, q, h, retrace, sq, out, ctrl);
        else XGB_LAUNCH((k_trace_world<ANY, COUNT, OneScene, false, true>))(one, q, h, retrace, sq, out, ctrl);
    } else {
        if (sc.world.enters) XGB_LAUNCH((k_trace_world<ANY, COUNT, OneScene, true, false>))(one, q, h, retrace, sq, out, ctrl);
        else XGB_LAUNCH((k_trace_world<ANY, COUNT, OneScene, false, false>))(one, q, h, retrace, sq, out, ctrl);
    }
    if (ANY || sc.nInstances == 1) return 1;
    XGB_LAUNCH(k_retrace<OneScene>)(one, q, h, retrace, ctrl);
    return 2;
}
int launchExtend(const SceneDev& scene, PathQueue q, HitQueue h, unsigned int* retrace, Ctrl* ctrl, int numSMs, bool count,
                 bool teams, cudaStream_t s) {
    const SceneDev sc = withTeams(scene, false, teams && !count);
    if (sc.teams) XGB_LAUNCH((k_trace_team<false, OneScene>))(OneScene{sc, RenderParams{}}, q, h, ShadowQueue{}, PathQueue{}, ctrl);
    const int before = sc.teams ? 1 : 0;
    RenderParams none{};
    if (useWorld(sc, false)) {
        const int n = count ? launchWorld<false, true>(sc, none, q, h, retrace, ShadowQueue{}, PathQueue{}, ctrl, numSMs, s)
                            : launchWorld<false, false>(sc, none, q, h, retrace, ShadowQueue{}, PathQueue{}, ctrl, numSMs, s);
        return n + before;
    }
    if (sc.listed && sc.blasLayout == 1) {
        if (count) XGB_LAUNCH((k_trace_wide<false, true>))(sc, none, q, h, ShadowQueue{}, PathQueue{}, ctrl);
        else XGB_LAUNCH((k_trace_wide<false, false>))(sc, none, q, h, ShadowQueue{}, PathQueue{}, ctrl);
    } else if (sc.listed && sc.shell) {
        if (count) XGB_LAUNCH((k_trace_flat2<false, true, OneScene, true>))(OneScene{sc, none}, q, h, ShadowQueue{}, PathQueue{}, ctrl);
        else XGB_LAUNCH((k_trace_flat2<false, false, OneScene, true>))(OneScene{sc, none}, q, h, ShadowQueue{}, PathQueue{}, ctrl);
    } else if (sc.listed) {
        if (count) XGB_LAUNCH((k_trace_flat2<false, true, OneScene>))(OneScene{sc, none}, q, h, ShadowQueue{}, PathQueue{}, ctrl);
        else XGB_LAUNCH((k_trace_flat2<false, false, OneScene>))(OneScene{sc, none}, q, h, ShadowQueue{}, PathQueue{}, ctrl);
    } else if (count) {
        XGB_LAUNCH((k_extend<true>))(sc, q, h, ctrl);
    } else {
        XGB_LAUNCH((k_extend<false>))(sc, q, h, ctrl);
    }
    return 1 + before;
}
int launchShadow(const SceneDev& scene, const RenderParams& rp, ShadowQueue sq, PathQueue out, Ctrl* ctrl, int numSMs,
                 bool teams, cudaStream_t s) {
    const SceneDev sc = withTeams(scene, true, teams);
    if (sc.teams) XGB_LAUNCH((k_trace_team<true, OneScene>))(OneScene{sc, rp}, PathQueue{}, HitQueue{}, sq, out, ctrl);
    const int before = sc.teams ? 1 : 0;
    if (useWorld(sc, true)) {
        return before + launchWorld<true, false>(sc, rp, PathQueue{}, HitQueue{}, nullptr, sq, out, ctrl, numSMs, s);
    }
    if (sc.listed && sc.blasLayout == 1) XGB_LAUNCH((k_trace_wide<true, false>))(sc, rp, PathQueue{}, HitQueue{}, sq, out, ctrl);
    else if (sc.listed && sc.shell)
        XGB_LAUNCH((k_trace_flat2<true, false, OneScene, true>))(OneScene{sc, rp}, PathQueue{}, HitQueue{}, sq, out, ctrl);
    else if (sc.listed)
        XGB_LAUNCH((k_trace_flat2<true, false, OneScene>))(OneScene{sc, rp}, PathQueue{}, HitQueue{}, sq, out, ctrl);
    else XGB_LAUNCH(k_shadow)(sc, rp, sq, out, ctrl);
    return 1 + before;
}

int batchKernels(const SceneDev* scenes, int n) {
    bool world = true, enters = false, flat = true, single = true;
    for (int j = 0; j < n; ++j) {
        const SceneDev& sc = scenes[j];
        world = world && !sc.shell && useWorld(sc, true);
        enters = enters || sc.world.enters;
        flat = flat && sc.nInstances <= kFlatInstances && sc.blasLayout == 0 && !sc.shell;
        single = single && sc.nInstances == 1;
    }
    if (world && single) return kBatchWorldSingle;
    // scenes of few instances take the world BVH for their shadow rays, and for the others
    // only beside scenes of many
    if (flat) return world && !enters ? kBatchFlatWorldShadow : kBatchFlat;
    return world ? (enters ? kBatchWorldEnter : kBatchWorld) : kBatchGeneral;
}
int launchExtendBatch(const BatchView& b, PathQueue q, HitQueue h, unsigned int* retrace, Ctrl* ctrl, int numSMs,
                      cudaStream_t s) {
    const BatchScenes sc{b};
    if (b.teams) XGB_LAUNCH((k_trace_team<false, BatchScenes>))(sc, q, h, ShadowQueue{}, PathQueue{}, ctrl);
    int launches = b.teams ? 2 : 1;
    switch (b.kernels) {
    case kBatchWorldSingle:
    case kBatchWorld:
        XGB_LAUNCH((k_trace_world<false, false, BatchScenes, false, false>))(sc, q, h, retrace, ShadowQueue{}, PathQueue{}, ctrl);
        break;
    case kBatchWorldEnter:
        XGB_LAUNCH((k_trace_world<false, false, BatchScenes, true, false>))(sc, q, h, retrace, ShadowQueue{}, PathQueue{}, ctrl);
        break;
    case kBatchFlat:
    case kBatchFlatWorldShadow: XGB_LAUNCH((k_trace_flat2<false, false, BatchScenes>))(sc, q, h, ShadowQueue{}, PathQueue{}, ctrl); break;
    default: XGB_LAUNCH(k_extend_batch)(b, q, h, ctrl);
    }
    if (b.kernels == kBatchWorld || b.kernels == kBatchWorldEnter) {
        XGB_LAUNCH(k_retrace<BatchScenes>)(sc, q, h, retrace, ctrl);
        ++launches;
    }
    return launches;
}
int launchShadowBatch(const BatchView& b, ShadowQueue sq, PathQueue out, Ctrl* ctrl, int numSMs, cudaStream_t s) {
    const BatchScenes sc{b};
    if (b.teams) XGB_LAUNCH((k_trace_team<true, BatchScenes>))(sc, PathQueue{}, HitQueue{}, sq, out, ctrl);
    switch (b.kernels) {
    case kBatchWorldSingle:
    case kBatchWorld:
    case kBatchFlatWorldShadow: XGB_LAUNCH((k_trace_world<true, false, BatchScenes, false, false>))(sc, PathQueue{}, HitQueue{}, nullptr, sq, out, ctrl); break;
    case kBatchWorldEnter: XGB_LAUNCH((k_trace_world<true, false, BatchScenes, true, false>))(sc, PathQueue{}, HitQueue{}, nullptr, sq, out, ctrl); break;
    case kBatchFlat: XGB_LAUNCH((k_trace_flat2<true, false, BatchScenes>))(sc, PathQueue{}, HitQueue{}, sq, out, ctrl); break;
    default: XGB_LAUNCH(k_shadow_batch)(b, sq, out, ctrl);
    }
    return b.teams ? 2 : 1;
}

// One instance takes the persistent per-lane kernel: 300,000 closest hits on a terrain of
// 520,000 triangles 0.63 -> 0.57 ms for the whole call, most of it copies. Traversal limits
// other than the defaults count traceScene's steps, one per node and leaf.
void launchQuery(const SceneDev& sc, const float* rays, int n, int any, float* hits, int* occluded, Ctrl* ctrl, int numSMs,
                 cudaStream_t s) {
    const bool limits = sc.maxSteps != kDefaultMaxSteps || sc.stackLimit != kMaxStackLimit;
    if (sc.nInstances == 1 && sc.world.tris && !sc.shell && !limits) {
        const QueryRays in{sc, rays, hits, occluded};
        if (any)
            XGB_LAUNCH((k_trace_world<true, false, QueryRays, false, false>))(in, PathQueue{}, HitQueue{}, nullptr, ShadowQueue{}, PathQueue{}, ctrl);
        else
            XGB_LAUNCH((k_trace_world<false, false, QueryRays, false, false>))(in, PathQueue{}, HitQueue{}, nullptr, ShadowQueue{}, PathQueue{}, ctrl);
    } else if (any) {
        XGB_LAUNCH((k_query<true>))(sc, rays, n, hits, occluded, ctrl);
    } else {
        XGB_LAUNCH((k_query<false>))(sc, rays, n, hits, occluded, ctrl);
    }
}
#undef XGB_LAUNCH

}  // namespace xgb
