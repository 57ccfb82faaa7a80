// Launch wrappers shared between the host API (api.cu) and the kernel
// translation units. No CUDA types beyond cudaStream_t cross this boundary.
#pragma once
#include <cuda_runtime.h>
#include <stddef.h>
#include <stdint.h>

#include "xgb_types.h"

namespace xgb {

// ---- BVH build (bvh_build.cu) ------------------------------------------------
constexpr int kBuilderPloc = 0;  // locally-ordered clustering (default)
constexpr int kBuilderLbvh = 1;  // Morton-split linear BVH
constexpr int kLayoutBinary = 0;  // Node2, two children per 64-byte node
constexpr int kLayoutWide = 1;    // WNode, eight quantised children per 80-byte node
struct BlasBuildInput {
    const float4* pos;  // device, object space
    const int* idx;     // device, 3 per triangle
    int nTris;
    int builder;        // kBuilderPloc or kBuilderLbvh
    int layout;         // kLayoutBinary or kLayoutWide
    cudaMemPool_t pool; // scratch memory and the wide nodes come from it
};
struct BlasBuildOutput {
    WNode* nodes;       // wide layout: device, allocated by buildBlas (nWide entries; the caller frees it)
    int nWide;
    Node2* nodes2;      // binary layout: device, nTris - 1 entries, allocated by the caller
    int wide;
    TriV* tris;         // device, nTris entries (leaf order), allocated by the caller
    float4* gnrm;       // device, nTris entries (original order)
    float* triArea;     // device, nTris entries (original order)
    int rootIsLeaf;
    int rootLeaf;
    float boundsLo[3], boundsHi[3];  // object-space bounds of the vertices used
};
// Builds a binary BVH over the triangles (PLOC or LBVH), in the binary layout or
// converted into an 8-wide compressed BVH, on `stream`, and synchronises it.
// Returns a CUDA error code (cudaSuccess on success).
cudaError_t buildBlas(const BlasBuildInput& in, BlasBuildOutput* out, cudaStream_t stream);

// Rows of `stride` floats (3 or 4) -> float4 with w = 0; of 2 or 4 floats -> float2.
void expandVec3(const float* src, int stride, size_t n, float4* dst, cudaStream_t s);
void expandUv(const float* src, int stride, size_t n, float2* dst, cudaStream_t s);

// An instance's share of a world BVH (WorldDev): the mesh's nodes (none when its root is a
// leaf) renumbered to start at nodeBase, its triangles at triBase with the instance's number.
struct WorldPart {
    const Node2* nodes;
    const TriV* tris;
    int nodeBase, triBase, inst;
};
// Parts on the device, in ascending order of both bases: the world's nodes [nTop, nNodes) and
// triangles [0, nTris). codes: the world's nodes [0, nTop) are those of `top`, its leaf i
// with codes[i] in its place (nullptr: they are there already).
void worldCopy(const WorldPart* parts, int nParts, const Node2* top, const int* codes, int nTop, int nNodes, int nTris,
               Node2* worldNodes, TriV* worldTris, cudaStream_t s);

// SVNDF fit of a displacement map (svndf.cu): lobes [resV][resU][5] float4, low
// heights [resV][resU] float4 (red channel). rate in [1, 16].
cudaError_t svndfFit(const TextureDev& src, float scale, int rate, uint32_t seed, int resU, int resV, float4* lobes,
                     float4* low, cudaStream_t s);

// ---- wavefront (integrator.cu / trace.cu) --------------------------------------
struct Ctrl {
    unsigned long long nextPath;   // next camera path id to generate
    unsigned long long totalPaths;
    unsigned long long firstNew;   // id of the first path generated this iteration
    unsigned int nCont;            // paths carried over into this iteration's input queue
    unsigned int nActive;          // paths in this iteration's input queue
    unsigned int nOut;             // paths written to the output queue by shade
    unsigned int nShadow;          // shadow rays written by shade (counted with nOut as one 64-bit word)
    unsigned int extendHead;       // persistent work counters
    unsigned int shadowHead;
    unsigned int errors;           // bit 0: traversal stack overflow
    unsigned int nRetrace;         // rays whose hits the instance order decides (k_trace_world)
    unsigned int nShadowDue;       // shadow rays of the previous shade launch, traced beside the next rays
    unsigned int nTail;            // paths the next tail launch finishes (0: it does nothing)
    unsigned int retraceHead;      // rays of nRetrace that k_retrace has taken
    unsigned long long extensionRays;
    unsigned long long shadowRays;
    unsigned long long iterations;
    unsigned long long pathsDone;
    unsigned long long nodeVisits;  // profiling counters (extension rays)
    unsigned long long triTests;
};

static_assert(offsetof(Ctrl, nOut) % 8 == 0 && offsetof(Ctrl, nShadow) == offsetof(Ctrl, nOut) + 4, "one 64-bit counter");

// ERR_WAIT: a bounded mbarrier wait of the tensor-memory inference kernels gave up.
enum ErrorBits : unsigned int { ERR_STACK = 1u, ERR_QUEUE = 2u, ERR_LOOP = 4u, ERR_WAIT = 8u };

struct PathQueue {
    float4* o;          // o.xyz, w = pdf of the BSDF sample that produced this ray (-1: specular)
    float4* d;          // d.xyz, w = bits: pathLength | flags << 16
    float4* thr;        // throughput.xyz, w = bits: pixel index
    uint2* rng;         // PCG state
    int* grec;          // guide training: record of the vertex this ray left (-1: none)
    unsigned int* pid;  // guide training: index of the path within the render call
};

// One training sample of the guiding network: a guided vertex, the direction
// sampled there and, once the path has finished, the incident radiance found
// along it: (contributions of the later vertices) / (throughput after this vertex).
struct __align__(16) GuideRecord {
    float3 p;
    float pdf;        // density wi was sampled with (mixture of BSDF and network)
    float3 n;
    float fcos;       // luminance of bsdfCos(wi) (product target)
    float3 wo;
    unsigned int pid; // path index within the render call
    float3 wi;
    float radiance;   // training target (luminance), filled in when the call ends
    float3 snap;      // the path's accumulated contribution before the next vertex (NaN: none)
    float pad0;
    float3 thr;       // path throughput after this vertex
    float pad1;
};
static_assert(sizeof(GuideRecord) == 96, "GuideRecord size");

struct HitQueue {
    float4* h;    // t, b0, b1, bits(prim); prim = -1 on a miss
    int* inst;
};
struct ShadowQueue {
    float4* o;          // o.xyz, tMax
    float4* d;          // d.xyz, bits(pixel)
    float4* c;          // contribution rgb, bits(output-queue index of the path or -1)
    uint2* rng;         // PCG state after a stochastic bsdfCos (committed if visible)
    unsigned int* pid;  // guide training: path credited with the contribution
};

enum PathFlags : int { FLAG_PRIMARY = 1, FLAG_STOCHASTIC_NEE = 2 };

struct RenderParams {
    int width, height;
    uint32_t sppBegin;
    uint32_t seed;
    int integrator;
    int maxDepth;
    int rrStart;
    float rrProb;
    unsigned int capacity;
    int filmFp64;
    void* film;  // float4* or double4*
    void* aov;   // first-hit albedo plane then normal plane (same type as film), nullptr: off
    int dropNonFinite;  // film additions with a non-finite component are skipped (opt-in fix)
    // learned proposal (0 / nullptr when off)
    int guided;
    int train;
    float bsdfFrac;           // one-sample MIS: probability of sampling the BSDF
    const float4* mix;        // per input path: 8 x (mu, kappa) then 8 weights
    GuideRecord* arena;       // training records of this call
    unsigned int* arenaCount; // may run past arenaCap (writers drop)
    int arenaCap;
    float recordProb;         // probability that a guided vertex becomes a record
    float4* pathAcc;          // per path of the call: contributions so far (rgb)
    // order of the camera paths of a sample pass: tileW x tileH pixel blocks
    // (k_generate), 0 = scanline rows
    int tileW, tileH;
    // order of the samples: sampleGroup (> 1) consecutive camera paths are
    // consecutive samples of one pixel, in passes of sampleGroup samples over
    // the film; 0 or 1 = one sample pass over the film after the other.
    // sppCount = samples of this call.
    int sampleGroup;
    unsigned int sppCount;
};

// Device arrays of a batch of render jobs sharing one wavefront (xgb_render_batch):
// a path of job j carries j << 24 | pixel in its pixel field.
// Which traversal kernels a batch takes: every scene has a world BVH (without / with
// instances to enter, or all of one instance, where no hit is marked to be traced again);
// every scene has <= 16 instances and binary mesh BVHs (and a world BVH for the shadow
// rays); any other.
enum BatchKernels : int {
    kBatchGeneral = 0,
    kBatchFlat = 1,
    kBatchWorld = 2,
    kBatchWorldEnter = 3,
    kBatchFlatWorldShadow = 4,
    kBatchWorldSingle = 5
};
struct BatchView {
    const SceneDev* scenes;
    const RenderParams* params;
    const unsigned long long* start;  // nJobs + 1 prefix sums of the jobs' path counts
    int nJobs;
    int kernels; // BatchKernels
    int nested;   // some scene has a material that evaluates another (the shade kernel with that code)
    int teams;    // small queues go to teams of lanes
    int counted;  // some scene bounds the steps of a ray
};
int batchCounted(const SceneDev* scenes, int n);
int batchTeams(const SceneDev* scenes, int n);
int batchKernels(const SceneDev* scenes, int n);
void launchGenerateBatch(const BatchView& b, PathQueue q, Ctrl* ctrl, int grid, cudaStream_t s);
void launchShadeBatch(const BatchView& b, PathQueue in, HitQueue h, PathQueue out, ShadowQueue sq, Ctrl* ctrl,
                      int numSMs, cudaStream_t s);
// Both return the number of kernels launched.
int launchExtendBatch(const BatchView& b, PathQueue q, HitQueue h, unsigned int* retrace, Ctrl* ctrl, int numSMs,
                      cudaStream_t s);
int launchShadowBatch(const BatchView& b, ShadowQueue sq, PathQueue out, Ctrl* ctrl, int numSMs, cudaStream_t s);

// Queue bookkeeping of an iteration. mode kPlanWave: a wavefront iteration; kPlanTail: the
// new camera paths go to a tail launch; kPlanTailIfFew: nothing happens (and the tail launch
// that follows does nothing) unless every camera path has started and at most tailMax paths
// are left, or at most tailOpen and fewer than half of those before the last vertex; they then
// go to the tail launch.
// A wavefront iteration also hands the shadow rays of the last shade launch to launchShadow;
// kPlanShadow does only that.
enum PlanMode : int { kPlanWave = 0, kPlanTail = 1, kPlanTailIfFew = 2, kPlanShadow = 3 };
// A call that fails after it has put work on its stream waits for that work all the same:
// the caller frees or reuses next what it reads and writes.
struct WaitOnFailure {
    cudaStream_t stream;
    bool done = false;
    ~WaitOnFailure() { if (!done) cudaStreamSynchronize(stream); }
};
// A second stream for the launches that run beside others, with its two events.
struct SideLane {
    cudaStream_t stream = nullptr;
    cudaEvent_t fork = nullptr, join = nullptr;
    bool create();
    void destroy();
    // Work of `stream` starts after what `s` has enqueued; and `s` goes on after it.
    void begin(cudaStream_t s) const { cudaEventRecord(fork, s); cudaStreamWaitEvent(stream, fork, 0); }
    void end() const { cudaEventRecord(join, stream); }
    void wait(cudaStream_t s) const { cudaStreamWaitEvent(s, join, 0); }
};
void launchPlan(Ctrl* ctrl, unsigned int capacity, cudaStream_t s, int mode = kPlanWave, unsigned int tailMax = 0,
                unsigned int tailOpen = 0);
// Paths up to which a tail launch beats the remaining wavefront iterations. Measured with
// 4,096 / 16,384 / 65,536 / 131,072 paths (none: no tail launches), ms per call: occluded
// room 384^2 x 8 55.6 / 51.1 / 46.6 / 45.9 (73.8), shell-mapped cloth 320^2 x 4 27.3 / 23.8 /
// 21.5 / 22.6 (40.9), its SVBRDF variant 26.7 / 24.4 / 23.0 / 25.7 (33.4); microfacet normal
// mapping, whose walks of up to 100 facets per BSDF call make a warp's lanes wait for one
// another and its code overflow the instruction cache, 400^2 x 4 6.4 / 7.3 / 10.3 / 10.3 (6.5).
// A tail thread walks a top-level BVH, or 8-wide nodes, by itself and slowly: those scenes take
// 8,192 where paths stay (metal rooms of 18 and 11 instances, 65,024 camera paths: 3.1 and 1.4 ms
// per call with 65,536, 1.0 and 0.7 without tail launches; of 18 and 25 instances, 16,256 camera
// paths: 1.57 and 1.77 with 16,384, 0.80 and 0.87 with 8,192, 1.20 and 1.39 without). Over 130
// random scenes of each kind, 6,000 to 200,000 paths, a call takes 0.25 / 0.41 of the time without
// tail launches in the mean, at worst 0.84 / 0.96 (with 65,536 for all 0.28 / 0.36, at worst 1.04 /
// 1.47); of 2 to 16 instances and binary meshes, with 65,536, 0.34, above 1 in two of 675.
//
// Up to tailOpen where paths leave fast, fewer than half of them having lived through the last
// vertex (under an open sky 10 to 25 % do): 65,536, and 524,288 in scenes without lights whose
// instances are walked as a list. With 65,536 / 262,144 / 524,288 / 1,048,576 paths the terrain took
// at 700,000 camera paths 1.70 / 1.45 / 1.31 / 1.53, 2.1 million 2.35 / 2.36 / 2.06 / 2.00, 67 million
// 30.5 / 30.4 / 30.4 / 30.4. In closed rooms most paths stay, and the wavefront is faster: with five
// clouds of triangles, 204,000 camera paths, 3.2 with 65,536, 5.8 with 524,288, 3.6 without tail
// launches. So is it over a top-level BVH (30 boxes on the terrain, 507,000 paths: 0.91 / 2.15;
// 300 boxes 1.73 / 7.2), and with lights (Cornell box, 262,000 paths: 0.58 / 1.30).
//
// A scene of one instance without lights takes two paths per thread of a full grid (155,648)
// whether they stay or not: the terrain at 134,000 camera paths 0.51 -> 0.31, closed rooms as one
// mesh 0.17 to 0.86 of the time without tail launches, but up to 1.34 of it at 320,000. Over 380
// random scenes without lights, 66,000 to 2 million paths, a call takes 0.44 of the time without tail
// launches in the mean and 0.99 at worst.
constexpr unsigned int kTailThreadsPerSM = 512;
inline unsigned int tailMaxPaths(const SceneDev& sc, int numSMs) {
    if (sc.nested & 1) return 4096u;
    if (!sc.listed || sc.blasLayout != 0) return 8192u;
    return sc.nLights == 0 && !sc.nested && sc.nInstances == 1 ? 2u * kTailThreadsPerSM * (unsigned int)numSMs : 65536u;
}
inline unsigned int tailOpenPaths(const SceneDev& sc) {
    if (sc.nested & 1) return 4096u;
    return sc.nLights == 0 && !sc.nested && sc.listed ? 524288u : 65536u;
}
// Finishes the ctrl->nTail paths of `in`; those that outlive the launch's bound go to `out` (tail.cuh).
void launchTail(const SceneDev& sc, const RenderParams& rp, PathQueue in, PathQueue out, Ctrl* ctrl, int numSMs,
                cudaStream_t s);
void launchGenerate(const SceneDev& sc, const RenderParams& rp, PathQueue q, Ctrl* ctrl, int grid, cudaStream_t s);
// Extension / shadow rays and shading of the wavefront; grids sized from the
// launched kernel's occupancy on numSMs SMs (one full wave).
// teams: whether small queues go to teams of lanes, where the scene allows it (not where a tail
// launch takes over before a queue gets that small).
// retrace: room for one number per path in the queue (the output queue, which is empty then).
// Both return the number of kernels launched.
int launchExtend(const SceneDev& sc, PathQueue q, HitQueue h, unsigned int* retrace, Ctrl* ctrl, int numSMs, bool count, bool teams,
                  cudaStream_t s);
void launchShade(const SceneDev& sc, const RenderParams& rp, PathQueue in, HitQueue h, PathQueue out, ShadowQueue sq,
                 Ctrl* ctrl, int numSMs, cudaStream_t s);
int launchShadow(const SceneDev& sc, const RenderParams& rp, ShadowQueue sq, PathQueue out, Ctrl* ctrl, int numSMs,
                  bool teams, cudaStream_t s);
// Film plane (float4 or double4 per pixel) -> packed float RGB, strideFloats 3 or 4 (image.cu).
void launchPackFilm(const void* film, int fp64, size_t n, int strideFloats, float* out, int grid, cudaStream_t s);
// Ray queries on a built scene: rays of 7 floats (o, d, tMax); closest hits as 5 floats per ray
// (t, instance, triangle, b0, b1; -1 for none) or any-hit flags. ctrl: zero but for nActive
// and nShadowDue = n.
void launchQuery(const SceneDev& sc, const float* rays, int n, int any, float* hits, int* occluded, Ctrl* ctrl, int numSMs,
                 cudaStream_t s);

}  // namespace xgb
