// The tail of a render: few paths left, each finished by one thread in one launch.
// Included by the units that instantiate k_tail (tail*.cu), each
// compiled with -fmad=false as every unit that shades.
#pragma once
#include "shade.cuh"
#include "trace.cuh"

namespace xgb {

// A wavefront iteration lasts at least as long as its slowest ray: with a few thousand
// paths left, the occluded room's 120 last iterations took 0.3-0.4 ms each for rays that
// average 15 us, and the launches themselves 20 us. Here a thread keeps its path in
// registers and alternates closest hit, shading and shadow ray until the path ends, so
// the launch lasts as long as the longest path, not as the sum over the iterations of
// the slowest ray of each. The work per vertex is that of the wavefront (shadeVertex,
// the same traversal order), so the film is the same up to the order of its sums.
//
// Threads of a warp wait for one another at every phase, so the paths are spread over as
// many warps as the GPU holds: a warp takes only ceil(n / warps) of them at a time.
//
// A path that is still alive after kTailVertices vertices goes to the output queue, from
// where the next launch takes it, so that a launch ends in bounded time.
constexpr int kTailBlock = 128;
constexpr int kTailBlocksPerSM = 4;  // 128 registers
constexpr int kTailVertices = 1024;
static_assert(kTailBlocksPerSM * kTailBlock == (int)kTailThreadsPerSM, "threads of a full grid");

template <class J, int NESTED>
__global__ void __launch_bounds__(kTailBlock, kTailBlocksPerSM) k_tail(J jobs, PathQueue in, PathQueue out, Ctrl* ctrl) {
    const unsigned int n = ctrl->nTail;
    const unsigned int warps = gridDim.x * (kTailBlock / 32);
    const unsigned int lanes = min(32u, (n + warps - 1u) / warps);  // paths a warp holds at a time
    const unsigned int lane = threadIdx.x & 31;
    if (lane >= lanes) return;
    const unsigned int laneMask = lanes == 32u ? kFull : (1u << lanes) - 1u;
    const unsigned int warp = blockIdx.x * (kTailBlock / 32) + (threadIdx.x >> 5);
    unsigned int extension = 0, shadows = 0, ended = 0;
    for (unsigned int i = warp * lanes + lane; i < n; i = warps * lanes + atomicAdd(&ctrl->extendHead, 1u)) {
        ShadeOut r;
        r.o = in.o[i];
        r.d = in.d[i];
        r.thr = in.thr[i];
        r.rng = in.rng[i];
        bool cont = true;
        for (int v = 0; cont && v < kTailVertices; ++v) {
            int job, pix;
            jobs.decode(__float_as_int(r.thr.w), job, pix);
            const SceneDev& sc = jobs.scene(job);
            TraceHit hit;
            const V3 o(r.o.x, r.o.y, r.o.z), d(r.d.x, r.d.y, r.d.z);
            ++extension;
            traceCall(sc, o, d, __int_as_float(0x7f800000), false, hit, &ctrl->errors);
            bool shadow = false, done = false;
            cont = false;
            r.stochastic = false;
            shadeVertex<J, NESTED, kAov>(jobs, in, i, r.o, r.d, r.thr, r.rng,
                                         make_float4(hit.t, hit.b0, hit.b1, __int_as_float(hit.prim)), hit.inst, r, cont,
                                         shadow, done);
            if (shadow) {
                ++shadows;
                const V3 so(r.so.x, r.so.y, r.so.z), sd(r.sd.x, r.sd.y, r.sd.z);
                if (!traceCall(sc, so, sd, r.so.w, true, hit, &ctrl->errors)) {
                    filmAddS(jobs.params(job), pix, V3(r.sc.x, r.sc.y, r.sc.z));
                    if (r.stochastic && cont) r.rng = r.srng;  // as the shadow kernels commit it
                }
            }
            ended += done ? 1u : 0u;
        }
        if (cont) {
            const unsigned int slot = atomicAdd(&ctrl->nOut, 1u);
            out.o[slot] = r.o;
            out.d[slot] = r.d;
            out.thr[slot] = r.thr;
            out.rng[slot] = r.rng;
        }
    }
    __syncwarp(laneMask);
    extension = __reduce_add_sync(laneMask, extension);
    shadows = __reduce_add_sync(laneMask, shadows);
    ended = __reduce_add_sync(laneMask, ended);
    if (lane == 0 && extension) {
        atomicAdd(&ctrl->extensionRays, (unsigned long long)extension);
        atomicAdd(&ctrl->shadowRays, (unsigned long long)shadows);
        atomicAdd(&ctrl->pathsDone, (unsigned long long)ended);
    }
}

void launchTailMask1(const OneJob& job, PathQueue in, PathQueue out, Ctrl* ctrl, int numSMs, cudaStream_t s);
void launchTailMask2(const OneJob& job, PathQueue in, PathQueue out, Ctrl* ctrl, int numSMs, cudaStream_t s);
void launchTailMask3(const OneJob& job, PathQueue in, PathQueue out, Ctrl* ctrl, int numSMs, cudaStream_t s);

}  // namespace xgb
