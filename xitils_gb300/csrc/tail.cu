// The tail kernel for scenes without nested materials and its launch; see tail.cuh.
// Compiled with -fmad=false.
#include "tail.cuh"

namespace xgb {

void launchTail(const SceneDev& sc, const RenderParams& rp, PathQueue in, PathQueue out, Ctrl* ctrl, int numSMs,
                cudaStream_t s) {
    const OneJob job{sc, rp};
    switch (sc.nested & 3) {
    case 1: launchTailMask1(job, in, out, ctrl, numSMs, s); break;
    case 2: launchTailMask2(job, in, out, ctrl, numSMs, s); break;
    case 3: launchTailMask3(job, in, out, ctrl, numSMs, s); break;
    default:
        // As in launchShade, a scene of Lambert materials only takes a variant with that code
        // alone: a path's first vertices wait for instructions (Cornell box 64 x 48 x 1 with planes
        // 0.203 -> 0.192 ms per call). GGX metal gained nothing (180,000 triangles, 317 x 211 x 2:
        // 1.67 ms both ways), nor did more blocks per SM (six 0.200, eight 0.207).
        if (rp.integrator == 0 && (sc.kinds & ~(1 << MAT_EMISSION)) == (1 << MAT_DIFFUSE))
            k_tail<OneJob, kOnlyDiffuse><<<numSMs * kTailBlocksPerSM, kTailBlock, 0, s>>>(job, in, out, ctrl);
        else k_tail<OneJob, 0><<<numSMs * kTailBlocksPerSM, kTailBlock, 0, s>>>(job, in, out, ctrl);
    }
}

}  // namespace xgb
