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
    default: k_tail<OneJob, 0><<<numSMs * kTailBlocksPerSM, kTailBlock, 0, s>>>(job, in, out, ctrl);
    }
}

}  // namespace xgb
