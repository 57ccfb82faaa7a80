// The tail kernel for scenes with both nested materials (mask 3); see tail.cuh. Compiled with -fmad=false.
#include "tail.cuh"

namespace xgb {

void launchTailMask3(const OneJob& job, PathQueue in, PathQueue out, Ctrl* ctrl, int numSMs, cudaStream_t s) {
    k_tail<OneJob, 3><<<numSMs * kTailBlocksPerSM, kTailBlock, 0, s>>>(job, in, out, ctrl);
}

}  // namespace xgb
