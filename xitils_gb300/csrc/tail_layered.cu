// The tail kernels for scenes with microfacet normal mapping (mask 1) or with
// MultiLobeSVBRDF (mask 2); see tail.cuh. Compiled with -fmad=false.
#include "tail.cuh"

namespace xgb {

void launchTailMask1(const OneJob& job, PathQueue in, PathQueue out, Ctrl* ctrl, int numSMs, cudaStream_t s) {
    k_tail<OneJob, 1><<<numSMs * kTailBlocksPerSM, kTailBlock, 0, s>>>(job, in, out, ctrl);
}
void launchTailMask2(const OneJob& job, PathQueue in, PathQueue out, Ctrl* ctrl, int numSMs, cudaStream_t s) {
    k_tail<OneJob, 2><<<numSMs * kTailBlocksPerSM, kTailBlock, 0, s>>>(job, in, out, ctrl);
}

}  // namespace xgb
