// FP32 instances of the pair kernels' force pass.
#include "pairs_launch.cuh"

namespace n2p2b200 {

void launchPairForcesF32(DevModel const& m, DevPairTable const& gt, BatchView const& b, int sms, cudaStream_t st, int variant)
{
    pairForcesT<float>(m, gt, b, sms, st, variant);
}

} // namespace n2p2b200
