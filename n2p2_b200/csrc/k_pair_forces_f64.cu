// FP64 instances of the pair kernels' force pass.
#include "pairs_launch.cuh"

namespace n2p2b200 {

void launchPairForcesF64(DevModel const& m, DevPairTable const& gt, BatchView const& b, int sms, cudaStream_t st, int variant)
{
    pairForcesT<double>(m, gt, b, sms, st, variant);
}

} // namespace n2p2b200
