// FP32 instances of the pair kernels' G pass.
#include "pairs_launch.cuh"

namespace n2p2b200 {

void launchPairValuesF32(DevModel const& m, DevPairTable const& gt, BatchView const& b, int sms, cudaStream_t st, int variant)
{
    pairValuesT<float>(m, gt, b, sms, st, variant);
}

} // namespace n2p2b200
