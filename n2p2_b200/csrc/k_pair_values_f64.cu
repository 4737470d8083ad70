// FP64 instances of the pair kernels' G pass.
#include "pairs_launch.cuh"

namespace n2p2b200 {

void launchPairValuesF64(DevModel const& m, DevPairTable const& gt, BatchView const& b, int sms, cudaStream_t st, int variant)
{
    pairValuesT<double>(m, gt, b, sms, st, variant);
}

} // namespace n2p2b200
