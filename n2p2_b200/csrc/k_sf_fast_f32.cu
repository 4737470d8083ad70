// FP32 instances of the symmetry-function passes (mixed precision form).
#include "sf_launch.cuh"

namespace n2p2b200 {

void launchSFValuesF32(DevModel const& m, BatchView const& b, int sms, cudaStream_t st)
{
    valuesT<float>(m, b, sms, st);
}

void launchSFForcesF32(DevModel const& m, BatchView const& b, int sms, cudaStream_t st)
{
    forcesT<float>(m, b, sms, st);
}

} // namespace n2p2b200
