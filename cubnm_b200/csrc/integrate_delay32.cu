// FP32 instantiation of the delay kernel (node states and coupling in FP32).
#include "integrate_delay.cuh"

namespace cbnm {

cudaError_t delay_config32(int model, const IntegrateArgs &a, int sms, DelayLaunch *c) {
    return delayblk::config<float>(model, a, sms, c);
}
cudaError_t launch_delay32(int model, const IntegrateArgs &a, const DelayLaunch &c, cudaStream_t st) {
    return delayblk::launch<float>(model, a, c, st);
}

}  // namespace cbnm
