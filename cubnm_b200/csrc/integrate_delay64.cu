// FP64 instantiation of the delay kernel (compiled with --fmad=false: the node update
// keeps the reference's operation order; the coupling sum uses fma explicitly).
#include "integrate_delay.cuh"

namespace cbnm {

cudaError_t delay_config64(int model, const IntegrateArgs &a, int sms, DelayLaunch *c) {
    return delayblk::config<double>(model, a, sms, c);
}
cudaError_t launch_delay64(int model, const IntegrateArgs &a, const DelayLaunch &c, cudaStream_t st) {
    return delayblk::launch<double>(model, a, c, st);
}

}  // namespace cbnm
