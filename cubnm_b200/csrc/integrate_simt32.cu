// FP32 per-simulation integrator: the FP32-mode kernel for what the tiles
// (integrate_mma.cu, integrate_fp32.cu: up to 224 nodes without delays) and the delay
// kernel (integrate_delay.cuh) do not take -- numerical FIC without delays, Kuramoto, more
// than 224 nodes without delays, tiles with few simulations each, simulations with too many
// delays below 32 steps, forced coupling forms.
//
// The per-simulation kernel of integrate_sim.cuh with R = float: node state,
// parameters, SC, noise and delay ring buffers in FP32 (half the bytes of the
// FP64 path where the delayed coupling is gather-bound, MUFU exp instead of the
// FP64 software exp), Balloon-Windkessel state and BOLD in FP64.  Compiled with
// FMA contraction.
#include "integrate_sim.cuh"

namespace cbnm {

cudaError_t launch_integrate_simt32(int model, const IntegrateArgs &a, cudaStream_t st) {
    return launch_sim_model<float>(model, a, st);
}

}  // namespace cbnm
