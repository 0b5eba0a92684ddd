// The FP32 instances of the stencil kernels (a translation unit of their own:
// the build compiles the two precisions side by side).
#include "lbm_flux.cuh"

namespace uqlbm {
template cudaError_t launch_flux<float>(int, const KArgs<float> &, int, int, cudaStream_t);
template cudaError_t prepare_flux<float>();
}  // namespace uqlbm
