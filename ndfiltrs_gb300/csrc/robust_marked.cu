// Robust window statistics of the float32 outputs that the tile kernel marked (the
// kernels of robust.cuh, instantiated apart from the others so that they compile in
// parallel).
#include "robust.cuh"

namespace ndf {

cudaError_t launch_robust_marked(const Plan& p, const float* in, float* out, cudaStream_t s) {
  return launch_robust_t<float, true>(p, in, out, s);
}

}  // namespace ndf
