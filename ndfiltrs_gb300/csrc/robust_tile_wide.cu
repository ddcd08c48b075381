// The robust tile kernels of 50 to 128 samples.
#include "robust_tile.cuh"

namespace ndf {

cudaError_t launch_robust_tile_wide(const Plan& p, const float* in, float* out, cudaStream_t s) {
  switch (p.robust_width) {
    case 64: return robust_tile::launch_kind<64>(p, in, out, s);
    case 81: return robust_tile::launch_kind<81>(p, in, out, s);
    case 128: return robust_tile::launch_kind<128>(p, in, out, s);
    default: return cudaErrorInvalidValue;
  }
}

}  // namespace ndf
