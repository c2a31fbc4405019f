// The register-tile kernel (step_tile.cuh) for FP32 shots with few points: its
// instances, apart from the others for compile time.
#include "step_tile.cuh"

namespace fdtd2d {

namespace {

template <int RP>
const void* kernel_of(bool lossless, bool aux) {
  if (aux) return lossless ? (const void*)step_tmat_kernel<Tile<RP>, true, true, true, float> : (const void*)step_tmat_kernel<Tile<RP>, false, true, true, float>;
  return lossless ? (const void*)step_tmat_kernel<Tile<RP>, true, false, true, float> : (const void*)step_tmat_kernel<Tile<RP>, false, false, true, float>;
}

}  // namespace

const void* tile_kernel_few(int shape, bool lossless, bool aux) {
  return shape == 0 ? kernel_of<kShapes[0]>(lossless, aux) : kernel_of<kShapes[1]>(lossless, aux);
}

}  // namespace fdtd2d
