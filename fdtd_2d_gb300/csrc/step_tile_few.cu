// The register-tile kernel (step_tile.cuh) for shots with few points: its
// instances, apart from the others for compile time.
#include "step_tile.cuh"

namespace fdtd2d {

namespace {

template <int RP, bool AUX, class T>
const void* kernel_of(bool lossless) {
  return lossless ? (const void*)step_tmat_kernel<Tile<RP>, true, AUX, true, T> : (const void*)step_tmat_kernel<Tile<RP>, false, AUX, true, T>;
}
template <int RP>
const void* kernel_of(int store, bool lossless, bool aux) {
  if (store != 0) return aux || store != 1 ? nullptr : kernel_of<RP, false, __half>(lossless);
  return aux ? kernel_of<RP, true, float>(lossless) : kernel_of<RP, false, float>(lossless);
}

}  // namespace

const void* tile_kernel_few(int shape, int store, bool lossless, bool aux) {
  return shape == 0 ? kernel_of<kShapes[0]>(store, lossless, aux) : kernel_of<kShapes[1]>(store, lossless, aux);
}

}  // namespace fdtd2d
