// The on-chip kernel (step_resident.cuh) on 16-bit fields, one form for lossy
// and lossless media (a product by 1 is exact; half the instances to compile).
#include "step_resident.cuh"

namespace fdtd2d {

namespace {

template <class T>
const void* kernel_of(int R) {
  switch (R) {
    case 6: return (const void*)step_persist_tile_kernel<6, false, false, false, T>;
    case 4: return (const void*)step_persist_tile_kernel<4, false, false, false, T>;
    default: return (const void*)step_persist_tile_kernel<2, false, false, false, T>;
  }
}

}  // namespace

const void* resident_kernel16(int R, int store) { return store == 1 ? kernel_of<__half>(R) : kernel_of<__nv_bfloat16>(R); }

}  // namespace fdtd2d
