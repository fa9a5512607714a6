// The RK4 run from patches that tests the waits between blocks, for the default scheme pair. It has a
// file of its own, so that the kernels of patch.cu are not built any differently for it: with the limit
// and the silent block as launch parameters of k_patch_rk4, one tendency of hexagon 3, a kernel it does
// not touch, took 16.2 us instead of 15.9 by the place its code got.
#include "model.hpp"
#include "patch.cuh"

namespace trisk {

namespace {

__global__ void __launch_bounds__(512, 1) k_patch_rk4_expire(const PatchParams A) {
  patch_rk4_run<PVM_TRISK, KE_CELL, true>(A);
}

}  // namespace

const void* patch_expire_kernel() {
  const void* kernel = reinterpret_cast<const void*>(k_patch_rk4_expire);
  patch_allow_smem(kernel);
  return kernel;
}

}  // namespace trisk
