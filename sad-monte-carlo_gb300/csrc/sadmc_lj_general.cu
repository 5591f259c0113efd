// The LJ move kernel for the methods without a lean path: canonical and 1/t-WL.
#include "sadmc_lj_kernel.cuh"

namespace sadmc {

cudaError_t launch_lj_move_general(const MoveLaunch& m, const LjSys& s, int lpw, cudaStream_t st) {
  SADMC_LJ_ALL_SHAPES(dev::FAM_GENERAL, false)
  return cudaErrorInvalidConfiguration;
}

}  // namespace sadmc
