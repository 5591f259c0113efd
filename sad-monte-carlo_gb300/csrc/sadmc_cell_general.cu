// The periodic-cell move kernel for the methods without a lean path: canonical and 1/t-WL.
#include "sadmc_cell_kernel.cuh"

namespace sadmc {

cudaError_t launch_cell_move_general(const MoveLaunch& m, const CellSys& s, int lpw, cudaStream_t st) {
  SADMC_CELL_ALL_SHAPES(dev::FAM_GENERAL)
  return cudaErrorInvalidConfiguration;
}

}  // namespace sadmc
