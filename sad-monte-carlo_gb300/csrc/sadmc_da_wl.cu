// Delayed-acceptance kernels of the other methods (Wang-Landau, 1/t), told apart at run time.
#include "sadmc_da_kernel.cuh"

namespace sadmc {

DaKernel da_kernel_any(int tiles) { return da_kernel_of<dev::FAM_ANY>(tiles); }

}  // namespace sadmc
