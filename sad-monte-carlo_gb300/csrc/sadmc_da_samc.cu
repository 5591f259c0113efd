// Delayed-acceptance kernels of SAMC walkers.
#include "sadmc_da_kernel.cuh"

namespace sadmc {

DaKernel da_kernel_samc(int tiles) { return da_kernel_of<M_SAMC>(tiles); }

}  // namespace sadmc
