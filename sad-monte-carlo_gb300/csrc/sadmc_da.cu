// Launch of the delayed-acceptance kernels, and their SAD instances (each method's are compiled in
// a file of their own).
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>

#include "sadmc_da_kernel.cuh"

namespace sadmc {

namespace {
DaKernel da_kernel(int tiles, int method) {
  return method == M_SAD ? da_kernel_of<M_SAD>(tiles) : method == M_SAMC ? da_kernel_samc(tiles) : da_kernel_any(tiles);
}
}  // namespace

cudaError_t launch_lj_da(const MoveLaunch& m, const LjSys& s, const SgWeights& w, int max_atoms,
                         int refresh_interval, uint64_t* stats, cudaStream_t st) {
  if ((s.np != 32 && s.np != 64) || max_atoms < 2 || max_atoms > s.np) return cudaErrorInvalidConfiguration;
  const int tiles = std::max(dev::da_rows(max_atoms) / 16, s.np == 32 ? 1 : 3);
  // The limit is set once per device and shape.  Host threads launching on
  // one device may race to set it; setting it twice is harmless, and the flags are atomic.
  static std::atomic<bool> attr[64][4] = {};
  int device = 0;
  cudaError_t e = cudaGetDevice(&device);
  if (e != cudaSuccess) return e;
  const size_t bytes = dev::da_smem_bytes(16 * tiles);
  if (device < 0 || device >= 64 || !attr[device][tiles - 1].load(std::memory_order_acquire)) {
    for (int method : {(int)M_SAD, (int)M_SAMC, (int)M_WL})
      if (e == cudaSuccess)
        e = cudaFuncSetAttribute(da_kernel(tiles, method), cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
    if (e != cudaSuccess) return e;
    if (device >= 0 && device < 64) attr[device][tiles - 1].store(true, std::memory_order_release);
  }
  const int blocks = (m.n_walkers + dev::DA_WPB - 1) / dev::DA_WPB;
  da_kernel(tiles, m.method)<<<blocks, 32 * dev::DA_WPB, bytes, st>>>(m, s, w, refresh_interval, stats);
  return cudaGetLastError();
}

}  // namespace sadmc
