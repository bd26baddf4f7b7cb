// The multi-step kernels (wave_kernel.cuh) and their launch, in a translation
// unit of their own so that the library's sources compile side by side.
#include <map>
#include <mutex>

#include "wave_kernel.cuh"

namespace ertm {

namespace {

template <int ENG, int C>
cudaError_t launch(const WaveSet& S, int grid, int smem, int smem_max, cudaStream_t st) {
  static std::mutex mu;
  static std::map<int, bool> set;
  {
    int dev = 0;
    if (cudaError_t e = cudaGetDevice(&dev)) return e;
    std::lock_guard<std::mutex> lock(mu);
    if (!set[dev]) {
      if (cudaError_t e = cudaFuncSetAttribute(k_wave<ENG, C>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem_max))
        return e;
      set[dev] = true;
    }
  }
  void* args[1] = {const_cast<WaveSet*>(&S)};
  return cudaLaunchCooperativeKernel(reinterpret_cast<const void*>(k_wave<ENG, C>), dim3(grid), dim3(WAVE_NT),
                                     args, (size_t)smem, st);
}

template <int ENG>
cudaError_t launch_e(int cells, const WaveSet& S, int grid, int smem, int smem_max, cudaStream_t st) {
  return cells == 1 ? launch<ENG, 1>(S, grid, smem, smem_max, st) : launch<ENG, 2>(S, grid, smem, smem_max, st);
}

}  // namespace

cudaError_t wave_launch(int engine, int cells, const WaveSet& S, int grid, int smem, int smem_max, cudaStream_t st) {
  if (engine == ENGINE_ACOUSTIC) return launch_e<ENGINE_ACOUSTIC>(cells, S, grid, smem, smem_max, st);
  if (engine == ENGINE_ELASTIC) return launch_e<ENGINE_ELASTIC>(cells, S, grid, smem, smem_max, st);
  return launch_e<ENGINE_VISCO>(cells, S, grid, smem, smem_max, st);
}

}  // namespace ertm
