// mbir_sweep_f32_batch_tab.cu -- persistent batched sweep kernels, table-driven step.
#include "mbir_sweep.cuh"

namespace mbir {

int launch_batch_sweep_tab(const BatchArgs& b, int group, int threads, size_t smem, int grid,
                           void* stream) {
  return sweep::launch_batch_pick<3, true>(b, group, threads, smem, grid,
                                           static_cast<cudaStream_t>(stream));
}

}  // namespace mbir
