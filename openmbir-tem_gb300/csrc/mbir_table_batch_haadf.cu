// mbir_table_batch_haadf.cu -- persistent batched sweeps of table-driven HAADF series.
#include "mbir_table.cuh"

namespace mbir {

int launch_batch_table_haadf(const BatchArgs& b, int group, int threads, size_t smem, int grid,
                             void* stream) {
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  const int shape = batch_group_shape(group);
  return batch_group_staged(group)
             ? sweep::launch_batch_table<true, false>(b, shape, threads, smem, grid, s)
             : sweep::launch_batch_table<false, false>(b, shape, threads, smem, grid, s);
}

}  // namespace mbir
