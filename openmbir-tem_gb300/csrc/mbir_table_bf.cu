// mbir_table_bf.cu -- table-driven bright-field sweeps (scheduled calls and row walks).
#include "mbir_table.cuh"

namespace mbir {

int launch_table_bf(const SweepArgs& a, size_t smem, void* stream) {
  return sweep::launch_table_pick<true>(a, smem, static_cast<cudaStream_t>(stream));
}

}  // namespace mbir
