// mbir_table_haadf.cu -- table-driven HAADF sweeps and forward projections.
#include "mbir_table.cuh"

namespace mbir {

int launch_table_haadf(const SweepArgs& a, size_t smem, void* stream) {
  return sweep::launch_table_pick<false>(a, smem, static_cast<cudaStream_t>(stream));
}

size_t table_smem_bytes(int n_theta, int n_x, int n_rs, bool stage, int n_sp, bool project,
                        int nbuf) {
  return sweep::table_layout(n_theta, n_x, n_rs, stage, n_sp, project, nbuf).total;
}

size_t table_walk_bytes(int n_theta, int n_x, int n_rs, bool stage, int n_sp, bool project,
                        size_t limit) {
  for (int nbuf = 2; nbuf > 0; --nbuf) {
    const size_t b = table_smem_bytes(n_theta, n_x, n_rs, stage, n_sp, project, nbuf);
    if (b <= limit) return b;
  }
  return 0;
}

}  // namespace mbir
