// mbir_sweep_f64.cu -- FP64 instantiations of the sweep and reference-order kernels (the
// reference's own precision; used for order-exact parity and precision studies).
#include "mbir_sweep.cuh"

namespace mbir {

int launch_sweep_f64(const SweepArgs& a, int nb, size_t smem, void* stream) {
  using namespace sweep;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  const bool st = a.smem_rows != 0;
  // The FP64 pipe (2 lanes per clock and SM) bounds an FP64 sweep: ~450 FP64 operations per voxel
  // and lane take ~7k cycles of its SM whatever the memory does, and a small volume has a few
  // slices per colour on 152 SMs.  So while twice the slices fit the device, a cluster of 2, 4 or
  // 8 CTAs shares each slice, in HBM instead of shared memory (the same bits either way).  A sweep
  // of the small HAADF configuration (16 slices, 71 views): 58 ms with one CTA per slice.
  if (nb == 3 && a.g.n_theta <= kMaxViewsShaped) {
    SweepArgs b = a;
    b.smem_rows = 0;
    b.n_rs = 0;
    const size_t bytes = smem_layout(a.g.n_theta, a.g.n_x, 0, 1, a.g.bins, false, 8, 0).total;
    for (int ctas = 8; ctas > 1; ctas >>= 1) {
      if (a.n_slices * ctas > 152) continue;
      bool launched = false;
      const int rc =
          a.bf ? launch_clusters<cluster_sweep_kernel<double, 3, 32, 5, true>>(b, bytes, ctas, s,
                                                                               launched)
               : launch_clusters<cluster_sweep_kernel<double, 3, 32, 5, false>>(b, bytes, ctas, s,
                                                                                launched);
      if (rc || launched) return rc;
    }
  }
  if (a.g.n_theta > kMaxViewsShaped) {  // 32 lanes x 8 views, slices in HBM
    if (st) return -7;
    if (nb == 3) return launch_sweep_m<double, 3, 32, 8, false>(a, smem, s);
    if (nb == 5) return launch_sweep_m<double, 5, 32, 8, false>(a, smem, s);
    if (nb == 9) return launch_sweep_m<double, 9, 32, 8, false>(a, smem, s);
    return -7;
  }
  if (nb == 3)
    return st ? launch_sweep_m<double, 3, 32, 5, true>(a, smem, s)
              : launch_sweep_m<double, 3, 32, 5, false>(a, smem, s);
  if (nb == 5)
    return st ? launch_sweep_m<double, 5, 32, 5, true>(a, smem, s)
              : launch_sweep_m<double, 5, 32, 5, false>(a, smem, s);
  if (nb == 9)
    return st ? launch_sweep_m<double, 9, 32, 5, true>(a, smem, s)
              : launch_sweep_m<double, 9, 32, 5, false>(a, smem, s);
  return -7;
}

int launch_ref_order_f64(const RefOrderArgs& a, int nb, void* stream) {
  using namespace sweep;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  if (nb == 3) return launch_ref_t<double, 3, 5>(a, s);
  if (nb == 5) return launch_ref_t<double, 5, 5>(a, s);
  if (nb == 9) return launch_ref_t<double, 9, 5>(a, s);
  return -7;
}

size_t sweep_smem_bytes(int n_theta, int n_x, int n_rs, int t_rows, int bins, int fp64,
                        int n_sp, bool sched) {
  return sweep::smem_layout(n_theta, n_x, n_rs, t_rows, bins, n_rs > 0, fp64 ? 8 : 4, n_sp, sched)
      .total;
}

}  // namespace mbir
