// mbir_kernels.cu -- sm_103a kernels of the MBIR hot path.
//
// The ICD sweep / projection kernels live in mbir_sweep.cuh (instantiated by
// mbir_sweep_f32.cu, mbir_sweep_f32_hbm.cu and mbir_sweep_f64.cu).  This file holds the rest:
//   view_sums_kernel  FP64 per-view reductions for gain/offset and variance estimation.
//   prior_cost_kernel FP64 accumulation of the QGGMRF prior term of the MAP cost.
// Every kernel is instantiated for Real = float (production) and Real = double (the
// reference's own precision, for order-exact parity and precision studies).
//
// Reference semantics follow Code/MBIRLib/HAADF/HAADF_ReconstructionEngine_UpdateVoxels.cpp
// (UpdateYSlice::execute :149-484), Code/MBIRLib/Common/AMatrixCol.cpp:82-239 (A-column),
// Code/MBIRLib/Reconstruction/QGGMRF_Functions.cpp:82-206 (prior), and
// HAADF_ReconstructionEngine_Extra.cpp:419-881 / HAADF_ReconstructionEngine.cpp:1147-1364.
#include <cuda_runtime.h>

#include <algorithm>
#include <type_traits>

#include "mbir_internal.h"
#include "mbir_wide.cuh"

namespace mbir {

namespace {

constexpr unsigned kFull = 0xffffffffu;
// ---- warp reductions ------------------------------------------------------------------
template <typename T>
__device__ __forceinline__ T warp_sum(T v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(kFull, v, o);
  return v;
}

// ---- layout conversions ----------------------------------------------------------------
template <typename Real>
__global__ void sino_to_dev_kernel(const float* __restrict__ h, Real* __restrict__ d, int n_theta,
                                   int n_r, int n_rp, int n_t) {
  const size_t total = static_cast<size_t>(n_t) * n_theta * n_rp;
  for (size_t i = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x; i < total;
       i += static_cast<size_t>(gridDim.x) * blockDim.x) {
    const int r = static_cast<int>(i % n_rp);
    const size_t rest = i / n_rp;
    const int v = static_cast<int>(rest % n_theta);
    const int t = static_cast<int>(rest / n_theta);
    d[i] = (r < n_r) ? static_cast<Real>(h[(static_cast<size_t>(v) * n_r + r) * n_t + t]) : Real(0);
  }
}
template <typename Real>
__global__ void sino_to_host_kernel(const Real* __restrict__ d, float* __restrict__ h, int n_theta,
                                    int n_r, int n_rp, int n_t) {
  const size_t total = static_cast<size_t>(n_theta) * n_r * n_t;
  for (size_t i = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x; i < total;
       i += static_cast<size_t>(gridDim.x) * blockDim.x) {
    const int t = static_cast<int>(i % n_t);
    const size_t rest = i / n_t;
    const int r = static_cast<int>(rest % n_r);
    const int v = static_cast<int>(rest / n_r);
    h[i] = static_cast<float>(d[(static_cast<size_t>(t) * n_theta + v) * n_rp + r]);
  }
}
template <typename Real>
__global__ void fill_volume_kernel(Real* __restrict__ x, Real value,
                                   const uint8_t* __restrict__ lineok, int n_lines, int n_y) {
  for (int l = blockIdx.x * blockDim.x + threadIdx.x; l < n_lines; l += gridDim.x * blockDim.x) {
    const Real v = lineok[l] ? value : Real(0);
    for (int y = blockIdx.y; y < n_y; y += gridDim.y)
      x[static_cast<size_t>(y) * n_lines + l] = v;
  }
}
template <typename Real>
__global__ void vol_to_dev_kernel(const float* __restrict__ zxy, Real* __restrict__ yzx, int n_z,
                                  int n_x, int n_y) {
  const size_t total = static_cast<size_t>(n_z) * n_x * n_y;
  for (size_t i = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x; i < total;
       i += static_cast<size_t>(gridDim.x) * blockDim.x) {
    const int x = static_cast<int>(i % n_x);
    const size_t rest = i / n_x;
    const int z = static_cast<int>(rest % n_z);
    const int y = static_cast<int>(rest / n_z);
    yzx[i] = static_cast<Real>(zxy[(static_cast<size_t>(z) * n_x + x) * n_y + y]);
  }
}
template <typename Real>
__global__ void vol64_to_dev_kernel(const double* __restrict__ zxy, Real* __restrict__ yzx,
                                    int n_z, int n_x, int n_y) {
  const size_t total = static_cast<size_t>(n_z) * n_x * n_y;
  for (size_t i = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x; i < total;
       i += static_cast<size_t>(gridDim.x) * blockDim.x) {
    const int x = static_cast<int>(i % n_x);
    const size_t rest = i / n_x;
    const int z = static_cast<int>(rest % n_z);
    const int y = static_cast<int>(rest / n_z);
    yzx[i] = static_cast<Real>(zxy[(static_cast<size_t>(z) * n_x + x) * n_y + y]);
  }
}
template <typename Real>
__global__ void vol_to_host_kernel(const Real* __restrict__ yzx, float* __restrict__ zxy, int n_z,
                                   int n_x, int n_y) {
  const size_t total = static_cast<size_t>(n_z) * n_x * n_y;
  for (size_t i = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x; i < total;
       i += static_cast<size_t>(gridDim.x) * blockDim.x) {
    const int y = static_cast<int>(i % n_y);
    const size_t rest = i / n_y;
    const int x = static_cast<int>(rest % n_x);
    const int z = static_cast<int>(rest / n_x);
    zxy[i] = static_cast<float>(yzx[(static_cast<size_t>(y) * n_z + z) * n_x + x]);
  }
}

// e = y - yest - mu_theta (calculateMeasurementWeight, HAADF_ReconstructionEngine_Extra.cpp:693-771)
template <typename Real>
__global__ void error_from_projection_kernel(const Real* __restrict__ y,
                                             const Real* __restrict__ yest, Real* __restrict__ e,
                                             const double* __restrict__ mu, int n_theta, int n_rp,
                                             int n_r, int n_t) {
  const size_t total = static_cast<size_t>(n_t) * n_theta * n_rp;
  for (size_t i = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x; i < total;
       i += static_cast<size_t>(gridDim.x) * blockDim.x) {
    const int r = static_cast<int>(i % n_rp);
    const int v = static_cast<int>((i / n_rp) % n_theta);
    e[i] = (r < n_r) ? static_cast<Real>(static_cast<double>(y[i]) -
                                         static_cast<double>(yest[i]) - mu[v])
                     : Real(0);
  }
}

// Per-view FP64 sums.  kind 0 (jointEstimation, HAADF_ReconstructionEngine_Extra.cpp:474-517):
//   [0] sum y w, [1] sum w, [2] sum yh w, [3] sum yh w y, [4] sum y^2 w, [5] sum yh^2 w,
//   yh = (y - e - mu)/I.  kind 1 (updateWeights :825-833): [0] sum e^2.
//
// The gain/offset solve subtracts these sums from one another and a sweep's zero skipping turns a
// last-bit difference of its inputs into another path, so every rounding of the sums is kept.
// The FP64 pipe bounds the kernel (2 lanes per clock and SM): kind 0 took ~23 FP64 operations per
// entry, ~10 of them the division by the view's gain.  wide::div_by gives the same quotient in
// five; the FP32 engine leaves out sum y^2 w (Y2 false), which its solve does not use.
template <typename Real, int K, bool Y2>
__global__ void view_sums_kernel(const Real* __restrict__ y, const Real* __restrict__ e,
                                 const double* __restrict__ mu, const double* __restrict__ gain,
                                 const double* __restrict__ wv, double* __restrict__ partial,
                                 int n_theta, int n_rp, int n_r, int t_begin, int t_end,
                                 int n_chunk) {
  const int v = blockIdx.x, ch = blockIdx.y;
  const int n_t = t_end - t_begin;
  const int t0 = t_begin + static_cast<int>(static_cast<long long>(ch) * n_t / n_chunk);
  const int t1 = t_begin + static_cast<int>(static_cast<long long>(ch + 1) * n_t / n_chunk);
  double acc[K];
#pragma unroll
  for (int k = 0; k < K; ++k) acc[k] = 0.0;
  const double m = mu[v], gi = gain[v], w = wv[v];
  const double inv = K > 1 ? 1.0 / gi : 0.0;
  const bool mid = wide::divides(gi);
  for (int t = t0; t < t1; ++t) {
    const size_t base = (static_cast<size_t>(t) * n_theta + v) * n_rp;
    for (int r = threadIdx.x; r < n_r; r += blockDim.x) {
      const double ev = e[base + r];
      if (K == 1) {
        acc[0] += ev * ev;
      } else {
        const double yv = y[base + r];
        const double yh = wide::div_by(yv - ev - m, gi, inv, mid);
        acc[0] += yv * w;
        acc[1] += w;
        acc[2] += yh * w;
        acc[K > 3 ? 3 : 0] += yh * w * yv;
        if constexpr (Y2) acc[K > 4 ? 4 : 0] += yv * yv * w;
        acc[K > 5 ? 5 : 0] += yh * yh * w;
      }
    }
  }
  __shared__ double red[32][K];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int k = 0; k < K; ++k) {
    const double s = warp_sum(acc[k]);
    if (lane == 0) red[warp][k] = s;
  }
  __syncthreads();
  if (threadIdx.x < K) {
    double s = 0.0;
    for (int w2 = 0; w2 < static_cast<int>(blockDim.x >> 5); ++w2) s += red[w2][threadIdx.x];
    partial[(static_cast<size_t>(v) * n_chunk + ch) * K + threadIdx.x] = s;
  }
}

__global__ void view_sums_final_kernel(const double* __restrict__ partial, double* __restrict__ out,
                                       int n_theta, int n_chunk, int K) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n_theta * K) return;
  const int v = i / K, k = i % K;
  double s = 0.0;
  for (int c = 0; c < n_chunk; ++c) s += partial[(static_cast<size_t>(v) * n_chunk + c) * K + k];
  out[i] = s;
}

// e = y - mu_new - I_new * yh, yh = (y - e - mu_old)/I_old
// (jointEstimation, HAADF_ReconstructionEngine_Extra.cpp:464-472 and :600-612)
template <typename Real>
__global__ void rebuild_error_kernel(const Real* __restrict__ y, Real* __restrict__ e,
                                     const double* __restrict__ mu_old,
                                     const double* __restrict__ gain_old,
                                     const double* __restrict__ mu_new,
                                     const double* __restrict__ gain_new, int n_theta, int n_rp,
                                     int n_r, int n_t) {
  const size_t total = static_cast<size_t>(n_t) * n_theta * n_rp;
  for (size_t i = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x; i < total;
       i += static_cast<size_t>(gridDim.x) * blockDim.x) {
    const int r = static_cast<int>(i % n_rp);
    if (r >= n_r) continue;
    const int v = static_cast<int>((i / n_rp) % n_theta);
    const double yv = y[i];
    const double yh = (yv - static_cast<double>(e[i]) - mu_old[v]) / gain_old[v];
    // the product is rounded on its own (no fused multiply-subtract), as in the reference
    e[i] = static_cast<Real>(yv - mu_new[v] - __dmul_rn(gain_new[v], yh));
  }
}

// rebuild_error_kernel of the FP32 engine: the same bits (mbir_wide.cuh)
__global__ void __launch_bounds__(256)
    rebuild_error_f32_kernel(const float* __restrict__ y, float* __restrict__ e,
                             const double* __restrict__ mu_old, const double* __restrict__ gain_old,
                             const double* __restrict__ mu_new, const double* __restrict__ gain_new,
                             int n_theta, int n_rp, int n_r, int n_t, int n_chunk) {
  const int v = blockIdx.x, ch = blockIdx.y;
  const int t0 = static_cast<int>(static_cast<long long>(ch) * n_t / n_chunk);
  const int t1 = static_cast<int>(static_cast<long long>(ch + 1) * n_t / n_chunk);
  const double mo = mu_old[v], go = gain_old[v], mn = mu_new[v], gn = gain_new[v];
  const wide::F2 mof = wide::neg(wide::split(mo)), mnf = wide::neg(wide::split(mn));
  const wide::F2 ratio = wide::neg(wide::split(gn / go));
  const float ra = fabsf(ratio.hi), fixed = fabsf(mnf.hi) + fabsf(mof.hi) * ra;
  wide::for_view_rows(
      v, t0, t1, n_theta, n_rp,
      [&](size_t row, int r) {
        const size_t base = row * n_rp;
        const float4 y4 = *reinterpret_cast<const float4*>(y + base + r);
        const float4 e4 = *reinterpret_cast<const float4*>(e + base + r);
        const float yv[4] = {y4.x, y4.y, y4.z, y4.w}, ev[4] = {e4.x, e4.y, e4.z, e4.w};
        float o[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const wide::F2 d = wide::add(wide::two_diff(yv[j], ev[j]), mof);
          const wide::F2 a = wide::add(wide::two_sum(yv[j], mnf.hi), wide::F2{mnf.lo, 0.f});
          const float size = fabsf(yv[j]) * (1.f + ra) + fabsf(ev[j]) * ra + fixed;
          if (!wide::rounds_to(wide::add(a, wide::mul(d, ratio)), 1.2e-13f * size, o[j])) {
            const double yd = yv[j];
            const double yh = (yd - static_cast<double>(ev[j]) - mo) / go;
            o[j] = static_cast<float>(yd - mn - __dmul_rn(gn, yh));
          }
          if (r + j >= n_r) o[j] = ev[j];
        }
        *reinterpret_cast<float4*>(e + base + r) = make_float4(o[0], o[1], o[2], o[3]);
      },
      [](auto) {});
}

// QGGMRF prior term of computeCost (HAADF_ReconstructionEngine.cpp:1285-1359): 13 forward
// neighbours per voxel, FP64 accumulation.  Offsets are (dz, dx, dy) with weight index
// [dy+1][dz+1][dx+1].
__constant__ int c_fwd[13][3] = {{0, 0, 1},  {0, 1, -1}, {0, 1, 0},   {0, 1, 1},   {1, -1, 0},
                                 {1, 0, 0},  {1, 1, 0},  {1, -1, -1}, {1, -1, 1},  {1, 0, -1},
                                 {1, 1, -1}, {1, 1, 1},  {1, 0, 1}};

__global__ void prior_cost_kernel(const double* __restrict__ x, DevFilter q, int n_z, int n_x,
                                  int n_y, double* __restrict__ partial) {
  // one (y, z) row of n_x voxels at a time: 32-bit index arithmetic, coalesced row reads
  const int rows = n_y * n_z;
  double acc = 0.0;
  for (int r = blockIdx.x; r < rows; r += gridDim.x) {
    const int yi = r / n_z, zi = r - yi * n_z;
    const double* row = x + static_cast<size_t>(r) * n_x;
    for (int xi = threadIdx.x; xi < n_x; xi += blockDim.x) {
      const double c = row[xi];
      for (int k = 0; k < 13; ++k) {
        const int zz = zi + c_fwd[k][0], xx = xi + c_fwd[k][1], yy = yi + c_fwd[k][2];
        if (zz < 0 || zz >= n_z || xx < 0 || xx >= n_x || yy < 0 || yy >= n_y) continue;
        const double nv = x[(static_cast<size_t>(yy) * n_z + zz) * n_x + xx];
        const int fi = 9 * (c_fwd[k][2] + 1) + 3 * (c_fwd[k][0] + 1) + (c_fwd[k][1] + 1);
        const double ad = fabs(c - nv);
        const double num = pow(ad, q.mrf_p);
        const double pq = pow(ad, q.mrf_p - q.mrf_q);
        acc += q.f[fi] * ((num / q.sig_p) / (q.mrf_c + pq / q.sig_pq));
      }
    }
  }
  acc = warp_sum(acc);
  __shared__ double red[32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (lane == 0) red[warp] = acc;
  __syncthreads();
  if (threadIdx.x == 0) {
    double s = 0.0;
    for (int w = 0; w < static_cast<int>(blockDim.x >> 5); ++w) s += red[w];
    partial[blockIdx.x] = s;
  }
}

// The FP32 engine's: each voxel's 13 pair terms in FP32 (relative error ~1e-6 of the term),
// summed per voxel and accumulated in FP64.  The pair weights are FP32 arguments (converted per
// pair they took a third of the kernel on the FP64 pipe).  A pair of equal voxels adds nothing (its
// numerator is 0) and is passed over: how much that saves depends on the volume.  The MAP cost of
// 512 x 256 x 128 voxels at 61 views takes 0.41 ms for a piecewise constant phantom, where nearly
// every pair is equal, and 0.97 ms for a reconstruction after eight sweeps; with FP64 conversions
// and every pair 1.3 and 1.4 ms.
struct PriorCostF {
  float f[13];           // pair weights in c_fwd order
  float P, PQ, isp, ispq, c;
  int p2, skip_equal;
};
__global__ void __launch_bounds__(256)
    prior_cost_f32_kernel(const float* __restrict__ x, const PriorCostF q, int n_z, int n_x,
                          int n_y, double* __restrict__ partial) {
  const int rows = n_y * n_z;
  double acc = 0.0;
  for (int r = blockIdx.x; r < rows; r += gridDim.x) {
    const int yi = r / n_z, zi = r - yi * n_z;
    const float* row = x + static_cast<size_t>(r) * n_x;
    for (int xi = threadIdx.x; xi < n_x; xi += blockDim.x) {
      const float c = row[xi];
      float vsum = 0.f;
      constexpr int fwd[13][3] = {{0, 0, 1},  {0, 1, -1}, {0, 1, 0},   {0, 1, 1},   {1, -1, 0},
                                  {1, 0, 0},  {1, 1, 0},  {1, -1, -1}, {1, -1, 1},  {1, 0, -1},
                                  {1, 1, -1}, {1, 1, 1},  {1, 0, 1}};  // c_fwd
#pragma unroll
      for (int k = 0; k < 13; ++k) {
        const int xx = xi + fwd[k][1], yy = yi + fwd[k][2];
        if (zi + fwd[k][0] >= n_z || yy < 0 || yy >= n_y) continue;  // (the same for the row)
        if (xx < 0 || xx >= n_x) continue;
        const float ad =
            fabsf(c - row[(static_cast<long long>(fwd[k][2]) * n_z + fwd[k][0]) * n_x + xx]);
        if (q.skip_equal && ad == 0.f) continue;
        const float num = q.p2 ? ad * ad : powf(ad, q.P);
        const float pq = powf(ad, q.PQ);
        vsum += q.f[k] * ((num * q.isp) / (q.c + pq * q.ispq));
      }
      acc += static_cast<double>(vsum);
    }
  }
  const double a1[1] = {acc};
  const double s = wide::block_sums<1>(a1);
  if (threadIdx.x == 0) partial[blockIdx.x] = s;
}

// One warp per column, the sum that additions in row order give.  The values are non-negative
// multiples of 2^-32 (or counts), so a sum below 2^21 is exact in any order; larger ones (of |x| over
// millions of voxels) round and are added again one after another (for 256 rows 5 us more, which
// every call of a bright-field reconstruction would pay).
__global__ void reduce_rows_kernel(const double* __restrict__ in, int n_rows, int n_cols,
                                   double* __restrict__ out, const int* __restrict__ err,
                                   const int* __restrict__ count) {
  if (threadIdx.x == 0 && err != nullptr) {
    int* tail = reinterpret_cast<int*>(out + n_cols);
    tail[0] = *err;
    tail[1] = count != nullptr ? count[0] : 0;
    tail[2] = count != nullptr ? count[1] : 0;
  }
  const int c = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (c >= n_cols) return;
  double s = 0.0;
  for (int r = lane; r < n_rows; r += 32) s += in[static_cast<size_t>(r) * n_cols + c];
  s = warp_sum(s);
  if (s < 2097152.0) {
    if (lane == 0) out[c] = s;
    return;
  }
  s = 0.0;
  for (int r0 = 0; r0 < n_rows; r0 += 32) {
    const double v = r0 + lane < n_rows ? in[static_cast<size_t>(r0 + lane) * n_cols + c] : 0.0;
    const int n = min(32, n_rows - r0);
    if (n == 32) {
#pragma unroll
      for (int k = 0; k < 32; ++k) s += __shfl_sync(kFull, v, k);
    } else {
      for (int k = 0; k < n; ++k) s += __shfl_sync(kFull, v, k);
    }
  }
  if (lane == 0) out[c] = s;
}

inline int ok_or(cudaError_t e) { return e == cudaSuccess ? 0 : -3; }
inline int grid_for(size_t n, int block) {
  size_t g = (n + block - 1) / block;
  if (g > 152 * 32) g = 152 * 32;
  if (g < 1) g = 1;
  return static_cast<int>(g);
}

}  // namespace

int launch_sweep_f32_smem(const SweepArgs& a, int nb, size_t smem, void* stream) {
  return a.bf ? launch_sweep_f32_smem_bf(a, nb, smem, stream)
              : launch_sweep_f32_smem_haadf(a, nb, smem, stream);
}

int launch_batch_sweep(const BatchArgs& b, int nb, int group, int threads, size_t smem, int grid,
                       void* stream) {
  if (batch_group_table(group))
    return batch_group_bf(group) ? launch_batch_table_bf(b, group, threads, smem, grid, stream)
                                 : launch_batch_table_haadf(b, group, threads, smem, grid, stream);
  if (nb == 3) return launch_batch_sweep_nb3(b, group, threads, smem, grid, stream);
  if (nb == 5) return launch_batch_sweep_nb5(b, group, threads, smem, grid, stream);
  return -7;
}

int launch_sweep(const SweepArgs& a, int nb, size_t smem, void* stream) {
  if (a.fp64) return launch_sweep_f64(a, nb, smem, stream);
  if (table_driven(a, nb))
    return a.bf ? launch_table_bf(a, smem, stream) : launch_table_haadf(a, smem, stream);
  return a.smem_rows ? launch_sweep_f32_smem(a, nb, smem, stream)
                     : launch_sweep_f32_hbm(a, nb, smem, stream);
}

int launch_ref_order(const RefOrderArgs& a, int nb, void* stream) {
  return a.fp64 ? launch_ref_order_f64(a, nb, stream) : launch_ref_order_f32(a, nb, stream);
}

template <typename Real>
static inline Real* RP(void* p) {
  return static_cast<Real*>(p);
}
template <typename Real>
static inline const Real* RP(const void* p) {
  return static_cast<const Real*>(p);
}

int launch_sino_to_dev(const float* h, void* d, int n_theta, int n_r, int n_rp, int n_t, int fp64,
                       void* stream) {
  const size_t n = static_cast<size_t>(n_t) * n_theta * n_rp;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  if (fp64)
    sino_to_dev_kernel<double><<<grid_for(n, 256), 256, 0, s>>>(h, RP<double>(d), n_theta, n_r,
                                                                 n_rp, n_t);
  else
    sino_to_dev_kernel<float><<<grid_for(n, 256), 256, 0, s>>>(h, RP<float>(d), n_theta, n_r,
                                                                n_rp, n_t);
  return ok_or(cudaGetLastError());
}
int launch_sino_to_host(const void* d, float* h, int n_theta, int n_r, int n_rp, int n_t,
                        int fp64, void* stream) {
  const size_t n = static_cast<size_t>(n_theta) * n_r * n_t;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  if (fp64)
    sino_to_host_kernel<double><<<grid_for(n, 256), 256, 0, s>>>(RP<double>(d), h, n_theta, n_r,
                                                                  n_rp, n_t);
  else
    sino_to_host_kernel<float><<<grid_for(n, 256), 256, 0, s>>>(RP<float>(d), h, n_theta, n_r,
                                                                 n_rp, n_t);
  return ok_or(cudaGetLastError());
}
int launch_fill_volume(void* yzx, double value, const uint8_t* lineok, int n_lines, int n_y,
                       int fp64, void* stream) {
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  const dim3 grid(std::max(1, std::min((n_lines + 255) / 256, 1024)), std::max(1, std::min(n_y, 32)));
  if (fp64)
    fill_volume_kernel<double><<<grid, 256, 0, s>>>(RP<double>(yzx), value, lineok, n_lines, n_y);
  else
    fill_volume_kernel<float><<<grid, 256, 0, s>>>(RP<float>(yzx), static_cast<float>(value), lineok,
                                                   n_lines, n_y);
  return ok_or(cudaGetLastError());
}
int launch_vol_to_dev(const float* zxy, void* yzx, int n_z, int n_x, int n_y, int fp64,
                      void* stream) {
  const size_t n = static_cast<size_t>(n_z) * n_x * n_y;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  if (fp64)
    vol_to_dev_kernel<double><<<grid_for(n, 256), 256, 0, s>>>(zxy, RP<double>(yzx), n_z, n_x, n_y);
  else
    vol_to_dev_kernel<float><<<grid_for(n, 256), 256, 0, s>>>(zxy, RP<float>(yzx), n_z, n_x, n_y);
  return ok_or(cudaGetLastError());
}
int launch_vol64_to_dev(const double* zxy, void* yzx, int n_z, int n_x, int n_y, int fp64,
                        void* stream) {
  const size_t n = static_cast<size_t>(n_z) * n_x * n_y;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  if (fp64)
    vol64_to_dev_kernel<double><<<grid_for(n, 256), 256, 0, s>>>(zxy, RP<double>(yzx), n_z, n_x,
                                                                  n_y);
  else
    vol64_to_dev_kernel<float><<<grid_for(n, 256), 256, 0, s>>>(zxy, RP<float>(yzx), n_z, n_x, n_y);
  return ok_or(cudaGetLastError());
}
int launch_vol_to_host(const void* yzx, float* zxy, int n_z, int n_x, int n_y, int fp64,
                       void* stream) {
  const size_t n = static_cast<size_t>(n_z) * n_x * n_y;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  if (fp64)
    vol_to_host_kernel<double><<<grid_for(n, 256), 256, 0, s>>>(RP<double>(yzx), zxy, n_z, n_x, n_y);
  else
    vol_to_host_kernel<float><<<grid_for(n, 256), 256, 0, s>>>(RP<float>(yzx), zxy, n_z, n_x, n_y);
  return ok_or(cudaGetLastError());
}
int launch_error_from_projection(const void* y, const void* yest, void* e, const double* mu,
                                 int n_theta, int n_rp, int n_r, int n_t, int fp64, void* stream) {
  const size_t n = static_cast<size_t>(n_t) * n_theta * n_rp;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  if (fp64)
    error_from_projection_kernel<double><<<grid_for(n, 256), 256, 0, s>>>(
        RP<double>(y), RP<double>(yest), RP<double>(e), mu, n_theta, n_rp, n_r, n_t);
  else
    error_from_projection_kernel<float><<<grid_for(n, 256), 256, 0, s>>>(
        RP<float>(y), RP<float>(yest), RP<float>(e), mu, n_theta, n_rp, n_r, n_t);
  return ok_or(cudaGetLastError());
}
int launch_view_sums(int kind, const void* y, const void* e, const double* mu,
                     const double* gain, const double* wv, double* partial, double* out,
                     int n_theta, int n_rp, int n_r, int n_t, int n_chunk, int fp64,
                     void* stream) {
  return launch_view_sums_rows(kind, y, e, mu, gain, wv, partial, out, n_theta, n_rp, n_r, 0, n_t,
                               n_chunk, fp64, false, stream);
}

int launch_view_sums_rows(int kind, const void* y, const void* e, const double* mu,
                          const double* gain, const double* wv, double* partial, double* out,
                          int n_theta, int n_rp, int n_r, int t_begin, int t_end, int n_chunk,
                          int fp64, bool all_sums, void* stream) {
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  dim3 grid(n_theta, n_chunk);
  const int K = kind == 0 ? 6 : 1;
  auto go = [&](auto kern, auto zero) {
    using Real = decltype(zero);
    kern<<<grid, 256, 0, s>>>(RP<Real>(y), RP<Real>(e), mu, gain, wv, partial, n_theta, n_rp, n_r,
                              t_begin, t_end, n_chunk);
  };
  if (fp64) {
    if (kind == 0)
      go(view_sums_kernel<double, 6, true>, 0.0);
    else
      go(view_sums_kernel<double, 1, false>, 0.0);
  } else if (kind == 0) {
    if (all_sums)
      go(view_sums_kernel<float, 6, true>, 0.f);
    else
      go(view_sums_kernel<float, 6, false>, 0.f);
  } else {
    go(view_sums_kernel<float, 1, false>, 0.f);
  }
  const int n = n_theta * K;
  view_sums_final_kernel<<<(n + 127) / 128, 128, 0, s>>>(partial, out, n_theta, n_chunk, K);
  return ok_or(cudaGetLastError());
}
int launch_rebuild_error(const void* y, void* e, const double* mu_old, const double* gain_old,
                         const double* mu_new, const double* gain_new, int n_theta, int n_rp,
                         int n_r, int n_t, int fp64, void* stream) {
  const size_t n = static_cast<size_t>(n_t) * n_theta * n_rp;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  if (fp64)
    rebuild_error_kernel<double><<<grid_for(n, 256), 256, 0, s>>>(
        RP<double>(y), RP<double>(e), mu_old, gain_old, mu_new, gain_new, n_theta, n_rp, n_r, n_t);
  else
    rebuild_error_f32_kernel<<<dim3(n_theta, std::min(32, n_t)), 256, 0, s>>>(
        RP<float>(y), RP<float>(e), mu_old, gain_old, mu_new, gain_new, n_theta, n_rp, n_r, n_t,
        std::min(32, n_t));
  return ok_or(cudaGetLastError());
}
int launch_prior_cost(const void* x, const DevFilter& f, int n_z, int n_x, int n_y,
                      double* partial, int n_blocks, int fp64, void* stream) {
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  if (fp64)
    prior_cost_kernel<<<n_blocks, 256, 0, s>>>(RP<double>(x), f, n_z, n_x, n_y, partial);
  else {
    PriorCostF q{};
    constexpr int fwd[13][3] = {{0, 0, 1},  {0, 1, -1}, {0, 1, 0},   {0, 1, 1},   {1, -1, 0},
                                {1, 0, 0},  {1, 1, 0},  {1, -1, -1}, {1, -1, 1},  {1, 0, -1},
                                {1, 1, -1}, {1, 1, 1},  {1, 0, 1}};  // c_fwd
    for (int k = 0; k < 13; k++)
      q.f[k] = static_cast<float>(f.f[9 * (fwd[k][2] + 1) + 3 * (fwd[k][0] + 1) + fwd[k][1] + 1]);
    q.P = static_cast<float>(f.mrf_p);
    q.PQ = static_cast<float>(f.mrf_p - f.mrf_q);
    q.isp = static_cast<float>(1.0 / f.sig_p);
    q.ispq = static_cast<float>(1.0 / f.sig_pq);
    q.c = static_cast<float>(f.mrf_c);
    q.p2 = f.mrf_p == 2.0 ? 1 : 0;
    // a pair of equal voxels: 0 / c, or 0 / inf, unless the constants make it 0 / 0 or inf 0
    q.skip_equal = f.mrf_p > 0 && q.c > 0.f && q.isp <= 3e38f && q.ispq >= 0.f ? 1 : 0;
    prior_cost_f32_kernel<<<n_blocks, 256, 0, s>>>(RP<float>(x), q, n_z, n_x, n_y, partial);
  }
  return ok_or(cudaGetLastError());
}
int launch_reduce_stats(const double* in, int n_rows, int n_cols, double* out, void* stream,
                        const int* err, const int* count) {
  reduce_rows_kernel<<<1, 32 * n_cols, 0, static_cast<cudaStream_t>(stream)>>>(in, n_rows, n_cols,
                                                                              out, err, count);
  return ok_or(cudaGetLastError());
}

}  // namespace mbir
