// mbir_bf.cu -- bright-field sinogram-wide kernels (compiled with -fmad=false).
//
//   layout_from_double   host-layout FP64 staging [theta][r][t] -> device [t][theta][r_pad]
//   offset sums / apply  BFForwardModel::jointEstimation (BFForwardModel.cpp:390-441): per view
//                        the offset (log dosage) step num/den, e -= step
//   selector             BFForwardModel::updateSelector (:517-531): sel = e^2 w < T^2
//   variance sums        BFForwardModel::updateWeights (:447-511): w *= alpha_view, then the
//                        global sums over selected (e^2 w) and rejected (|e| sqrt(alpha w))
//                        entries; scale_weights then divides by the new common variance
//   cost sums            BFForwardModel::forwardCost (:812-846), data term
//   magnitude map        per-line sum |dx| of a call (fixed point -> FP64), the 5x5 Hamming
//                        VSC filter (BFReconstructionEngine_Extra.cpp:888-947), the NHICD
//                        list mask (GenNonHomList :1016-1047) and the stop-rule ROI sums
//                        (roiVolumeSum :1200-1215, stopCriteria :1239-1248)
//
// Each reduction has a parallel form (fixed-shape tree: deterministic, not the reference's
// order) and a reference-order form (one thread, the reference's loop order) used by the
// reference-exact mode; without fused multiply-adds the latter reproduce the reference's FP64
// arithmetic.  Elementwise passes are the same in both modes.
#include <cuda_runtime.h>

#include <algorithm>

#include "mbir_internal.h"
#include "mbir_wide.cuh"

namespace mbir {

namespace {

constexpr int kRedBlocks = 152 * 4;  // grid of the global parallel reductions

inline int ok_or(cudaError_t e) { return e == cudaSuccess ? 0 : -3; }
inline int grid_for(size_t n, int block) {
  size_t g = (n + block - 1) / block;
  if (g > 152 * 32) g = 152 * 32;
  if (g < 1) g = 1;
  return static_cast<int>(g);
}
template <typename Real>
inline Real* RP(void* p) {
  return static_cast<Real*>(p);
}
template <typename Real>
inline const Real* RP(const void* p) {
  return static_cast<const Real*>(p);
}

__device__ __forceinline__ double warp_sum_d(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// Block sum of K values (blockDim.x a multiple of 32, <= 1024); result valid in thread 0.
template <int K>
__device__ __forceinline__ void block_sum(double (&acc)[K]) {
  __shared__ double red[32][K];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int k = 0; k < K; ++k) {
    const double s = warp_sum_d(acc[k]);
    if (lane == 0) red[warp][k] = s;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
#pragma unroll
    for (int k = 0; k < K; ++k) {
      double s = 0.0;
      for (int w = 0; w < static_cast<int>(blockDim.x >> 5); ++w) s += red[w][k];
      acc[k] = s;
    }
  }
}

template <typename Real>
__global__ void layout_from_double_kernel(const double* __restrict__ h, Real* __restrict__ d,
                                          int n_theta, int n_r, int n_rp, int n_t) {
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

// one offset-sum term (BFForwardModel.cpp:405-420)
__device__ __forceinline__ void offset_term(double ev, double w, bool sel, double T, double dl,
                                            double& num, double& den) {
  if (sel) {
    num += (ev * w);
    den += w;
  } else {
    num += (T * dl * ev / fabs(ev)) * sqrt(w);
    den += ((T * dl * sqrt(w)) / fabs(ev));
  }
}

// one variance-sum term (BFForwardModel.cpp:470-480); w already multiplied by alpha_view
__device__ __forceinline__ void variance_term(double ev, double w, double a, bool sel,
                                              double& s1, double& s2) {
  if (sel)
    s1 += (ev * ev * w);
  else
    s2 += fabs(ev) * sqrt(a * w);
}

// one data-term entry of forwardCost (BFForwardModel.cpp:822-830)
__device__ __forceinline__ double cost_term(double ev, double w, bool sel, double T, double dl) {
  if (sel) return (ev * ev * w);
  return (2 * T * dl * fabs(ev) * sqrt(w) + T * T * (1 - 2 * dl));
}

template <typename Real>
__global__ void offset_sums_kernel(const Real* __restrict__ e, const Real* __restrict__ w,
                                   const uint8_t* __restrict__ sel, double T, double dl,
                                   int n_theta, int n_rp, int n_sp, int n_r, int n_t, int n_chunk,
                                   double* __restrict__ partial) {
  const int v = blockIdx.x, ch = blockIdx.y;
  const int t0 = static_cast<int>(static_cast<long long>(ch) * n_t / n_chunk);
  const int t1 = static_cast<int>(static_cast<long long>(ch + 1) * n_t / n_chunk);
  double acc[2] = {0.0, 0.0};
  for (int t = t0; t < t1; ++t) {
    const size_t base = (static_cast<size_t>(t) * n_theta + v) * n_rp;
    const size_t sb = (static_cast<size_t>(t) * n_theta + v) * n_sp;
    for (int r = threadIdx.x; r < n_r; r += blockDim.x)
      offset_term(e[base + r], w[base + r], sel[sb + r] == 1, T, dl, acc[0], acc[1]);
  }
  block_sum<2>(acc);
  if (threadIdx.x == 0) {
    partial[(static_cast<size_t>(v) * n_chunk + ch) * 2 + 0] = acc[0];
    partial[(static_cast<size_t>(v) * n_chunk + ch) * 2 + 1] = acc[1];
  }
}

__global__ void chunk_final_kernel(const double* __restrict__ partial, double* __restrict__ out,
                                   int n_theta, int n_chunk, int K) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n_theta * K) return;
  const int v = i / K, k = i % K;
  double s = 0.0;
  for (int c = 0; c < n_chunk; ++c) s += partial[(static_cast<size_t>(v) * n_chunk + c) * K + k];
  out[i] = s;
}

// ---- FP32 engine: the same passes with FP64-accurate sums and roundings on the FP32 units
// (mbir_wide.cuh).  With their arithmetic in FP64 the five passes of an offset and a variance
// update took 0.5 ms of 8 M entries (73 MB, in L2 mostly: about 60 us); the two updates now make
// four: offset sums, offset step and selector, variance sums, new weights and selector.

// four selector bytes (rows of a multiple of 16)
__device__ __forceinline__ void sel4(const uint8_t* sel, size_t i, bool (&on)[4]) {
  const uchar4 s = *reinterpret_cast<const uchar4*>(sel + i);
  on[0] = s.x == 1;
  on[1] = s.y == 1;
  on[2] = s.z == 1;
  on[3] = s.w == 1;
}
__device__ __forceinline__ void load4(const float* p, float (&v)[4]) {
  const float4 q = *reinterpret_cast<const float4*>(p);
  v[0] = q.x;
  v[1] = q.y;
  v[2] = q.z;
  v[3] = q.w;
}

// Per view and chunk of rows two sums of selected entries (WideSum) and rejected ones (FP64).
// term(e, w, a) is the selected entry's contribution, kind by kind.
enum SumKind { kOffsetSums = 0, kVarianceSums = 1, kCostSums = 2 };

// (float)((double)w * a)
__device__ __forceinline__ float weight_times(float w, double a, wide::F2 af) {
  const wide::F2 p = wide::mul(af, w);
  float r;
  if (!wide::rounds_to(p, 1.2e-13f * fabsf(p.hi), r))
    r = wide::times_fp64(w, a);
  return r;
}

// The terms of the entries that the selector rejects, with FP64 roots and divisions (~40
// operations, each 16 cycles of the SM per warp however few lanes take part).  A warp collects such
// entries of detector rows [t0, t1) and evaluates 32 at a time (20 offset and 20 variance updates
// at 75 x 333 x 97 entries with T = 3, with the division of the sums moved into the passes: 6.4 ->
// 4.7 ms).
template <int KIND>
__device__ __forceinline__ void rejected_sums(const float* __restrict__ e, const float* w,
                                              const uint8_t* __restrict__ sel, double a,
                                              wide::F2 af, int store, double T, double dl, int v,
                                              int t0, int t1, int n_theta, int n_rp, int n_sp,
                                              int n_r, double (&acc)[2]) {
  __shared__ float2 queue[8][64];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  float2* q = queue[warp];
  auto term = [&](float2 ew) {
    if constexpr (KIND == kOffsetSums)
      offset_term(ew.x, ew.y, false, T, dl, acc[0], acc[1]);
    else if constexpr (KIND == kVarianceSums)
      variance_term(ew.x, ew.y, a, false, acc[0], acc[1]);
    else
      acc[0] += cost_term(ew.x, ew.y, false, T, dl);
  };
  const int n = (t1 - t0) * n_r;
  int held = 0;
  for (int i0 = 32 * warp; i0 < n; i0 += 256) {
    const int i = i0 + lane, dt = i / n_r, r = i - dt * n_r;
    const size_t row = static_cast<size_t>(t0 + dt) * n_theta + v;
    const bool off = i < n && sel[row * n_sp + r] != 1;
    const unsigned m = __ballot_sync(0xffffffffu, off);
    if (!m) continue;
    if (off) {
      float wv = w[row * n_rp + r];
      if (KIND == kVarianceSums && !store) wv = weight_times(wv, a, af);
      q[held + __popc(m & ((1u << lane) - 1u))] = make_float2(e[row * n_rp + r], wv);
    }
    held += __popc(m);
    __syncwarp();
    if (held >= 32) {
      term(q[lane]);
      held -= 32;
      const float2 next = q[32 + lane];
      __syncwarp();
      if (lane < held) q[lane] = next;
      __syncwarp();
    }
  }
  if (lane < held) term(q[lane]);
}

template <int KIND>
__global__ void __launch_bounds__(256)
    sums_f32_kernel(const float* __restrict__ e, float* __restrict__ w,
                    const uint8_t* __restrict__ sel, const double* __restrict__ alpha, int store,
                    double T, double dl, int n_theta, int n_rp, int n_sp, int n_r, int n_t,
                    int n_chunk, double* __restrict__ partial) {
  const int v = blockIdx.x, ch = blockIdx.y;
  const int t0 = static_cast<int>(static_cast<long long>(ch) * n_t / n_chunk);
  const int t1 = static_cast<int>(static_cast<long long>(ch + 1) * n_t / n_chunk);
  const double a = KIND == kVarianceSums ? alpha[v] : 1.0;
  const wide::F2 af = wide::split_factor(a);
  double acc[2] = {0.0, 0.0};
  wide::WideSum sum[2];
  bool any = false, rejected = false;
  wide::for_view_rows(
      v, t0, t1, n_theta, n_rp,
      [&](size_t row, int r) {
        const size_t base = row * n_rp;
        float ev[4], wv[4];
        bool on[4];
        load4(e + base + r, ev);
        load4(w + base + r, wv);
        sel4(sel, row * n_sp + r, on);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          if (r + j >= n_r) continue;
          if constexpr (KIND == kVarianceSums) wv[j] = weight_times(wv[j], a, af);
          if (on[j]) {
            any = true;
            if constexpr (KIND == kOffsetSums) {
              sum[0].add(wide::two_prod(ev[j], wv[j]));
              sum[1].add(wv[j]);
            } else {
              sum[0].add_square_times(ev[j], wv[j]);
            }
          } else {
            rejected = true;
          }
        }
        if constexpr (KIND == kVarianceSums) {
          if (store) *reinterpret_cast<float4*>(w + base + r) = make_float4(wv[0], wv[1], wv[2], wv[3]);
        }
      },
      [&](auto again) {
        const bool sound = sum[0].sound() && (KIND != kOffsetSums || sum[1].sound());
        if (sound) {
          acc[0] += sum[0].value();
          if constexpr (KIND == kOffsetSums) acc[1] += sum[1].value();
        } else if (any) {
          again([&](size_t row, int r) {
            const size_t base = row * n_rp;
            for (int j = 0; j < 4 && r + j < n_r; ++j) {
              if (sel[row * n_sp + r + j] != 1) continue;
              const double ed = e[base + r + j];
              double wd = w[base + r + j];
              if constexpr (KIND == kOffsetSums) {
                acc[0] += ed * wd;
                acc[1] += wd;
              } else {
                if constexpr (KIND == kVarianceSums)
                  if (!store) wd = static_cast<float>(wd * a);
                acc[0] += ed * ed * wd;
              }
            }
          });
        }
        sum[0] = wide::WideSum();
        sum[1] = wide::WideSum();
        any = false;
      });
  if (__syncthreads_or(rejected))
    rejected_sums<KIND>(e, w, sel, a, af, store, T, dl, v, t0, t1, n_theta, n_rp, n_sp, n_r, acc);
  const double s = wide::block_sums<2>(acc);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (warp < 2 && lane == 0) partial[(static_cast<size_t>(v) * n_chunk + ch) * 2 + warp] = s;
}

// e -= step of the view (its num / den of the offset sums, the host's division), then the selector
// (offset_apply_kernel and selector_kernel)
__global__ void __launch_bounds__(256)
    offset_step_f32_kernel(float* __restrict__ e, const float* __restrict__ w,
                           uint8_t* __restrict__ sel, const double* __restrict__ sums, double T,
                           int n_theta, int n_rp, int n_sp, int n_r, int n_t, int n_chunk) {
  const int v = blockIdx.x, ch = blockIdx.y;
  const int t0 = static_cast<int>(static_cast<long long>(ch) * n_t / n_chunk);
  const int t1 = static_cast<int>(static_cast<long long>(ch + 1) * n_t / n_chunk);
  __shared__ double s_step;
  if (threadIdx.x == 0) s_step = sums[2 * v] / sums[2 * v + 1];
  __syncthreads();
  const double st = s_step, t2 = T * T;
  const wide::F2 sf = wide::neg(wide::split(st));
  const float t2f = static_cast<float>(t2);
  wide::for_view_rows(
      v, t0, t1, n_theta, n_rp,
      [&](size_t row, int r) {
        const size_t base = row * n_rp;
        float ev[4], wv[4];
        load4(e + base + r, ev);
        load4(w + base + r, wv);
        const size_t si = row * n_sp + r;
        uint8_t on[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          on[j] = 0;
          if (r + j >= n_r) continue;
          const wide::F2 d = wide::add(wide::two_sum(ev[j], sf.hi), wide::F2{sf.lo, 0.f});
          float o;
          if (!wide::rounds_to(d, 1.2e-13f * (fabsf(ev[j]) + fabsf(sf.hi)), o))
            o = wide::minus_fp64(ev[j], st);
          ev[j] = o;
          on[j] = wide::below(o, wv[j], t2, t2f) ? 1 : 0;
        }
        *reinterpret_cast<float4*>(e + base + r) = make_float4(ev[0], ev[1], ev[2], ev[3]);
        if (r + 3 < n_r) {
          *reinterpret_cast<uchar4*>(sel + si) = make_uchar4(on[0], on[1], on[2], on[3]);
        } else {
          for (int j = 0; j < 4 && r + j < n_r; ++j) sel[si + j] = on[j];
        }
      },
      [](auto) {});
}

// w = (float)((float)(w alpha_view) / upd), then the selector (variance_sums_kernel's scaling,
// scale_weights_kernel and selector_kernel)
__global__ void __launch_bounds__(256)
    new_weights_f32_kernel(const float* __restrict__ e, float* __restrict__ w,
                           uint8_t* __restrict__ sel, const double* __restrict__ alpha,
                           const double* __restrict__ sums, double dT, double count, double T,
                           int n_theta, int n_rp, int n_sp, int n_r, int n_t, int n_chunk) {
  const int v = blockIdx.x, ch = blockIdx.y;
  const int t0 = static_cast<int>(static_cast<long long>(ch) * n_t / n_chunk);
  const int t1 = static_cast<int>(static_cast<long long>(ch + 1) * n_t / n_chunk);
  const double a = alpha[v], t2 = T * T;
  __shared__ double s_upd[2];  // the new variance, once per block (FP64 divisions), its inverse
  if (threadIdx.x == 0) {
    s_upd[0] = (sums[0] + dT * sums[1]) / count;
    s_upd[1] = 1.0 / s_upd[0];
  }
  __syncthreads();
  const double upd = s_upd[0];
  const wide::F2 af = wide::split_factor(a), inv = wide::split_factor(s_upd[1]);
  const float t2f = static_cast<float>(t2);
  wide::for_view_rows(
      v, t0, t1, n_theta, n_rp,
      [&](size_t row, int r) {
        const size_t base = row * n_rp;
        float ev[4], wv[4];
        load4(e + base + r, ev);
        load4(w + base + r, wv);
        const size_t si = row * n_sp + r;
        uint8_t on[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          on[j] = 0;
          if (r + j >= n_r) continue;
          const float w1 = weight_times(wv[j], a, af);
          const wide::F2 q = wide::mul(inv, w1);
          if (!wide::rounds_to(q, 1.2e-13f * fabsf(q.hi), wv[j]))
            wv[j] = wide::over_fp64(w1, upd);
          on[j] = wide::below(ev[j], wv[j], t2, t2f) ? 1 : 0;
        }
        *reinterpret_cast<float4*>(w + base + r) = make_float4(wv[0], wv[1], wv[2], wv[3]);
        if (r + 3 < n_r) {
          *reinterpret_cast<uchar4*>(sel + si) = make_uchar4(on[0], on[1], on[2], on[3]);
        } else {
          for (int j = 0; j < 4 && r + j < n_r; ++j) sel[si + j] = on[j];
        }
      },
      [](auto) {});
}

// Column sums of partial [n][K] (256 threads)
template <int K>
__global__ void __launch_bounds__(256)
    partials_final_kernel(const double* __restrict__ partial, double* __restrict__ out, int n) {
  double acc[K];
#pragma unroll
  for (int k = 0; k < K; ++k) acc[k] = 0.0;
  for (int i = threadIdx.x; i < n; i += 256)
#pragma unroll
    for (int k = 0; k < K; ++k) acc[k] += partial[static_cast<size_t>(i) * K + k];
  const double s = wide::block_sums<K>(acc);
  if ((threadIdx.x & 31) == 0 && (threadIdx.x >> 5) < K) out[threadIdx.x >> 5] = s;
}

// Row chunks per view: about 2000 blocks, their partials within the 4096 doubles of the engine's
// bright-field scratch
inline int view_chunks(const BfSino& b) {
  return std::max(1, std::min(b.n_t, 2000 / std::max(1, b.n_theta)));
}

// reference order: one thread per view, r then t
template <typename Real>
__global__ void offset_sums_ref_kernel(const Real* __restrict__ e, const Real* __restrict__ w,
                                       const uint8_t* __restrict__ sel, double T, double dl,
                                       int n_theta, int n_rp, int n_sp, int n_r, int n_t,
                                       double* __restrict__ out) {
  const int v = blockIdx.x * blockDim.x + threadIdx.x;
  if (v >= n_theta) return;
  double num = 0, den = 0;
  for (int r = 0; r < n_r; r++)
    for (int t = 0; t < n_t; t++) {
      const size_t i = (static_cast<size_t>(t) * n_theta + v) * n_rp + r;
      const size_t si = (static_cast<size_t>(t) * n_theta + v) * n_sp + r;
      offset_term(e[i], w[i], sel[si] == 1, T, dl, num, den);
    }
  out[v * 2 + 0] = num;
  out[v * 2 + 1] = den;
}

template <typename Real>
__global__ void offset_apply_kernel(Real* __restrict__ e, const double* __restrict__ step,
                                    int n_theta, int n_rp, int n_r, int n_t) {
  const size_t total = static_cast<size_t>(n_t) * n_theta * n_rp;
  for (size_t i = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x; i < total;
       i += static_cast<size_t>(gridDim.x) * blockDim.x) {
    const int r = static_cast<int>(i % n_rp);
    if (r >= n_r) continue;
    const int v = static_cast<int>((i / n_rp) % n_theta);
    e[i] = static_cast<Real>(static_cast<double>(e[i]) - step[v]);
  }
}

template <typename Real>
__global__ void selector_kernel(const Real* __restrict__ e, const Real* __restrict__ w,
                                uint8_t* __restrict__ sel, double T, int n_theta, int n_rp,
                                int n_sp, int n_r, int n_t) {
  const size_t total = static_cast<size_t>(n_t) * n_theta * n_sp;
  for (size_t i = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x; i < total;
       i += static_cast<size_t>(gridDim.x) * blockDim.x) {
    const int r = static_cast<int>(i % n_sp);
    if (r >= n_r) continue;
    const size_t row = i / n_sp;
    const size_t k = row * n_rp + r;
    const double ev = e[k];
    sel[i] = (ev * ev * static_cast<double>(w[k]) < T * T) ? 1 : 0;
  }
}

template <typename Real>
__global__ void variance_sums_kernel(const Real* __restrict__ e, Real* __restrict__ w,
                                     const uint8_t* __restrict__ sel,
                                     const double* __restrict__ alpha, int n_theta, int n_rp,
                                     int n_sp, int n_r, int n_t, double* __restrict__ partial) {
  const size_t total = static_cast<size_t>(n_t) * n_theta * n_rp;
  double acc[2] = {0.0, 0.0};
  for (size_t i = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x; i < total;
       i += static_cast<size_t>(gridDim.x) * blockDim.x) {
    const int r = static_cast<int>(i % n_rp);
    if (r >= n_r) continue;
    const size_t row = i / n_rp;
    const int v = static_cast<int>(row % n_theta);
    const double a = alpha[v];
    const Real wn = static_cast<Real>(static_cast<double>(w[i]) * a);
    w[i] = wn;
    variance_term(e[i], wn, a, sel[row * n_sp + r] == 1, acc[0], acc[1]);
  }
  block_sum<2>(acc);
  if (threadIdx.x == 0) {
    partial[blockIdx.x * 2 + 0] = acc[0];
    partial[blockIdx.x * 2 + 1] = acc[1];
  }
}

__global__ void blocks_final_kernel(const double* __restrict__ partial, double* __restrict__ out,
                                    int n_blocks, int K) {
  const int k = threadIdx.x;
  if (k >= K) return;
  double s = 0.0;
  for (int b = 0; b < n_blocks; ++b) s += partial[b * K + k];
  out[k] = s;
}

// reference order (one thread): first w *= alpha everywhere, then theta, r, t sums
template <typename Real>
__global__ void variance_sums_ref_kernel(const Real* __restrict__ e, Real* __restrict__ w,
                                         const uint8_t* __restrict__ sel,
                                         const double* __restrict__ alpha, int n_theta, int n_rp,
                                         int n_sp, int n_r, int n_t, double* __restrict__ out) {
  if (blockIdx.x != 0 || threadIdx.x != 0) return;
  for (int th = 0; th < n_theta; th++)
    for (int r = 0; r < n_r; r++)
      for (int t = 0; t < n_t; t++) {
        const size_t i = (static_cast<size_t>(t) * n_theta + th) * n_rp + r;
        w[i] = static_cast<Real>(static_cast<double>(w[i]) * alpha[th]);
      }
  double s1 = 0, s2 = 0;
  for (int th = 0; th < n_theta; th++)
    for (int r = 0; r < n_r; r++)
      for (int t = 0; t < n_t; t++) {
        const size_t i = (static_cast<size_t>(t) * n_theta + th) * n_rp + r;
        const size_t si = (static_cast<size_t>(t) * n_theta + th) * n_sp + r;
        variance_term(e[i], w[i], alpha[th], sel[si] == 1, s1, s2);
      }
  out[0] = s1;
  out[1] = s2;
}

template <typename Real>
__global__ void scale_weights_kernel(Real* __restrict__ w, double alpha, int n_theta, int n_rp,
                                     int n_r, int n_t) {
  const size_t total = static_cast<size_t>(n_t) * n_theta * n_rp;
  for (size_t i = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x; i < total;
       i += static_cast<size_t>(gridDim.x) * blockDim.x) {
    const int r = static_cast<int>(i % n_rp);
    if (r >= n_r) continue;
    w[i] = static_cast<Real>(static_cast<double>(w[i]) / alpha);
  }
}

template <typename Real>
__global__ void cost_sums_kernel(const Real* __restrict__ e, const Real* __restrict__ w,
                                 const uint8_t* __restrict__ sel, double T, double dl, int n_theta,
                                 int n_rp, int n_sp, int n_r, int n_t,
                                 double* __restrict__ partial) {
  const size_t total = static_cast<size_t>(n_t) * n_theta * n_rp;
  double acc[1] = {0.0};
  for (size_t i = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x; i < total;
       i += static_cast<size_t>(gridDim.x) * blockDim.x) {
    const int r = static_cast<int>(i % n_rp);
    if (r >= n_r) continue;
    const size_t row = i / n_rp;
    acc[0] += cost_term(e[i], w[i], sel[row * n_sp + r] == 1, T, dl);
  }
  block_sum<1>(acc);
  if (threadIdx.x == 0) partial[blockIdx.x] = acc[0];
}

template <typename Real>
__global__ void cost_sums_ref_kernel(const Real* __restrict__ e, const Real* __restrict__ w,
                                     const uint8_t* __restrict__ sel, double T, double dl,
                                     int n_theta, int n_rp, int n_sp, int n_r, int n_t,
                                     double* __restrict__ out) {
  if (blockIdx.x != 0 || threadIdx.x != 0) return;
  double c = 0;
  for (int th = 0; th < n_theta; th++)
    for (int r = 0; r < n_r; r++)
      for (int t = 0; t < n_t; t++) {
        const size_t i = (static_cast<size_t>(t) * n_theta + th) * n_rp + r;
        const size_t si = (static_cast<size_t>(t) * n_theta + th) * n_sp + r;
        c += cost_term(e[i], w[i], sel[si] == 1, T, dl);
      }
  out[0] = c;
}

__global__ void mag_reset_kernel(unsigned long long* __restrict__ fx,
                                 const uint8_t* __restrict__ active, int n) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n && active[i]) fx[i] = 0ull;
}

__global__ void mag_update_kernel(const unsigned long long* __restrict__ fx,
                                  const uint8_t* __restrict__ active, double* __restrict__ mag,
                                  int n) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n && active[i]) mag[i] = static_cast<double>(fx[i]) / kFixScale;
}

// 5x5 Hamming window of BFReconstructionEngine.cpp:157-185
__constant__ double c_hamming[5][5] = {{0.0013, 0.0086, 0.0159, 0.0086, 0.0013},
                                       {0.0086, 0.0581, 0.1076, 0.0581, 0.0086},
                                       {0.0159, 0.1076, 0.1993, 0.1076, 0.0159},
                                       {0.0086, 0.0581, 0.1076, 0.0581, 0.0086},
                                       {0.0013, 0.0086, 0.0159, 0.0086, 0.0013}};

__global__ void vsc_kernel(const double* __restrict__ mag, double* __restrict__ filt, int n_z,
                           int n_x) {
  const int idx = blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= n_z * n_x) return;
  const int i = idx / n_x, j = idx % n_x;
  double f = 0;
  for (int p = -2; p <= 2; p++)
    for (int q = -2; q <= 2; q++)
      if (i + p >= 0 && i + p < n_z && j + q >= 0 && j + q < n_x)
        f += c_hamming[p + 2][q + 2] * mag[static_cast<size_t>(i + p) * n_x + (j + q)];
  filt[idx] = f;
}

// The lines of a homogeneous call: active mask, and their magnitudes restart at 0
__global__ void h_list_kernel(const uint8_t* __restrict__ slot, int j, uint8_t* __restrict__ active,
                              unsigned long long* __restrict__ fx, int n) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const bool on = slot[i] == j;
  active[i] = on ? 1 : 0;
  if (on) fx[i] = 0ull;
}

// The lines of a non-homogeneous call (SetNonHomThreshold, GenNonHomList): those whose filtered
// magnitude exceeds the order statistic `rank` (0-based, ascending).  One CTA: the order
// statistic by radix selection on the bits of the (non-negative) magnitudes, 8 at a time from
// the top, until the bucket holds at most kTail values, which are then ranked directly; then the
// active mask, the magnitudes' restart and the ascending list of the active lines with an
// A-column.  On the host (read-back of the map, nth_element, list, upload) this took ~0.25 ms of
// a call's 2.1 on 512 x 128 lines; with one load in flight per thread 0.217 ms, with kAtOnce and a
// tail of 256 instead of 1024 values 0.104 (under a profiler, caches cold; a call took 0.09 less).
constexpr int kTail = 256;
constexpr int kAtOnce = 8;  // loads of a thread in flight: one SM reads the values, latency counts
__global__ void __launch_bounds__(1024)
    nh_list_kernel(const double* __restrict__ filt, const uint8_t* __restrict__ lineok, int n,
                   int rank, uint8_t* __restrict__ active, unsigned long long* __restrict__ fx,
                   int* __restrict__ vis, int* __restrict__ n_vis) {
  __shared__ int hist[256];
  __shared__ unsigned long long tail[kTail];
  __shared__ unsigned long long s_prefix;
  __shared__ int s_rank, s_count, s_n;
  __shared__ int before[kAtOnce][32], row_n[kAtOnce];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const unsigned long long* bits = reinterpret_cast<const unsigned long long*>(filt);
  unsigned long long prefix = 0ull;  // the bits above `shift + 8` of the order statistic
  int r = rank, count = n, shift = 64;
  while (count > kTail && shift > 0) {
    shift -= 8;
    if (tid < 256) hist[tid] = 0;
    __syncthreads();
    for (int i0 = 0; i0 < n; i0 += kAtOnce * 1024) {
      unsigned long long v[kAtOnce];
#pragma unroll
      for (int k = 0; k < kAtOnce; ++k) {
        const int i = i0 + k * 1024 + tid;
        v[k] = i < n ? bits[i] : 0ull;
      }
#pragma unroll
      for (int k = 0; k < kAtOnce; ++k) {
        const bool in = i0 + k * 1024 + tid < n && (shift == 56 || (v[k] >> (shift + 8)) == prefix);
        if (!__any_sync(0xffffffffu, in)) continue;
        const int d = in ? static_cast<int>((v[k] >> shift) & 255u) : -1;
        // the values of a warp share their upper digits: one addition per distinct digit
        const unsigned same = __match_any_sync(0xffffffffu, d);
        if (in && lane == __ffs(same) - 1) atomicAdd(&hist[d], __popc(same));
      }
    }
    __syncthreads();
    if (warp == 0) {  // the bucket of rank r: eight digits per lane, summed across the warp
      int c[8], t = 0;
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        c[k] = hist[8 * lane + k];
        t += c[k];
      }
      int before = t;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int u = __shfl_up_sync(0xffffffffu, before, o);
        if (lane >= o) before += u;
      }
      before -= t;
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        if (r >= before && r < before + c[k]) {
          s_prefix = (prefix << 8) | static_cast<unsigned>(8 * lane + k);
          s_rank = r - before;
          s_count = c[k];
        }
        before += c[k];
      }
    }
    __syncthreads();
    prefix = s_prefix;
    r = s_rank;
    count = s_count;
    __syncthreads();
  }
  if (shift > 0) {  // rank the bucket's values
    if (tid == 0) s_n = 0;
    __syncthreads();
    for (int i0 = 0; i0 < n; i0 += kAtOnce * 1024) {
      unsigned long long v[kAtOnce];
#pragma unroll
      for (int k = 0; k < kAtOnce; ++k) {
        const int i = i0 + k * 1024 + tid;
        v[k] = i < n ? bits[i] : 0ull;
      }
#pragma unroll
      for (int k = 0; k < kAtOnce; ++k)
        if (i0 + k * 1024 + tid < n && (shift == 64 || (v[k] >> shift) == prefix))
          tail[atomicAdd(&s_n, 1)] = v[k];
    }
    __syncthreads();
    if (tid < count) {
      const unsigned long long v = tail[tid];
      int less = 0, same = 0;
      for (int k = 0; k < count; ++k) {
        less += tail[k] < v;
        same += tail[k] == v;
      }
      if (less <= r && r < less + same) s_prefix = v;
    }
    __syncthreads();
    prefix = s_prefix;
  }
  const double thr = __longlong_as_double(static_cast<long long>(prefix));
  int base = 0;
  for (int i0 = 0; i0 < n; i0 += kAtOnce * 1024) {
    double f[kAtOnce];
    uint8_t ok[kAtOnce];
#pragma unroll
    for (int k = 0; k < kAtOnce; ++k) {
      const int i = i0 + k * 1024 + tid;
      f[k] = i < n ? filt[i] : 0.0;
      ok[k] = i < n ? lineok[i] : 0;
    }
    unsigned m[kAtOnce];
#pragma unroll
    for (int k = 0; k < kAtOnce; ++k) {
      const int i = i0 + k * 1024 + tid;
      const bool on = i < n && f[k] > thr;
      if (i < n) active[i] = on ? 1 : 0;
      if (on) fx[i] = 0ull;
      m[k] = __ballot_sync(0xffffffffu, on && ok[k] != 0);
      if (lane == 0) before[k][warp] = __popc(m[k]);
    }
    __syncthreads();
    if (warp < kAtOnce) {  // the lines of the warps before, row by row
      const int c = before[warp][lane];
      int sum = c;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int u = __shfl_up_sync(0xffffffffu, sum, o);
        if (lane >= o) sum += u;
      }
      before[warp][lane] = sum - c;
      if (lane == 31) row_n[warp] = sum;
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < kAtOnce; ++k) {
      if (m[k] >> lane & 1u)
        vis[base + before[k][warp] + __popc(m[k] & ((1u << lane) - 1u))] = i0 + k * 1024 + tid;
      base += row_n[k];
    }
    __syncthreads();
  }
  if (tid == 0) *n_vis = base;
}

// ROI sums: kind 0 = sum of the magnitude map over ROI lines, kind 1 = sum of the volume over
// ROI lines and all y.  The ROI is the index box [x0,x1] x [z0,z1].
template <typename Real>
__global__ void roi_sums_kernel(const DevGeom g, int kind, const double* __restrict__ mag,
                                const Real* __restrict__ x, double* __restrict__ partial) {
  const size_t nl = static_cast<size_t>(g.n_z) * g.n_x;
  const size_t total = kind == 0 ? nl : nl * g.n_y;
  double acc[1] = {0.0};
  for (size_t i = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x; i < total;
       i += static_cast<size_t>(gridDim.x) * blockDim.x) {
    const size_t l = i % nl;
    const int z = static_cast<int>(l / g.n_x), xx = static_cast<int>(l % g.n_x);
    if (xx < g.roi_x0 || xx > g.roi_x1 || z < g.roi_z0 || z > g.roi_z1) continue;
    acc[0] += kind == 0 ? mag[l] : static_cast<double>(x[i]);  // x: [y][z][x]
  }
  block_sum<1>(acc);
  if (threadIdx.x == 0) partial[blockIdx.x] = acc[0];
}

template <typename Real>
__global__ void roi_sums_ref_kernel(const DevGeom g, int kind, const double* __restrict__ mag,
                                    const Real* __restrict__ x, double* __restrict__ out) {
  if (blockIdx.x != 0 || threadIdx.x != 0) return;
  double s = 0;
  const size_t plane = static_cast<size_t>(g.n_z) * g.n_x;
  for (int j = 0; j < g.n_z; j++)
    for (int k = 0; k < g.n_x; k++) {
      if (k < g.roi_x0 || k > g.roi_x1 || j < g.roi_z0 || j > g.roi_z1) continue;
      if (kind == 0) {
        s += mag[static_cast<size_t>(j) * g.n_x + k];
      } else {
        for (int i = 0; i < g.n_y; i++)
          s += static_cast<double>(x[static_cast<size_t>(i) * plane + static_cast<size_t>(j) * g.n_x + k]);
      }
    }
  out[0] = s;
}

}  // namespace

int launch_layout_from_double(const double* h, void* d, int n_theta, int n_r, int n_rp, int n_t,
                              int fp64, void* stream) {
  const size_t n = static_cast<size_t>(n_t) * n_theta * n_rp;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  if (fp64)
    layout_from_double_kernel<double><<<grid_for(n, 256), 256, 0, s>>>(h, RP<double>(d), n_theta,
                                                                        n_r, n_rp, n_t);
  else
    layout_from_double_kernel<float><<<grid_for(n, 256), 256, 0, s>>>(h, RP<float>(d), n_theta,
                                                                       n_r, n_rp, n_t);
  return ok_or(cudaGetLastError());
}

int launch_bf_offset_sums(const BfSino& b, int exact, double T, double dl, double* partial,
                          int n_chunk, double* out, void* stream) {
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  if (exact) {
    const int grid = (b.n_theta + 63) / 64;
    if (b.fp64)
      offset_sums_ref_kernel<double><<<grid, 64, 0, s>>>(RP<double>(b.e), RP<double>(b.w), b.sel, T,
                                                         dl, b.n_theta, b.n_rp, b.n_sp, b.n_r, b.n_t,
                                                         out);
    else
      offset_sums_ref_kernel<float><<<grid, 64, 0, s>>>(RP<float>(b.e), RP<float>(b.w), b.sel, T, dl,
                                                        b.n_theta, b.n_rp, b.n_sp, b.n_r, b.n_t, out);
    return ok_or(cudaGetLastError());
  }
  const dim3 grid(b.n_theta, n_chunk);
  if (b.fp64)
    offset_sums_kernel<double><<<grid, 256, 0, s>>>(RP<double>(b.e), RP<double>(b.w), b.sel, T, dl,
                                                    b.n_theta, b.n_rp, b.n_sp, b.n_r, b.n_t, n_chunk,
                                                    partial);
  else
    sums_f32_kernel<kOffsetSums><<<grid, 256, 0, s>>>(RP<float>(b.e), RP<float>(b.w), b.sel, nullptr,
                                                      0, T, dl, b.n_theta, b.n_rp, b.n_sp, b.n_r,
                                                      b.n_t, n_chunk, partial);
  const int n = b.n_theta * 2;
  chunk_final_kernel<<<(n + 127) / 128, 128, 0, s>>>(partial, out, b.n_theta, n_chunk, 2);
  return ok_or(cudaGetLastError());
}

int launch_bf_offset_apply(const BfSino& b, const double* step, void* stream) {
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  const size_t n = static_cast<size_t>(b.n_t) * b.n_theta * b.n_rp;
  if (b.fp64)
    offset_apply_kernel<double><<<grid_for(n, 256), 256, 0, s>>>(RP<double>(b.e), step, b.n_theta,
                                                                 b.n_rp, b.n_r, b.n_t);
  else
    offset_apply_kernel<float><<<grid_for(n, 256), 256, 0, s>>>(RP<float>(b.e), step, b.n_theta,
                                                                b.n_rp, b.n_r, b.n_t);
  return ok_or(cudaGetLastError());
}

int launch_bf_selector(const BfSino& b, double T, void* stream) {
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  const size_t n = static_cast<size_t>(b.n_t) * b.n_theta * b.n_sp;
  if (b.fp64)
    selector_kernel<double><<<grid_for(n, 256), 256, 0, s>>>(RP<double>(b.e), RP<double>(b.w), b.sel,
                                                             T, b.n_theta, b.n_rp, b.n_sp, b.n_r,
                                                             b.n_t);
  else
    selector_kernel<float><<<grid_for(n, 256), 256, 0, s>>>(RP<float>(b.e), RP<float>(b.w), b.sel, T,
                                                            b.n_theta, b.n_rp, b.n_sp, b.n_r, b.n_t);
  return ok_or(cudaGetLastError());
}

int launch_bf_variance_sums(const BfSino& b, int exact, const double* alpha, bool scale,
                            double* partial, double* out, void* stream) {
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  if (exact) {
    if (b.fp64)
      variance_sums_ref_kernel<double><<<1, 32, 0, s>>>(RP<double>(b.e), RP<double>(b.w), b.sel,
                                                        alpha, b.n_theta, b.n_rp, b.n_sp, b.n_r,
                                                        b.n_t, out);
    else
      variance_sums_ref_kernel<float><<<1, 32, 0, s>>>(RP<float>(b.e), RP<float>(b.w), b.sel, alpha,
                                                       b.n_theta, b.n_rp, b.n_sp, b.n_r, b.n_t, out);
    return ok_or(cudaGetLastError());
  }
  if (b.fp64) {
    variance_sums_kernel<double><<<kRedBlocks, 256, 0, s>>>(RP<double>(b.e), RP<double>(b.w), b.sel,
                                                            alpha, b.n_theta, b.n_rp, b.n_sp, b.n_r,
                                                            b.n_t, partial);
    blocks_final_kernel<<<1, 32, 0, s>>>(partial, out, kRedBlocks, 2);
    return ok_or(cudaGetLastError());
  }
  const int chunks = view_chunks(b);
  sums_f32_kernel<kVarianceSums><<<dim3(b.n_theta, chunks), 256, 0, s>>>(
      RP<float>(b.e), RP<float>(b.w), b.sel, alpha, scale ? 1 : 0, 0.0, 0.0, b.n_theta, b.n_rp,
      b.n_sp, b.n_r, b.n_t, chunks, partial);
  partials_final_kernel<2><<<1, 256, 0, s>>>(partial, out, b.n_theta * chunks);
  return ok_or(cudaGetLastError());
}

// FP32 engine: the offset step and the selector that follows it, in one pass
int launch_bf_offset_step(const BfSino& b, const double* sums, double T, void* stream) {
  const int chunks = view_chunks(b);
  offset_step_f32_kernel<<<dim3(b.n_theta, chunks), 256, 0, static_cast<cudaStream_t>(stream)>>>(
      RP<float>(b.e), RP<float>(b.w), b.sel, sums, T, b.n_theta, b.n_rp, b.n_sp, b.n_r, b.n_t,
      chunks);
  return ok_or(cudaGetLastError());
}

// FP32 engine: the weights of the new common variance (after variance sums that did not scale
// them) and the selector that follows, in one pass
int launch_bf_new_weights(const BfSino& b, const double* alpha, const double* sums, double dT,
                          double count, double T, void* stream) {
  const int chunks = view_chunks(b);
  new_weights_f32_kernel<<<dim3(b.n_theta, chunks), 256, 0, static_cast<cudaStream_t>(stream)>>>(
      RP<float>(b.e), RP<float>(b.w), b.sel, alpha, sums, dT, count, T, b.n_theta, b.n_rp, b.n_sp,
      b.n_r, b.n_t, chunks);
  return ok_or(cudaGetLastError());
}

int launch_bf_scale_weights(const BfSino& b, double alpha, void* stream) {
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  const size_t n = static_cast<size_t>(b.n_t) * b.n_theta * b.n_rp;
  if (b.fp64)
    scale_weights_kernel<double><<<grid_for(n, 256), 256, 0, s>>>(RP<double>(b.w), alpha, b.n_theta,
                                                                  b.n_rp, b.n_r, b.n_t);
  else
    scale_weights_kernel<float><<<grid_for(n, 256), 256, 0, s>>>(RP<float>(b.w), alpha, b.n_theta,
                                                                 b.n_rp, b.n_r, b.n_t);
  return ok_or(cudaGetLastError());
}

int launch_bf_cost_sums(const BfSino& b, int exact, double T, double dl, double* partial,
                        double* out, void* stream) {
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  if (exact) {
    if (b.fp64)
      cost_sums_ref_kernel<double><<<1, 32, 0, s>>>(RP<double>(b.e), RP<double>(b.w), b.sel, T, dl,
                                                    b.n_theta, b.n_rp, b.n_sp, b.n_r, b.n_t, out);
    else
      cost_sums_ref_kernel<float><<<1, 32, 0, s>>>(RP<float>(b.e), RP<float>(b.w), b.sel, T, dl,
                                                   b.n_theta, b.n_rp, b.n_sp, b.n_r, b.n_t, out);
    return ok_or(cudaGetLastError());
  }
  if (b.fp64) {
    cost_sums_kernel<double><<<kRedBlocks, 256, 0, s>>>(RP<double>(b.e), RP<double>(b.w), b.sel, T,
                                                        dl, b.n_theta, b.n_rp, b.n_sp, b.n_r, b.n_t,
                                                        partial);
    blocks_final_kernel<<<1, 32, 0, s>>>(partial, out, kRedBlocks, 1);
    return ok_or(cudaGetLastError());
  }
  const int chunks = view_chunks(b);
  sums_f32_kernel<kCostSums><<<dim3(b.n_theta, chunks), 256, 0, s>>>(
      RP<float>(b.e), RP<float>(b.w), b.sel, nullptr, 0, T, dl, b.n_theta, b.n_rp, b.n_sp, b.n_r,
      b.n_t, chunks, partial);
  partials_final_kernel<2><<<1, 256, 0, s>>>(partial, out, b.n_theta * chunks);
  return ok_or(cudaGetLastError());
}

int launch_bf_mag_reset(unsigned long long* fx, const uint8_t* active, int n, void* stream) {
  mag_reset_kernel<<<(n + 255) / 256, 256, 0, static_cast<cudaStream_t>(stream)>>>(fx, active, n);
  return ok_or(cudaGetLastError());
}

int launch_bf_mag_update(const unsigned long long* fx, const uint8_t* active, double* mag, int n,
                         void* stream) {
  mag_update_kernel<<<(n + 255) / 256, 256, 0, static_cast<cudaStream_t>(stream)>>>(fx, active,
                                                                                   mag, n);
  return ok_or(cudaGetLastError());
}

int launch_bf_vsc(const double* mag, double* filt, int n_z, int n_x, void* stream) {
  const int n = n_z * n_x;
  vsc_kernel<<<(n + 255) / 256, 256, 0, static_cast<cudaStream_t>(stream)>>>(mag, filt, n_z, n_x);
  return ok_or(cudaGetLastError());
}

int launch_bf_h_list(const uint8_t* slot, int j, uint8_t* active, unsigned long long* fx, int n,
                     void* stream) {
  h_list_kernel<<<(n + 255) / 256, 256, 0, static_cast<cudaStream_t>(stream)>>>(slot, j, active, fx,
                                                                               n);
  return ok_or(cudaGetLastError());
}

int launch_bf_nh_list(const double* filt, const uint8_t* lineok, int n, int rank, uint8_t* active,
                      unsigned long long* fx, int* vis, int* n_vis, void* stream) {
  nh_list_kernel<<<1, 1024, 0, static_cast<cudaStream_t>(stream)>>>(filt, lineok, n, rank, active,
                                                                    fx, vis, n_vis);
  return ok_or(cudaGetLastError());
}

int launch_roi_sum(const DevGeom& g, int exact, int kind, const double* mag, const void* x,
                   int fp64, double* partial, double* out, void* stream) {
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  if (exact) {
    if (fp64)
      roi_sums_ref_kernel<double><<<1, 32, 0, s>>>(g, kind, mag, RP<double>(x), out);
    else
      roi_sums_ref_kernel<float><<<1, 32, 0, s>>>(g, kind, mag, RP<float>(x), out);
    return ok_or(cudaGetLastError());
  }
  if (fp64)
    roi_sums_kernel<double><<<kRedBlocks, 256, 0, s>>>(g, kind, mag, RP<double>(x), partial);
  else
    roi_sums_kernel<float><<<kRedBlocks, 256, 0, s>>>(g, kind, mag, RP<float>(x), partial);
  blocks_final_kernel<<<1, 32, 0, s>>>(partial, out, kRedBlocks, 1);
  return ok_or(cudaGetLastError());
}

}  // namespace mbir
