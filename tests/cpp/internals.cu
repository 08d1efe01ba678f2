// Entries for tests of what has no C entry of its own: shared-memory layouts (host only) and the
// sinogram passes on arrays of the caller's.
#include <cuda_runtime.h>

#include <cstdint>
#include <vector>

#include "mbir_engine.h"
#include "mbir_internal.h"
#include "mbir_wide.cuh"

using namespace mbir;

namespace {

// A host array [n_t][n_theta][n_r] in the device layout (rows padded to `pitch` entries)
template <typename T>
struct Rows {
  T* d = nullptr;
  int n_r, pitch;
  size_t rows;
  Rows(const T* h, int n_theta, int n_r_, int n_t, int pitch_)
      : n_r(n_r_), pitch(pitch_), rows(static_cast<size_t>(n_theta) * n_t) {
    cudaMalloc(&d, rows * pitch * sizeof(T));
    cudaMemset(d, 0, rows * pitch * sizeof(T));
    cudaMemcpy2D(d, pitch * sizeof(T), h, n_r * sizeof(T), n_r * sizeof(T), rows,
                 cudaMemcpyHostToDevice);
  }
  void get(T* h) const {
    cudaMemcpy2D(h, n_r * sizeof(T), d, pitch * sizeof(T), n_r * sizeof(T), rows,
                 cudaMemcpyDeviceToHost);
  }
  ~Rows() { cudaFree(d); }
};

template <typename T>
struct Dev {
  T* d = nullptr;
  size_t n;
  Dev(const T* h, size_t n_) : n(n_) {
    cudaMalloc(&d, n * sizeof(T));
    if (h) cudaMemcpy(d, h, n * sizeof(T), cudaMemcpyHostToDevice);
  }
  void get(T* h, size_t k) const { cudaMemcpy(h, d, k * sizeof(T), cudaMemcpyDeviceToHost); }
  ~Dev() { cudaFree(d); }
};

struct Sino {
  Rows<float> e, w;
  Rows<uint8_t> sel;
  BfSino b{};
  Sino(const float* he, const float* hw, const uint8_t* hs, int n_theta, int n_r, int n_t)
      : e(he, n_theta, n_r, n_t, (n_r + 3) / 4 * 4),
        w(hw, n_theta, n_r, n_t, (n_r + 3) / 4 * 4),
        sel(hs, n_theta, n_r, n_t, (n_r + 15) / 16 * 16) {
    b.e = e.d;
    b.w = w.d;
    b.sel = sel.d;
    b.fp64 = 0;
    b.n_theta = n_theta;
    b.n_rp = e.pitch;
    b.n_sp = sel.pitch;
    b.n_r = n_r;
    b.n_t = n_t;
  }
};

__global__ void div_by_kernel(const double* x, const double* g, double* q, int n) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
    q[i] = wide::div_by(x[i], g[i], 1.0 / g[i], wide::divides(g[i]));
}

int done() { return cudaDeviceSynchronize() == cudaSuccess ? 0 : -3; }

}  // namespace

extern "C" {

// layouts of one detector row per slice and 64 response bins, FP32
int t_general_bytes(int n_theta, int n_x, int n_rs, int n_sp) {
  return static_cast<int>(sweep_smem_bytes(n_theta, n_x, n_rs, 1, 64, 0, n_sp));
}
int t_table_bytes_of(int n_theta, int n_x, int n_rs, int staged, int n_sp, int nbuf) {
  return static_cast<int>(table_smem_bytes(n_theta, n_x, n_rs, staged != 0, n_sp, false, nbuf));
}
int t_walk_bytes(int n_theta, int n_x, int n_rs, int staged, int n_sp, long limit) {
  return static_cast<int>(table_walk_bytes(n_theta, n_x, n_rs, staged != 0, n_sp, false, limit));
}
int t_sched_bytes(int n_theta, int n_rs, int staged, int n_sp) {
  return static_cast<int>(table_smem_bytes(n_theta, 0, n_rs, staged != 0, n_sp, false, 2));
}

// kind 0: variance sums (out: sum e^2 (w a), sum |e| sqrt(a w a)), kind 1: cost sum
int t_bf_sums(int kind, const float* e, const float* w, const uint8_t* sel, const double* alpha,
              double T, double dl, int n_theta, int n_r, int n_t, double* out) {
  Sino s(e, w, sel, n_theta, n_r, n_t);
  Dev<double> a(alpha, n_theta), part(nullptr, 4096), o(nullptr, 16);
  const int rc = kind == 0
                     ? launch_bf_variance_sums(s.b, 0, a.d, false, part.d, o.d, nullptr)
                     : launch_bf_cost_sums(s.b, 0, T, dl, part.d, o.d, nullptr);
  if (rc || done()) return rc ? rc : -3;
  o.get(out, kind == 0 ? 2 : 1);
  return 0;
}

// e -= num / den of each view, then the selector: in one pass (fused) or by the passes of a slab
int t_offset_step(int fused, float* e, const float* w, uint8_t* sel, const double* sums, double T,
                  int n_theta, int n_r, int n_t) {
  Sino s(e, w, sel, n_theta, n_r, n_t);
  Dev<double> d(sums, 2 * n_theta);
  std::vector<double> step(n_theta);
  for (int v = 0; v < n_theta; v++) step[v] = sums[2 * v] / sums[2 * v + 1];
  Dev<double> ds(step.data(), n_theta);
  int rc;
  if (fused) {
    rc = launch_bf_offset_step(s.b, d.d, T, nullptr);
  } else if ((rc = launch_bf_offset_apply(s.b, ds.d, nullptr)) == 0) {
    rc = launch_bf_selector(s.b, T, nullptr);
  }
  if (rc || done()) return rc ? rc : -3;
  s.e.get(e);
  s.sel.get(sel);
  return 0;
}

// w = (float)((float)(w alpha) / upd), then the selector, likewise
int t_new_weights(int fused, const float* e, float* w, uint8_t* sel, const double* alpha,
                  const double* sums, double dT, double count, double T, int n_theta, int n_r,
                  int n_t) {
  Sino s(e, w, sel, n_theta, n_r, n_t);
  Dev<double> a(alpha, n_theta), d(sums, 2), part(nullptr, 4096), o(nullptr, 16);
  int rc;
  if (fused) {
    rc = launch_bf_new_weights(s.b, a.d, d.d, dT, count, T, nullptr);
  } else {
    // the scaling by alpha is that of the variance sums' pass
    const double upd = (sums[0] + dT * sums[1]) / count;
    if ((rc = launch_bf_variance_sums(s.b, 0, a.d, true, part.d, o.d, nullptr)) == 0 &&
        (rc = launch_bf_scale_weights(s.b, upd, nullptr)) == 0)
      rc = launch_bf_selector(s.b, T, nullptr);
  }
  if (rc || done()) return rc ? rc : -3;
  s.w.get(w);
  s.sel.get(sel);
  return 0;
}

// e = y - mu_new - gain_new ((y - e - mu_old) / gain_old)
int t_rebuild_error(const float* y, float* e, const double* mu_old, const double* gain_old,
                    const double* mu_new, const double* gain_new, int n_theta, int n_r, int n_t) {
  const int pitch = (n_r + 3) / 4 * 4;
  Rows<float> dy(y, n_theta, n_r, n_t, pitch), de(e, n_theta, n_r, n_t, pitch);
  Dev<double> a(mu_old, n_theta), b(gain_old, n_theta), c(mu_new, n_theta), d(gain_new, n_theta);
  const int rc = launch_rebuild_error(dy.d, de.d, a.d, b.d, c.d, d.d, n_theta, pitch, n_r, n_t, 0,
                                      nullptr);
  if (rc || done()) return rc ? rc : -3;
  de.get(e);
  return 0;
}

// q = x / g by the view sums' division
int t_div_by(const double* x, const double* g, double* q, int n) {
  Dev<double> dx(x, n), dg(g, n), dq(nullptr, n);
  div_by_kernel<<<152, 256>>>(dx.d, dg.d, dq.d, n);
  if (cudaGetLastError() != cudaSuccess || done()) return -3;
  dq.get(q, n);
  return 0;
}

// The engine's optional A-column table; all of a device's given back; an allocation that no device
// has room for
long t_optional_table_bytes(void* engine) {
  return static_cast<long>((*static_cast<Engine**>(engine))->optional_table_bytes());
}
void t_reclaim_tables(int device) { reclaim_tables(device); }
int t_huge_allocation_fails(int device) {
  void* p = nullptr;
  const bool failed = device_malloc(&p, size_t{1} << 50, device) == cudaErrorMemoryAllocation;
  cudaGetLastError();
  return failed && p == nullptr ? 1 : 0;
}

int t_reduce_stats(const double* in, int n_rows, int n_cols, double* out) {
  Dev<double> d(in, static_cast<size_t>(n_rows) * n_cols), o(nullptr, n_cols + 2);
  const int rc = launch_reduce_stats(d.d, n_rows, n_cols, o.d, nullptr);
  if (rc || done()) return rc ? rc : -3;
  o.get(out, n_cols);
  return 0;
}

}  // extern "C"
