// mbir_wide.cuh -- FP64-accurate sums and roundings of FP32 arrays on the FP32 units.
//
// The sinogram-wide passes of the FP32 engine are defined in FP64: sums of products over a view or
// the whole sinogram, and elementwise updates whose FP64 result is rounded to FP32.  GB300's FP64
// pipe takes 2 lanes per clock and SM, so 5 to 30 FP64 operations per element (conversions among
// them) bound those passes at 5 to 30 times their memory time.  Here
//   * sums use the error-free transformations of Knuth (two_sum) and Dekker/FMA (two_prod):
//     a product of two or three FP32 numbers enters as the pairs whose sum it is exactly, WideSum
//     holds the sum as three FP32 numbers whose rounding error is near 2^-70 of it, and is added
//     to an FP64 accumulator once per thread and chunk, so that fewer FP64 roundings take part than
//     when every term was multiplied and added in FP64;
//   * elementwise results are computed to ~2^-44 and rounded to FP32 when no rounding boundary is
//     near (Ziv's test); otherwise, about once in 10^5 elements, the FP64 expression is evaluated.
//     Results are the same bits as the FP64 expression's.
// Chunks whose sum is not finite or so small that the FP32 products may have lost bits to
// underflow are summed again in FP64 by the caller.
#pragma once
#include <cuda_runtime.h>

namespace mbir {
namespace wide {

struct F2 {
  float hi, lo;  // hi = rn(hi + lo)
};

__device__ __forceinline__ F2 two_sum(float a, float b) {
  const float s = __fadd_rn(a, b);
  const float t = __fsub_rn(s, a);
  return {s, __fadd_rn(__fsub_rn(a, __fsub_rn(s, t)), __fsub_rn(b, t))};
}
__device__ __forceinline__ F2 two_diff(float a, float b) { return two_sum(a, -b); }
__device__ __forceinline__ F2 two_prod(float a, float b) {
  const float p = __fmul_rn(a, b);
  return {p, __fmaf_rn(a, b, -p)};
}
// |a| >= |b|
__device__ __forceinline__ F2 fast_two_sum(float a, float b) {
  const float s = __fadd_rn(a, b);
  return {s, __fsub_rn(b, __fsub_rn(s, a))};
}
__device__ __forceinline__ F2 add(F2 a, F2 b) {
  const F2 s = two_sum(a.hi, b.hi);
  return fast_two_sum(s.hi, __fadd_rn(s.lo, __fadd_rn(a.lo, b.lo)));
}
__device__ __forceinline__ F2 neg(F2 a) { return {-a.hi, -a.lo}; }
__device__ __forceinline__ F2 mul(F2 a, F2 b) {
  const F2 p = two_prod(a.hi, b.hi);
  return fast_two_sum(p.hi, __fmaf_rn(a.hi, b.lo, __fmaf_rn(a.lo, b.hi, p.lo)));
}
__device__ __forceinline__ F2 mul(F2 a, float b) {
  const F2 p = two_prod(a.hi, b);
  return fast_two_sum(p.hi, __fmaf_rn(a.lo, b, p.lo));
}
__device__ __forceinline__ F2 split(double v) {
  const float h = static_cast<float>(v);
  return {h, static_cast<float>(v - static_cast<double>(h))};
}
// v as a factor of a product that is rounded to FP32 (rounds_to): below 2^-90 the low part would be
// subnormal and short of bits, so a product takes the FP64 expression there (no F2 rounds with NaN)
__device__ __forceinline__ F2 split_factor(double v) {
  return fabs(v) >= 8.1e-28 ? split(v) : F2{__int_as_float(0x7fc00000), 0.f};
}

struct WideSum {
  float s0 = 0.f, s1 = 0.f, s2 = 0.f;
  __device__ __forceinline__ void add(float x) {
    const F2 a = two_sum(s0, x);
    const F2 b = two_sum(s1, a.lo);
    s0 = a.hi;
    s1 = b.hi;
    s2 = __fadd_rn(s2, b.lo);
  }
  __device__ __forceinline__ void add(F2 x) {
    const F2 a = two_sum(s0, x.hi);
    const F2 b = two_sum(s1, a.lo);
    const F2 c = two_sum(b.hi, x.lo);
    s0 = a.hi;
    s1 = c.hi;
    s2 = __fadd_rn(s2, __fadd_rn(b.lo, c.lo));
  }
  // e^2 w, exact to the sum's own rounding: both parts of e^2 times w, the two low ends combined
  __device__ __forceinline__ void add_square_times(float e, float w) {
    const F2 q = two_prod(e, e), p = two_prod(q.hi, w), t = two_prod(q.lo, w);
    const F2 r = two_sum(p.lo, t.hi);
    add(F2{p.hi, r.hi});
    s2 = __fadd_rn(s2, __fadd_rn(r.lo, t.lo));
  }
  __device__ __forceinline__ double value() const {
    return static_cast<double>(s0) + (static_cast<double>(s1) + static_cast<double>(s2));
  }
  // the FP32 products behind the sum kept all their bits
  __device__ __forceinline__ bool sound() const {
    const float a = fabsf(s0);
    return a >= 1e-24f && a <= 1e36f;
  }
};

// v.hi + v.lo rounded to FP32 in `r` when no rounding boundary lies within `eps` (absolute) of it
__device__ __forceinline__ bool rounds_to(F2 v, float eps, float& r) {
  const F2 s = two_sum(v.hi, v.lo);
  r = s.hi;
  const float a = fabsf(r);
  const unsigned bits = __float_as_uint(a);
  const float half = __fmul_rn(0.5f, __fsub_rn(__uint_as_float(bits + 1u), a));
  return a >= 1e-24f && a <= 1e36f && (bits & 0x7fffffu) != 0u &&
         fabsf(__fsub_rn(fabsf(s.lo), half)) > eps;
}

// Calls of their own: inlined, a fallback's few FP64 instructions are predicated instead of branched
// over and take their turns on the FP64 pipe for every entry (50 of the 84 to 90 us that the
// bright-field offset step and weight update took at 61 x 512 x 256 entries).
static __device__ __noinline__ bool below_fp64(float e, float w, double t2) {
  const double ev = e;
  return ev * ev * static_cast<double>(w) < t2;
}
static __device__ __noinline__ float minus_fp64(float e, double step) {
  return static_cast<float>(static_cast<double>(e) - step);
}
static __device__ __noinline__ float over_fp64(float w, double by) {
  return static_cast<float>(static_cast<double>(w) / by);
}
static __device__ __noinline__ float times_fp64(float w, double by) {
  return static_cast<float>(static_cast<double>(w) * by);
}

// e^2 w < t2 as the FP64 expression decides it; t2f = (float)t2
__device__ __forceinline__ bool below(float e, float w, double t2, float t2f) {
  const float q = __fmul_rn(e, e), p = __fmul_rn(q, w);
  // FP32 product within 2^-22 of the true one unless it or e^2 under- or overflows
  if (q >= 1e-30f && p >= 1e-30f && p <= 1e36f &&
      (t2f > 1e38f || fabsf(__fsub_rn(p, t2f)) > 1e-6f * t2f))
    return p < t2f;
  return below_fp64(e, w, t2);
}

// The entries of one view in detector rows [t0, t1), four at a time (the padded rows are whole
// float4s): f(row, r) with `row` = t n_theta + v and r..r+3 the bins, for the entries of
// this thread in batches; after(again) closes a batch, whose entries again(g) passes over once
// more.
template <typename F, typename After>
__device__ __forceinline__ void for_view_rows(int v, int t0, int t1, int n_theta, int n_rp, F f,
                                              After after) {
  constexpr int kBatch = 8;
  const int q = n_rp >> 2;
  int t = t0, c = threadIdx.x;
  while (c >= q) {
    c -= q;
    ++t;
  }
  while (t < t1) {
    const int tb = t, cb = c;
    for (int k = 0; k < kBatch && t < t1; ++k) {
      f(static_cast<size_t>(t) * n_theta + v, 4 * c);
      c += blockDim.x;
      while (c >= q) {
        c -= q;
        ++t;
      }
    }
    after([&](auto g) {
      int t2 = tb, c2 = cb;
      for (int k = 0; k < kBatch && t2 < t1; ++k) {
        g(static_cast<size_t>(t2) * n_theta + v, 4 * c2);
        c2 += blockDim.x;
        while (c2 >= q) {
          c2 -= q;
          ++t2;
        }
      }
    });
  }
}

// Block sums of K values (256 threads), each in all lanes of warp k; one FP64 addition per value
// instead of the five that a butterfly of every warp makes (FP64 additions take 16 cycles of the
// SM per warp).
template <int K>
__device__ __forceinline__ double block_sums(const double (&acc)[K]) {
  __shared__ double red[K][256];
#pragma unroll
  for (int k = 0; k < K; ++k) red[k][threadIdx.x] = acc[k];
  __syncthreads();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  double s = 0.0;
  if (warp < K) {
    for (int i = lane; i < 256; i += 32) s += red[warp][i];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  }
  return s;
}

// x / g, correctly rounded, from inv = rn(1 / g): one refinement makes the quotient faithful, a
// second one correctly rounded (Markstein, "Computation of elementary functions on the IBM RISC
// System/6000 processor", 1990), while neither the quotient nor the residuals leave the normal
// range: here both magnitudes within 2^-400 to 2^401, the quotient then within 2^-801 to 2^801.
__device__ __forceinline__ bool mid_range(double x) {
  const unsigned e = (static_cast<unsigned>(__double2hiint(x)) >> 20) & 0x7ffu;
  return e - 623u < 801u;
}
// whether div_by may use g's inverse (a mantissa of ones only is outside the theorem)
__device__ __forceinline__ bool divides(double g) {
  return mid_range(g) && (__double_as_longlong(g) & 0xfffffffffffffLL) != 0xfffffffffffffLL;
}
__device__ __forceinline__ double div_by(double x, double g, double inv, bool mid) {
  if (!mid || !mid_range(x)) return x / g;
  double q = __dmul_rn(x, inv);
  q = fma(fma(-q, g, x), inv, q);
  return fma(fma(-q, g, x), inv, q);
}

}  // namespace wide
}  // namespace mbir
