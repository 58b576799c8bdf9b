// kernels.cuh — built-in interaction kernels f(x, y) as device functions,
// their gradients (adjoint) and compile-time dispatch over (kernel, dim).
//
// The ids and formulas match include/fmma_b200.h and the CPU oracle.  The
// reference's default functor is include/fmma/fmma.hpp:55-63 (1/|x-y|).
#pragma once

#include <cuda_runtime.h>

#include "../../include/fmma_b200.h"

namespace fmma_b200 {

template <int KID>
struct KernelTraits {
  static constexpr bool translation_invariant = KID != FMMA_KERNEL_SUM2_OVER_R2;
  static constexpr bool symmetric = KID != FMMA_KERNEL_INV_DIFF && KID != FMMA_KERNEL_SUM_OVER_R2;
};

inline bool kernel_translation_invariant(int kid) { return kid != FMMA_KERNEL_SUM2_OVER_R2; }

// 1/sqrt(x) for a positive normal x: the hardware's approximation (about 20
// bits) refined by one step of Householder's third-order iteration for
// y^-2 = x, y (1 + e/2 + 3 e^2/8) with e = 1 - x y^2, whose remainder
// 5 e^3 / 16 is far below an ulp; the roundings leave at most one ulp, as a
// square root and a division do.  Five FP64 operations against about 9 for
// rsqrt() and 23 for the square root and division (measured rates, 1.57e12
// and 0.77e12 a second).
__device__ __forceinline__ double inv_sqrt_normal(double x) {
  double y;
  asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
  const double e = fma(-(x * y), y, 1.0);
  return fma(y * e, fma(e, 0.375, 0.5), y);
}
// Zero, subnormal, infinite, NaN or negative: not for inv_sqrt_normal.
__device__ __forceinline__ bool not_normal(double x) {
  return (unsigned)(__double2hiint(x) - 0x00100000) >= 0x7fe00000u;
}
__device__ __forceinline__ double inv_sqrt(double x) { return not_normal(x) ? rsqrt(x) : inv_sqrt_normal(x); }

// r2 / p0 with ip = 1 / p0 rounded (Markstein's division step: the quotient by
// the reciprocal and one exact remainder give the rounded quotient).  Both
// within 2^+-500, so that nothing over- or underflows.
__device__ __forceinline__ double div_by(double r2, double p0, double ip) {
  const double q = r2 * ip;
  return fma(fma(-q, p0, r2), ip, q);
}
__device__ __forceinline__ bool not_mid_range(double x) {
  return (unsigned)(__double2hiint(x) - ((1023 - 500) << 20)) >= (unsigned)(1000 << 20);
}

// FP64 evaluation.
template <int KID, int D>
__device__ __forceinline__ double keval(const double* x, const double* y, double p0) {
  double r2 = 0.0, s = 0.0;
  if (KID == FMMA_KERNEL_INV_DIFF) {
    double t = x[0] - y[0];
    return t != 0.0 ? 1.0 / t : 0.0;
  }
#pragma unroll
  for (int q = 0; q < D; ++q) {
    double t = x[q] - y[q];
    r2 += t * t;
    if (KID == FMMA_KERNEL_SUM_OVER_R2) s += t;
    if (KID == FMMA_KERNEL_SUM2_OVER_R2) { double u = x[q] + y[q]; s += u * u; }
  }
  switch (KID) {
    case FMMA_KERNEL_INV_R: return inv_sqrt(r2);
    case FMMA_KERNEL_INV_R_SAFE: return r2 > 0.0 ? inv_sqrt(r2) : 0.0;
    case FMMA_KERNEL_LOG_R: return r2 > 0.0 ? 0.5 * log(r2) : 0.0;
    case FMMA_KERNEL_GAUSSIAN: return exp(-r2 / p0);
    case FMMA_KERNEL_MULTIQUADRIC: return sqrt(r2 + p0);
    case FMMA_KERNEL_SUM_OVER_R2: return s / r2;
    case FMMA_KERNEL_SUM2_OVER_R2: return s / r2;
    default: return 0.0;
  }
}

// The kernel from its parts, U pairs at once (the checks for operands outside
// the fast steps' ranges are made once per batch).  r2 = |x - y|^2; s: what
// kparts leaves there; ip = 1 / p0 for the Gaussian (kinv).
template <int KID>
__device__ __forceinline__ double kinv(double p0) {
  // 0: always take the plain division
  return KID == FMMA_KERNEL_GAUSSIAN && !not_mid_range(p0) ? 1.0 / p0 : 0.0;
}
template <int KID, int D>
__device__ __forceinline__ void kparts(const double* x, const double* y, double& r2, double& s) {
  r2 = 0.0;
  s = 0.0;
#pragma unroll
  for (int q = 0; q < D; ++q) {
    const double t = x[q] - y[q];
    r2 += t * t;
    if (KID == FMMA_KERNEL_SUM_OVER_R2 || KID == FMMA_KERNEL_INV_DIFF) s += t;
    if (KID == FMMA_KERNEL_SUM2_OVER_R2) { const double u = x[q] + y[q]; s += u * u; }
  }
}
// MID: every r2 is known to lie within 2^+-500.
template <int KID, int U, bool MID = false>
__device__ __forceinline__ void kvals(const double (&r2)[U], const double (&s)[U], double p0, double ip,
                                      double (&f)[U]) {
  if constexpr (MID && (KID == FMMA_KERNEL_INV_R || KID == FMMA_KERNEL_INV_R_SAFE)) {
#pragma unroll
    for (int u = 0; u < U; ++u) f[u] = inv_sqrt_normal(r2[u]);
  } else if constexpr (KID == FMMA_KERNEL_INV_R || KID == FMMA_KERNEL_INV_R_SAFE) {
    bool odd = false;
#pragma unroll
    for (int u = 0; u < U; ++u) {
      f[u] = inv_sqrt_normal(r2[u]);
      odd = odd || not_normal(r2[u]);
    }
    if (odd) {
#pragma unroll
      for (int u = 0; u < U; ++u)
        if (not_normal(r2[u])) f[u] = KID == FMMA_KERNEL_INV_R || r2[u] > 0.0 ? rsqrt(r2[u]) : 0.0;
    }
  } else if constexpr (KID == FMMA_KERNEL_GAUSSIAN) {
    bool odd = ip == 0.0;
    double a[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      a[u] = div_by(r2[u], p0, ip);
      odd = odd || not_mid_range(r2[u]);
    }
    if (odd) {
#pragma unroll
      for (int u = 0; u < U; ++u)
        if (ip == 0.0 || not_mid_range(r2[u])) a[u] = r2[u] / p0;
    }
#pragma unroll
    for (int u = 0; u < U; ++u) f[u] = exp(-a[u]);
  } else {
#pragma unroll
    for (int u = 0; u < U; ++u) {
      switch (KID) {
        case FMMA_KERNEL_INV_DIFF: f[u] = s[u] != 0.0 ? 1.0 / s[u] : 0.0; break;
        case FMMA_KERNEL_LOG_R: f[u] = r2[u] > 0.0 ? 0.5 * log(r2[u]) : 0.0; break;
        case FMMA_KERNEL_MULTIQUADRIC: f[u] = sqrt(r2[u] + p0); break;
        default: f[u] = s[u] / r2[u]; break;
      }
    }
  }
}
// f and the factor c of grad_x f = c (x - y), for the radial kernels.
template <int KID, int U>
__device__ __forceinline__ void kvals_grad(const double (&r2)[U], double p0, double ip, double (&f)[U],
                                           double (&c)[U]) {
  const double none[U] = {};
  kvals<KID, U>(r2, none, p0, ip, f);
#pragma unroll
  for (int u = 0; u < U; ++u) {
    switch (KID) {
      case FMMA_KERNEL_INV_R:  // the gradient is guarded, the value is not
      case FMMA_KERNEL_INV_R_SAFE: c[u] = r2[u] > 0.0 ? -f[u] * f[u] * f[u] : 0.0; break;
      case FMMA_KERNEL_LOG_R: c[u] = r2[u] > 0.0 ? 1.0 / r2[u] : 0.0; break;
      case FMMA_KERNEL_GAUSSIAN: c[u] = -2.0 / p0 * f[u]; break;
      default: c[u] = 1.0 / f[u]; break;  // multiquadric
    }
  }
}

// FP32 evaluation on a difference vector t = x - y (translation-invariant
// kernels only; the mixed-precision P2P forms t from box-local offsets).
template <int KID, int D>
__device__ __forceinline__ float keval_diff_f32(const float* t, float p0) {
  if (KID == FMMA_KERNEL_INV_DIFF) return t[0] != 0.f ? 1.f / t[0] : 0.f;
  float r2 = 0.f, s = 0.f;
#pragma unroll
  for (int q = 0; q < D; ++q) {
    r2 = fmaf(t[q], t[q], r2);
    if (KID == FMMA_KERNEL_SUM_OVER_R2) s += t[q];
  }
  switch (KID) {
    case FMMA_KERNEL_INV_R: return rsqrtf(r2);
    case FMMA_KERNEL_INV_R_SAFE: return r2 > 0.f ? rsqrtf(r2) : 0.f;
    case FMMA_KERNEL_LOG_R: return r2 > 0.f ? 0.5f * __logf(r2) : 0.f;
    case FMMA_KERNEL_GAUSSIAN: return __expf(-r2 / p0);
    case FMMA_KERNEL_MULTIQUADRIC: return sqrtf(r2 + p0);
    case FMMA_KERNEL_SUM_OVER_R2: return s / r2;
    default: return 0.f;
  }
}

// Gradient of f with respect to its first argument x, FP64 (adjoint).
// grad_y f = -grad_x f for translation-invariant kernels.
template <int KID, int D>
__device__ __forceinline__ void kgrad_x(const double* x, const double* y, double p0, double* g) {
  double t[D];
  double r2 = 0.0, s = 0.0;
#pragma unroll
  for (int q = 0; q < D; ++q) {
    t[q] = x[q] - y[q];
    r2 += t[q] * t[q];
    s += t[q];
  }
  double c = 0.0;
  switch (KID) {
    case FMMA_KERNEL_INV_R:
    case FMMA_KERNEL_INV_R_SAFE: {
      if (r2 > 0.0) { double ir = inv_sqrt(r2); c = -ir * ir * ir; }
      break;
    }
    case FMMA_KERNEL_LOG_R: c = r2 > 0.0 ? 1.0 / r2 : 0.0; break;
    case FMMA_KERNEL_GAUSSIAN: c = -2.0 / p0 * exp(-r2 / p0); break;
    case FMMA_KERNEL_MULTIQUADRIC: c = 1.0 / sqrt(r2 + p0); break;
    case FMMA_KERNEL_INV_DIFF: {
      g[0] = t[0] != 0.0 ? -1.0 / (t[0] * t[0]) : 0.0;
      return;
    }
    case FMMA_KERNEL_SUM_OVER_R2: {
#pragma unroll
      for (int q = 0; q < D; ++q) g[q] = r2 > 0.0 ? (1.0 / r2 - 2.0 * s * t[q] / (r2 * r2)) : 0.0;
      return;
    }
    default: {
#pragma unroll
      for (int q = 0; q < D; ++q) g[q] = 0.0;
      return;
    }
  }
#pragma unroll
  for (int q = 0; q < D; ++q) g[q] = c * t[q];
}

// Host dispatch helper: calls F::template run<KID, D>(args...).
template <typename F, typename... Args>
void dispatch_kernel(int kid, int dim, Args&&... args) {
#define FMMA_DISPATCH_D(KID_)                                          \
  switch (dim) {                                                        \
    case 1: F::template run<KID_, 1>(args...); return;                  \
    case 2: F::template run<KID_, 2>(args...); return;                  \
    default: F::template run<KID_, 3>(args...); return;                 \
  }
  switch (kid) {
    case FMMA_KERNEL_INV_R: FMMA_DISPATCH_D(FMMA_KERNEL_INV_R)
    case FMMA_KERNEL_INV_R_SAFE: FMMA_DISPATCH_D(FMMA_KERNEL_INV_R_SAFE)
    case FMMA_KERNEL_INV_DIFF: F::template run<FMMA_KERNEL_INV_DIFF, 1>(args...); return;
    case FMMA_KERNEL_LOG_R: FMMA_DISPATCH_D(FMMA_KERNEL_LOG_R)
    case FMMA_KERNEL_GAUSSIAN: FMMA_DISPATCH_D(FMMA_KERNEL_GAUSSIAN)
    case FMMA_KERNEL_MULTIQUADRIC: FMMA_DISPATCH_D(FMMA_KERNEL_MULTIQUADRIC)
    case FMMA_KERNEL_SUM_OVER_R2: FMMA_DISPATCH_D(FMMA_KERNEL_SUM_OVER_R2)
    default: FMMA_DISPATCH_D(FMMA_KERNEL_SUM2_OVER_R2)
  }
#undef FMMA_DISPATCH_D
}

}  // namespace fmma_b200
