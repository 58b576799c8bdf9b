// m2p.cuh — the inner loop shared by the far-field sums of the tree and
// nrnmm solvers (M2P: a target against the P Chebyshev nodes of a box,
// weighted by the box's expansion; src/fmm_core.cpp:624-661,
// src/nrnmm.cpp:86-97).
//
// A box is staged in shared memory as its 1-D node coordinates X[q][o]
// (D x n) and its weights W[r][k] (RB x P); node k = (o_0, .., o_{D-1}) with
// the last dimension fastest.  The innermost loop is unrolled so that the
// evaluations of consecutive nodes (each a chain of a square root or
// logarithm and a divide) overlap in the FP64 pipe.
#pragma once

#include <cuda_runtime.h>

#include "kernels.cuh"

namespace fmma_b200 {

// For the radial kernels the node grid saves work: the squares of the outer
// dimensions are formed once per row of nodes, the innermost differences once
// per box, so a pair costs one multiply-add for r^2, f (5 operations for 1/r)
// and one multiply-add per right-hand side: 7 FP64 operations for 1/r instead
// of 16 with rsqrt() and all differences per pair.  N nodes per dimension, at
// compile time: a row's N evaluations are independent.  FP64 pipe bound.
// Against the general loop: tree solver's far sums, 200k points in 3-D, 6 nodes
// 29.9 -> 13.3 ms (16 warps an SM at 117 registers, 20 in blocks of 64; 24 at 80
// were 10 % slower), nrnmm 100k points 51.1 -> 27.9 ms a call; the FP64 pipe is
// 55 to 61 % busy.
template <int KID, int D, int RB, int N>
__device__ __forceinline__ void far_box_row(const double* x, const double* __restrict__ X,
                                            const double* __restrict__ W, int P, double p0, double ip, double* acc) {
  double t[N];  // innermost differences
#pragma unroll
  for (int o = 0; o < N; ++o) t[o] = x[D - 1] - X[(D - 1) * N + o];
  // exponents of the outer part a and of the smallest and largest |t| that
  // keep every r^2 = a + t^2 of a row within 2^+-500
  constexpr int kLo = (1023 - 500) << 20, kHi = (1023 + 498) << 20;
  int tlo = 0x7fffffff, thi = 0;
#pragma unroll
  for (int o = 0; o < N; ++o) {
    const int h = __double2hiint(t[o]) & 0x7fffffff;
    tlo = min(tlo, h);
    thi = max(thi, h);
  }
  const bool top = thi < ((1023 + 248) << 20), bottom = tlo >= ((1023 - 249) << 20);
  const double none[N] = {};
  auto row = [&](double a, const double* Wk) {
    double r2[N], f[N];
#pragma unroll
    for (int o = 0; o < N; ++o) r2[o] = fma(t[o], t[o], a);
    const int h = __double2hiint(a);
    if (top && h < kHi && (bottom || h >= kLo)) kvals<KID, N, true>(r2, none, p0, ip, f);
    else kvals<KID, N>(r2, none, p0, ip, f);
#pragma unroll
    for (int rr = 0; rr < RB; ++rr) {
      if constexpr (N % 2 == 0) {  // rows of weights on 16 bytes
#pragma unroll
        for (int o = 0; o < N; o += 2) {
          const double2 w = *reinterpret_cast<const double2*>(Wk + rr * P + o);
          acc[rr] = fma(f[o], w.x, acc[rr]);
          acc[rr] = fma(f[o + 1], w.y, acc[rr]);
        }
      } else {
#pragma unroll
        for (int o = 0; o < N; ++o) acc[rr] = fma(f[o], Wk[rr * P + o], acc[rr]);
      }
    }
  };
  if constexpr (D == 1) {
    row(0.0, W);
  } else {
#pragma unroll 1
    for (int o0 = 0; o0 < N; ++o0) {
      const double d0 = x[0] - X[o0], a0 = d0 * d0;
      if constexpr (D == 2) {
        row(a0, W + o0 * N);
      } else {
#pragma unroll 1
        for (int o1 = 0; o1 < N; ++o1) {
          const double d1 = x[1] - X[N + o1];
          row(fma(d1, d1, a0), W + (o0 * N + o1) * N);
        }
      }
    }
  }
}

// Kernels and right-hand sides that far_box_row is made for, and the node
// counts.  The kernels that hold it (ROW) are compiled apart from those of the
// general loop, which needs fewer registers and more warps: in one kernel the
// loop ran at the rows' 16 warps an SM (nrnmm, 2-D, 10 nodes, 100k points:
// 1/r 12.87 ms against 11.41 at 24, Gaussian 31.99 against 30.75).
template <int KID, int RB>
constexpr bool far_row_kernel() {
  return RB == 1 && (KID == FMMA_KERNEL_INV_R || KID == FMMA_KERNEL_INV_R_SAFE || KID == FMMA_KERNEL_LOG_R ||
                     KID == FMMA_KERNEL_GAUSSIAN || KID == FMMA_KERNEL_MULTIQUADRIC);
}
inline bool far_row_nodes(int n) { return n >= 2 && n <= 8; }

// far_box_row for the boxes j < nb of a staged batch that `skip(j)` lets
// through, for n in far_row_nodes.
template <int KID, int D, int RB, typename Skip>
__device__ __forceinline__ void far_batch(const double* x, const double* X, const double* W, int nb, int n, int P,
                                          double p0, double ip, double* acc, const Skip& skip) {
#define FMMA_FAR_N(N_)                                                                                         \
  case N_:                                                                                                     \
    for (int j = 0; j < nb; ++j)                                                                               \
      if (!skip(j)) far_box_row<KID, D, RB, N_>(x, X + j * D * N_, W + (size_t)j * RB * P, P, p0, ip, acc);    \
    break;
  switch (n) {
    FMMA_FAR_N(2) FMMA_FAR_N(3) FMMA_FAR_N(4) FMMA_FAR_N(5) FMMA_FAR_N(6) FMMA_FAR_N(7) FMMA_FAR_N(8)
    default: break;
  }
#undef FMMA_FAR_N
}

// Kernel value of the general loop below: 1/r through rsqrt(), whose operands
// outside the normal range cost no branch of their own; with one pair at a time
// that beats inv_sqrt's fewer operations behind a check (nrnmm, 2-D, 10 nodes
// 1.61 against 1.93 ms; 3-D, 6 nodes x 3 rhs 7.92 against 8.77; tree, 3-D, 6
// nodes x 3 rhs 24.4 against 25.8).
template <int KID, int D>
__device__ __forceinline__ double kfar(const double* x, const double* y, double p0) {
  if constexpr (KID == FMMA_KERNEL_INV_R || KID == FMMA_KERNEL_INV_R_SAFE) {
    double r2 = 0.0;
#pragma unroll
    for (int q = 0; q < D; ++q) {
      const double t = x[q] - y[q];
      r2 += t * t;
    }
    if constexpr (KID == FMMA_KERNEL_INV_R_SAFE) return r2 > 0.0 ? rsqrt(r2) : 0.0;
    return rsqrt(r2);
  } else {
    return keval<KID, D>(x, y, p0);
  }
}

template <int KID, int D, int RB>
__device__ __forceinline__ void far_box_sum(const double* x, const double* __restrict__ X,
                                            const double* __restrict__ W, int n, int P, double p0, double* acc) {
  double y[D];
  if constexpr (D == 1) {
#pragma unroll 4
    for (int o0 = 0; o0 < n; ++o0) {
      y[0] = X[o0];
      const double f = kfar<KID, D>(x, y, p0);
#pragma unroll
      for (int rr = 0; rr < RB; ++rr) acc[rr] += f * W[rr * P + o0];
    }
  } else if constexpr (D == 2) {
    for (int o0 = 0; o0 < n; ++o0) {
      y[0] = X[o0];
      const double* Wk = W + o0 * n;
#pragma unroll 4
      for (int o1 = 0; o1 < n; ++o1) {
        y[1] = X[n + o1];
        const double f = kfar<KID, D>(x, y, p0);
#pragma unroll
        for (int rr = 0; rr < RB; ++rr) acc[rr] += f * Wk[rr * P + o1];
      }
    }
  } else {
    for (int o0 = 0; o0 < n; ++o0) {
      y[0] = X[o0];
      for (int o1 = 0; o1 < n; ++o1) {
        y[1] = X[n + o1];
        const double* Wk = W + (o0 * n + o1) * n;
#pragma unroll 4
        for (int o2 = 0; o2 < n; ++o2) {
          y[2] = X[2 * n + o2];
          const double f = kfar<KID, D>(x, y, p0);
#pragma unroll
          for (int rr = 0; rr < RB; ++rr) acc[rr] += f * Wk[rr * P + o2];
        }
      }
    }
  }
}

}  // namespace fmma_b200
