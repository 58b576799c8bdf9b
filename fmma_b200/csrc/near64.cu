// near64.cu — FP64 sums over point pairs: the near field of the leaves
// (src/fmm.cpp:121-141), with or without gradients, and the exact direct sum
// (src/fmma.cpp:80-101).
//
// Both are bound by the FP64 pipe: per pair 2 D operations for |x - y|^2, 5
// for 1/r (47 for log r, 25 for the Gaussian, by measured rates) and one
// multiply-add per right-hand side.  What the kernels arrange is that the
// pipe always has independent pairs: sources come in tiles through shared
// memory, four pairs of a lane are evaluated at a time, and the work is cut so
// that small problems fill the GPU too (the exact sum over source ranges, a
// leaf's near field over the warps of a unit), with the partial sums added in
// a fixed order.
// Against a thread (exact) or warp (near) that walked its sources in global
// memory with 1/r by square root and division: exact 2-D 131072^2 34.2 -> 12.9
// ms (10 FP64 operations a pair are 9.7 ms at the pipe's 17.7e12 a second),
// 2048^2 303 -> 57 us a call of which the kernel is 12; near field of 200k
// points x 2 rhs in 3-D 2.08 -> 0.36 ms.
#include <algorithm>
#include <type_traits>

#include "fmm_stages.cuh"
#include "fmma_internal.cuh"
#include "kernels.cuh"
#include "solver.cuh"

namespace fmma_b200 {

namespace {

constexpr int kNearThreads = 256;
constexpr int kNearWarps = kNearThreads / 32;
constexpr int kNearTile = 32;  // sources staged per step of a warp

// Targets of the next chunk of `rem` remaining ones and the lanes (a power of
// two) it occupies: 32, or all of them when they fill three quarters of the
// next power of two, else the largest power of two below.  The 32 / lanes
// groups of lanes share the chunk's sources.
__device__ __forceinline__ int chunk_of(int rem, int* lanes) {
  int np = 1;
  while (np < rem && np < 32) np <<= 1;
  if (rem >= np) {
    *lanes = np;
    return np;
  }
  if (4 * rem >= 3 * np) {
    *lanes = np;
    return rem;
  }
  *lanes = np >> 1;
  return np >> 1;
}

struct NearArgs {
  const int* row_box;
  int64_t nrow;
  const int* near;
  int nnear;
  const int *tb, *te, *sb, *se;
  const double* tx;
  int64_t nt;
  const double* sx;
  int64_t ns;
  const double* ws;
  int R;
  double p0;
  const double *pot, *potg;
  const int* perm_t;
  int slots, wpu;  // units per row; warps per unit (1 or kNearWarps / 2)
};

// The sums of sorted target t from right-hand side r0, and its gradient, with
// the far field's added, to the caller's order.
template <int D, int RB, bool GRAD, typename T>
__device__ __forceinline__ void near_store(const NearArgs& a, const double* acc, int r0, int t, T* __restrict__ out,
                                           double* __restrict__ grad) {
  const int64_t ot = a.perm_t[t];
#pragma unroll
  for (int r = 0; r < RB; ++r)
    if (r0 + r < a.R && out)
      out[(int64_t)(r0 + r) * a.nt + ot] = (T)(acc[r] + (a.pot ? a.pot[(int64_t)(r0 + r) * a.nt + t] : 0.0));
  if constexpr (GRAD) {
#pragma unroll
    for (int q = 0; q < D; ++q)
      grad[((int64_t)r0 * a.nt + ot) * D + q] =
          acc[RB + q] + (a.potg ? a.potg[((int64_t)r0 * a.nt + t) * D + q] : 0.0);
  }
}

// A unit is every `slots`-th target chunk of a leaf row, taken by wpu warps
// that share its sources tile by tile.  The 3^d neighbour leaves form one list
// of sources (lane k holds neighbour k's range and the prefix sum of the
// counts), so tiles are full across neighbour boundaries.
// GRAD: also grad[r][t][q] = potg + sum w d f / d x_q (RB = 1).
template <int KID, int D, int RB, bool GRAD, typename T>
__global__ void __launch_bounds__(kNearThreads, GRAD || RB > 2 ? 2 : 3) k_near64(const NearArgs a, T* __restrict__ out,
                                                                       double* __restrict__ grad) {
  constexpr int U = 4, NA = RB + (GRAD ? D : 0);
  __shared__ double s_y[kNearWarps][D][kNearTile];
  __shared__ double s_w[kNearWarps][RB][kNearTile];
  __shared__ double s_red[kNearWarps][NA][32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int wpu = a.wpu, upb = kNearWarps / wpu, unit_in = warp / wpu, wu = warp - unit_in * wpu;
  const double p0 = a.p0, ip = kinv<KID>(p0);
  const int64_t nunits = a.nrow * a.slots;
  for (int64_t unit = (int64_t)blockIdx.x * upb + unit_in; unit < nunits; unit += (int64_t)gridDim.x * upb) {
    const int64_t row = unit / a.slots;
    const int slot = (int)(unit - row * a.slots);
    const int b = a.row_box[row];
    const int t0 = a.tb[b], t1 = a.te[b];
    if (t0 >= t1) continue;
    int nb_box = -1, nb_cnt = 0, nb_first = 0;
    if (lane < a.nnear) {
      nb_box = a.near[row * a.nnear + lane];
      if (nb_box >= 0) {
        nb_first = a.sb[nb_box];
        nb_cnt = a.se[nb_box] - nb_first;
      }
    }
    int nb_end = nb_cnt;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int v = __shfl_up_sync(0xffffffffu, nb_end, o);
      if (lane >= o) nb_end += v;
    }
    const int total = __shfl_sync(0xffffffffu, nb_end, 31);
    const int nb_base = nb_first - (nb_end - nb_cnt);  // source of list entry e: nb_base + e
    int k = 0, lanes = 32;
    for (int tc = t0, cnt = 0; tc < t1; tc += cnt, ++k) {
      cnt = chunk_of(t1 - tc, &lanes);
      if (k % a.slots != slot) continue;
      const int G = 32 / lanes, ti = lane & (lanes - 1), g = lane / lanes;
      const bool tv = ti < cnt;
      double x[D];
#pragma unroll
      for (int q = 0; q < D; ++q) x[q] = tv ? a.tx[(int64_t)q * a.nt + tc + ti] : 0.0;
      for (int r0 = 0; r0 < a.R; r0 += RB) {
        double acc[NA];
#pragma unroll
        for (int r = 0; r < NA; ++r) acc[r] = 0.0;
        // this lane's source of the tile at e0, a tile ahead of its use
        double yn[D], wn[RB];
        auto fetch = [&](int e0) {
          const int e = e0 + lane;
          int n = 0;  // the first neighbour whose range ends beyond e
#pragma unroll
          for (int step = 16; step > 0; step >>= 1)
            if (__shfl_sync(0xffffffffu, nb_end, n + step - 1) <= e) n += step;
          const int j = __shfl_sync(0xffffffffu, nb_base, n & 31) + e;
          const bool ok = e < total;
#pragma unroll
          for (int q = 0; q < D; ++q) yn[q] = ok ? a.sx[(int64_t)q * a.ns + j] : 0.0;
#pragma unroll
          for (int r = 0; r < RB; ++r)
            wn[r] = ok && r0 + r < a.R ? a.ws[(int64_t)(r0 + r) * a.ns + j] : 0.0;
        };
        const int stride = kNearTile * wpu;
        int e0 = wu * kNearTile;
        if (e0 < total) fetch(e0);
        for (; e0 < total; e0 += stride) {
          __syncwarp();
#pragma unroll
          for (int q = 0; q < D; ++q) s_y[warp][q][lane] = yn[q];
#pragma unroll
          for (int r = 0; r < RB; ++r) s_w[warp][r][lane] = wn[r];
          __syncwarp();
          if (e0 + stride < total) fetch(e0 + stride);
          const int m = min(kNearTile, total - e0);
          auto pairs = [&](int i0, auto u_c) {  // list entries i0 + G u, u < UU
            constexpr int UU = decltype(u_c)::value;
            double r2[UU], s[UU], f[UU], c[UU], t[UU][D];
#pragma unroll
            for (int u = 0; u < UU; ++u) {
              double y[D];
#pragma unroll
              for (int q = 0; q < D; ++q) y[q] = s_y[warp][q][i0 + G * u];
              kparts<KID, D>(x, y, r2[u], s[u]);
              if constexpr (GRAD) {
#pragma unroll
                for (int q = 0; q < D; ++q) t[u][q] = x[q] - y[q];
              }
            }
            if constexpr (!GRAD) {
              kvals<KID, UU>(r2, s, p0, ip, f);
            } else if constexpr (KID == FMMA_KERNEL_INV_DIFF || KID == FMMA_KERNEL_SUM_OVER_R2 ||
                                 KID == FMMA_KERNEL_SUM2_OVER_R2) {
              kvals<KID, UU>(r2, s, p0, ip, f);
            } else {
              kvals_grad<KID, UU>(r2, p0, ip, f, c);
            }
#pragma unroll
            for (int u = 0; u < UU; ++u) {
#pragma unroll
              for (int r = 0; r < RB; ++r) acc[r] = fma(s_w[warp][r][i0 + G * u], f[u], acc[r]);
              if constexpr (GRAD) {
                const double w = s_w[warp][0][i0 + G * u];
                if constexpr (KID == FMMA_KERNEL_INV_DIFF) {
                  acc[RB] += w * (t[u][0] != 0.0 ? -1.0 / (t[u][0] * t[u][0]) : 0.0);
                } else if constexpr (KID == FMMA_KERNEL_SUM_OVER_R2) {
#pragma unroll
                  for (int q = 0; q < D; ++q)
                    acc[RB + q] +=
                        w * (r2[u] > 0.0 ? 1.0 / r2[u] - 2.0 * s[u] * t[u][q] / (r2[u] * r2[u]) : 0.0);
                } else if constexpr (KID != FMMA_KERNEL_SUM2_OVER_R2) {  // that one has no gradient: zero
                  const double wc = w * c[u];
#pragma unroll
                  for (int q = 0; q < D; ++q) acc[RB + q] = fma(wc, t[u][q], acc[RB + q]);
                }
              }
            }
          };
          int i = g;
          for (; i + (U - 1) * G < m; i += U * G) pairs(i, std::integral_constant<int, U>{});
          for (; i < m; i += G) pairs(i, std::integral_constant<int, 1>{});
        }
        // over the lane groups, then over the unit's warps
#pragma unroll
        for (int r = 0; r < NA; ++r)
          for (int o = lanes; o < 32; o <<= 1) acc[r] += __shfl_xor_sync(0xffffffffu, acc[r], o);
        if (wpu > 1) {
#pragma unroll
          for (int r = 0; r < NA; ++r) s_red[warp][r][lane] = acc[r];
          asm volatile("bar.sync %0, %1;" ::"r"(1 + unit_in), "r"(wpu * 32) : "memory");
          if (wu == 0) {
#pragma unroll
            for (int r = 0; r < NA; ++r)
              for (int w = 1; w < wpu; ++w) acc[r] += s_red[warp + w][r][lane];
          }
          asm volatile("bar.sync %0, %1;" ::"r"(1 + unit_in), "r"(wpu * 32) : "memory");
        }
        if (wu == 0 && g == 0 && tv) near_store<D, RB, GRAD>(a, acc, r0, tc + ti, out, grad);
      }
    }
  }
}

// Sparse leaves in 1-D and 2-D: a warp per leaf row, its lanes split as
// (target, source subset), that walks the row's few neighbours in global
// memory.  With a handful of sources in all, the latency of the row's loads is
// what counts, and this form keeps twice the warps of k_near64 and has no list
// to make: against it, us, 262,144 clustered points in 1-D 95 -> 46 (3 rhs 211
// -> 117), in 2-D 158 -> 97 (gradient 291 -> 135), 20,000 uniform points in 2-D
// 25 -> 19.  From about five points a leaf in 1-D and two in 2-D k_near64 is as
// fast or faster (10 points, 1-D, 256 leaves x 4 rhs 15 against 27), and in 3-D,
// with up to 27 neighbours, at one point a leaf already.
template <int KID, int D, int RB, bool GRAD, typename T>
__global__ void __launch_bounds__(kNearThreads) k_near64_sparse(const NearArgs a, T* __restrict__ out,
                                                                double* __restrict__ grad) {
  constexpr int NA = RB + (GRAD ? D : 0);
  const int lane = threadIdx.x & 31;
  const int64_t nw = ((int64_t)gridDim.x * kNearThreads) >> 5;
  for (int64_t row = ((int64_t)blockIdx.x * kNearThreads + threadIdx.x) >> 5; row < a.nrow; row += nw) {
    const int b = a.row_box[row];
    const int t0 = a.tb[b], t1 = a.te[b];
    for (int tc = t0; tc < t1; tc += 32) {
      const int cnt = min(32, t1 - tc);
      int lanes = 1;
      while (lanes < cnt) lanes <<= 1;
      const int G = 32 / lanes, ti = lane & (lanes - 1), g = lane / lanes;
      const bool tv = ti < cnt;
      double x[D];
#pragma unroll
      for (int q = 0; q < D; ++q) x[q] = tv ? a.tx[(int64_t)q * a.nt + tc + ti] : 0.0;
      for (int r0 = 0; r0 < a.R; r0 += RB) {
        double acc[NA];
#pragma unroll
        for (int r = 0; r < NA; ++r) acc[r] = 0.0;
        if (tv) {
          for (int k = 0; k < a.nnear; ++k) {
            const int s = a.near[row * a.nnear + k];
            if (s < 0) continue;
            const int j1 = a.se[s];
            for (int j = a.sb[s] + g; j < j1; j += G) {
              double y[D];
#pragma unroll
              for (int q = 0; q < D; ++q) y[q] = a.sx[(int64_t)q * a.ns + j];
              const double f = keval<KID, D>(x, y, a.p0);
#pragma unroll
              for (int r = 0; r < RB; ++r)
                if (r0 + r < a.R) acc[r] += a.ws[(int64_t)(r0 + r) * a.ns + j] * f;
              if constexpr (GRAD) {
                double gr[D];
                kgrad_x<KID, D>(x, y, a.p0, gr);
                const double w = a.ws[(int64_t)r0 * a.ns + j];
#pragma unroll
                for (int q = 0; q < D; ++q) acc[RB + q] += w * gr[q];
              }
            }
          }
        }
#pragma unroll
        for (int r = 0; r < NA; ++r)
          for (int o = lanes; o < 32; o <<= 1) acc[r] += __shfl_xor_sync(0xffffffffu, acc[r], o);
        if (g == 0 && tv) near_store<D, RB, GRAD>(a, acc, r0, tc + ti, out, grad);
      }
    }
  }
}

// Where the sparse form runs: fewer than 16 sources in a mean row's list, all
// of whose neighbours are taken to exist.
bool near_sparse(const NearArgs& a, int d, int64_t nbox) {
  return d < 3 && a.ns * a.nnear < 16 * nbox;
}

// The two cuts of the near field.  slots: a row's chunks of 32 targets, so
// that every chunk of a mean row is a unit.  wpu: four warps share a unit's
// sources, tile by tile, where the lists are long enough for the reduction over
// them: from 48 sources when the units fill less than a quarter of the warps
// the GPU holds (24 an SM), from 192 when less than all, from 400 below eight
// waves.  That is in pairs of 1/r; a pair of another kernel counts by what it
// costs against it (log r 4, the Gaussian 3, a root or division 2.5), but the
// last line takes 192 sources, six tiles, at least.  us with one warp and with four, 1/r, uniform points, one
// rhs: 96 units x 240 sources 23 and 13, 128 x 30 both 9; 2,048 x 360 40 and 36,
// x 60 13 and 21; 8,192 x 1,080 284 and 232, x 60 30 and 56; 32,768 x 30 54 and
// 150 (four rhs 118 and 365).  The list's length is estimated from the mean
// leaf, all of whose neighbours are taken to exist.
NearArgs near_args(fmma_ctx* ctx, int nnear, const Tree& tr, const double* tx, const double* sx, const double* ws,
                   int R, const double* pot, const double* potg) {
  const Level& Lf = tr.lev[0];
  NearArgs a{tr.near_row_box, tr.nnear_rows, tr.near, nnear, Lf.tb, Lf.te, Lf.sb, Lf.se, tx, tr.nt, sx, tr.ns, ws, R,
             ctx->p0, pot, potg, tr.perm_t, 1, 1};
  const int64_t mean = (tr.nt + tr.nnear_rows - 1) / tr.nnear_rows;
  a.slots = (int)std::max<int64_t>(1, std::min<int64_t>(64, (mean + 31) / 32));
  const int64_t units = a.nrow * a.slots, warps = (int64_t)ctx->sm_count * 24;
  const int k = ctx->kernel_id;
  const int cost = k == FMMA_KERNEL_INV_R || k == FMMA_KERNEL_INV_R_SAFE
                       ? 10
                       : (k == FMMA_KERNEL_LOG_R ? 40 : (k == FMMA_KERNEL_GAUSSIAN ? 30 : 25));
  const int64_t list = tr.ns * nnear / std::max<int64_t>(1, Lf.nbox), work = list * cost / 10;  // of a unit
  const int64_t most = work >= 400 && list >= 192 ? 8 * warps : (work >= 192 ? warps : (work >= 48 ? warps / 4 : 0));
  a.wpu = units < most ? kNearWarps / 2 : 1;
  return a;
}

unsigned near_grid(fmma_ctx* ctx, const NearArgs& a) {
  const int upb = kNearWarps / a.wpu;
  return (unsigned)std::max<int64_t>(1, std::min<int64_t>((a.nrow * a.slots + upb - 1) / upb,
                                                          (int64_t)ctx->sm_count * 64));
}

template <typename T>
struct NearLaunch {
  template <int KID, int D>
  static void run(fmma_ctx* ctx, const Tree& tr, const double* tx, const double* sx, const double* ws, int R,
                  const double* pot, T* out) {
    const NearArgs a = near_args(ctx, D == 1 ? 3 : (D == 2 ? 9 : 27), tr, tx, sx, ws, R, pot, nullptr);
    if constexpr (D < 3) {
      if (near_sparse(a, D, tr.lev[0].nbox)) {
        const unsigned g = grid_for(a.nrow * 32, kNearThreads, (int64_t)ctx->sm_count * 16);
        if (R == 1) FMMA_LAUNCH(ctx, (k_near64_sparse<KID, D, 1, false, T>), g, kNearThreads, 0, a, out, nullptr);
        else if (R <= 4) FMMA_LAUNCH(ctx, (k_near64_sparse<KID, D, 4, false, T>), g, kNearThreads, 0, a, out, nullptr);
        else FMMA_LAUNCH(ctx, (k_near64_sparse<KID, D, 8, false, T>), g, kNearThreads, 0, a, out, nullptr);
        return;
      }
    }
    const unsigned g = near_grid(ctx, a);
    if (R == 1) FMMA_LAUNCH(ctx, (k_near64<KID, D, 1, false, T>), g, kNearThreads, 0, a, out, nullptr);
    else if (R == 2) FMMA_LAUNCH(ctx, (k_near64<KID, D, 2, false, T>), g, kNearThreads, 0, a, out, nullptr);
    else if (R <= 4) FMMA_LAUNCH(ctx, (k_near64<KID, D, 4, false, T>), g, kNearThreads, 0, a, out, nullptr);
    else FMMA_LAUNCH(ctx, (k_near64<KID, D, 8, false, T>), g, kNearThreads, 0, a, out, nullptr);
  }
};

struct NearGradLaunch {
  template <int KID, int D>
  static void run(fmma_ctx* ctx, const Tree& tr, const double* tx, const double* sx, const double* ws, int R,
                  const double* pot, const double* potg, double* out, double* grad) {
    const NearArgs a = near_args(ctx, D == 1 ? 3 : (D == 2 ? 9 : 27), tr, tx, sx, ws, R, pot, potg);
    if constexpr (D < 3) {
      if (near_sparse(a, D, tr.lev[0].nbox)) {
        FMMA_LAUNCH(ctx, (k_near64_sparse<KID, D, 1, true, double>),
                    grid_for(a.nrow * 32, kNearThreads, (int64_t)ctx->sm_count * 16), kNearThreads, 0, a, out, grad);
        return;
      }
    }
    FMMA_LAUNCH(ctx, (k_near64<KID, D, 1, true, double>), near_grid(ctx, a), kNearThreads, 0, a, out, grad);
  }
};

// ---------------------------------------------------------------------------
// exact
// ---------------------------------------------------------------------------
constexpr int kExThreads = 128;
constexpr int kExTargets = 2;  // targets per thread
constexpr int kExTile = 128;   // sources staged per step

// ans[r][i] = sum_j w[r][j] f(tgt[rows ? rows[i] : i], src[j]), RB right-hand
// sides per pass.  Block (x, y) takes the targets of tile x and the sources of
// range y.  With several ranges its sums go to part[(y * R + r) * nt + i], and
// the tile's last block to finish (done[x], back to zero when it leaves) adds
// the ranges in order: no second launch.
template <int KID, int D, int RB, typename T>
__global__ void __launch_bounds__(kExThreads) k_exact(const T* __restrict__ tgt, int64_t nt,
                                                      const int64_t* __restrict__ rows, const T* __restrict__ src,
                                                      int64_t ns, const T* __restrict__ w, int R, double p0,
                                                      int64_t range, double* part, unsigned* done,
                                                      T* __restrict__ ans) {
  constexpr int U = 4 / kExTargets;
  __shared__ double sy[D][kExTile];
  __shared__ double sw[RB][kExTile];
  const double ip = kinv<KID>(p0);
  const int64_t j_begin = (int64_t)blockIdx.y * range, j_end = min(ns, j_begin + range);
  int64_t ti[kExTargets];
  double x[kExTargets][D];
#pragma unroll
  for (int k = 0; k < kExTargets; ++k) {
    ti[k] = ((int64_t)blockIdx.x * kExTargets + k) * kExThreads + threadIdx.x;
    const int64_t t = ti[k] < nt ? (rows ? rows[ti[k]] : ti[k]) : -1;
#pragma unroll
    for (int q = 0; q < D; ++q) x[k][q] = t >= 0 ? (double)tgt[t * D + q] : 0.0;
  }
  for (int r0 = 0; r0 < R; r0 += RB) {
    double acc[kExTargets][RB];
#pragma unroll
    for (int k = 0; k < kExTargets; ++k)
#pragma unroll
      for (int r = 0; r < RB; ++r) acc[k][r] = 0.0;
    for (int64_t j0 = j_begin; j0 < j_end; j0 += kExTile) {
      const int cnt = (int)min((int64_t)kExTile, j_end - j0);
      __syncthreads();
      if ((int)threadIdx.x < cnt) {
        const int64_t j = j0 + threadIdx.x;
#pragma unroll
        for (int q = 0; q < D; ++q) sy[q][threadIdx.x] = (double)src[j * D + q];
#pragma unroll
        for (int r = 0; r < RB; ++r)
          sw[r][threadIdx.x] = r0 + r < R ? (w ? (double)w[(int64_t)(r0 + r) * ns + j] : 1.0) : 0.0;
      }
      __syncthreads();
      auto pairs = [&](int i, auto u_c) {  // sources i .. i + UU - 1 with both targets
        constexpr int UU = decltype(u_c)::value, NP = UU * kExTargets;
        double r2[NP], s[NP], f[NP];
#pragma unroll
        for (int u = 0; u < UU; ++u) {
          double y[D];
#pragma unroll
          for (int q = 0; q < D; ++q) y[q] = sy[q][i + u];
#pragma unroll
          for (int k = 0; k < kExTargets; ++k) kparts<KID, D>(x[k], y, r2[u * kExTargets + k], s[u * kExTargets + k]);
        }
        kvals<KID, NP>(r2, s, p0, ip, f);
#pragma unroll
        for (int u = 0; u < UU; ++u)
#pragma unroll
          for (int r = 0; r < RB; ++r)
#pragma unroll
            for (int k = 0; k < kExTargets; ++k)
              acc[k][r] = fma(sw[r][i + u], f[u * kExTargets + k], acc[k][r]);
      };
      int i = 0;
#pragma unroll 2
      for (; i + U <= cnt; i += U) pairs(i, std::integral_constant<int, U>{});
      for (; i < cnt; ++i) pairs(i, std::integral_constant<int, 1>{});
    }
#pragma unroll
    for (int k = 0; k < kExTargets; ++k)
      if (ti[k] < nt)
#pragma unroll
        for (int r = 0; r < RB; ++r)
          if (r0 + r < R) {
            if (gridDim.y == 1) ans[(int64_t)(r0 + r) * nt + ti[k]] = (T)acc[k][r];
            else part[((int64_t)blockIdx.y * R + r0 + r) * nt + ti[k]] = acc[k][r];
          }
  }
  if (gridDim.y == 1) return;
  __shared__ bool s_last;
  __threadfence();  // this thread's sums before the count
  __syncthreads();
  if (threadIdx.x == 0) s_last = atomicInc(&done[blockIdx.x], gridDim.y - 1) == gridDim.y - 1;
  __syncthreads();
  if (!s_last) return;
  __threadfence();
  for (int r = 0; r < R; ++r)
#pragma unroll
    for (int k = 0; k < kExTargets; ++k)
      if (ti[k] < nt) {
        const double* p = part + (int64_t)r * nt + ti[k];
        const int64_t step = (int64_t)R * nt;
        double sum = 0.0;
        int y = 0;
        for (; y + 8 <= (int)gridDim.y; y += 8) {
          double v[8];
#pragma unroll
          for (int u = 0; u < 8; ++u) v[u] = __ldcg(p + (y + u) * step);
#pragma unroll
          for (int u = 0; u < 8; ++u) sum += v[u];
        }
        for (; y < (int)gridDim.y; ++y) sum += __ldcg(p + y * step);
        ans[(int64_t)r * nt + ti[k]] = (T)sum;
      }
}

template <typename T>
struct ExactLaunch {
  template <int KID, int D>
  static void run(fmma_ctx* ctx, const T* tgt, int64_t nt, const int64_t* rows, const T* src, int64_t ns, const T* w,
                  int R, double p0, T* ans) {
    // Source ranges: the cut that wastes least of its last wave (four blocks
    // an SM), where a block's set-up and partial sums cost about as much as 32
    // sources; a range holds at least 64.
    const int64_t tiles = (nt + kExThreads * kExTargets - 1) / (kExThreads * kExTargets);
    const int64_t cap = (int64_t)ctx->sm_count * 4;
    const int64_t most = std::max<int64_t>(1, std::min<int64_t>({(ns + 63) / 64, 8 * cap / tiles + 1, 1024}));
    int64_t best = 1;
    double best_t = 0.0;
    for (int64_t s = 1; s <= most; ++s) {
      const double t = (double)((tiles * s + cap - 1) / cap) * (1.0 / (double)s + 32.0 / (double)ns);
      if (s == 1 || t < best_t) {
        best = s;
        best_t = t;
      }
    }
    int64_t range = (ns + best - 1) / best;
    int nranges = (int)((ns + range - 1) / range);
    double* part = nullptr;
    unsigned* done = nullptr;
    if (nranges > 1) {
      part = static_cast<double*>(ctx_buf_try(ctx, "exact_part", sizeof(double) * (size_t)nranges * R * nt));
      const size_t had = ctx->bufs["exact_done"].bytes;
      if (part) done = static_cast<unsigned*>(ctx_buf_try(ctx, "exact_done", sizeof(unsigned) * (size_t)tiles));
      if (done && ctx->bufs["exact_done"].bytes != had)  // a new buffer: every launch leaves it at zero
        FMMA_CHECK_CUDA(cudaMemsetAsync(done, 0, ctx->bufs["exact_done"].bytes, ctx->stream));
      if (!done) {  // no scratch to be had: one range, which needs none
        range = ns;
        nranges = 1;
      }
    }
    const dim3 grid((unsigned)tiles, (unsigned)nranges);
    if (R == 1)
      FMMA_LAUNCH(ctx, (k_exact<KID, D, 1, T>), grid, kExThreads, 0, tgt, nt, rows, src, ns, w, R, p0, range, part,
                  done, ans);
    else
      FMMA_LAUNCH(ctx, (k_exact<KID, D, 4, T>), grid, kExThreads, 0, tgt, nt, rows, src, ns, w, R, p0, range, part,
                  done, ans);
  }
};

}  // namespace

template <typename T>
void near_field_f64(fmma_ctx* ctx, int d, int R, const Tree& tr, const double* tx, const double* sx, const double* ws,
                    const double* pot, T* ans) {
  if (tr.nnear_rows == 0) return;
  if (ctx->kernel_id == kUserKernel) {
    const Level& Lf = tr.lev[0];
    fmma_user_launch ua{};
    ua.what = FMMA_USER_P2P;
    ua.dim = d;
    ua.nrhs = R;
    ua.nrow = tr.nnear_rows;
    ua.row_box = tr.near_row_box;
    ua.near = tr.near;
    ua.nnear = d == 1 ? 3 : (d == 2 ? 9 : 27);
    ua.tb = Lf.tb;
    ua.te = Lf.te;
    ua.sb = Lf.sb;
    ua.se = Lf.se;
    ua.tx = tx;
    ua.nt = tr.nt;
    ua.sx = sx;
    ua.ns = tr.ns;
    ua.ws = ws;
    ua.pot = pot;
    ua.perm_t = tr.perm_t;
    ua.out = ans;
    ua.out_f32 = sizeof(T) == 4;
    call_user_hook(ctx, ua);
  } else {
    dispatch_kernel<NearLaunch<T>>(ctx->kernel_id, d, ctx, tr, tx, sx, ws, R, pot, ans);
  }
}

void near_field_grad_f64(fmma_ctx* ctx, int d, int R, const Tree& tr, const double* tx, const double* sx,
                         const double* ws, const double* pot, const double* potg, double* ans, double* grad) {
  if (tr.nnear_rows == 0) return;
  FMMA_REQUIRE(ctx->kernel_id != kUserKernel, "gradients need a built-in kernel");
  dispatch_kernel<NearGradLaunch>(ctx->kernel_id, d, ctx, tr, tx, sx, ws, R, pot, potg, ans, grad);
}

template <typename T>
void solve_exact(fmma_ctx* ctx, int dim, int64_t nt, const T* tgt, int64_t ns, const T* src, int R, const T* w,
                 T* ans, const int64_t* rows) {
  if (nt == 0) return;
  if (ns == 0) {
    FMMA_CHECK_CUDA(cudaMemsetAsync(ans, 0, sizeof(T) * (size_t)(nt * R), ctx->stream));
    return;
  }
  if (ctx->kernel_id == kUserKernel) {
    fmma_user_launch a{};
    a.what = FMMA_USER_EXACT;
    a.dim = dim;
    a.nrhs = R;
    a.nt = nt;
    a.ns = ns;
    a.tgt = tgt;
    a.src = src;
    a.w = w;
    a.rows = rows;
    a.out = ans;
    a.out_f32 = sizeof(T) == 4;
    call_user_hook(ctx, a);
    return;
  }
  dispatch_kernel<ExactLaunch<T>>(ctx->kernel_id, dim, ctx, tgt, nt, rows, src, ns, w, R, ctx->p0, ans);
}

template void near_field_f64<double>(fmma_ctx*, int, int, const Tree&, const double*, const double*, const double*,
                                     const double*, double*);
template void near_field_f64<float>(fmma_ctx*, int, int, const Tree&, const double*, const double*, const double*,
                                    const double*, float*);
template void solve_exact<double>(fmma_ctx*, int, int64_t, const double*, int64_t, const double*, int, const double*,
                                  double*, const int64_t*);
template void solve_exact<float>(fmma_ctx*, int, int64_t, const float*, int64_t, const float*, int, const float*,
                                 float*, const int64_t*);

}  // namespace fmma_b200
