// p2m.cu — P2M at the leaves for 2 to 8 nodes per dimension
// (src/fmm_core.cpp:269-280): Wm[b][r][k] = sum_s w_rs prod_q S_n(x_kq, rel_sq).
//
// A warp walks a run of consecutive leaves, whose sources are consecutive, in
// tiles of 32 sources.  Lanes over sources: each computes the d n factors of
// its source (T_j by the recurrence once, then n sums of n - 1 terms with the
// T_j(x_k) as constant operands) into shared memory.  Lanes over coefficients:
// lane c owns the coefficients of the node pair (k_0, k_1) = c, reads that
// pair's two factors of a source and sums over the third dimension's factors,
// which all lanes share.  What bounds it is instruction issue (FP64 pipe and
// shared loads next): about 30 instructions a source at 6 nodes in 3-D against
// about 110 when the factors were computed by one lane each per source and
// gathered by shuffles (a shuffle moves 4 bytes a lane).  With 16 or fewer
// node pairs the warp takes two or four sources at a time in lane groups.
// P2M stage, us: 1 rhs, 2-D 1M 6 nodes 281 -> 48, 2-D 131k 4 nodes 94 -> 10, 3-D
// 333k 5 nodes 172 -> 25, 3-D 4M clustered 6 nodes 2220 -> 860; 16 rhs, 19M
// sources in 2-D, 5 nodes 3730 -> 2630.
#include "fmm_stages.cuh"
#include "fmma_internal.cuh"

namespace fmma_b200 {

namespace {

constexpr int kTileWarps = 4;
constexpr int kTileMaxLeaves = 32;  // leaves of a warp's run: their ranges sit in the lanes
constexpr int kFRow = 33;           // doubles between factor rows: distinct banks for the rows of a source

template <int D, int N>
struct P2MShape {
  static constexpr int C = D == 1 ? N : N * N;        // node pairs (single nodes in 1-D)
  static constexpr int SLOTS = (C + 31) / 32;         // per lane
  static constexpr int GL = C > 16 ? 32 : (C > 8 ? 16 : 8);  // lanes of a group
  static constexpr int K2 = D == 3 ? N : 1;
};

template <int D, int N, int RB>
__global__ void __launch_bounds__(32 * kTileWarps) k_p2m_tile(
    const uint64_t* __restrict__ key, const int* __restrict__ sb, const int* __restrict__ se, int64_t nbox, int run,
    const double* __restrict__ sx, int64_t ns, const double* __restrict__ ws, int R, const Cube* __restrict__ cubes,
    const int* __restrict__ depth, bool isf, int Kpad, const __grid_constant__ NodeTable<N> tn,
    double* __restrict__ Wm, bool many, int grid_n) {
  using S = P2MShape<D, N>;
  constexpr int SLOTS = S::SLOTS, GL = S::GL, G = 32 / GL, K2 = S::K2, C = S::C;
  constexpr int P = C * K2, WROW = RB == 1 ? 1 : RB + 2;  // weights of a source: rows of 16-byte multiples
  __shared__ __align__(16) double s_w[kTileWarps][32 * WROW];
  __shared__ double s_f[kTileWarps][D * N * kFRow];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  double* const F = s_f[warp];
  double* const Ws = s_w[warp];
  const int grp = lane / GL, gl = lane & (GL - 1);
  int row0[SLOTS], row1[SLOTS];  // factor rows of the lane's node pairs
#pragma unroll
  for (int s = 0; s < SLOTS; ++s) {
    const int c = min(gl + 32 * s, C - 1);
    row0[s] = (D == 1 ? c : c / N) * kFRow;
    row1[s] = (N + c % N) * kFRow;
  }
  const int64_t nw = (int64_t)gridDim.x * kTileWarps;
  const int64_t nrun = (nbox + run - 1) / run;
  for (int64_t u = (int64_t)blockIdx.x * kTileWarps + warp; u < nrun; u += nw) {
    const int64_t b0 = u * run;
    const int nb = (int)min((int64_t)run, nbox - b0);
    const int my_sb = lane < nb ? sb[b0 + lane] : 0, my_se = lane < nb ? se[b0 + lane] : 0;
    // one problem: its cube and leaf width once
    const int pid0 = many || grid_n > 0 ? 0 : key_pid(key[b0]);
    const int Nl0 = grid_n > 0 ? grid_n : (many ? 1 : 1 << (depth[pid0] - 1));
    const LeafWidth lw0 = leaf_width(cubes[pid0], Nl0, isf);
    for (int r0 = 0; r0 < R; r0 += RB) {
      int t0 = 0, t1 = 0;  // sources of the tile in shared memory
      for (int l = 0; l < nb; ++l) {
        const int s0 = __shfl_sync(0xffffffffu, my_sb, l), s1 = __shfl_sync(0xffffffffu, my_se, l);
        if (s1 <= s0) continue;
        double acc[SLOTS][K2][RB];
#pragma unroll
        for (int s = 0; s < SLOTS; ++s)
#pragma unroll
          for (int k = 0; k < K2; ++k)
#pragma unroll
            for (int r = 0; r < RB; ++r) acc[s][k][r] = 0.0;
        for (int p = s0; p < s1;) {
          if (p < t0 || p >= t1) {  // the next tile: sources p .. p + 31 of the run's leaves
            __syncwarp();           // every lane is done with the last one
            t0 = p;
            const int last = __shfl_sync(0xffffffffu, my_se, nb - 1);
            t1 = min(p + 32, grid_n > 0 ? s1 : last);
            const int i = p + lane;
            int pid = pid0, Nl = Nl0;
            if (many) {  // the source's leaf: the first whose range ends beyond it
              int n = 0;
#pragma unroll
              for (int step = 16; step > 0; step >>= 1) {
                const int e = __shfl_sync(0xffffffffu, my_se, n + step - 1);
                if (n + step <= nb && e <= i) n += step;
              }
              pid = key_pid(key[b0 + min(n, nb - 1)]);
              Nl = 1 << (depth[pid] - 1);
            }
            if (i < t1) {
              const Cube& c = cubes[pid];
              const LeafWidth lw = many ? leaf_width(c, Nl, isf) : lw0;
#pragma unroll
              for (int q = 0; q < D; ++q) {
                const double y = point_rel(sx[(int64_t)q * ns + i], c, lw, q, Nl, isf);
                double T[N];
                T[0] = 1.0;
                if (N > 1) T[1] = y;
#pragma unroll
                for (int j = 2; j < N; ++j) T[j] = 2.0 * y * T[j - 1] - T[j - 2];
#pragma unroll
                for (int k = 0; k < N; ++k) {
                  double s = 0.0;
#pragma unroll
                  for (int j = 1; j < N; ++j) s += tn.T[k * N + j] * T[j];
                  F[(q * N + k) * kFRow + lane] = 1.0 / N + 2.0 * (1.0 / N) * s;
                }
              }
              if constexpr (RB == 1) Ws[lane] = ws[(int64_t)r0 * ns + i];
              else {
#pragma unroll
                for (int r = 0; r < RB; ++r) Ws[lane * WROW + r] = r0 + r < R ? ws[(int64_t)(r0 + r) * ns + i] : 0.0;
              }
            }
            __syncwarp();
          }
          const int e = min(s1, t1) - t0;
          for (int i = p - t0 + grp; i < e; i += G) {
            double w[RB], f2[K2];
            if constexpr (RB == 1) w[0] = Ws[i];
            else {
#pragma unroll
              for (int r = 0; r < RB; r += 2) {
                const double2 v = *reinterpret_cast<const double2*>(Ws + i * WROW + r);
                w[r] = v.x;
                w[r + (RB > 1 ? 1 : 0)] = v.y;
              }
            }
            if constexpr (D == 3) {
#pragma unroll
              for (int k = 0; k < K2; ++k) f2[k] = F[(2 * N + k) * kFRow + i];
            }
#pragma unroll
            for (int s = 0; s < SLOTS; ++s) {
              double f = F[row0[s] + i];
              if constexpr (D >= 2) f *= F[row1[s] + i];
              if constexpr (D == 3 && RB == 1) {
                const double g = w[0] * f;
#pragma unroll
                for (int k = 0; k < K2; ++k) acc[s][k][0] = fma(g, f2[k], acc[s][k][0]);
              } else {
#pragma unroll
                for (int k = 0; k < K2; ++k) {
                  const double g = D == 3 ? f * f2[D == 3 ? k : 0] : f;
#pragma unroll
                  for (int r = 0; r < RB; ++r) acc[s][k][r] = fma(w[r], g, acc[s][k][r]);
                }
              }
            }
          }
          p = t0 + e;
        }
        // over the lane groups, then the leaf's rows
        if constexpr (G > 1) {
#pragma unroll
          for (int k = 0; k < K2; ++k)
#pragma unroll
            for (int r = 0; r < RB; ++r)
#pragma unroll
              for (int o = GL; o < 32; o <<= 1) acc[0][k][r] += __shfl_xor_sync(0xffffffffu, acc[0][k][r], o);
        }
#pragma unroll
        for (int r = 0; r < RB; ++r) {
          if (r0 + r >= R) break;
          double* dst = Wm + ((b0 + l) * R + r0 + r) * Kpad;
          if (grp == 0) {
#pragma unroll
            for (int s = 0; s < SLOTS; ++s) {
              const int c = gl + 32 * s;
              if (c < C) {
#pragma unroll
                for (int k = 0; k < K2; ++k) dst[c * K2 + k] = acc[s][k][r];
              }
            }
          }
          if (P + lane < Kpad) dst[P + lane] = 0.0;
        }
      }
    }
  }
}

template <int D, int N, int RB>
void p2m_tile(fmma_ctx* ctx, const Level& Lf, const double* sx, int64_t ns, const double* ws, int R,
              const Cube* cubes, const int* depth, bool isf, int Kpad, double* Wm, int nprob, int grid_n) {
  // Leaves per warp: sparse leaves share tiles of 32 sources, as long as the
  // runs fill the GPU four times (16 warps an SM)
  const int64_t want = Lf.nbox / ((int64_t)ctx->sm_count * 64);
  const int run = (int)(want < 1 ? 1 : (want > kTileMaxLeaves ? kTileMaxLeaves : want));
  const int64_t nrun = (Lf.nbox + run - 1) / run;
  FMMA_LAUNCH(ctx, (k_p2m_tile<D, N, RB>), grid_for(nrun, kTileWarps, (int64_t)ctx->sm_count * 64), 32 * kTileWarps, 0,
              Lf.key, Lf.sb, Lf.se, Lf.nbox, run, sx, ns, ws, R, cubes, depth, isf, Kpad, node_table<N>(), Wm,
              nprob > 1 && grid_n == 0, grid_n);
}

template <int D, int N>
void p2m_tile_rb(fmma_ctx* ctx, const Level& Lf, const double* sx, int64_t ns, const double* ws, int R,
                 const Cube* cubes, const int* depth, bool isf, int Kpad, double* Wm, int nprob, int grid_n) {
  // right-hand sides per pass: as many as keep the lane's sums near 24
  constexpr int kSums = P2MShape<D, N>::SLOTS * P2MShape<D, N>::K2;
  constexpr int kMost = kSums == 1 ? 16 : (kSums == 2 ? 8 : (kSums <= 6 ? 4 : 2));
  if (R == 1)
    p2m_tile<D, N, 1>(ctx, Lf, sx, ns, ws, R, cubes, depth, isf, Kpad, Wm, nprob, grid_n);
  else if (kMost > 4 && R <= 4)
    p2m_tile<D, N, kMost < 4 ? kMost : 4>(ctx, Lf, sx, ns, ws, R, cubes, depth, isf, Kpad, Wm, nprob, grid_n);
  else
    p2m_tile<D, N, kMost>(ctx, Lf, sx, ns, ws, R, cubes, depth, isf, Kpad, Wm, nprob, grid_n);
}

template <int D>
bool p2m_tile_n(fmma_ctx* ctx, const Level& Lf, const double* sx, int64_t ns, const double* ws, int R,
                const Cube* cubes, const int* depth, bool isf, int n, int Kpad, double* Wm, int nprob, int grid_n) {
#define FMMA_P2M_N(N_) \
  case N_: p2m_tile_rb<D, N_>(ctx, Lf, sx, ns, ws, R, cubes, depth, isf, Kpad, Wm, nprob, grid_n); return true;
  switch (n) {
    FMMA_P2M_N(2) FMMA_P2M_N(3) FMMA_P2M_N(4) FMMA_P2M_N(5) FMMA_P2M_N(6) FMMA_P2M_N(7) FMMA_P2M_N(8)
    default: return false;
  }
#undef FMMA_P2M_N
}

}  // namespace

bool launch_p2m_tile(fmma_ctx* ctx, const Level& Lf, const double* sx, int64_t ns, const double* ws, int R,
                     const Cube* cubes, const int* depth, int d, bool isf, int n, int P, int Kpad, double* Wm,
                     int nprob, int grid_n) {
  (void)P;
  if (d == 1) return p2m_tile_n<1>(ctx, Lf, sx, ns, ws, R, cubes, depth, isf, n, Kpad, Wm, nprob, grid_n);
  if (d == 2) return p2m_tile_n<2>(ctx, Lf, sx, ns, ws, R, cubes, depth, isf, n, Kpad, Wm, nprob, grid_n);
  return p2m_tile_n<3>(ctx, Lf, sx, ns, ws, R, cubes, depth, isf, n, Kpad, Wm, nprob, grid_n);
}

}  // namespace fmma_b200
