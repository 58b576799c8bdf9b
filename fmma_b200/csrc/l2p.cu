// l2p.cu — L2P at the leaves for 2 to 8 nodes per dimension
// (src/fmm_core.cpp:580-615): pot[r][t] = sum_k Wl[b][r][k] prod_q S_n(x_kq, rel_tq).
//
// A contraction over the coefficients on the FP64 tensor cores (DMMA m8n8k4),
// eight targets of a leaf as rows.  A warp walks a run of consecutive leaves,
// whose targets are consecutive, in tiles of 32 targets: lanes over targets
// compute the d n factors S_n of theirs into shared memory once, the A
// fragments are products of two or three of them, the B fragments are read
// from Wl as they lie there.  Two forms:
//  - plain: the columns are 8 right-hand sides, the sum runs over all n^d nodes;
//  - split (few right-hand sides): the columns are the n nodes of the last
//    dimension, the sum runs over the n^(d-1) nodes of the others, and each
//    target takes the product with its last factors at the end, so that the
//    tensor cores' columns are filled at one right-hand side too: n^(d-1) / 4
//    DMMAs for 8 targets instead of n^d / 4.
// What bounds it is the factors' FP64 arithmetic and shared stores at one
// right-hand side, and the stores of pot with 16 (2.5 GB at 19M targets).
// Against one lane a target with the sum over the nodes in its registers, us:
// 1 rhs, 250k targets, 5 nodes in 3-D 61.6 -> 22.2; 1 rhs, 131072 targets, 4
// nodes in 2-D 20.7 -> 10.0; 2 rhs, 200k targets, 5 nodes in 3-D 53.8 -> 24.4;
// 16 rhs, 19M targets in 2-D leaves of about 40, 5 nodes 4250 -> 2150.  On
// sparse leaves it stands against lanes over coefficients with the leaf's L2L
// fused in: 1M targets in 2-D leaves of 15, 6 nodes 251 -> 45 + 63 for the
// L2L; 262k clustered in 3-D 346 -> 99 + 262; 4M clustered 4360 -> 960 + 3300.
// With the gradient, against a lane a target in a block a leaf: 1M targets, 5
// nodes in 3-D 465 -> 128.
#include "fmm_stages.cuh"
#include "fmma_internal.cuh"

namespace fmma_b200 {

namespace {

template <bool GRAD>
__host__ __device__ constexpr int l2p_warps() {
  return GRAD ? 2 : 4;  // per block
}
constexpr int kL2PMaxLeaves = 32;  // leaves of a warp's run: their ranges sit in the lanes
// doubles between factor rows: 4 mod 16, so that the four rows and eight
// targets of a fragment lie in distinct banks; a fragment that begins at a
// tile's last targets reads up to 3 doubles into the next row, unused ones
constexpr int kL2PRow = 36;

template <int D, int N>
struct L2PShape {
  static constexpr int P = D == 1 ? N : (D == 2 ? N * N : N * N * N);
  static constexpr int K = D == 1 ? N : P / N;          // nodes of all dimensions but the last
  static constexpr int KSP = (P + 3) / 4;               // K steps, plain form
  static constexpr int KSS = (K + 3) / 4;               // and split form
  // right-hand sides up to which the split form has fewer DMMAs
  static constexpr int kSplitMost = D == 1 ? 0 : (KSP - 1) / KSS;
};

__device__ __forceinline__ void l2p_dmma(double& d0, double& d1, double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};\n"
               : "+d"(d0), "+d"(d1)
               : "d"(a), "d"(b));
}

// Product of the factors of node k (over the first Q dimensions) at F[row][i].
template <int Q, int N>
__device__ __forceinline__ double l2p_product(const double* F, int k) {
  if constexpr (Q == 1) return F[k * kL2PRow];
  else if constexpr (Q == 2) return F[(k / N) * kL2PRow] * F[(N + k % N) * kL2PRow];
  else
    return F[(k / (N * N)) * kL2PRow] * F[(N + k / N % N) * kL2PRow] * F[(2 * N + k % N) * kL2PRow];
}

// RT: column groups of 8 right-hand sides a pass (plain), 0: the split form.
// GRAD (split form, coordinates in double): the gradient potg[r][t][q] too.
// The derivative along a dimension takes that dimension's factor's derivative
// in the product; those of all but the last dimension are sums of their own,
// the last one's shares the potential's.
template <int D, int N, int RT, bool GRAD>
__global__ void __launch_bounds__(32 * l2p_warps<GRAD>(), GRAD ? 8 : 5) k_l2p_mma(
    const uint64_t* __restrict__ key, const int* __restrict__ tb, const int* __restrict__ te, int64_t nbox, int run,
    const double* __restrict__ tx, int64_t nt, const Cube* __restrict__ cubes, const int* __restrict__ depth, bool isf,
    int Kpad, int R, const __grid_constant__ NodeTable<N> tn, const double* __restrict__ Wl, double* __restrict__ pot,
    double* __restrict__ potg, bool many) {
  using S = L2PShape<D, N>;
  constexpr int W = l2p_warps<GRAD>();
  constexpr int NS = GRAD && RT == 0 ? D : 1;  // sums: the potential's, the gradient's of all but the last dimension
  constexpr int kG = D * N * kL2PRow;          // the factors' derivatives behind the factors
  __shared__ double s_f[W][(GRAD ? 2 : 1) * kG + 4];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int kk = lane & 3, row = lane >> 2;  // of a fragment: K index or column pair, target (or column of B)
  double* const F = s_f[warp];
  const int64_t nw = (int64_t)gridDim.x * W;
  const int64_t nrun = (nbox + run - 1) / run;
  for (int64_t u = (int64_t)blockIdx.x * W + warp; u < nrun; u += nw) {
    const int64_t b0 = u * run;
    const int nb = (int)min((int64_t)run, nbox - b0);
    const int my_tb = lane < nb ? tb[b0 + lane] : 0, my_te = lane < nb ? te[b0 + lane] : 0;
    // a problem with Depth < 3 has no local expansions
    const bool on = lane < nb && my_te > my_tb && (!many || depth[key_pid(key[b0 + lane])] >= 3);
    const unsigned leaves = __ballot_sync(0xffffffffu, on);
    const int last = __shfl_sync(0xffffffffu, my_te, nb - 1);
    // one problem: its cube and leaf width once
    const int pid0 = many ? 0 : key_pid(key[b0]);
    const int Nl0 = many ? 1 : 1 << (depth[pid0] - 1);
    const LeafWidth lw0 = leaf_width(cubes[pid0], Nl0, isf);
    int t0 = 0, t1 = 0;  // targets of the tile in shared memory
    for (unsigned todo = leaves; todo != 0; todo &= todo - 1) {
      const int l = __ffs(todo) - 1;
      const int s0 = __shfl_sync(0xffffffffu, my_tb, l), s1 = __shfl_sync(0xffffffffu, my_te, l);
      const double* const wl = Wl + (b0 + l) * R * Kpad;
      for (int p = s0; p < s1;) {
        if (p < t0 || p >= t1) {  // the next tile: targets p .. p + 31 of the run's leaves
          __syncwarp();           // every lane is done with the last one
          t0 = p;
          t1 = min(p + 32, last);
          const int i = p + lane;
          int pid = pid0, Nl = Nl0;
          if (many) {  // the target's leaf: the first whose range ends beyond it
            int m = 0;
#pragma unroll
            for (int step = 16; step > 0; step >>= 1) {
              const int e = __shfl_sync(0xffffffffu, my_te, m + step - 1);
              if (m + step <= nb && e <= i) m += step;
            }
            pid = key_pid(key[b0 + min(m, nb - 1)]);
            Nl = 1 << (depth[pid] - 1);
          }
          if (i < t1) {
            const Cube& c = cubes[pid];
            const LeafWidth lw = many ? leaf_width(c, Nl, isf) : lw0;
#pragma unroll
            for (int q = 0; q < D; ++q) {
              const double y = point_rel(tx[(int64_t)q * nt + i], c, lw, q, Nl, isf);
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
                F[(q * N + k) * kL2PRow + lane] = 1.0 / N + 2.0 * (1.0 / N) * s;
              }
              if constexpr (GRAD) {  // T_j' = j U_{j-1}
                double V[N];         // j U_{j-1}
                double u0 = 0.0, u1 = 1.0;
#pragma unroll
                for (int j = 1; j < N; ++j) {
                  V[j] = (double)j * u1;
                  const double u2 = 2.0 * y * u1 - u0;
                  u0 = u1;
                  u1 = u2;
                }
#pragma unroll
                for (int k = 0; k < N; ++k) {
                  double s = 0.0;
#pragma unroll
                  for (int j = 1; j < N; ++j) s += tn.T[k * N + j] * V[j];
                  F[kG + (q * N + k) * kL2PRow + lane] = 2.0 * (1.0 / N) * s;
                }
              }
            }
          }
          __syncwarp();
        }
        const int e = min(s1, t1) - t0, i0 = p - t0, nm = (e - i0 + 7) >> 3;  // 1 to 4 groups of 8 targets
        const double* const Fi = F + i0 + row;
        if constexpr (RT == 0) {
          double scale = 1.0;
          if constexpr (GRAD) {
            const int pid = key_pid(key[b0 + l]);
            scale = 2.0 * (double)(1 << (depth[pid] - 1)) / cubes[pid].Len;
          }
          for (int r = 0; r < R; ++r) {
            double b[S::KSS], acc[4][NS][2];
#pragma unroll
            for (int ks = 0; ks < S::KSS; ++ks) {
              const int k = ks * 4 + kk;
              b[ks] = k < S::K && row < N ? wl[(int64_t)r * Kpad + k * N + row] : 0.0;
            }
#pragma unroll
            for (int m = 0; m < 4; ++m) {
#pragma unroll
              for (int c = 0; c < NS; ++c) acc[m][c][0] = acc[m][c][1] = 0.0;
              if (m >= nm) continue;
#pragma unroll
              for (int ks = 0; ks < S::KSS; ++ks) {
                const int k = min(ks * 4 + kk, S::K - 1);
                if constexpr (!GRAD) {
                  l2p_dmma(acc[m][0][0], acc[m][0][1], l2p_product<D == 1 ? 1 : D - 1, N>(Fi + m * 8, k), b[ks]);
                } else if constexpr (D == 2) {
                  const double* const f0 = Fi + m * 8 + k * kL2PRow;
                  l2p_dmma(acc[m][0][0], acc[m][0][1], f0[0], b[ks]);
                  l2p_dmma(acc[m][NS - 1][0], acc[m][NS - 1][1], f0[kG], b[ks]);
                } else if constexpr (D == 3) {
                  const double* const p0 = Fi + m * 8 + (k / N) * kL2PRow;
                  const double* const p1 = Fi + m * 8 + (N + k % N) * kL2PRow;
                  const double f0 = p0[0], f1 = p1[0];
                  l2p_dmma(acc[m][0][0], acc[m][0][1], f0 * f1, b[ks]);
                  l2p_dmma(acc[m][1 % NS][0], acc[m][1 % NS][1], p0[kG] * f1, b[ks]);
                  l2p_dmma(acc[m][NS - 1][0], acc[m][NS - 1][1], f0 * p1[kG], b[ks]);
                }
              }
            }
            const double* const fl = Fi + (D - 1) * N * kL2PRow;
#pragma unroll
            for (int m = 0; m < 4; ++m) {
              if (m >= nm) continue;
              // columns beyond N are zeros
              const int c0 = min(2 * kk, N - 1) * kL2PRow + m * 8, c1 = min(2 * kk + 1, N - 1) * kL2PRow + m * 8;
              const bool store = kk == 0 && i0 + m * 8 + row < e;
              const int64_t t = (int64_t)r * nt + p + m * 8 + row;
              auto total = [&](const double* a, int at) {
                double v = a[0] * fl[at + c0];
                v += a[1] * fl[at + c1];
                v += __shfl_xor_sync(0xffffffffu, v, 1);
                v += __shfl_xor_sync(0xffffffffu, v, 2);
                return v;
              };
              const double v = total(acc[m][0], 0);
              if (store) pot[t] = v;
              if constexpr (GRAD) {
#pragma unroll
                for (int q = 0; q < D; ++q) {
                  const double g = q == D - 1 ? total(acc[m][0], kG) : total(acc[m][(q + 1) % NS], 0);
                  if (store) potg[t * D + q] = g * scale;
                }
              }
            }
          }
        } else {
          constexpr int UB = S::KSP < 8 ? S::KSP : 8;  // K steps whose B fragments load together
          for (int r0 = 0; r0 < R; r0 += 8 * RT) {
            double acc[4][RT > 0 ? RT : 1][2] = {};
#pragma unroll 1
            for (int kb = 0; kb < S::KSP; kb += UB) {
              double b[UB][RT > 0 ? RT : 1];
#pragma unroll
              for (int j = 0; j < UB; ++j)
#pragma unroll
                for (int c = 0; c < RT; ++c) {
                  const int k = (kb + j) * 4 + kk, r = r0 + c * 8 + row;
                  b[j][c] = k < S::P && r < R ? wl[(int64_t)r * Kpad + k] : 0.0;
                }
#pragma unroll
              for (int j = 0; j < UB; ++j) {
                const int k = min((kb + j) * 4 + kk, S::P - 1);
#pragma unroll
                for (int m = 0; m < 4; ++m) {
                  if (m >= nm) continue;
                  const double a = l2p_product<D, N>(Fi + m * 8, k);
#pragma unroll
                  for (int c = 0; c < RT; ++c) l2p_dmma(acc[m][c][0], acc[m][c][1], a, b[j][c]);
                }
              }
            }
#pragma unroll
            for (int m = 0; m < 4; ++m) {
              if (i0 + m * 8 + row >= e) continue;
#pragma unroll
              for (int c = 0; c < RT; ++c)
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                  const int r = r0 + c * 8 + 2 * kk + h;
                  if (r < R) pot[(int64_t)r * nt + p + m * 8 + row] = acc[m][c][h];
                }
            }
          }
        }
        p = t0 + e;
      }
    }
  }
}

template <int D, int N, int RT, bool GRAD>
void l2p_mma(fmma_ctx* ctx, const Level& Lf, const double* tx, int64_t nt, const Cube* cubes, const int* depth,
             bool isf, int Kpad, int R, const double* Wl, double* pot, double* potg, int nprob) {
  // Leaves per warp: leaves share tiles of 32 targets, as long as the runs
  // fill the GPU four times (16 warps an SM)
  const int64_t want = Lf.nbox / ((int64_t)ctx->sm_count * 64);
  const int run = (int)(want < 1 ? 1 : (want > kL2PMaxLeaves ? kL2PMaxLeaves : want));
  const int64_t nrun = (Lf.nbox + run - 1) / run;
  FMMA_LAUNCH(ctx, (k_l2p_mma<D, N, RT, GRAD>),
              grid_for(nrun, l2p_warps<GRAD>(), (int64_t)ctx->sm_count * 64), 32 * l2p_warps<GRAD>(), 0,
              Lf.key, Lf.tb, Lf.te, Lf.nbox, run, tx, nt, cubes, depth, isf, Kpad, R, node_table<N>(), Wl, pot, potg,
              nprob > 1);
}

template <int D>
bool l2p_mma_n(fmma_ctx* ctx, const Level& Lf, const double* tx, int64_t nt, const Cube* cubes, const int* depth,
               bool isf, int n, int Kpad, int R, const double* Wl, double* pot, int nprob) {
#define FMMA_L2P_CALL(N_, RT_) \
  l2p_mma<D, N_, RT_, false>(ctx, Lf, tx, nt, cubes, depth, isf, Kpad, R, Wl, pot, nullptr, nprob)
#define FMMA_L2P_N(N_)                                \
  case N_:                                            \
    if (R <= L2PShape<D, N_>::kSplitMost) {           \
      if constexpr (D > 1) FMMA_L2P_CALL(N_, 0);      \
    } else if (R <= 8) {                              \
      FMMA_L2P_CALL(N_, 1);                           \
    } else {                                          \
      FMMA_L2P_CALL(N_, 2);                           \
    }                                                 \
    return true;
  switch (n) {
    FMMA_L2P_N(2) FMMA_L2P_N(3) FMMA_L2P_N(4) FMMA_L2P_N(5) FMMA_L2P_N(6) FMMA_L2P_N(7) FMMA_L2P_N(8)
    default: return false;
  }
#undef FMMA_L2P_N
#undef FMMA_L2P_CALL
}

template <int D>
bool l2p_grad_n(fmma_ctx* ctx, const Level& Lf, const double* tx, int64_t nt, const Cube* cubes, const int* depth,
                int n, int Kpad, int R, const double* Wl, double* pot, double* potg, int nprob) {
#define FMMA_L2P_N(N_) \
  case N_: l2p_mma<D, N_, 0, true>(ctx, Lf, tx, nt, cubes, depth, false, Kpad, R, Wl, pot, potg, nprob); return true;
  switch (n) {
    FMMA_L2P_N(2) FMMA_L2P_N(3) FMMA_L2P_N(4) FMMA_L2P_N(5) FMMA_L2P_N(6) FMMA_L2P_N(7) FMMA_L2P_N(8)
    default: return false;
  }
#undef FMMA_L2P_N
}

}  // namespace

bool launch_l2p_mma(fmma_ctx* ctx, const Level& Lf, const double* tx, int64_t nt, const Cube* cubes, const int* depth,
                    int d, bool isf, int n, int Kpad, int R, const double* Wl, double* pot, int nprob) {
  if (d == 1) return l2p_mma_n<1>(ctx, Lf, tx, nt, cubes, depth, isf, n, Kpad, R, Wl, pot, nprob);
  if (d == 2) return l2p_mma_n<2>(ctx, Lf, tx, nt, cubes, depth, isf, n, Kpad, R, Wl, pot, nprob);
  return l2p_mma_n<3>(ctx, Lf, tx, nt, cubes, depth, isf, n, Kpad, R, Wl, pot, nprob);
}

bool launch_l2p_grad(fmma_ctx* ctx, const Level& Lf, const double* tx, int64_t nt, const Cube* cubes, const int* depth,
                     int d, int n, int Kpad, int R, const double* Wl, double* pot, double* potg, int nprob) {
  if (d == 2) return l2p_grad_n<2>(ctx, Lf, tx, nt, cubes, depth, n, Kpad, R, Wl, pot, potg, nprob);
  if (d == 3) return l2p_grad_n<3>(ctx, Lf, tx, nt, cubes, depth, n, Kpad, R, Wl, pot, potg, nprob);
  return false;
}

}  // namespace fmma_b200
