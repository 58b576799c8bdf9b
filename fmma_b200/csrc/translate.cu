// translate.cu — M2M and L2L (src/fmm_core.cpp:319-336, :524-541) for 1 to 8
// nodes per dimension, in 1-D for 1 to 16.
//
// The operator of a child is a product of 1-D operators A_0 or A_1 along the
// dimensions, so a parent's sum over its 2^d children is taken dimension by
// dimension: along the last one the pairs of children that differ in it are
// translated and added (A_0 x_0 + A_1 x_1), which leaves 2^(d-1) half-way
// expansions, and so on: 2^d - 1 fibre sets of 2 n^2 multiply-adds where child
// by child takes d 2^d sets of n^2 (14 against 24 n^2-sets in 3-D).  L2L is
// the same tree downwards with the transposes.
//
// A warp takes U (parent, right-hand side) units at a time, U so that the
// fibres fill its lanes; the children lie in shared memory (cp.async, missing
// ones as zeros), a lane takes a fibre, the n values that differ in one
// dimension's digit, into registers, multiplies them by operators that are
// constants of the launch, and writes the results where they came from.  Rows
// of the last dimension are padded to an odd length against bank conflicts.
// What bounds it is latency (of a unit's child ranges and expansions, and of
// shared memory between the passes) at 16 to 32 warps an SM, not HBM: the
// largest M2M below moves 2.9 GB (with 16 rhs in 2-D the passes' shared memory,
// 76 % of its throughput).  Against child by child with the operators
// read from shared memory (a load per multiply-add), and for P <= 32 dense
// P x P operators, M2M and L2L of all levels, us: 4M clustered, 6 nodes
// 3390 -> 2160 and 4360 -> 2780; 262k clustered 482 -> 285 and 399 -> 353; 1M
// in 2-D, 6 nodes 103 -> 48 and 112 -> 60; 250k in 3-D, 5 nodes 35 -> 12 and
// 18 -> 25; 19M in 2-D x 16 rhs, 5 nodes 3040 -> 2040 and 3430 -> 2070.
// Tried and slower: a second buffer for the next units' expansions (2260 and
// 2520 in the last case; it costs warps).
#include "fmm_stages.cuh"
#include "fmma_internal.cuh"

namespace fmma_b200 {

namespace {

constexpr int kTransWarps = 4;

template <int D, int N>
struct TransShape {
  static constexpr int NC = 1 << D;                                 // children of a parent
  static constexpr int NF = D == 1 ? 1 : (D == 2 ? N : N * N);      // fibres of an expansion
  static constexpr int P = N * NF;
  static constexpr int NP = N % 4 == 0 ? N + 1 : N;                 // padded row of the last dimension
  static constexpr int SS = NF * NP;                                // doubles of an expansion in shared memory
  static constexpr int U = D == 1 ? 32 : (D == 2 ? 32 / N : (N <= 2 ? 8 : (N == 3 ? 3 : (N == 4 ? 2 : 1))));
  // loads and stores of an expansion: GL lanes, EPL coefficients each
  static constexpr int GL = P > 16 ? 32 : (P > 8 ? 16 : 8), EPL = (P + GL - 1) / GL;
  static constexpr int X = U * NC * SS;                             // doubles of a warp's units
  static constexpr int kBlocks = D < 3 ? 8 : (N >= 7 ? 2 : (N >= 5 ? 4 : 6));  // for the registers
  static constexpr size_t kSmem = sizeof(double) * kTransWarps * X;
};

// A_0 and A_1 [i][j], as constants of the launch.
template <int N>
struct TransOps {
  double a[2][N * N];
};

// First element of fibre f along dimension Q, and the fibre's stride.
template <int D, int N, int Q>
__device__ __forceinline__ int fibre_base(int f) {
  constexpr int NP = TransShape<D, N>::NP;
  if constexpr (Q == D - 1) return f * NP;
  else if constexpr (Q == 1) return (f / N) * (N * NP) + f % N;
  else if constexpr (D == 2) return f;
  else return (f / N) * NP + f % N;
}
template <int D, int N, int Q>
__device__ __forceinline__ constexpr int fibre_stride() {
  constexpr int NP = TransShape<D, N>::NP;
  return Q == D - 1 ? 1 : (Q == D - 2 ? NP : N * NP);
}

// Dimension Q of all units' expansions X[unit][child][SS].  The children that
// differ in it only are `half` apart (bit D - 1 - Q of the child).  UP: the
// lower one of a pair becomes A_0 lower + A_1 upper; else the lower one's
// A_0^T and A_1^T images become the pair.
template <int D, int N, int Q, bool UP>
__device__ __forceinline__ void trans_pass(double* X, const TransOps<N>& op, int lane) {
  using S = TransShape<D, N>;
  constexpr int s = D - 1 - Q, G = S::NC >> (s + 1), half = S::SS << s, st = fibre_stride<D, N, Q>();
#pragma unroll 1
  for (int i = lane; i < S::U * G * S::NF; i += 32) {
    const int f = i % S::NF, pair = i / S::NF;  // pair: (unit, pair of children)
    double* const x = X + (pair << (s + 1)) * S::SS + fibre_base<D, N, Q>(f);
    double a[N], b[N];
#pragma unroll
    for (int j = 0; j < N; ++j) a[j] = x[j * st];
    if constexpr (UP) {
#pragma unroll
      for (int j = 0; j < N; ++j) b[j] = x[half + j * st];
#pragma unroll
      for (int k = 0; k < N; ++k) {
        double y = 0.0;
#pragma unroll
        for (int j = 0; j < N; ++j) y = fma(op.a[0][k * N + j], a[j], y);
#pragma unroll
        for (int j = 0; j < N; ++j) y = fma(op.a[1][k * N + j], b[j], y);
        x[k * st] = y;
      }
    } else {
#pragma unroll
      for (int k = 0; k < N; ++k) {
        double y = 0.0, z = 0.0;
#pragma unroll
        for (int j = 0; j < N; ++j) {
          y = fma(op.a[0][j * N + k], a[j], y);
          z = fma(op.a[1][j * N + k], a[j], z);
        }
        x[k * st] = y;
        x[half + k * st] = z;
      }
    }
  }
  __syncwarp();
}

// Rows (box * R + right-hand side) of the children level of (unit, child) into
// row[U][NC], -1 where there is none in use (begin, end: the points that count).
template <int D, int U>
__device__ __forceinline__ void trans_children(int64_t* row, int64_t u0, int64_t nunit, int R, const uint64_t* ckey,
                                               const int* cbeg, const int* cend, const int* pcb, const int* pce,
                                               const int* pbeg, const int* pend, const uint64_t* pkey,
                                               const int* depth, int vpar, int lane) {
  constexpr int NC = 1 << D;
  for (int s = lane; s < U * NC; s += 32) row[s] = -1;
  __syncwarp();
  // lanes over (unit, child by its place in the parent's range)
  for (int s = lane; s < U * NC; s += 32) {
    const int64_t unit = u0 + s / NC;
    if (unit >= nunit) continue;
    const int64_t p = R == 1 ? unit : unit / R;
    const int ch = pcb[p] + s % NC;
    if (ch >= pce[p] || pend[p] <= pbeg[p]) continue;
    if (depth[key_pid(pkey[p])] - 1 - vpar < 2) continue;  // expansions are used on levels >= 2 only
    if (cend[ch] > cbeg[ch])
      row[s / NC * NC + (int)(ckey[ch] & (uint64_t)(NC - 1))] = (int64_t)ch * R + (unit - p * R);
  }
  __syncwarp();
}

// Where coefficient k of an expansion lies in shared memory.
template <int D, int N>
__device__ __forceinline__ int trans_at(int k) {
  constexpr int NP = TransShape<D, N>::NP;
  return NP == N ? k : (k / N) * NP + k % N;
}

template <int D, int N>
__global__ void __launch_bounds__(32 * kTransWarps, TransShape<D, N>::kBlocks) k_m2m_tree(
    const uint64_t* __restrict__ ckey, const int* __restrict__ csb, const int* __restrict__ cse,
    const uint64_t* __restrict__ pkey, const int* __restrict__ pcb, const int* __restrict__ pce,
    const int* __restrict__ psb, const int* __restrict__ pse, int64_t npar, int vpar, const int* __restrict__ depth,
    int Kpad, int R, const __grid_constant__ TransOps<N> op, const double* __restrict__ Wc, double* __restrict__ Wp) {
  using S = TransShape<D, N>;
  constexpr int GL = S::GL, EPL = S::EPL;
  extern __shared__ __align__(16) double sm[];
  __shared__ int64_t s_row[kTransWarps][2][S::U * S::NC];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int grp = lane / GL, gl = lane % GL;
  double* const X = sm + (size_t)warp * S::X;
  int at[EPL];
#pragma unroll
  for (int i = 0; i < EPL; ++i) at[i] = trans_at<D, N>(gl + GL * i);
  const int64_t nunit = npar * R, nw = (int64_t)gridDim.x * kTransWarps * S::U;
  auto rows = [&](int64_t u0, int64_t* row) {
    trans_children<D, S::U>(row, u0, nunit, R, ckey, csb, cse, pcb, pce, psb, pse, pkey, depth, vpar, lane);
  };
  auto load = [&](const int64_t* row) {
#pragma unroll 1
    for (int s = grp; s < S::U * S::NC; s += 32 / GL) {
      const int64_t rw = row[s];
      const double* const src = Wc + rw * Kpad + gl;
      double* const dst = X + s * S::SS;
      if (rw >= 0) {
#pragma unroll
        for (int i = 0; i < EPL; ++i)
          if (gl + GL * i < S::P) cp_async8_zfill(dst + at[i], src + GL * i, true);
      } else {
#pragma unroll
        for (int i = 0; i < EPL; ++i)
          if (gl + GL * i < S::P) dst[at[i]] = 0.0;
      }
    }
  };
  int64_t u0 = ((int64_t)blockIdx.x * kTransWarps + warp) * S::U;
  if (u0 >= nunit) return;
  rows(u0, s_row[warp][0]);
  load(s_row[warp][0]);
  cp_async_commit();
  for (int cur = 0; u0 < nunit; u0 += nw, cur ^= 1) {
    // the next units' rows come under these ones' copies
    int64_t* const row = s_row[warp][cur];
    const bool more = u0 + nw < nunit;
    if (more) rows(u0 + nw, s_row[warp][cur ^ 1]);
    cp_async_wait<0>();
    __syncwarp();
    trans_pass<D, N, D - 1, true>(X, op, lane);
    if constexpr (D >= 2) trans_pass<D, N, D - 2, true>(X, op, lane);
    if constexpr (D == 3) trans_pass<D, N, 0, true>(X, op, lane);
    for (int u = grp; u < S::U; u += 32 / GL) {
      bool any = false;  // a parent in use has a child with sources
#pragma unroll
      for (int c = 0; c < S::NC; ++c) any |= row[u * S::NC + c] >= 0;
      if (!any) continue;
      const double* const x = X + u * S::NC * S::SS;
      double* const dst = Wp + (u0 + u) * Kpad;
#pragma unroll
      for (int i = 0; i < EPL; ++i)
        if (gl + GL * i < S::P) dst[gl + GL * i] = x[at[i]];
      if (S::P + gl < Kpad) dst[S::P + gl] = 0.0;
    }
    __syncwarp();  // every lane is done with the expansions and the rows
    if (more) load(s_row[warp][cur ^ 1]);
    cp_async_commit();
  }
}

// Wl[b] += op^T Wl[parent(b)] for the children b with targets of the parents.
template <int D, int N>
__global__ void __launch_bounds__(32 * kTransWarps, TransShape<D, N>::kBlocks) k_l2l_tree(
    const uint64_t* __restrict__ ckey, const int* __restrict__ ctb, const int* __restrict__ cte,
    const uint64_t* __restrict__ pkey, const int* __restrict__ pcb, const int* __restrict__ pce,
    const int* __restrict__ ptb, const int* __restrict__ pte, int64_t npar, int vpar, const int* __restrict__ depth,
    int Kpad, int R, const __grid_constant__ TransOps<N> op, const double* __restrict__ Wp, double* __restrict__ Wc) {
  using S = TransShape<D, N>;
  constexpr int GL = S::GL, EPL = S::EPL, G = 32 / GL, NS = S::U * S::NC;
  extern __shared__ __align__(16) double sm[];
  __shared__ int64_t s_row[kTransWarps][2][NS];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int grp = lane / GL, gl = lane % GL;
  double* const X = sm + (size_t)warp * S::X;
  int at[EPL];
#pragma unroll
  for (int i = 0; i < EPL; ++i) at[i] = trans_at<D, N>(gl + GL * i);
  const int64_t nunit = npar * R, nw = (int64_t)gridDim.x * kTransWarps * S::U;
  auto rows = [&](int64_t u0, int64_t* row) {
    trans_children<D, S::U>(row, u0, nunit, R, ckey, ctb, cte, pcb, pce, ptb, pte, pkey, depth, vpar, lane);
  };
  auto load = [&](int64_t u0) {
    for (int u = grp; u < S::U; u += G) {
      const double* const src = Wp + min(u0 + u, nunit - 1) * Kpad + gl;
      double* const dst = X + u * S::NC * S::SS;
#pragma unroll
      for (int i = 0; i < EPL; ++i)
        if (gl + GL * i < S::P) cp_async8_zfill(dst + at[i], src + GL * i, true);
    }
  };
  int64_t u0 = ((int64_t)blockIdx.x * kTransWarps + warp) * S::U;
  if (u0 >= nunit) return;
  load(u0);
  cp_async_commit();
  rows(u0, s_row[warp][0]);
  for (int flip = 0; u0 < nunit; u0 += nw, flip ^= 1) {
    // the next units' rows come under these ones' copies
    int64_t* const row = s_row[warp][flip];
    const bool more = u0 + nw < nunit;
    if (more) rows(u0 + nw, s_row[warp][flip ^ 1]);
    cp_async_wait<0>();
    __syncwarp();
    trans_pass<D, N, 0, false>(X, op, lane);
    if constexpr (D >= 2) trans_pass<D, N, 1, false>(X, op, lane);
    if constexpr (D == 3) trans_pass<D, N, 2, false>(X, op, lane);
    // coefficients k < P of each child's row (the padding stays as it is), a
    // batch of children's loads in flight, the next batch's ahead
    constexpr int NB = EPL >= 8 ? 1 : 8 / EPL;
    double cur[NB][EPL], nxt[NB][EPL];
    auto fetch = [&](double (*v)[EPL], int s0) {
#pragma unroll
      for (int j = 0; j < NB; ++j) {
        const int s = s0 + G * j;
        const int64_t rw = s < NS ? row[s] : -1;
        const double* const src = Wc + rw * Kpad + gl;
#pragma unroll
        for (int i = 0; i < EPL; ++i) v[j][i] = rw >= 0 && gl + GL * i < S::P ? src[GL * i] : 0.0;
      }
    };
    fetch(cur, grp);
#pragma unroll 1
    for (int s0 = grp; s0 < NS; s0 += G * NB) {
      if (s0 + G * NB < NS) fetch(nxt, s0 + G * NB);
#pragma unroll
      for (int j = 0; j < NB; ++j) {
        const int s = s0 + G * j;
        const int64_t rw = s < NS ? row[s] : -1;
        double* const dst = Wc + rw * Kpad + gl;
        const double* const x = X + s * S::SS;
        if (rw >= 0) {
#pragma unroll
          for (int i = 0; i < EPL; ++i)
            if (gl + GL * i < S::P) dst[GL * i] = cur[j][i] + x[at[i]];
        }
#pragma unroll
        for (int i = 0; i < EPL; ++i) cur[j][i] = nxt[j][i];
      }
    }
    __syncwarp();  // every lane is done with the expansions and the rows
    if (more) load(u0 + nw);
    cp_async_commit();
  }
}

template <int D, int N, bool UP>
void trans_launch(fmma_ctx* ctx, const Level& C, const Level& Pl, int vpar, const int* depth, int Kpad, int R,
                  const double* in, double* out) {
  using S = TransShape<D, N>;
  static const TransOps<N> op = [] {
    const ChebTables ct = make_cheb_tables(N);
    TransOps<N> t;
    for (int s = 0; s < 2; ++s)
      for (int i = 0; i < N * N; ++i) t.a[s][i] = ct.A[s][i];
    return t;
  }();
  const unsigned grid = grid_for((Pl.nbox * R + S::U - 1) / S::U, kTransWarps, (int64_t)ctx->sm_count * 32);
  auto* const kernel = UP ? k_m2m_tree<D, N> : k_l2l_tree<D, N>;
  if (S::kSmem > 48 * 1024 && !ctx->capturing)
    FMMA_CHECK_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)S::kSmem));
  FMMA_LAUNCH(ctx, kernel, grid, 32 * kTransWarps, S::kSmem, C.key, UP ? C.sb : C.tb, UP ? C.se : C.te, Pl.key, Pl.cb,
              Pl.ce, UP ? Pl.sb : Pl.tb, UP ? Pl.se : Pl.te, Pl.nbox, vpar, depth, Kpad, R, op, in, out);
}

template <bool UP>
bool trans_any(fmma_ctx* ctx, const Level& C, const Level& Pl, int vpar, const int* depth, int d, int n, int Kpad,
               int R, const double* in, double* out) {
#define FMMA_TRANS(D_, N_) \
  case 16 * D_ + N_: trans_launch<D_, N_, UP>(ctx, C, Pl, vpar, depth, Kpad, R, in, out); return true;
#define FMMA_TRANS_3(N_) FMMA_TRANS(1, N_) FMMA_TRANS(2, N_) FMMA_TRANS(3, N_)
  if (n < 1 || n > 16) return false;
  switch (16 * d + n) {
    FMMA_TRANS_3(1) FMMA_TRANS_3(2) FMMA_TRANS_3(3) FMMA_TRANS_3(4) FMMA_TRANS_3(5) FMMA_TRANS_3(6) FMMA_TRANS_3(7)
    FMMA_TRANS_3(8)
    FMMA_TRANS(1, 9) FMMA_TRANS(1, 10) FMMA_TRANS(1, 11) FMMA_TRANS(1, 12) FMMA_TRANS(1, 13) FMMA_TRANS(1, 14)
    FMMA_TRANS(1, 15) FMMA_TRANS(1, 16)
    default: return false;
  }
#undef FMMA_TRANS_3
#undef FMMA_TRANS
}

}  // namespace

bool launch_m2m_tree(fmma_ctx* ctx, const Level& C, const Level& Pl, int vpar, const int* depth, int d, int n, int Kpad,
                     int R, const double* Wc, double* Wp) {
  return trans_any<true>(ctx, C, Pl, vpar, depth, d, n, Kpad, R, Wc, Wp);
}

bool launch_l2l_tree(fmma_ctx* ctx, const Level& C, const Level& Pl, int vpar, const int* depth, int d, int n, int Kpad,
                     int R, const double* Wp, double* Wc) {
  return trans_any<false>(ctx, C, Pl, vpar, depth, d, n, Kpad, R, Wp, Wc);
}

}  // namespace fmma_b200
