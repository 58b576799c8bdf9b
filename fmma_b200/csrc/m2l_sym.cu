// m2l_sym.cu — FP64 M2L in three dimensions for radial kernels, on the
// reflection symmetry of the Chebyshev grid.
//
// The sum is that of src/fmm_core.cpp:375-455: Wl[b] = sum over the far slots
// of K(offset) Wm[source].  The node set is symmetric (node n-1-k = -node k),
// so for f(x, y) = g(|x - y|) the operator of an offset with some components
// negated is the operator of |offset| with rows and columns reversed along
// those dimensions.  In the basis of even and odd parts along every dimension
// (x_k + x_{n-1-k}, x_k - x_{n-1-k}) a reversal is a sign per parity block, so
// the up to eight sources at the offsets (+-o_0, +-o_1, +-o_2) of one target
// share the 8 x 8 parity blocks of one operator:
//
//   y_a += sum_b K_ab z_{a^b, b},   z_{c, b} = sum_g (-1)^{c.g} x_{g, b}
//
// (a, b: parity of the target and source block, one bit per dimension; g: the
// signs of the offset): P^2 multiply-adds for eight sources instead of 8 P^2,
// and the z by an 8-point Walsh-Hadamard butterfly of the gathered sources.
// Along a dimension with o_q = 0 there is one source and K_ab = 0 unless
// a_q = b_q, which halves the operator instead; along one with |o_q| = 3 the
// far list has one side only, so there is one source and nothing to combine
// (on the negative side the operator's a_q != b_q blocks change sign).  The 189 far slots of a target
// fall into 56 orbits worth 39.5 P^2 multiply-adds (189 P^2 before).
//
// FP64 tensor (DMMA) bound.  A block owns 8 MB target rows (box x rhs) of one
// child-parity class.  Eight multiplying warps hold the rows' sums, a warp the
// outputs of one parity, or with an odd node count of the parities a and 7 - a
// for half of the rows, so that every warp has the same number of columns
// (an even-parity block is larger).  Eight gathering warps read the 8 source
// values of a (row, k), run the butterfly in registers and store the z of a
// stage (two K steps of 4) into a ring of four in shared memory; a full and an
// empty mbarrier per slot tie the two sides.  Operator fragments are read from
// L2 straight into registers (with an even node count a warp shares them with
// no other warp of the block), a stage ahead.  Orbits with no source for a
// tile are skipped, and so are a tile's unused row groups of 8, by kernels
// compiled for 1, 2, half and all of them (a DMMA that is predicated off still
// takes its turn on the pipe).
// Measured on the 262k clustered level (6 nodes, 1945 tiles), on a million
// points of the adjoint's two solves and on 4096 boxes x 2 rhs (5 nodes), ms of
// all levels: gather, butterfly and multiply in the same warps 41.7, - and
// 1.68; warps of their own 34.6, - and 1.40; straight-line multiplying,
// one-sided dimensions and fragments loaded ahead 28.9, 10.2 and 0.98; row
// groups at compile time and the prologue's loads all in flight 28.3, 9.4 and
// 0.88.  A stage then takes 2750 cycles (6 nodes), of which the DMMAs need
// 2048 and the butterfly's additions, which take turns on the same pipe, 390
// (without them 2400).  Tried and slower: the operators in shared memory by
// bulk copies (29.9, 10.0, 0.90), the butterfly ahead of the wait for a free
// slot (31.1, 10.5, 0.94), a ring of three (28.5, 9.5, 0.88).
#include <algorithm>
#include <cmath>

#include "fmm_stages.cuh"
#include "fmma_internal.cuh"
#include "kernels.cuh"
#include "solver.cuh"

namespace fmma_b200 {

namespace {

constexpr int kOrbits = 56;       // |o| in {0..3}^3 without {0,1}^3
constexpr int kSymThreads = 512;  // 8 multiplying warps, 8 gathering warps
constexpr int kSymRing = 4;       // stages of z in shared memory
constexpr long long kSymWaitCycles = 4000000000ll;  // default bound of a pipeline wait (~2 s)
constexpr int kSymMaxStages = 64; // stages of one orbit: 8 blocks of up to 16 K steps, two per stage
constexpr int kSymSlots = 189;

// Constant geometry of one node count, uploaded in front of the operators.
struct SymGeom {
  int n, he, ho;         // nodes per dimension, even and odd parts per dimension
  int KB, NB, MB;        // padded block length, column groups of 8 per warp, row groups of 8 per block
  int P, total;          // coefficients, pipeline stages of one operator set
  int size[8], off[8];   // coefficients of a parity block and its offset in a folded row of P
  int nst[8];            // stages of an orbit by its zero mask
  int zmask[kOrbits];    // bit q: o_q = 0
  int umask[kOrbits];    // bit q: |o_q| = 3, which a class has on one side only ...
  int neg[8];            // ... the negative one where bit q is set (by class)
  int stage0[kOrbits];   // first stage of the orbit's operator
  int desc[8][kSymMaxStages][2];  // K step: b0 | k4 << 3, or -1 (no step)
  int slot[8][kOrbits][8];        // far slot of (class, orbit, signs), -1 where there is none
  int rep[kOrbits][3];            // |o|
};

int block_size(int he, int ho, int b) {
  int s = 1;
  for (int q = 0; q < 3; ++q) s *= ((b >> q) & 1) ? ho : he;
  return s;
}

SymGeom make_geom(int n) {
  SymGeom g;
  g.n = n;
  g.he = (n + 1) / 2;
  g.ho = n / 2;
  g.P = n * n * n;
  const int full = g.he * g.he * g.he;
  g.KB = (full + 3) / 4 * 4;
  g.NB = full <= 8 ? 1 : (full <= 32 ? 4 : 8);
  g.MB = g.NB == 8 ? 4 : 8;
  int o = 0;
  for (int b = 0; b < 8; ++b) {
    g.size[b] = block_size(g.he, g.ho, b);
    g.off[b] = o;
    o += g.size[b];
  }
  // K steps by zero mask: the blocks b0 over the nonzero dimensions; along
  // the zero ones the step spans the blocks of both parities (the even one
  // is the longer)
  for (int z = 0; z < 8; ++z) {
    int steps = 0;
    for (int s = 0; s < kSymMaxStages; ++s) g.desc[z][s][0] = g.desc[z][s][1] = -1;
    if (z != 7)
      for (int b0 = 0; b0 < 8; ++b0) {
        if (b0 & z) continue;
        const int k4s = (g.size[b0] + 3) / 4;
        for (int k4 = 0; k4 < k4s; ++k4, ++steps) g.desc[z][steps / 2][steps % 2] = b0 | (k4 << 3);
      }
    g.nst[z] = (steps + 1) / 2;
  }
  int w = 0;
  g.total = 0;
  int orbit_of[64];
  for (int i = 0; i < 64; ++i) {
    const int r[3] = {i / 16, (i / 4) % 4, i % 4};
    orbit_of[i] = -1;
    if (r[0] <= 1 && r[1] <= 1 && r[2] <= 1) continue;
    orbit_of[i] = w;
    int z = 0, u = 0;
    for (int q = 0; q < 3; ++q) {
      g.rep[w][q] = r[q];
      if (r[q] == 0) z |= 1 << q;
      if (r[q] == 3) u |= 1 << q;
    }
    g.zmask[w] = z;
    g.umask[w] = u;
    g.stage0[w] = g.total;
    g.total += g.nst[z];
    ++w;
  }
  const FarTables& F = far_tables(3);
  for (int c = 0; c < 8; ++c) {
    g.neg[c] = 0;
    for (int i = 0; i < kOrbits; ++i)
      for (int s = 0; s < 8; ++s) g.slot[c][i][s] = -1;
    for (int q = 0; q < F.nfar; ++q) {
      const int* v = F.off_vec[F.slot_off[c][q]];
      int sg = 0;
      for (int e = 0; e < 3; ++e) {
        sg |= v[e] < 0 ? 1 << e : 0;
        if (v[e] == -3) g.neg[c] |= 1 << e;
      }
      g.slot[c][orbit_of[std::abs(v[0]) * 16 + std::abs(v[1]) * 4 + std::abs(v[2])]][sg] = q;
    }
  }
  return g;
}

const SymGeom& sym_geom(int n) {
  static const SymGeom g[6] = {make_geom(3), make_geom(4), make_geom(5), make_geom(6), make_geom(7), make_geom(8)};
  return g[n - 3];
}

// Half-index h of a node triple, its parity block offsets and node numbers.
struct Half {
  int j[3], mid;  // mid bit q: j_q is the centre node (odd n), which has no odd part
  __device__ __forceinline__ Half(int h, int he, int ho) {
    j[2] = h % he;
    j[1] = (h / he) % he;
    j[0] = h / (he * he);
    mid = 0;
#pragma unroll
    for (int q = 0; q < 3; ++q) mid |= j[q] >= ho ? 1 << q : 0;
  }
  __device__ __forceinline__ int in_block(int b, int he, int ho) const {
    const int s1 = (b & 2) ? ho : he, s2 = (b & 4) ? ho : he;
    return (j[0] * s1 + j[1]) * s2 + j[2];
  }
  __device__ __forceinline__ int node(int sg, int n) const {
    int k = 0;
#pragma unroll
    for (int q = 0; q < 3; ++q) k = k * n + (((sg >> q) & 1) ? n - 1 - j[q] : j[q]);
    return k;
  }
};

__device__ __forceinline__ void butterfly8(double* v) {
#pragma unroll
  for (int q = 1; q < 8; q <<= 1)
#pragma unroll
    for (int i = 0; i < 8; ++i)
      if (!(i & q)) {
        const double u = v[i], t = v[i | q];
        v[i] = u + t;
        v[i | q] = u - t;
      }
}

// s + e = a + b exactly (Knuth).
__device__ __forceinline__ void two_sum(double a, double b, double& s, double& e) {
  const double t = __dadd_rn(a, b), bb = __dsub_rn(t, a);
  e = __dadd_rn(__dsub_rn(a, __dsub_rn(t, bb)), __dsub_rn(b, bb));
  s = t;
}

// (len (x/2 - (o + y/2)))^2 with its rounding error.
__device__ __forceinline__ void sym_square(double x, double y, int o, double len, double& s, double& e) {
  double a, al, t, tl;
  two_sum(x / 2, -y / 2, a, al);
  two_sum(a, -(double)o, t, tl);
  const double p = len * t, pl = fma(len, t, -p) + len * (tl + al);
  s = p * p;
  e = fma(p, p, -s) + 2.0 * p * pl;
}

// Kernel values at offset o (in box widths) between a source node y and the
// target nodes x0 and x1, which differ in the last dimension only.  The
// Gaussian's argument is formed and divided with its rounding error, which its
// value takes r^2/p0 times over otherwise; the other kernels as everywhere.
template <int KID>
__device__ __forceinline__ void sym_values(const double* x0, const double* x1, const double* y, const int* o,
                                           double len, double p0, double ip, double (&f)[2]) {
  if constexpr (KID == FMMA_KERNEL_GAUSSIAN) {
    double r, e, s0, e0, s1, e1;
    sym_square(x0[0], y[0], o[0], len, s0, e0);
    sym_square(x0[1], y[1], o[1], len, s1, e1);
    two_sum(s0, s1, r, e);
    e += e0 + e1;
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      double s, es, r2, rl;
      sym_square(u ? x1[2] : x0[2], y[2], o[2], len, s, es);
      two_sum(r, s, r2, rl);
      rl += e + es;
      const double a = ip != 0.0 ? r2 * ip : r2 / p0;  // and what is left of r^2
      const double d = fma(-a, p0, r2) + rl;
      f[u] = exp(-a);
      if (f[u] > 0.0) f[u] -= f[u] * (ip != 0.0 ? d * ip : d / p0);
    }
  } else {
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      double v[3], w[3];
#pragma unroll
      for (int q = 0; q < 3; ++q) {
        v[q] = len * ((u ? x1[q] : x0[q]) / 2);
        w[q] = len * ((double)o[q] + y[q] / 2);
      }
      f[u] = keval<KID, 3>(v, w, p0);
    }
  }
}

// Operators in the parity basis, one warp per (table, orbit, i, j) with i, j
// half-indices: the 64 values of f over the reversals of i and j (two per
// lane), transformed along both by shuffles, give the entry (i, j) of all 64
// blocks.  The halves of the inverse transforms on both sides, 1/64 in all, are
// in the folded sources.  Error of the M2L against long double over that of
// k_m2l_f64, median over 3 to 8 nodes, four kernels and all levels: 0.25 (the
// sums are 39.5/189 as long); what the care for the Gaussian's argument is for
// (36 -> 41 us a level at 5 nodes, once a geometry): p0 = 0.01 in the unit cube,
// level 2, 4 nodes, 1.13 -> 0.16.
template <int KID>
__global__ void __launch_bounds__(256) k_sym_table(const double* __restrict__ lens, int ntab,
                                                   const double* __restrict__ node_all,
                                                   const SymGeom* __restrict__ gp, double p0,
                                                   double* __restrict__ tab) {
  const SymGeom& g = *gp;
  const int n = g.n, he = g.he, ho = g.ho, NB = g.NB;
  const int nh = he * he * he, lane = threadIdx.x & 31;
  const double ip = kinv<KID>(p0);
  const int64_t total = (int64_t)ntab * kOrbits * nh * nh;
  const int64_t nw = ((int64_t)gridDim.x * blockDim.x) >> 5;
  for (int64_t e = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; e < total; e += nw) {
    const int hj = (int)(e % nh), hi = (int)(e / nh % nh), w = (int)(e / ((int64_t)nh * nh) % kOrbits);
    const int64_t t = e / ((int64_t)nh * nh * kOrbits);
    const double len = lens[t];
    const Half I(hi, he, ho), J(hj, he, ho);
    double v[2];  // index = row reversal * 8 + column reversal = lane + 32 u
    sym_values<KID>(node_all + 3 * I.node(lane >> 3, n), node_all + 3 * I.node((lane >> 3) + 4, n),
                    node_all + 3 * J.node(lane & 7, n), g.rep[w], len, p0, ip, v);
    const double s = v[0] + v[1], d = v[0] - v[1];
    v[0] = s;
    v[1] = d;
#pragma unroll
    for (int q = 1; q < 32; q <<= 1)
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        const double o = __shfl_xor_sync(0xffffffffu, v[u], q);
        v[u] = (lane & q) ? o - v[u] : v[u] + o;
      }
    const int z = g.zmask[w], b = lane & 7, b0 = b & ~z;
    if (b & J.mid) continue;
    const int k = J.in_block(b, he, ho);
    int step = k >> 2;  // K steps of the blocks before b0
    for (int c = 0; c < b0; ++c)
      if (!(c & z)) step += (g.size[c] + 3) / 4;
    double* base = tab + (t * g.total + g.stage0[w] + (step >> 1)) * (int64_t)(8 * 2 * 32) * NB;
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      const int a = (lane >> 3) + 4 * u;
      if ((a & I.mid) || ((a ^ b) & z)) continue;
      const int col = I.in_block(a, he, ho);
      const int l = (col & 7) * 4 + (k & 3), nb = col >> 3;  // lane and column group of the fragment
      const int64_t at = ((int64_t)a * 2 + (step & 1)) * (32 * NB) + (NB == 1 ? l : (nb >> 1) * 64 + l * 2 + (nb & 1));
      base[at] = v[u];
    }
  }
}

// out[row][b][KB]: the even and odd parts of Wm's rows (box x rhs) by 1/64, zero
// padded, and a row of zeros behind them (the source of an empty slot).  The
// factor is exact, and taken here it keeps the sums of up to 64 coefficients,
// in the fold and in the butterfly, within the largest of them: no weight
// overflows that did not in the sum offset by offset.
__global__ void __launch_bounds__(256) k_sym_fold(const double* __restrict__ Wm, int64_t nrows, int Kpad,
                                                  const SymGeom* __restrict__ gp, double* __restrict__ out) {
  const int n = gp->n, he = gp->he, ho = gp->ho, KB = gp->KB;
  const int nh = he * he * he, lane = threadIdx.x & 31;
  const int64_t nw = ((int64_t)gridDim.x * blockDim.x) >> 5;
  for (int64_t row = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; row <= nrows; row += nw) {
    const double* w = Wm + row * Kpad;
    double* o = out + row * 8 * KB;
    if (row == nrows) {
      for (int k = lane; k < 8 * KB; k += 32) o[k] = 0.0;
      break;
    }
    for (int h = lane; h < nh; h += 32) {
      const Half H(h, he, ho);
      double v[8];
#pragma unroll
      for (int s = 0; s < 8; ++s) v[s] = (s & H.mid) ? 0.0 : w[H.node(s, n)] * (1.0 / 64);
      butterfly8(v);
#pragma unroll
      for (int b = 0; b < 8; ++b)
        if (!(b & H.mid)) o[b * KB + H.in_block(b, he, ho)] = v[b];
    }
#pragma unroll
    for (int b = 0; b < 8; ++b)
      for (int k = gp->size[b] + lane; k < KB; k += 32) o[b * KB + k] = 0.0;
  }
}

// Wl rows from their parity blocks: the nparts partial sums in order, then the
// inverse transform (its halves are in the folded sources).  With one part the
// blocks lie in Wl itself and a warp turns a row in place.
// Latency bound: a part's loads are all in flight before its sums (coefficient
// by coefficient over the parts 437, 351 and 67 us in the three cases above,
// now 296, 252 and 63).
__global__ void __launch_bounds__(256) k_sym_unfold(const double* __restrict__ part, int nparts, int64_t nv, int R,
                                                    const int* __restrict__ row_box, int Kpad,
                                                    const SymGeom* __restrict__ gp, double* __restrict__ Wl) {
  const int n = gp->n, he = gp->he, ho = gp->ho, P = gp->P;
  const int nh = he * he * he, lane = threadIdx.x & 31;
  const int64_t nw = ((int64_t)gridDim.x * blockDim.x) >> 5;
  for (int64_t v = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; v < nv; v += nw) {
    const int64_t brow = v / R;
    double* dst = Wl + ((int64_t)row_box[brow] * R + (v - brow * R)) * Kpad;
    const double* src = nparts > 1 ? part + v * P : dst;
    double y[2][8];  // at most 64 half-indices: two per lane
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      const int h = lane + 32 * u;
      const Half H(h < nh ? h : 0, he, ho);
      int k[8];  // -1: no such coefficient
#pragma unroll
      for (int a = 0; a < 8; ++a) {
        k[a] = h < nh && !(a & H.mid) ? gp->off[a] + H.in_block(a, he, ho) : -1;
        y[u][a] = k[a] >= 0 ? src[k[a]] : 0.0;
      }
      if (32 * u < nh) {
        const double* sp = src;
#pragma unroll 2
        for (int p = 1; p < nparts; ++p) {  // eight loads of a part in flight
          sp += nv * P;
#pragma unroll
          for (int a = 0; a < 8; ++a)
            if (k[a] >= 0) y[u][a] += sp[k[a]];
        }
      }
    }
    __syncwarp();
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      const int h = lane + 32 * u;
      if (h >= nh) continue;
      const Half H(h, he, ho);
      butterfly8(y[u]);
#pragma unroll
      for (int s = 0; s < 8; ++s)
        if (!(s & H.mid)) dst[H.node(s, n)] = y[u][s];
    }
    __syncwarp();
  }
}

struct SymParams {
  const int4* tiles;
  const int* il;
  const int* row_box;
  const SymGeom* geom;
  const double* W;     // folded sources [box * R + r][8][KB]
  const double* tab;   // [table][stage][a][step][column group pair][lane][2]
  const int* part_lo;  // [gridDim.y + 1] first orbit of each part
  double* Wl;          // parity blocks into Wl (one part) ...
  double* part;        // ... or [part][virtual row][P]
  int64_t nv;          // virtual rows (rows x rhs)
  int R, Kpad;
  int zero_row;        // the row of zeros of W
  int* err;            // set when a bounded wait gives up
  long long wait_cycles;  // the bound
  int hold;            // test hook: the gathering warps never report a stage
};

__device__ __forceinline__ uint32_t smem_addr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void bar_init(uint64_t* bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;\n" ::"r"(smem_addr(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void bar_arrive(uint64_t* bar) {
  asm volatile("{\n.reg .b64 st;\nmbarrier.arrive.shared::cta.b64 st, [%0];\n}\n" ::"r"(smem_addr(bar)) : "memory");
}
__device__ __forceinline__ bool bar_try(uint64_t* bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n.reg .pred p;\nmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\nselp.u32 %0, 1, 0, p;\n}\n"
      : "=r"(ok)
      : "r"(smem_addr(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}
// Whether the phase is complete, without waiting.
__device__ __forceinline__ bool bar_test(uint64_t* bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n.reg .pred p;\nmbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\nselp.u32 %0, 1, 0, p;\n}\n"
      : "=r"(ok)
      : "r"(smem_addr(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}
// Bounded wait of a whole warp: false, for all its lanes, when the bound passes
// or another warp has given up.  The vote is what keeps the warp together: the
// lanes poll on their own, and what follows (DMMAs, votes, shuffles) needs all
// of them, or none where the wait failed.
__device__ __forceinline__ bool bar_wait(uint64_t* bar, uint32_t parity, volatile int* abort, long long limit) {
  bool ok = bar_try(bar, parity);
  if (!ok) {
    const long long t0 = clock64();
    while (true) {
      for (int i = 0; i < 32 && !ok; ++i) ok = bar_try(bar, parity);
      if (ok || *abort) break;
      if (clock64() - t0 > limit) {
        *abort = 1;
        break;
      }
    }
  }
  return __all_sync(0xffffffffu, ok);
}

__device__ __forceinline__ void dmma(double& d0, double& d1, double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};\n"
               : "+d"(d0), "+d"(d1)
               : "d"(a), "d"(b));
}

template <int NB, int MB>
struct SymShape {
  static constexpr int TM = 8 * MB;
  static constexpr int TPR = 256 / TM;               // threads gathering one row
  static constexpr int EPT = 8 / TPR;                // values of a stage's 8 per thread
  static constexpr int PLANE = 8 * TM * 4 + 8;       // doubles of one K step's z (padded by 64 B)
  // registers a thread after the split: 256 (kMulRegs + kGatherRegs) = 512 * 128, the launch's
  static constexpr int kMulRegs = 176, kGatherRegs = 256 - kMulRegs;
  static constexpr int KB = NB == 1 ? 8 : (NB == 4 ? 28 : 64);  // SymGeom::KB of its node counts
  static constexpr int ILS = TM + 1;                 // stride of a slot's source list
  static constexpr int kTabStage = 8 * 2 * 32 * NB;  // doubles of a stage's operator
  static constexpr size_t kSmem = sizeof(double) * kSymRing * 2 * PLANE +
                                  sizeof(int) * (kSymSlots * ILS + 8 * kSymMaxStages * 2 + kOrbits * 8 + kOrbits * 5);
};

// What the multiplying warps read of the block.
struct SymBlock {
  const double* z;     // ring of z
  const double* tab;   // operators of the tile's table
  const int4* act;     // active orbits
  const int2* desc;    // K steps by zero mask and stage
  uint64_t *full, *empty;
  int* abort;
  long long limit;     // bound of a wait
  int nact, neg, v0, vcnt;
};

// One multiplying warp.  Its accumulators are two parts of row groups: with an
// even node count (PAIR false) the first G0 and the following G1 groups of the
// tile for one parity a0, with an odd one G0 = G1 groups of one half of the
// tile for the parities a0 and 7 - a0, whose column groups N0 + N1 are the
// same for every warp.  A stage is four units (K step, part) in a straight
// line: the source fragments of a unit load under the DMMAs of the one before,
// the next stage's first ones too when that stage is there already, and the
// operator fragments a stage ahead.
template <int NB, int MB, bool PAIR, int N0, int N1, int G0, int G1>
__device__ __forceinline__ bool sym_multiply(const SymParams& p, const SymBlock& sb, int warp, int lane) {
  using S = SymShape<NB, MB>;
  constexpr int TM = S::TM, H = MB / 2, NF = PAIR ? N0 + N1 : N0, GA = G0 > G1 ? G0 : G1, G1A = G1 > 0 ? G1 : 1;
  const int a0 = PAIR ? warp & 3 : (warp < 4 ? warp : 11 - warp);
  const int a1 = PAIR ? 7 - a0 : a0;
  const int row1 = PAIR ? 0 : G0 * 32, row0 = PAIR ? (warp >> 2) * H * 32 : 0;
  double acc0[G0][N0][2], acc1[G1A][N1][2], bf[2][NF], av[2][GA];
#pragma unroll
  for (int i = 0; i < G0; ++i)
#pragma unroll
    for (int j = 0; j < N0; ++j) acc0[i][j][0] = acc0[i][j][1] = 0.0;
#pragma unroll
  for (int i = 0; i < G1A; ++i)
#pragma unroll
    for (int j = 0; j < N1; ++j) acc1[i][j][0] = acc1[i][j][1] = 0.0;
  const double* const b0 = sb.tab + a0 * (2 * 32 * NB) + lane * (NB == 1 ? 1 : 2);
  const double* const b1 = sb.tab + a1 * (2 * 32 * NB) + lane * (NB == 1 ? 1 : 2);
  auto load_b = [&](int stage, int ks) {
#pragma unroll
    for (int part = 0; part < (PAIR ? 2 : 1); ++part) {
      const double* src = (part ? b1 : b0) + (int64_t)stage * S::kTabStage + ks * (32 * NB);
      const int n = part ? N1 : N0, f = part ? N0 : 0;
#pragma unroll
      for (int j = 0; j < n; j += 2) {
        if (NB > 1 && j + 1 < n) {
          const double2 t = __ldg(reinterpret_cast<const double2*>(src + (j >> 1) * 64));
          bf[ks][f + j] = t.x;
          bf[ks][f + j + 1 < NF ? f + j + 1 : 0] = t.y;
        } else {
          bf[ks][f + j] = __ldg(src + (j >> 1) * 64);
        }
      }
    }
  };
  struct Stage {
    int s0, s1, u, un, tab;  // un: the one-sided dimensions on the negative side
  };
  int oi = 0, st = -1, nst = 0, slot = 0, phase = 0;
  Stage cur, nxt{};
  const int2* ds = nullptr;
  // the next stage of the list; false at the end
  auto advance = [&]() -> bool {
    if (++st >= nst) {
      if (nst > 0) ++oi;
      if (oi >= sb.nact) return false;
      const int4 f = sb.act[oi];
      ds = sb.desc + ((f.x >> 8) & 7) * kSymMaxStages;
      nxt.u = f.x >> 16;
      nxt.un = nxt.u & sb.neg;
      nxt.tab = f.w - 1;
      nst = f.y;
      st = 0;
    }
    const int2 d = ds[st];
    nxt.s0 = d.x;
    nxt.s1 = d.y;
    ++nxt.tab;
    return true;
  };
  // z of (K step, part) of a stage, and the sign of its operator blocks
  const double* const z0 = sb.z + row0 + lane;
  auto load_a = [&](double* v, const Stage& s, int sl, int ks, int part) {
    const int c = (part ? a1 : a0) ^ ((ks ? s.s1 : s.s0) & 7);
    const double* src = z0 + (sl * 2 + ks) * S::PLANE + (c & ~s.u) * (TM * 4) + (part ? row1 : 0);
#pragma unroll
    for (int mb = 0; mb < (part ? G1 : G0); ++mb) v[mb] = src[mb * 32];
  };
  auto flip = [&](const Stage& s, int ks) {
    if (s.un == 0) return;
#pragma unroll
    for (int part = 0; part < (PAIR ? 2 : 1); ++part) {
      const int c = (part ? a1 : a0) ^ ((ks ? s.s1 : s.s0) & 7);
      if (__popc(c & s.un) & 1) {
#pragma unroll
        for (int j = 0; j < (part ? N1 : N0); ++j) bf[ks][(part ? N0 : 0) + j] = -bf[ks][(part ? N0 : 0) + j];
      }
    }
  };
  auto mul = [&](const double* v, int ks, int part) {
    if (part == 0) {
#pragma unroll
      for (int nb = 0; nb < N0; ++nb)
#pragma unroll
        for (int mb = 0; mb < G0; ++mb) dmma(acc0[mb][nb][0], acc0[mb][nb][1], v[mb], bf[ks][nb]);
    } else {
#pragma unroll
      for (int nb = 0; nb < N1; ++nb)
#pragma unroll
        for (int mb = 0; mb < G1; ++mb) dmma(acc1[mb][nb][0], acc1[mb][nb][1], v[mb], bf[ks][(PAIR ? N0 : 0) + nb]);
    }
  };
  bool have = advance(), ready = false;  // ready: the stage's first source fragments are in av[0]
  cur = nxt;
  if (have) {
    load_b(cur.tab, 0);
    load_b(cur.tab, 1);
  }
  while (have) {
    const bool more = advance();  // nxt: the stage behind this one
    const int nslot = slot + 1 == kSymRing ? 0 : slot + 1, nphase = slot + 1 == kSymRing ? phase ^ 1 : phase;
    if (!ready) {
      if (!bar_wait(&sb.full[slot], phase, sb.abort, sb.limit)) return false;
      load_a(av[0], cur, slot, 0, 0);
    }
    const bool two = cur.s1 >= 0;  // the last stage of an orbit may have one K step
    flip(cur, 0);
    load_a(av[1], cur, slot, 0, 1);
    mul(av[0], 0, 0);
    if (two) load_a(av[0], cur, slot, 1, 0);
    mul(av[1], 0, 1);
    load_b(nxt.tab, 0);
    if (two) {
      flip(cur, 1);
      load_a(av[1], cur, slot, 1, 1);
      mul(av[0], 1, 0);
    }
    ready = more && __all_sync(0xffffffffu, bar_test(&sb.full[nslot], nphase));
    if (ready) load_a(av[0], nxt, nslot, 0, 0);
    if (two) mul(av[1], 1, 1);
    load_b(nxt.tab, 1);
    __syncwarp();
    if (lane == 0) bar_arrive(&sb.empty[slot]);  // the stage's values are in registers
    slot = nslot;
    phase = nphase;
    cur = nxt;
    have = more;
  }

  const SymGeom& g = *p.geom;
#pragma unroll
  for (int part = 0; part < 2; ++part) {
    const int a = part ? a1 : a0;
    const int size = g.size[a], first = g.off[a];
#pragma unroll
    for (int mb = 0; mb < (part ? G1 : G0); ++mb) {
      const int i = (row0 + (part ? row1 : 0)) / 4 + mb * 8 + (lane >> 2);
      if (i >= sb.vcnt) continue;
      const int64_t v = sb.v0 + i;
      double* dst;
      if (gridDim.y > 1) {
        dst = p.part + ((int64_t)blockIdx.y * p.nv + v) * g.P + first;
      } else {
        const int64_t brow = v / p.R;
        dst = p.Wl + ((int64_t)p.row_box[brow] * p.R + (v - brow * p.R)) * p.Kpad + first;
      }
#pragma unroll
      for (int nb = 0; nb < (part ? N1 : N0); ++nb) {
        const int col = nb * 8 + (lane & 3) * 2;
        const double x = part ? acc1[part ? mb : 0][part ? nb : 0][0] : acc0[part ? 0 : mb][part ? 0 : nb][0];
        const double y = part ? acc1[part ? mb : 0][part ? nb : 0][1] : acc0[part ? 0 : mb][part ? 0 : nb][1];
        if (col < size) dst[col] = x;
        if (col + 1 < size) dst[col + 1] = y;
      }
    }
  }
  return true;
}

// A multiplying warp without rows (the upper half of a small tile): it frees
// the stages as they come.
__device__ __forceinline__ bool sym_pass(const SymBlock& sb, int nstages, int lane) {
  for (int it = 0, slot = 0, phase = 0; it < nstages; ++it) {
    if (!bar_wait(&sb.full[slot], phase, sb.abort, sb.limit)) return false;
    __syncwarp();
    if (lane == 0) bar_arrive(&sb.empty[slot]);
    if (++slot == kSymRing) {
      slot = 0;
      phase ^= 1;
    }
  }
  return true;
}

// The parity (pair) of a warp by its number, for G0 (and G1) row groups.
template <int N, int NB, int MB, int G0, int G1>
__device__ __forceinline__ bool sym_warp(const SymParams& p, const SymBlock& sb, int warp, int lane) {
  if constexpr (N % 2 == 0) {
    constexpr int C = (N / 2 * (N / 2) * (N / 2) + 7) / 8;  // column groups of every parity
    return sym_multiply<NB, MB, false, C, C, G0, G1>(p, sb, warp, lane);
  } else {
    // column groups by the number of odd dimensions of the parity; warp & 3
    // has 0, 1, 1 and 2 of them, its partner 3, 2, 2 and 1
    constexpr int E = (N + 1) / 2, O = N / 2;
    constexpr int C0 = (E * E * E + 7) / 8, C1 = (E * E * O + 7) / 8, C2 = (E * O * O + 7) / 8,
                  C3 = (O * O * O + 7) / 8;
    if ((warp & 3) == 0) return sym_multiply<NB, MB, true, C0, C3, G0, G0>(p, sb, warp, lane);
    if ((warp & 3) == 3) return sym_multiply<NB, MB, true, C2, C1, G0, G0>(p, sb, warp, lane);
    return sym_multiply<NB, MB, true, C1, C2, G0, G0>(p, sb, warp, lane);
  }
}

// N nodes per dimension.
template <int N, int NB, int MB>
__global__ void __launch_bounds__(kSymThreads, 1) k_m2l_sym(const SymParams p) {
  using S = SymShape<NB, MB>;
  constexpr int TM = S::TM, EPT = S::EPT, KB = S::KB, kTabStage = S::kTabStage;
  extern __shared__ __align__(128) double sym_smem[];
  double* const sZ = sym_smem;                                              // [ring][2][PLANE]
  // active orbits: (orbit | zero mask << 8 | one-sided mask << 16, stages, 0, first stage)
  int4* const sAct = reinterpret_cast<int4*>(sZ + 2 * kSymRing * S::PLANE);
  int2* const sDesc = reinterpret_cast<int2*>(sAct + kOrbits);   // [zero mask][stage] K steps
  int* const sSlot = reinterpret_cast<int*>(sDesc + 8 * kSymMaxStages);  // [orbit][8]
  int* const sOn = sSlot + kOrbits * 8;                          // [orbit] it has a source
  int* const sIl = sOn + kOrbits;                                // [slot][ILS] source row (box * R + r)
  __shared__ uint64_t s_full[kSymRing], s_empty[kSymRing];
  __shared__ int4 s_orb[kOrbits];  // sAct's entries of all orbits
  __shared__ int s_nact, s_nst, s_abort;
  const SymGeom& g = *p.geom;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int4 tile = p.tiles[blockIdx.x];
  const int cls = tile.x, v0 = tile.y, vcnt = tile.z;
  const int R = p.R, none = p.zero_row;
  const int lo = p.part_lo[blockIdx.y], hi = p.part_lo[blockIdx.y + 1];
  // row groups gathered (multiplied: rounded up to 1, 2, half or all)
  const int used = (vcnt + 7) >> 3;
  const int groups = used > MB / 2 ? MB : used;

  // far slots of the rows (a warp takes TM / 16 rows, all loads in flight)
  {
    constexpr int RPW = TM / 16, LPR = (kSymSlots + 31) / 32;
    int s[RPW][LPR];
#pragma unroll
    for (int k = 0; k < RPW; ++k) {
      const int r = warp + 16 * k;
      const int v = v0 + min(r, vcnt - 1), brow = v / R, rr = v - brow * R;
      const int* row = p.il + (int64_t)brow * kSymSlots;
#pragma unroll
      for (int j = 0; j < LPR; ++j) {
        const int q = lane + 32 * j;
        const int sb = q < kSymSlots && r < vcnt ? row[q] : -1;
        s[k][j] = sb >= 0 ? sb * R + rr : none;
      }
    }
    for (int i = tid; i < 8 * kSymMaxStages; i += kSymThreads)
      sDesc[i] = make_int2((&g.desc[0][0][0])[2 * i], (&g.desc[0][0][0])[2 * i + 1]);
    for (int i = tid; i < kOrbits * 8; i += kSymThreads) sSlot[i] = g.slot[cls][i >> 3][i & 7];
    if (tid < kOrbits) {
      const int z = g.zmask[tid];
      s_orb[tid] = make_int4(tid | (z << 8) | (g.umask[tid] << 16), g.nst[z], 0, g.stage0[tid]);
      sOn[tid] = 0;
    }
#pragma unroll
    for (int k = 0; k < RPW; ++k)
#pragma unroll
      for (int j = 0; j < LPR; ++j)
        if (lane + 32 * j < kSymSlots) sIl[(lane + 32 * j) * S::ILS + warp + 16 * k] = s[k][j];
  }
  if (tid == 0) {
    for (int s = 0; s < kSymRing; ++s) {
      bar_init(&s_full[s], 8);   // a lane of each gathering warp
      bar_init(&s_empty[s], 8);  // a lane of each multiplying warp
    }
    s_abort = 0;
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
  }
  __syncthreads();
  for (int i = tid; i < (hi - lo) * MB; i += kSymThreads) {
    const int w = lo + i / MB, mb = i % MB;
    bool any = false;
    for (int s = 0; s < 8; ++s) {
      const int q = sSlot[w * 8 + s];
      if (q < 0) continue;
#pragma unroll
      for (int r = 0; r < 8; ++r) any |= sIl[q * S::ILS + mb * 8 + r] != none;
    }
    if (any) sOn[w] = 1;
  }
  __syncthreads();
  if (warp == 0) {
    int base = 0, stages = 0;
    for (int w0 = 0; w0 < kOrbits; w0 += 32) {
      const int w = w0 + lane;
      const bool on = w < kOrbits && sOn[w] != 0;
      const unsigned m = __ballot_sync(0xffffffffu, on);
      if (on) {
        sAct[base + __popc(m & ((1u << lane) - 1u))] = s_orb[w];
        stages += s_orb[w].y;
      }
      base += __popc(m);
    }
    stages = __reduce_add_sync(0xffffffffu, stages);
    if (lane == 0) {
      s_nact = base;
      s_nst = stages;
    }
  }
  __syncthreads();
  const int nact = s_nact;

  if (warp >= 8) {
    // ---- gathering warps: one row, EPT consecutive k of one K step a thread ----
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;\n" ::"n"(S::kGatherRegs));
    const int gt = tid - 256;
    const int grow = gt / S::TPR, gp = gt % S::TPR;
    const int gks = EPT == 2 ? gp >> 1 : gp >> 2;
    const int gk = EPT == 2 ? (gp & 1) * 2 : gp & 3;
    const bool mine = (grow >> 3) < groups;  // warp-uniform
    double* const zdst = sZ + gks * S::PLANE + grow * 4 + gk;
    const int neg = g.neg[cls];
    int slot = 0, phase = 1;
    bool ok = true;
    for (int oi = 0; oi < nact && ok; ++oi) {
      const int4 f = sAct[oi];
      // u: the one-sided dimensions; only the planes j with no bit of u are made
      const int z = (f.x >> 8) & 7, u = f.x >> 16, nst = f.y;
      const int* sl = sSlot + (f.x & 255) * 8;
      const int* ds = reinterpret_cast<const int*>(sDesc + z * kSymMaxStages) + gks;
      unsigned off[8];  // the orbit's sources, in units of 4 doubles
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const int q = sl[(j & ~z & ~u) | (neg & u)];
        const int s = q >= 0 ? sIl[q * S::ILS + grow] : none;
        off[j] = (unsigned)s * (2u * KB) + (unsigned)((j & z) * (KB / 4));
      }
      for (int st = 0; st < nst; ++st) {
        double raw[8][EPT];
        if (mine) {
          const int step = max(ds[st * 2], 0);  // no step: any data, not multiplied
          const char* src = reinterpret_cast<const char*>(p.W + (step & 7) * KB + (step >> 3) * 4 + gk);
#pragma unroll
          for (int j = 0; j < 8; ++j)
            if (!(j & u)) {
              const char* sj = src + (uint64_t)off[j] * 32u;
              if constexpr (EPT == 2) {
                const double2 t = __ldg(reinterpret_cast<const double2*>(sj));
                raw[j][0] = t.x;
                raw[j][EPT - 1] = t.y;
              } else {
                raw[j][0] = __ldg(reinterpret_cast<const double*>(sj));
              }
            }
        }
        ok = bar_wait(&s_empty[slot], phase, &s_abort, p.wait_cycles);
        if (!ok) break;
        if (mine) {
#pragma unroll
          for (int q = 1; q < 8; q <<= 1)
            if (!((z | u) & q)) {
#pragma unroll
              for (int j = 0; j < 8; ++j)
                if (!(j & q)) {
                  if (j & u) continue;
#pragma unroll
                  for (int e = 0; e < EPT; ++e) {
                    const double x = raw[j][e], y = raw[j | q][e];
                    raw[j][e] = x + y;
                    raw[j | q][e] = x - y;
                  }
                }
            }
          double* dst = zdst + slot * 2 * S::PLANE;
#pragma unroll
          for (int j = 0; j < 8; ++j)
            if (!(j & u)) {
              if constexpr (EPT == 2)
                *reinterpret_cast<double2*>(dst + j * TM * 4) = make_double2(raw[j][0], raw[j][EPT - 1]);
              else
                dst[j * TM * 4] = raw[j][0];
            }
        }
        __syncwarp();
        if (lane == 0 && !p.hold) bar_arrive(&s_full[slot]);
        if (++slot == kSymRing) {
          slot = 0;
          phase ^= 1;
        }
      }
    }
    if (!ok) *p.err = 1;
    return;
  }

  // ---- multiplying warps ----
  asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;\n" ::"n"(S::kMulRegs));
  const SymBlock sb{sZ,      p.tab + (int64_t)tile.w * g.total * kTabStage, sAct, sDesc, s_full, s_empty,
                    &s_abort, p.wait_cycles, nact, g.neg[cls], v0, vcnt};
  constexpr int H = MB / 2;
  bool ok;
  if (groups > H) ok = sym_warp<N, NB, MB, H, H>(p, sb, warp, lane);
  else if (N % 2 == 1 && warp >= 4) ok = sym_pass(sb, s_nst, lane);
  else if (groups > 2) ok = sym_warp<N, NB, MB, H, 0>(p, sb, warp, lane);
  else if (groups == 2) ok = sym_warp<N, NB, MB, 2, 0>(p, sb, warp, lane);
  else ok = sym_warp<N, NB, MB, 1, 0>(p, sb, warp, lane);
  if (!ok) *p.err = 1;
}

template <int N, int NB, int MB>
void launch_sym(fmma_ctx* ctx, const SymParams& p, int ntiles, int nparts) {
  constexpr size_t smem = SymShape<NB, MB>::kSmem;
  if (!ctx->capturing)  // the attribute is the current device's
    FMMA_CHECK_CUDA(cudaFuncSetAttribute(k_m2l_sym<N, NB, MB>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  FMMA_LAUNCH(ctx, (k_m2l_sym<N, NB, MB>), dim3((unsigned)ntiles, (unsigned)nparts), kSymThreads, smem, p);
}

struct SymTableLaunch {
  template <int KID, int D>
  static void run(fmma_ctx* ctx, const double* lens, int ntab, const double* node_all, const SymGeom* g, int64_t total,
                  double p0, double* tab) {
    if constexpr (D == 3 && (KID == FMMA_KERNEL_INV_R || KID == FMMA_KERNEL_INV_R_SAFE || KID == FMMA_KERNEL_LOG_R ||
                             KID == FMMA_KERNEL_GAUSSIAN || KID == FMMA_KERNEL_MULTIQUADRIC))
      FMMA_LAUNCH(ctx, (k_sym_table<KID>), grid_for(total * 32, 256, (int64_t)ctx->sm_count * 16), 256, 0, lens, ntab,
                  node_all, g, p0, tab);
  }
};

constexpr int kSymMaxParts = 16;

// The orbits of a tile are split over blocks where that fills the last wave
// of a level: a block costs its share of a tile plus about 2 % of one (the
// prologue and the partial sums), and one block runs on an SM at a time.
int sym_parts(const fmma_ctx* ctx, int64_t ntiles, int most) {
  int nparts = 1;
  double best = 0.0;
  for (int s = 1; s <= most; ++s) {
    const int64_t waves = (ntiles * s + ctx->sm_count - 1) / ctx->sm_count;
    const double t = (double)waves * (1.0 / s + 0.02);
    if (s == 1 || t < best) {
      best = t;
      nparts = s;
    }
  }
  return nparts;
}

size_t sym_src_bytes(const Level& Lv, const SymGeom& g, int R) {
  return sizeof(double) * (size_t)(Lv.nbox * R + 1) * 8 * g.KB;
}

}  // namespace

bool m2l_sym_scratch(fmma_ctx* ctx, const std::vector<const Level*>& levels, int n, int R, int* most_parts) {
  const SymGeom& g = sym_geom(n);
  const int TM = 8 * g.MB;
  size_t src = 0, part = 0;
  for (const Level* Lv : levels) {
    int64_t ntiles = 0;  // as m2l_tiles cuts the segments
    for (const int4& sg : Lv->segs) ntiles += ((int64_t)(sg.w - sg.z) * R + TM - 1) / TM;
    const int nparts = sym_parts(ctx, ntiles, kSymMaxParts);
    src = std::max(src, sym_src_bytes(*Lv, g, R));
    if (nparts > 1) part = std::max(part, sizeof(double) * (size_t)(nparts * Lv->nrow * R) * g.P);
  }
  if (!ctx_buf_try(ctx, "sym_src", src)) return false;
  *most_parts = part == 0 || ctx_buf_try(ctx, "sym_part", part) ? kSymMaxParts : 1;
  return true;
}

bool m2l_sym_ok(const fmma_ctx* ctx, int d, int n, int64_t rows) {
  // source rows are addressed in units of 4 doubles, in 32 bits
  if (rows >= ((int64_t)1 << 25)) return false;
  switch (ctx->kernel_id) {
    case FMMA_KERNEL_INV_R:
    case FMMA_KERNEL_INV_R_SAFE:
    case FMMA_KERNEL_LOG_R:
    case FMMA_KERNEL_GAUSSIAN:
    case FMMA_KERNEL_MULTIQUADRIC: return d == 3 && n >= 3 && n <= 8;
    default: return false;
  }
}

void m2l_level_sym(fmma_ctx* ctx, const Level& Lv, int v, int n, int Kpad, int R, const std::vector<double>& lens,
                   const std::string& tabkey, const double* node_all, const double* Wm, double* Wl, int most_parts) {
  const SymGeom& g = sym_geom(n);
  const int ntab = (int)lens.size();
  // geometry and operators in one cached block
  constexpr size_t kGeomBytes = (sizeof(SymGeom) + 255) / 256 * 256;
  const size_t per_tab = (size_t)g.total * 8 * 2 * 32 * g.NB;
  bool fresh = false;
  char* blk = reinterpret_cast<char*>(cached_op(ctx, "sym_" + tabkey, kGeomBytes + sizeof(double) * per_tab * ntab,
                                                &fresh));
  const SymGeom* dg = reinterpret_cast<const SymGeom*>(blk);
  double* tab = reinterpret_cast<double*>(blk + kGeomBytes);
  if (fresh) {
    upload(ctx, blk, &g, sizeof(SymGeom));
    double* dl = ctx_buf_t<double>(ctx, "table_lens", (size_t)ntab);
    upload(ctx, dl, lens.data(), sizeof(double) * (size_t)ntab);
    FMMA_CHECK_CUDA(cudaMemsetAsync(tab, 0, sizeof(double) * per_tab * ntab, ctx->stream));
    const int64_t nh = (int64_t)g.he * g.he * g.he;
    dispatch_kernel<SymTableLaunch>(ctx->kernel_id, 3, ctx, dl, ntab, node_all, dg, (int64_t)ntab * kOrbits * nh * nh,
                                    ctx->p0, tab);
  }
  const int TM = 8 * g.MB;
  std::vector<int4> tiles = m2l_tiles(Lv, R, TM);
  const int ntiles = (int)tiles.size();
  int4* dt = ctx_buf_t<int4>(ctx, "m2l_tiles" + std::to_string(v), tiles.size());
  upload(ctx, dt, tiles.data(), sizeof(int4) * tiles.size());

  const int nparts = sym_parts(ctx, ntiles, most_parts);
  std::vector<int> lo((size_t)nparts + 1, 0);
  for (int s = 1, w = 0; s < nparts; ++s) {
    while (w < kOrbits && (int64_t)g.stage0[w] * nparts < (int64_t)s * g.total) ++w;
    lo[(size_t)s] = w;
  }
  lo[(size_t)nparts] = kOrbits;
  int* dlo = ctx_buf_t<int>(ctx, "sym_parts" + std::to_string(v), lo.size());
  upload(ctx, dlo, lo.data(), sizeof(int) * lo.size());

  const int64_t nv = Lv.nrow * R, nsrc = Lv.nbox * R;
  double* W = static_cast<double*>(ctx_buf(ctx, "sym_src", sym_src_bytes(Lv, g, R)));
  double* part = nullptr;
  if (nparts > 1) part = static_cast<double*>(ctx_buf(ctx, "sym_part", sizeof(double) * (size_t)(nparts * nv) * g.P));
  int* err = m2l_err_slot(ctx, v);
  FMMA_CHECK_CUDA(cudaMemsetAsync(err, 0, sizeof(int), ctx->stream));
  SymParams p{dt, Lv.il, Lv.row_box, dg, W, tab, dlo, Wl, part, nv, R, Kpad, (int)nsrc, err,
              ctx->tc_wait_cycles > 0 ? ctx->tc_wait_cycles : kSymWaitCycles, ctx->tc_hold ? 1 : 0};
  kernel_timer_begin(ctx);
  const int64_t wcap = (int64_t)ctx->sm_count * 32;
  FMMA_LAUNCH(ctx, k_sym_fold, grid_for((nsrc + 1) * 32, 256, wcap), 256, 0, Wm, nsrc, Kpad, dg, W);
  switch (n) {
    case 3: launch_sym<3, 1, 8>(ctx, p, ntiles, nparts); break;
    case 4: launch_sym<4, 1, 8>(ctx, p, ntiles, nparts); break;
    case 5: launch_sym<5, 4, 8>(ctx, p, ntiles, nparts); break;
    case 6: launch_sym<6, 4, 8>(ctx, p, ntiles, nparts); break;
    case 7: launch_sym<7, 8, 4>(ctx, p, ntiles, nparts); break;
    default: launch_sym<8, 8, 4>(ctx, p, ntiles, nparts); break;
  }
  FMMA_LAUNCH(ctx, k_sym_unfold, grid_for(nv * 32, 256, wcap), 256, 0, part, nparts, nv, R, Lv.row_box, Kpad, dg, Wl);
  kernel_timer_end(ctx, 2.0 * g.P * g.P * R, v);
  ctx->m2l_err_flags.push_back(err);
}

}  // namespace fmma_b200
