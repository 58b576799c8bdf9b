// tree.cu — integer tree build on the device: bounding cube, leaf binning
// (bit-exact with the reference), Morton keys, stable radix sort, leaf ranges,
// per-level box arrays, far (M2L) and near (P2P) interaction lists.
//
// Reference: binning src/fmm_core.cpp:255-267 and src/fmm.cpp:126-131, cube
// src/fmm_core.cpp:125-173, far list src/fmm_core.cpp:15-63, near list
// src/fmm_core.cpp:79-115.  The reference walks a dense 2^(d*l) grid; here
// only non-empty boxes exist (a box without sources contributes exact zeros
// to M2L/M2M/P2P, a box without targets receives nothing that is read).
#include <algorithm>
#include <cstring>

#include "fmm_stages.cuh"
#include "fmma_internal.cuh"

namespace fmma_b200 {

// ---------------------------------------------------------------------------
// far-slot tables
// ---------------------------------------------------------------------------
static FarTables make_far_tables(int d) {
  FarTables F;
  std::memset(&F, 0, sizeof(F));
  int p7 = 1, p6 = 1, p3 = 1;
  for (int q = 0; q < d; ++q) { p7 *= 7; p6 *= 6; p3 *= 3; }
  F.nfar = p6 - p3;
  F.noff = p7 - p3;
  F.nclass = 1 << d;
  // far offsets, row-major over (o + 3), last dimension fastest
  int offid[343];
  int cnt = 0;
  for (int s = 0; s < p7; ++s) {
    int o[3] = {0, 0, 0}, sc = s, dist = 0;
    for (int q = d - 1; q >= 0; --q) { o[q] = sc % 7 - 3; sc /= 7; dist = std::max(dist, std::abs(o[q])); }
    if (dist <= 1) { offid[s] = -1; continue; }
    offid[s] = cnt;
    for (int q = 0; q < d; ++q) F.off_vec[cnt][q] = o[q];
    ++cnt;
  }
  for (int c = 0; c < 8; ++c)
    for (int j = 0; j < 216; ++j) F.jslot[c][j] = -1;
  for (int c = 0; c < F.nclass; ++c) {
    int par[3] = {0, 0, 0};
    for (int q = 0; q < d; ++q) par[q] = (c >> (d - 1 - q)) & 1;
    int k = 0;
    for (int j = 0; j < p6; ++j) {
      int jd[3] = {0, 0, 0}, jc = j, dist = 0;
      for (int q = d - 1; q >= 0; --q) { jd[q] = jc % 6; jc /= 6; }
      int s7 = 0;
      for (int q = 0; q < d; ++q) {
        int o = jd[q] - 2 - par[q];
        dist = std::max(dist, std::abs(o));
        s7 = s7 * 7 + (o + 3);
      }
      if (dist <= 1) continue;
      F.slot_j[c][k] = j;
      F.slot_off[c][k] = offid[s7];
      F.jslot[c][j] = k;
      ++k;
    }
  }
  return F;
}

const FarTables& far_tables(int d) {  // made once, by whichever thread comes first
  static const FarTables F[kMaxDim] = {make_far_tables(1), make_far_tables(2), make_far_tables(3)};
  return F[d - 1];
}

// ---------------------------------------------------------------------------
// problem of each point, bounding cube per problem
// ---------------------------------------------------------------------------
__device__ __forceinline__ unsigned long long ord_enc(double x) {
  unsigned long long u = (unsigned long long)__double_as_longlong(x);
  return (u >> 63) ? ~u : (u | 0x8000000000000000ull);
}
__device__ __forceinline__ double ord_dec(unsigned long long u) {
  u = (u >> 63) ? (u & 0x7fffffffffffffffull) : ~u;
  return __longlong_as_double((long long)u);
}

__device__ __forceinline__ int find_seg(const int64_t* __restrict__ off, int np, int64_t i) {
  int lo = 0, hi = np;  // last p with off[p] <= i
  while (hi - lo > 1) {
    int m = (lo + hi) >> 1;
    if (off[m] <= i) lo = m; else hi = m;
  }
  return lo;
}

// problem id of each element of [targets | sources] (a single problem needs none:
// the kernels below take a null pid for 0)
__global__ void k_point_pid(const int64_t* __restrict__ toff, const int64_t* __restrict__ soff, int np, int64_t nt,
                            int64_t ns, int* __restrict__ pid) {
  const int64_t n = nt + ns;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    pid[i] = i < nt ? find_seg(toff, np, i) : find_seg(soff, np, i - nt);
}

__global__ void k_bbox_init(unsigned long long* mm, int np, int* flag) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < np * kMaxDim; i += gridDim.x * blockDim.x) {
    int p = i / kMaxDim, q = i % kMaxDim;
    mm[p * 2 * kMaxDim + q] = ~0ull;
    mm[p * 2 * kMaxDim + kMaxDim + q] = 0ull;
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) *flag = 0;
}

// Per-problem min/max of every coordinate over targets and sources: order
// free and exact (src/fmm_core.cpp:125-148).  Each warp scans one contiguous
// chunk (coalesced, 32 points per step) and each lane keeps running extrema
// for the problem it is in, flushing them with atomics only when the
// problem changes and once at the end (a warp reduction when the whole warp
// ends in one problem): a handful of atomics per warp instead of one per
// step.
__device__ __forceinline__ void bbox_flush(unsigned long long* mm, int p, int d, const unsigned long long* lo,
                                           const unsigned long long* hi) {
  for (int q = 0; q < d; ++q) {
    atomicMin(&mm[p * 2 * kMaxDim + q], lo[q]);
    atomicMax(&mm[p * 2 * kMaxDim + kMaxDim + q], hi[q]);
  }
}

template <typename T>
__global__ void k_bbox(const T* __restrict__ tgt, int64_t nt, const T* __restrict__ src, int64_t ns,
                       const int* __restrict__ pid, int d, unsigned long long* mm, int* flag) {
  const int64_t n = nt + ns;
  const int lane = threadIdx.x & 31;
  const int64_t nw = ((int64_t)gridDim.x * blockDim.x) >> 5;
  const int64_t wid = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int64_t chunk = ((n + nw - 1) / nw + 31) / 32 * 32;
  const int64_t b0 = wid * chunk, b1 = min(n, b0 + chunk);
  int bad = 0, cur = -1;
  unsigned long long lo[kMaxDim], hi[kMaxDim];
  for (int q = 0; q < kMaxDim; ++q) { lo[q] = ~0ull; hi[q] = 0ull; }
  for (int64_t i = b0 + lane; i < b1; i += 32) {
    const int p = pid ? pid[i] : 0;
    if (p != cur) {
      if (cur >= 0) bbox_flush(mm, cur, d, lo, hi);
      for (int q = 0; q < kMaxDim; ++q) { lo[q] = ~0ull; hi[q] = 0ull; }
      cur = p;
    }
    const T* x = i < nt ? tgt + i * d : src + (i - nt) * d;
    for (int q = 0; q < d; ++q) {
      const double v = (double)x[q];
      if (!isfinite(v)) bad = 1;
      const unsigned long long e = ord_enc(v);
      lo[q] = e < lo[q] ? e : lo[q];
      hi[q] = e > hi[q] ? e : hi[q];
    }
  }
  const unsigned same = __match_any_sync(0xffffffffu, cur);
  if (same == 0xffffffffu) {
    for (int q = 0; q < d; ++q)
      for (int o = 16; o > 0; o >>= 1) {
        const unsigned long long a = __shfl_xor_sync(0xffffffffu, lo[q], o);
        const unsigned long long bb = __shfl_xor_sync(0xffffffffu, hi[q], o);
        lo[q] = a < lo[q] ? a : lo[q];
        hi[q] = bb > hi[q] ? bb : hi[q];
      }
    if (lane == 0 && cur >= 0) bbox_flush(mm, cur, d, lo, hi);
  } else if (cur >= 0) {
    bbox_flush(mm, cur, d, lo, hi);
  }
  bad = __any_sync(0xffffffffu, bad);
  if (lane == 0 && bad) atomicOr(flag, 1);
}

// src/fmm_core.cpp:160-173 in the caller's precision, one problem per thread.
// A degenerate cube (every coordinate equal: the reference divides by zero
// there) gets Len = 1.
__global__ void k_cube(const unsigned long long* mm, const int* flag, int np, int d, Cube* cubes) {
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= np) return;
  const unsigned long long* m = mm + p * 2 * kMaxDim;
  double mn[kMaxDim], mx[kMaxDim];
  for (int q = 0; q < d; ++q) { mn[q] = ord_dec(m[q]); mx[q] = ord_dec(m[kMaxDim + q]); }
  Cube c;
  double L = 0.0;
  for (int q = 0; q < d; ++q) { double e = __dsub_rn(mx[q], mn[q]); L = L < e ? e : L; }
  if (!(L > 0.0)) L = 1.0;
  for (int q = 0; q < d; ++q) c.origin[q] = __dsub_rn(__dmul_rn(__dadd_rn(mx[q], mn[q]), 0.5), __dmul_rn(L, 0.5));
  c.Len = L;
  float Lf = 0.f;
  for (int q = 0; q < d; ++q) { float e = __fsub_rn((float)mx[q], (float)mn[q]); Lf = Lf < e ? e : Lf; }
  if (!(Lf > 0.f)) Lf = 1.f;
  for (int q = 0; q < d; ++q)
    c.originf[q] = __fsub_rn(__fmul_rn(__fadd_rn((float)mx[q], (float)mn[q]), 0.5f), __fmul_rn(Lf, 0.5f));
  c.Lenf = Lf;
  for (int q = d; q < kMaxDim; ++q) { c.origin[q] = 0.0; c.originf[q] = 0.f; }
  c.nonfinite = *flag;
  c.pad = 0;
  cubes[p] = c;
}

template <typename T>
__global__ void k_leaf_keys(const T* __restrict__ tgt, int64_t nt, const T* __restrict__ src, int64_t ns,
                            const int* __restrict__ pid, int d, const int* __restrict__ depth,
                            const Cube* __restrict__ cubes, uint64_t* __restrict__ keys, int* __restrict__ idx) {
  const int64_t n = nt + ns;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    const int p = pid ? pid[i] : 0;
    const Cube& c = cubes[p];
    const int bits = depth[p] - 1;
    const int N = 1 << bits;
    const T* x = i < nt ? tgt + i * d : src + (i - nt) * d;
    int cc[kMaxDim] = {0, 0, 0};
    for (int q = 0; q < d; ++q) cc[q] = bin_coord<T>(x[q], c, q, N);
    keys[i] = ((uint64_t)p << kPidShift) | morton_encode(cc, d, bits);
    if (idx) idx[i] = (int)i;
  }
}

// ---------------------------------------------------------------------------
// leaves and levels: every level from the sorted keys in three launches
//
// Key i opens a box at virtual level v when its level-v ancestor differs from
// key i-1's: at every level v <= hb / d, hb the highest bit in which the two
// Morton codes differ, and at every level when the problem changes, up to its
// problem's root (virtual level depth - 1).  With t_i the highest such level
// (-1: none), the box of key i at level v is number #{j <= i: t_j >= v} - 1 of
// that level, so all levels' boxes, parents, children and point ranges follow
// from one counting pass (per block and level), a scan over the blocks and one
// emitting pass.  The launches do not grow with the depth (12 per level
// before), which is what small trees cost.  Solves, launches and time: 1-D 4096
// points, 8 levels 133 -> 41, 1064 -> 583 us; 2-D 131k 110 -> 43, 1298 -> 976
// us; 3-D 4M clustered 240 -> 94, tree stage 5.7 -> 5.1 ms.
// ---------------------------------------------------------------------------
constexpr int kTreeThreads = 256;
constexpr int kTreeWarps = kTreeThreads / 32;
constexpr int kMaxLevels = 32;

// Highest level at which key i's ancestor differs from key i-1's (63: another
// problem, or the first key; -1: the same leaf).
__device__ __forceinline__ int key_diff(const uint64_t* __restrict__ keys, int64_t i, int d) {
  if (i == 0) return 63;
  const uint64_t k = keys[i], kp = keys[i - 1];
  if (key_pid(k) != key_pid(kp)) return 63;
  const uint64_t x = (k ^ kp) & kMortonMask;
  return x == 0 ? -1 : (63 - __clzll((long long)x)) / d;
}

// cnt[v * gridDim.x + block] = keys of the block's tile with t >= v (v < V);
// row V: targets.
__global__ void __launch_bounds__(kTreeThreads) k_tree_count(const uint64_t* __restrict__ keys,
                                                             const int* __restrict__ idx, int64_t n, int64_t nt,
                                                             int rounds, int d, const int* __restrict__ depth, int V,
                                                             int* __restrict__ cnt) {
  __shared__ int h[kMaxLevels + 1];
  if (threadIdx.x <= kMaxLevels) h[threadIdx.x] = 0;
  __syncthreads();
  const int64_t base = (int64_t)blockIdx.x * rounds * kTreeThreads;
  for (int r = 0; r < rounds; ++r) {
    const int64_t i = base + (int64_t)r * kTreeThreads + threadIdx.x;
    const int t = i < n ? min(key_diff(keys, i, d), depth[key_pid(keys[i])] - 1) : -1;
    if (t >= 0) atomicAdd(&h[t], 1);
    const unsigned m = __ballot_sync(0xffffffffu, i < n && idx[i] < nt);
    if ((threadIdx.x & 31) == 0 && m) atomicAdd(&h[kMaxLevels], __popc(m));
  }
  __syncthreads();
  if (threadIdx.x < V) {
    int s = 0;
    for (int t = threadIdx.x; t < V; ++t) s += h[t];
    cnt[(int64_t)threadIdx.x * gridDim.x + blockIdx.x] = s;
  }
  if (threadIdx.x == V) cnt[(int64_t)V * gridDim.x + blockIdx.x] = h[kMaxLevels];
}

// First box of each level in the arrays of all levels.
struct LevelOff {
  int64_t o[kMaxLevels + 1];
};

struct LevelArrays {
  uint64_t* key;
  int *tb, *te, *sb, *se, *cb, *ce, *parent;
};

// The boxes of every level and the point permutations.  off: the scanned
// counts (exclusive over the blocks).  The key that opens a box writes its
// key, begins and parent; the next key that leaves it (or the end) its ends.
__global__ void __launch_bounds__(kTreeThreads) k_tree_emit(const uint64_t* __restrict__ keys,
                                                            const int* __restrict__ idx, int64_t n, int64_t nt,
                                                            int rounds, int d, const int* __restrict__ depth, int V,
                                                            const int* __restrict__ off, const LevelOff lo,
                                                            const LevelArrays L, int* __restrict__ perm_t,
                                                            int* __restrict__ perm_s) {
  __shared__ int s_run[kMaxLevels + 1];                      // boxes (row V: targets) before these keys
  __shared__ int s_pre[kTreeWarps][kMaxLevels + 1];          // ... of the round before this warp
  __shared__ unsigned s_bal[kTreeWarps][kMaxLevels + 1];     // the warp's keys with t >= v
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const unsigned lt = (1u << lane) - 1u;
  if (threadIdx.x <= V) s_run[threadIdx.x] = off[(int64_t)threadIdx.x * gridDim.x + blockIdx.x];
  const int64_t base = (int64_t)blockIdx.x * rounds * kTreeThreads;
  for (int r = 0; r < rounds; ++r) {
    const int64_t i = base + (int64_t)r * kTreeThreads + threadIdx.x;
    const bool ok = i < n;
    const uint64_t k = ok ? keys[i] : 0;
    const int id = ok ? idx[i] : 0;
    const int diff = ok ? key_diff(keys, i, d) : -1;
    const int dp = ok ? depth[key_pid(k)] - 1 : -1;
    const int t = min(diff, dp);
    for (int v = 0; v < V; ++v) {
      const unsigned m = __ballot_sync(0xffffffffu, ok && t >= v);
      if (lane == 0) s_bal[warp][v] = m;
    }
    const unsigned mt = __ballot_sync(0xffffffffu, ok && id < nt);
    if (lane == 0) s_bal[warp][V] = mt;
    __syncthreads();
    if (threadIdx.x <= V) {
      int a = s_run[threadIdx.x];
      for (int w = 0; w < kTreeWarps; ++w) {
        s_pre[w][threadIdx.x] = a;
        a += __popc(s_bal[w][threadIdx.x]);
      }
      s_run[threadIdx.x] = a;
    }
    __syncthreads();
    if (ok) {
      auto before = [&](int v) { return s_pre[warp][v] + __popc(s_bal[warp][v] & lt); };  // exclusive
      const int tpos = before(V), spos = (int)i - tpos;
      if (id < nt) perm_t[tpos] = id;
      else perm_s[spos] = id - (int)nt;
      if (i > 0 && diff >= 0) {  // the boxes of key i-1 that end here
        const int top = min(diff, depth[key_pid(keys[i - 1])] - 1);
        for (int v = 0; v <= top; ++v) {
          const int64_t b = lo.o[v] + before(v) - 1;
          L.te[b] = tpos;
          L.se[b] = spos;
          L.ce[b] = v > 0 ? before(v - 1) : 0;
        }
      }
      for (int v = 0; v <= t; ++v) {
        const int64_t b = lo.o[v] + before(v);
        L.key[b] = (k & ~kMortonMask) | ((k & kMortonMask) >> (d * v));
        L.tb[b] = tpos;
        L.sb[b] = spos;
        L.cb[b] = v > 0 ? before(v - 1) : 0;
        // the enclosing box one level up: opened here (v < t) or before
        L.parent[b] = v < dp ? before(v + 1) - (v < t ? 0 : 1) : -1;
      }
      if (i == n - 1) {  // the last boxes
        const int e = id < nt ? 1 : 0;
        for (int v = 0; v <= dp; ++v) {
          const int64_t b = lo.o[v] + before(v) - (t >= v ? 0 : 1);
          L.te[b] = tpos + e;
          L.se[b] = spos + 1 - e;
          L.ce[b] = v > 0 ? before(v - 1) + (t >= v - 1 ? 1 : 0) : 0;
        }
      }
    }
    __syncthreads();  // s_bal and s_pre are rewritten
  }
}

// Sort keys of the rows of every level in one array: M2L rows of level v
// (boxes with targets at real level >= 2) by (v, problem, class), then the
// near-field rows (leaves with targets) as level V; boxes of neither kind last.
// V: the levels that can have rows; the boxes of the coarser ones have none.
// Entry i < total is box i - lo.o[v] of its level v, entry total + b leaf b.
__global__ void k_row_keys(const uint64_t* __restrict__ key, const int* __restrict__ tb, const int* __restrict__ te,
                           const LevelOff lo, int V, int64_t total, int64_t nleaf, int d, int np,
                           const int* __restrict__ depth, uint64_t* __restrict__ ck, int* __restrict__ cv) {
  const uint64_t mask = (1ull << d) - 1ull;
  const uint64_t none = (uint64_t)(V * (int64_t)np + 1) << d;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total + nleaf;
       i += (int64_t)gridDim.x * blockDim.x) {
    if (i >= total) {
      const int64_t b = i - total;
      ck[i] = te[b] > tb[b] ? (uint64_t)V * np << d : none;
      cv[i] = (int)b;
      continue;
    }
    int v = 0;
    while (v < V && i >= lo.o[v + 1]) ++v;
    if (v == V) {
      ck[i] = none;
      cv[i] = 0;
      continue;
    }
    const uint64_t k = key[i];
    const int p = key_pid(k);
    const bool row = te[i] > tb[i] && depth[p] - 1 - v >= 2;
    ck[i] = row ? (((uint64_t)v * np + p) << d) | (k & mask) : none;
    cv[i] = (int)(i - lo.o[v]);
  }
}

// begin[key] = first entry of the sorted row keys with that key (-1: none).
__global__ void k_row_segs(const uint64_t* __restrict__ ck, int64_t n, int* __restrict__ begin) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    if (i == 0 || ck[i] != ck[i - 1]) begin[ck[i]] = (int)i;
}

// First row of each level in the sorted rows.
struct RowOff {
  int64_t o[kMaxLevels + 1];
};

// row_of[box of any level] = its row within the level (pre-filled with -1).
__global__ void k_rows_of_boxes(const int* __restrict__ row_box, const RowOff ro, const LevelOff lo, int V,
                                int* __restrict__ row_of) {
  const int64_t n = ro.o[V];
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    int v = 0;
    while (i >= ro.o[v + 1]) ++v;
    row_of[lo.o[v] + row_box[i]] = (int)(i - ro.o[v]);
  }
}

// ---------------------------------------------------------------------------
// host driver
// ---------------------------------------------------------------------------
static int bits_for(int n) {
  int b = 0;
  while ((1 << b) < n) ++b;
  return b;
}

// Problem of every point and the cube of every problem (device and host).
template <typename T>
static void forest_cubes(fmma_ctx* ctx, int d, const std::vector<int64_t>& toff, const T* tgt,
                         const std::vector<int64_t>& soff, const T* src, Tree& tr, int* pid,
                         const char* cube_buf = "cube") {
  const int np = (int)toff.size() - 1;
  const int64_t nt = toff[(size_t)np], ns = soff[(size_t)np];
  if (pid) {
    int64_t* dto = ctx_buf_t<int64_t>(ctx, "forest_toff", (size_t)np + 1);
    int64_t* dso = ctx_buf_t<int64_t>(ctx, "forest_soff", (size_t)np + 1);
    upload(ctx, dto, toff.data(), sizeof(int64_t) * (size_t)(np + 1));
    upload(ctx, dso, soff.data(), sizeof(int64_t) * (size_t)(np + 1));
    FMMA_LAUNCH(ctx, k_point_pid, grid_for(nt + ns, 256, (int64_t)ctx->sm_count * 16), 256, 0, dto, dso, np, nt, ns,
                pid);
  }
  unsigned long long* mm = ctx_buf_t<unsigned long long>(ctx, "bbox_mm", (size_t)np * 2 * kMaxDim);
  int* flag = ctx_buf_t<int>(ctx, "bbox_flag", 1);
  FMMA_LAUNCH(ctx, k_bbox_init, grid_for((int64_t)np * kMaxDim, 256), 256, 0, mm, np, flag);
  FMMA_LAUNCH(ctx, (k_bbox<T>), grid_for(nt + ns, 256, (int64_t)ctx->sm_count * 8), 256, 0, tgt, nt, src, ns, pid, d,
              mm, flag);
  tr.d_cube = static_cast<Cube*>(ctx_buf(ctx, cube_buf, sizeof(Cube) * (size_t)np));
  FMMA_LAUNCH(ctx, k_cube, grid_for(np, 128), 128, 0, mm, flag, np, d, tr.d_cube);
  tr.h_cube.resize((size_t)np);
  Cube* hp = static_cast<Cube*>(ctx_pinned(ctx, sizeof(Cube) * (size_t)np));
  FMMA_CHECK_CUDA(cudaMemcpyAsync(hp, tr.d_cube, sizeof(Cube) * (size_t)np, cudaMemcpyDeviceToHost, ctx->stream));
  FMMA_CHECK_CUDA(cudaStreamSynchronize(ctx->stream));
  std::memcpy(tr.h_cube.data(), hp, sizeof(Cube) * (size_t)np);
  if (tr.h_cube[0].nonfinite) throw Error(FMMA_ERR_INVALID_ARG, "a coordinate is NaN or Inf");
}

// Leaf keys, sorted; leaves; all virtual levels (no lists).
template <typename T>
static void forest_levels(fmma_ctx* ctx, int d, const std::vector<int64_t>& toff, const T* tgt,
                          const std::vector<int64_t>& soff, const T* src, const std::vector<int>& depth) {
  Tree& tr = ctx->tree;
  const int np = (int)depth.size();
  FMMA_REQUIRE(np >= 1 && np <= kMaxProblems, "between 1 and 4096 problems");
  FMMA_REQUIRE((int)toff.size() == np + 1 && (int)soff.size() == np + 1, "bad offsets");
  tr.valid = false;
  tr.d_pairs = nullptr;
  tr.pairs_read = true;
  tr.dim = d;
  tr.nprob = np;
  tr.depth = depth;
  tr.vmax = 0;
  for (int p = 0; p < np; ++p) {
    FMMA_REQUIRE(depth[(size_t)p] >= 1 && d * (depth[(size_t)p] - 1) <= kPidShift && depth[(size_t)p] - 1 <= 30,
                 "Depth out of range");
    tr.vmax = std::max(tr.vmax, depth[(size_t)p]);
  }
  tr.nt = toff[(size_t)np];
  tr.ns = soff[(size_t)np];
  const int64_t nt = tr.nt, ns = tr.ns, n = nt + ns;
  tr.lev.assign((size_t)tr.vmax, Level());
  tr.d_depth = ctx_buf_t<int>(ctx, "forest_depth", (size_t)np);
  upload(ctx, tr.d_depth, depth.data(), sizeof(int) * (size_t)np);
  const int blk = 256;
  const unsigned g = grid_for(n, blk, (int64_t)ctx->sm_count * 16);

  int* pid = np > 1 ? ctx_buf_t<int>(ctx, "pt_pid", (size_t)(n > 0 ? n : 1)) : nullptr;
  forest_cubes<T>(ctx, d, toff, tgt, soff, src, tr, pid);

  uint64_t* keys = ctx_buf_t<uint64_t>(ctx, "pt_keys", (size_t)n);
  int* idx = ctx_buf_t<int>(ctx, "pt_idx", (size_t)n);
  uint64_t* keys2 = ctx_buf_t<uint64_t>(ctx, "pt_keys2", (size_t)n);
  int* idx2 = ctx_buf_t<int>(ctx, "pt_idx2", (size_t)n);
  FMMA_LAUNCH(ctx, (k_leaf_keys<T>), g, blk, 0, tgt, nt, src, ns, pid, d, tr.d_depth, tr.d_cube, keys, idx);
  radix_sort_swap(ctx, &keys, &idx, &keys2, &idx2, n, 0, d * (tr.vmax - 1));
  if (np > 1) radix_sort_swap(ctx, &keys, &idx, &keys2, &idx2, n, kPidShift, kPidShift + bits_for(np));

  // Boxes of every level, counted per block of keys, scanned and read back in
  // one wait (row V: the targets).
  const int V = tr.vmax;
  FMMA_REQUIRE(V < kMaxLevels, "Depth out of range");
  // keys per block: enough blocks for small trees, fewer counts for large ones
  const int rounds = (int)std::max<int64_t>(1, std::min<int64_t>(8, n / ((int64_t)kTreeThreads * ctx->sm_count * 4)));
  const int64_t tile = (int64_t)rounds * kTreeThreads;
  const int64_t nblk = std::max<int64_t>(1, (n + tile - 1) / tile);
  int* cnt = ctx_buf_t<int>(ctx, "tree_cnt", (size_t)(V + 1) * nblk);
  int* off = ctx_buf_t<int>(ctx, "tree_off", (size_t)(V + 1) * nblk);
  int* tot = ctx_buf_t<int>(ctx, "tree_tot", (size_t)V + 1);
  FMMA_LAUNCH(ctx, k_tree_count, (unsigned)nblk, kTreeThreads, 0, keys, idx, n, nt, rounds, d, tr.d_depth, V, cnt);
  scan_rows(ctx, cnt, off, nblk, V + 1, tot);
  std::vector<int> hl((size_t)V + 1, 0);
  read_ints(ctx, tot, hl.data(), V + 1);

  tr.perm_t = ctx_buf_t<int>(ctx, "perm_t", (size_t)(nt > 0 ? nt : 1));
  tr.perm_s = ctx_buf_t<int>(ctx, "perm_s", (size_t)(ns > 0 ? ns : 1));
  LevelOff lo{};
  for (int v = 0; v < V; ++v) lo.o[v + 1] = lo.o[v] + hl[(size_t)v];
  const size_t total = (size_t)std::max<int64_t>(1, lo.o[V]);
  LevelArrays L;
  L.key = ctx_buf_t<uint64_t>(ctx, "lev_key", total);
  L.tb = ctx_buf_t<int>(ctx, "lev_tb", total);
  L.te = ctx_buf_t<int>(ctx, "lev_te", total);
  L.sb = ctx_buf_t<int>(ctx, "lev_sb", total);
  L.se = ctx_buf_t<int>(ctx, "lev_se", total);
  L.cb = ctx_buf_t<int>(ctx, "lev_cb", total);
  L.ce = ctx_buf_t<int>(ctx, "lev_ce", total);
  L.parent = ctx_buf_t<int>(ctx, "lev_parent", total);
  for (int v = 0; v < V; ++v) {
    Level& Lv = tr.lev[(size_t)v];
    const int64_t o = lo.o[v];
    Lv.v = v;
    Lv.nbox = hl[(size_t)v];
    Lv.key = L.key + o;
    Lv.tb = L.tb + o;
    Lv.te = L.te + o;
    Lv.sb = L.sb + o;
    Lv.se = L.se + o;
    Lv.cb = L.cb + o;
    Lv.ce = L.ce + o;
    Lv.parent = L.parent + o;
  }
  FMMA_LAUNCH(ctx, k_tree_emit, (unsigned)nblk, kTreeThreads, 0, keys, idx, n, nt, rounds, d, tr.d_depth, V, off, lo,
              L, tr.perm_t, tr.perm_s);
}

template <typename T>
void build_forest(fmma_ctx* ctx, int d, const std::vector<int64_t>& toff, const T* tgt,
                  const std::vector<int64_t>& soff, const T* src, const std::vector<int>& depth, bool lists) {
  forest_levels<T>(ctx, d, toff, tgt, soff, src, depth);
  Tree& tr = ctx->tree;
  const int np = tr.nprob;
  const int blk = 256;
  if (lists) {
    const FarTables& F = far_tables(d);
    int* jslot = ctx_buf_t<int>(ctx, "jslot", 8 * 216);
    upload(ctx, jslot, F.jslot, sizeof(int) * 8 * 216);
    unsigned long long* pairs = ctx_buf_t<unsigned long long>(ctx, "il_pairs", (size_t)tr.vmax + 2);
    FMMA_CHECK_CUDA(cudaMemsetAsync(pairs, 0, sizeof(unsigned long long) * (size_t)(tr.vmax + 2), ctx->stream));
    const int V = tr.vmax;
    LevelOff lo{};
    for (int v = 0; v < V; ++v) lo.o[v + 1] = lo.o[v] + tr.lev[(size_t)v].nbox;
    const int64_t total = lo.o[V], nleaf = tr.lev[0].nbox, nkey = total + nleaf;
    const Level& first = tr.lev[0];  // the arrays of all levels start at the leaves
    // Rows of all levels and the near-field rows in one sort; the table of
    // segment begins by (level, problem, class) is read back in one wait.  Real
    // level >= 2 leaves the V - 2 finest levels (the table of 4000 problems of
    // Depth 2 in 3-D: 64,016 entries with all levels, 16 without).
    const int VR = std::max(0, V - 2);
    const int64_t ntable = ((int64_t)VR * np + 2) << d;
    uint64_t* ck = ctx_buf_t<uint64_t>(ctx, "row_ck", (size_t)nkey);
    int* cv = ctx_buf_t<int>(ctx, "row_cv", (size_t)nkey);
    uint64_t* ck2 = ctx_buf_t<uint64_t>(ctx, "row_ck2", (size_t)nkey);
    int* cv2 = ctx_buf_t<int>(ctx, "row_cv2", (size_t)nkey);
    int* begin = ctx_buf_t<int>(ctx, "row_begin", (size_t)ntable);
    FMMA_CHECK_CUDA(cudaMemsetAsync(begin, 0xff, sizeof(int) * (size_t)ntable, ctx->stream));
    FMMA_LAUNCH(ctx, k_row_keys, grid_for(nkey, blk), blk, 0, first.key, first.tb, first.te, lo, VR, total, nleaf, d,
                np, tr.d_depth, ck, cv);
    radix_sort_swap(ctx, &ck, &cv, &ck2, &cv2, nkey, 0, d + bits_for(VR * np + 2));
    FMMA_LAUNCH(ctx, k_row_segs, grid_for(nkey, blk), blk, 0, ck, nkey, begin);
    std::vector<int> hb((size_t)ntable);
    read_ints(ctx, begin, hb.data(), (int)ntable);
    // segment ends: the next begin present, in key order
    int64_t end = nkey;
    std::vector<int64_t> ends((size_t)ntable);
    for (int64_t k = ntable - 1; k >= 0; --k) {
      ends[(size_t)k] = end;
      if (hb[(size_t)k] >= 0) end = hb[(size_t)k];
    }
    RowOff ro{};
    for (int v = 0; v < V; ++v) {
      Level& Lv = tr.lev[(size_t)v];
      // operator tables: problems with a real level >= 2 at this virtual level
      Lv.pid_table.assign((size_t)np, -1);
      Lv.table_pid.clear();
      for (int p = 0; p < np; ++p)
        if (tr.depth[(size_t)p] - 1 - v >= 2) {
          Lv.pid_table[(size_t)p] = (int)Lv.table_pid.size();
          Lv.table_pid.push_back(p);
        }
      Lv.segs.clear();
      const int64_t r0 = ro.o[v];
      int64_t r1 = r0;
      for (int64_t k = ((int64_t)v * np) << d; v < VR && k < ((int64_t)(v + 1) * np) << d; ++k) {
        if (hb[(size_t)k] < 0) continue;
        r1 = ends[(size_t)k];
        Lv.segs.push_back(make_int4((int)(k >> d) - v * np, (int)(k & ((1 << d) - 1)), (int)(hb[(size_t)k] - r0),
                                    (int)(r1 - r0)));
      }
      ro.o[v + 1] = r1;
      Lv.nrow = r1 - r0;
    }
    const int64_t nrow = ro.o[V], knear = ((int64_t)VR * np) << d;
    tr.nnear_rows = hb[(size_t)knear] >= 0 ? ends[(size_t)knear] - hb[(size_t)knear] : 0;
    tr.near_row_box = cv + nrow;
    // neighbour lists of every level top-down, far lists of the rows on the way
    const int nnb = d == 1 ? 3 : (d == 2 ? 9 : 27);
    int* nbr = ctx_buf_t<int>(ctx, "nbr", (size_t)total * nnb);
    int* row_of = ctx_buf_t<int>(ctx, "row_of_box", (size_t)total);
    int* il = ctx_buf_t<int>(ctx, "il", (size_t)nrow * F.nfar + 1);
    unsigned* smask = ctx_buf_t<unsigned>(ctx, "slot_mask", (size_t)nrow * kSlotWords + 1);
    FMMA_CHECK_CUDA(cudaMemsetAsync(nbr, 0xff, sizeof(int) * (size_t)total * nnb, ctx->stream));
    if (nrow > 0) {
      FMMA_CHECK_CUDA(cudaMemsetAsync(row_of, 0xff, sizeof(int) * (size_t)total, ctx->stream));
      FMMA_CHECK_CUDA(cudaMemsetAsync(il, 0xff, sizeof(int) * (size_t)nrow * F.nfar, ctx->stream));
      FMMA_CHECK_CUDA(cudaMemsetAsync(smask, 0, sizeof(unsigned) * (size_t)nrow * kSlotWords, ctx->stream));
      FMMA_LAUNCH(ctx, k_rows_of_boxes, grid_for(nrow, blk), blk, 0, cv, ro, lo, V, row_of);
    }
    ListLevels ll{};
    for (int v = 0; v < V; ++v) {
      Level& Lv = tr.lev[(size_t)v];
      Lv.row_box = cv + ro.o[v];
      Lv.il = il + ro.o[v] * F.nfar;
      Lv.slot_mask = smask + ro.o[v] * kSlotWords;
      ll.box0[v] = lo.o[v];
      ll.row0[v] = ro.o[v];
      ll.nbox[v] = Lv.nbox;
      ll.rows[v] = Lv.nrow > 0;
    }
    ll.V = V;
    ll.d = d;
    ll.nfar = F.nfar;
    ll.key = first.key;
    ll.parent = first.parent;
    ll.tb = first.tb;
    ll.te = first.te;
    ll.sb = first.sb;
    ll.se = first.se;
    ll.cb = first.cb;
    ll.ce = first.ce;
    ll.row_of = row_of;
    ll.jslot = jslot;
    ll.nbr = nbr;
    ll.il = il;
    ll.slot_mask = smask;
    ll.pairs = pairs;
    launch_lists_topdown(ctx, ll);
    // near lists at the leaves (rows = leaves with targets, key order)
    tr.near = ctx_buf_t<int>(ctx, "near", (size_t)tr.nnear_rows * nnb + 1);
    launch_near_rows(ctx, nbr, tr.near_row_box, tr.nnear_rows, d, first.tb, first.te, first.sb, first.se, tr.near,
                     pairs + V);
    tr.d_pairs = pairs;  // read when needed (tree_read_pairs)
    tr.pairs_read = false;
  }
  tr.valid = true;
}

bool tree_fetch_pairs(fmma_ctx* ctx, void* pinned) {
  const Tree& tr = ctx->tree;
  if (tr.pairs_read || !tr.d_pairs) return false;
  FMMA_CHECK_CUDA(cudaMemcpyAsync(pinned, tr.d_pairs, sizeof(unsigned long long) * (size_t)(tr.vmax + 1),
                                  cudaMemcpyDeviceToHost, ctx->stream));
  return true;
}

void tree_take_pairs(fmma_ctx* ctx, const void* pinned) {
  Tree& tr = ctx->tree;
  const unsigned long long* hp = static_cast<const unsigned long long*>(pinned);
  tr.pairs_read = true;
  for (int v = 0; v < tr.vmax; ++v) tr.lev[(size_t)v].il_pairs = (int64_t)hp[v];
  tr.p2p_pairs = (int64_t)hp[tr.vmax];
}

void tree_read_pairs(fmma_ctx* ctx) {
  void* pp = ctx_pinned(ctx, 512);
  if (!tree_fetch_pairs(ctx, pp)) return;
  FMMA_CHECK_CUDA(cudaStreamSynchronize(ctx->stream));
  tree_take_pairs(ctx, pp);
}

template void build_forest<double>(fmma_ctx*, int, const std::vector<int64_t>&, const double*,
                                   const std::vector<int64_t>&, const double*, const std::vector<int>&, bool);
template void build_forest<float>(fmma_ctx*, int, const std::vector<int64_t>&, const float*,
                                  const std::vector<int64_t>&, const float*, const std::vector<int>&, bool);

template <typename T>
void build_tree(fmma_ctx* ctx, int d, int depth, int64_t nt, const T* tgt, int64_t ns, const T* src, bool lists) {
  build_forest<T>(ctx, d, {0, nt}, tgt, {0, ns}, src, {depth}, lists);
}

template void build_tree<double>(fmma_ctx*, int, int, int64_t, const double*, int64_t, const double*, bool);
template void build_tree<float>(fmma_ctx*, int, int, int64_t, const float*, int64_t, const float*, bool);

// ---------------------------------------------------------------------------
// occupancy and export
// ---------------------------------------------------------------------------
__global__ void k_max_run(const uint64_t* __restrict__ key, const int* __restrict__ tb, const int* __restrict__ te,
                          const int* __restrict__ sb, const int* __restrict__ se, int64_t nb, int* __restrict__ out) {
  for (int64_t b = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; b < nb;
       b += (int64_t)gridDim.x * blockDim.x) {
    const int p = key_pid(key[b]);
    atomicMax(&out[2 * p], te[b] - tb[b]);
    atomicMax(&out[2 * p + 1], se[b] - sb[b]);
  }
}

template <typename T>
void leaf_occupancy(fmma_ctx* ctx, int d, const std::vector<int64_t>& toff, const T* tgt,
                    const std::vector<int64_t>& soff, const T* src, const std::vector<int>& depth,
                    std::vector<int>* max_t, std::vector<int>* max_s) {
  forest_levels<T>(ctx, d, toff, tgt, soff, src, depth);
  const int np = (int)depth.size();
  Level& leaf = ctx->tree.lev[0];
  int* out = ctx_buf_t<int>(ctx, "occ", (size_t)2 * np);
  FMMA_CHECK_CUDA(cudaMemsetAsync(out, 0, sizeof(int) * 2 * (size_t)np, ctx->stream));
  FMMA_LAUNCH(ctx, k_max_run, grid_for(leaf.nbox, 256), 256, 0, leaf.key, leaf.tb, leaf.te, leaf.sb, leaf.se, leaf.nbox,
              out);
  std::vector<int> h((size_t)2 * np);
  read_ints(ctx, out, h.data(), 2 * np);
  max_t->resize((size_t)np);
  max_s->resize((size_t)np);
  for (int p = 0; p < np; ++p) {
    (*max_t)[(size_t)p] = h[(size_t)(2 * p)];
    (*max_s)[(size_t)p] = h[(size_t)(2 * p + 1)];
  }
  ctx->tree.valid = false;
}

template void leaf_occupancy<double>(fmma_ctx*, int, const std::vector<int64_t>&, const double*,
                                     const std::vector<int64_t>&, const double*, const std::vector<int>&,
                                     std::vector<int>*, std::vector<int>*);
template void leaf_occupancy<float>(fmma_ctx*, int, const std::vector<int64_t>&, const float*,
                                    const std::vector<int64_t>&, const float*, const std::vector<int>&,
                                    std::vector<int>*, std::vector<int>*);

__global__ void k_key_to_rowmajor(const uint64_t* __restrict__ keys, int64_t n, int d, int bits,
                                  int64_t* __restrict__ out) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x) {
    int c[kMaxDim] = {0, 0, 0};
    morton_decode(keys[i] & kMortonMask, d, bits, c);
    int64_t r = 0;
    for (int q = 0; q < d; ++q) r = (r << bits) | (int64_t)c[q];
    out[i] = r;
  }
}

template <typename T>
void export_bins(fmma_ctx* ctx, int d, int depth, int64_t nt, const T* tgt, int64_t ns, const T* src,
                 int64_t* tbox, int64_t* sbox, Cube* cube_out) {
  Tree tmp;
  const int64_t n = nt + ns;
  int* pid = nullptr;
  forest_cubes<T>(ctx, d, {0, nt}, tgt, {0, ns}, src, tmp, pid);
  *cube_out = tmp.h_cube[0];
  int* dd = ctx_buf_t<int>(ctx, "export_depth", 1);
  upload(ctx, dd, &depth, sizeof(int));
  uint64_t* keys = ctx_buf_t<uint64_t>(ctx, "pt_keys", (size_t)(n > 0 ? n : 1));
  const int bits = depth - 1;
  FMMA_LAUNCH(ctx, (k_leaf_keys<T>), grid_for(n, 256), 256, 0, tgt, nt, src, ns, pid, d, dd, tmp.d_cube, keys,
              (int*)nullptr);
  if (nt > 0) FMMA_LAUNCH(ctx, k_key_to_rowmajor, grid_for(nt, 256), 256, 0, keys, nt, d, bits, tbox);
  if (ns > 0) FMMA_LAUNCH(ctx, k_key_to_rowmajor, grid_for(ns, 256), 256, 0, keys + nt, ns, d, bits, sbox);
}

template <typename T>
const Cube* problem_cube(fmma_ctx* ctx, int d, int64_t nt, const T* tgt, int64_t ns, const T* src,
                         const char* cube_buf, Cube* host) {
  Tree tmp;
  forest_cubes<T>(ctx, d, {0, nt}, tgt, {0, ns}, src, tmp, nullptr, cube_buf);
  *host = tmp.h_cube[0];
  return tmp.d_cube;
}

template const Cube* problem_cube<double>(fmma_ctx*, int, int64_t, const double*, int64_t, const double*, const char*,
                                          Cube*);
template const Cube* problem_cube<float>(fmma_ctx*, int, int64_t, const float*, int64_t, const float*, const char*,
                                         Cube*);

template void export_bins<double>(fmma_ctx*, int, int, int64_t, const double*, int64_t, const double*, int64_t*, int64_t*, Cube*);
template void export_bins<float>(fmma_ctx*, int, int, int64_t, const float*, int64_t, const float*, int64_t*, int64_t*, Cube*);

}  // namespace fmma_b200
