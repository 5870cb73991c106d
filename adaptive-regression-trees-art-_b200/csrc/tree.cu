// tree.cu -- node-sorted stable partition of rows by a split plane, and
// batched tree routing + leaf prediction.
//
// Routing rule everywhere: w . x - z >= 0 goes right (builder.py:494,
// tree.py:159, splitters.py:618).  The side is the sign of the exact value
// of w . x - z (right_side: a compensated dot product, and exact expansion
// arithmetic for the rare scores within its error bound); numpy's own
// rounded X @ w - z can disagree only where its rounding error exceeds
// |w . x - z|.
#include <cooperative_groups.h>

#include <algorithm>
#include <atomic>
#include <type_traits>

#include "common.cuh"
#include "level_plan.cuh"
#include "rows.cuh"

namespace cg = cooperative_groups;

namespace art {
namespace {

// The nodes of a level differ by a factor of a thousand in rows, and their sizes
// are known on the device alone.  So a level call is two launches: the first deals
// the nodes of at most `joint` rows to single CTAs (or, with several nodes a CTA,
// those of at most `single` rows to its warps), the second each of the others to
// a cluster of CTAs (one CTA reads about 50 GB/s).  The second starts as soon as
// every CTA of the first has (programmatic dependent launch) and ends after it.
// What is added, and in which order, follows the node's own row count, so results
// depend on none of this.
// A node of the level.
struct LevelNode {
  int64_t r0, n;
  const double* x;
  int d, vec;
};
__device__ __forceinline__ int64_t level_rows(const ArtSegments& seg, int64_t k) {
  return seg.row_offsets[k + 1] - seg.row_offsets[k];
}
__device__ __forceinline__ LevelNode level_node(const ArtSegments& seg, const double* x, int64_t k) {
  LevelNode v;
  v.r0 = seg.row_offsets[k];
  v.n = seg.row_offsets[k + 1] - v.r0;
  v.x = x + seg.x_offsets[k];
  v.d = seg.dims[k];
  v.vec = row_vec(v.x, v.d);
  return v;
}
// f with the width of a node's loads as a constant: a branch on it in every row
// would keep the loads of several rows from being in flight together.
template <typename F>
__device__ __forceinline__ void by_width(int vec, F f) {
  if (vec == 4) f(std::integral_constant<int, 4>());
  else if (vec == 2) f(std::integral_constant<int, 2>());
  else f(std::integral_constant<int, 1>());
}

// The first launch: single(node) by a warp, range(node) by the CTA.
template <typename Range, typename Single>
__device__ __forceinline__ void level_small_work(const ArtSegments& seg, const LevelPlan& L, Range range, Single single) {
  asm volatile("griddepcontrol.launch_dependents;");
  const int64_t k0 = (int64_t)blockIdx.x * L.nodes;
  const int nk = (int)min((int64_t)L.nodes, L.count - k0);
  if (L.single >= 0)
    for (int i = threadIdx.x >> 5; i < nk; i += kLevelWarps)
      if (level_rows(seg, k0 + i) <= L.single) single(k0 + i);
  for (int i = 0; i < nk; ++i) {
    const int64_t n = level_rows(seg, k0 + i);
    if (n > L.single && n <= L.joint) range(k0 + i);
  }
}
// The second: range(node, how many before it) by the cluster; `hold`: what that
// leaves in shared memory stays until every CTA has read it.
template <bool hold, typename Range>
__device__ __forceinline__ void level_large_work(const ArtSegments& seg, const LevelPlan& L, Range range) {
  __shared__ unsigned big[kLevelWarps];
  const int64_t k0 = (int64_t)(blockIdx.x / cg::this_cluster().num_blocks()) * L.nodes;
  const int nk = (int)min((int64_t)L.nodes, L.count - k0), tid = threadIdx.x;
  const unsigned m = __ballot_sync(0xffffffffu, tid < nk && level_rows(seg, k0 + tid) > L.joint);
  if ((tid & 31) == 0) big[tid >> 5] = m;
  if (__syncthreads_or(m != 0u)) {
    int turn = 0;
    for (int w = 0; 32 * w < nk; ++w)
      for (unsigned left = big[w]; left; left &= left - 1u) range(k0 + 32 * w + __ffs(left) - 1, turn++);
    if (hold) cg::this_cluster().sync();
  }
  asm volatile("griddepcontrol.wait;" ::: "memory");
}

// The side (right_side) is decided by the plain score where that is further from zero
// than its error bound (gamma_{d+1} times sum |x_i w_i| + |z|, taken twice);
// w is zero-padded to a multiple of eight.  Two FMAs an input against eleven
// operations for the compensated score, which still decides the rest, NaN
// and infinite scores and products near underflow among them.
__device__ __forceinline__ void plain_score(const double* xr, const double* w, int d, int vec, double& s, double& mag) {
  s = mag = 0.0;
#pragma unroll 4
  for (int i = 0; i < d; i += 8) {
    double v[8];
    load8(xr, i, d, vec, v);
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      s = fma(v[q], w[i + q], s);
      mag = fma(fabs(v[q]), fabs(w[i + q]), mag);
    }
  }
}
__device__ __forceinline__ bool row_side(const double* xr, const double* w, int d, double z, int vec) {
  double s, mag;
  plain_score(xr, w, d, vec, s, mag);
  s = __dsub_rn(s, z);
  mag = __dadd_rn(mag, fabs(z));
  if (fabs(s) > 2.220446049250313e-16 * (d + 4) * mag && mag > 1e-280) return s >= 0.0;
  return right_side(xr, w, d, z);
}

struct PartArgs {
  ArtSegments seg;
  const double* x;
  const double* theta;
  int64_t ts;
  const int8_t* split;
  int64_t* perm;
  int32_t* n_right;
};

// Stable partition.  CTA r of a node's cluster takes the r-th range of its
// rows: it reads x once, keeps the sides as a bit mask in shared memory, learns
// the other ranges' right counts through distributed shared memory, and
// scatters its row numbers to their places.  Rows past the mask's capacity
// (2^18 a CTA) have their sides formed a second time.
constexpr int kMaskWords = 8192;
struct PartShared {
  double w[kLevelWarps][ART_MAX_DIM + 8];  // zero-padded
  int64_t right[2];
  int warp[kLevelWarps];
  unsigned mask[kMaskWords];
};
extern __shared__ __align__(16) unsigned char level_smem[];

// This warp's rows first, first + step, ... (lane 0's; below end) to mask words
// at, at + wstep, ... of shared memory, as far as there are any; returns the
// right rows' number.
__device__ __forceinline__ int mark_sides(const LevelNode& v, const double* w, double z, int64_t first, int64_t step, int64_t end,
                                          int at, int wstep) {
  PartShared& S = *(PartShared*)level_smem;
  const int lane = threadIdx.x & 31;
  int count = 0;
#pragma unroll 1
  for (int64_t r = first + lane; r - lane < end; r += step, at += wstep) {
    const bool right = r < end && row_side(v.x + r * v.d, w, v.d, z, v.vec);
    const unsigned m = __ballot_sync(0xffffffffu, right);
    if (lane == 0 && at < kMaskWords) S.mask[at] = m;
    count += __popc(m);
  }
  return count;
}

// This warp's words q of up to 32, a row per lane, to their places: `mine` is
// word `lane`, `pre` the right rows before it (from `first` on), left and right
// the next places.
__device__ __forceinline__ void place_words(unsigned mine, int pre, int q0, int words, int64_t first, int64_t end,
                                            int64_t r0, int64_t left, int64_t right, int64_t* perm) {
  const int lane = threadIdx.x & 31;
  for (int q = 0; q < 32; ++q) {
    const int wq = q0 + q;
    if (wq >= words) break;
    const unsigned m = __shfl_sync(0xffffffffu, mine, q);
    const int before = __shfl_sync(0xffffffffu, pre, q);
    const int64_t r = first + 32 * (int64_t)wq + lane;
    if (r < end) {
      const int ahead = before + __popc(m & ((1u << lane) - 1u));
      const int64_t pos = (m >> lane) & 1u ? right + ahead : left + (32 * wq + lane - ahead);
      perm[r0 + pos] = r0 + r;
    }
  }
}
__device__ __forceinline__ int warp_scan(int v) {  // inclusive
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int t = __shfl_up_sync(0xffffffffu, v, o);
    if (lane >= o) v += t;
  }
  return v;
}

// One warp's node of at most kSingleRows rows.
__device__ __forceinline__ void partition_warp(const PartArgs& A, int64_t k) {
  PartShared& S = *(PartShared*)level_smem;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const LevelNode v = level_node(A.seg, A.x, k);
  double* w = S.w[warp];
  unsigned* mask = S.mask + 32 * warp;
  __syncwarp();
  for (int i = lane; i < ((v.d + 7) & ~7); i += 32) w[i] = i < v.d ? A.theta[k * A.ts + i] : 0.0;
  mask[lane] = 0u;
  const double z = A.theta[k * A.ts + v.d];
  __syncwarp();
  const int n = (int)v.n;
  if (A.split == nullptr || A.split[k] != 0) mark_sides(v, w, z, 0, 32, n, 32 * warp, 1);
  __syncwarp();
  const unsigned mine = 32 * lane < n ? mask[lane] : 0u;
  const int cnt = __popc(mine), incl = warp_scan(cnt), total = __shfl_sync(0xffffffffu, incl, 31);
  if (A.n_right && lane == 0) A.n_right[k] = total;
  place_words(mine, incl - cnt, 0, (n + 31) / 32, 0, n, v.r0, 0, n - total, A.perm);
}

// A CTA's range of a node: all of it, or its part of the cluster's, whose nodes
// alternate between two slots for their counts (`turn`).
template <bool CLUSTER>
__device__ __forceinline__ void partition_range(const PartArgs& A, int64_t k, int turn) {
  cg::cluster_group cluster = cg::this_cluster();
  const int csize = CLUSTER ? (int)cluster.num_blocks() : 1, crank = CLUSTER ? (int)cluster.block_rank() : 0;
  PartShared& S = *(PartShared*)level_smem;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const LevelNode v = level_node(A.seg, A.x, k);
  const int64_t n = v.n;
  const bool do_split = A.split == nullptr || A.split[k] != 0;
  double* w = S.w[0];
  __syncthreads();  // the node before is done with what is shared
  for (int i = tid; i < ((v.d + 7) & ~7); i += kLevelThreads) w[i] = i < v.d ? A.theta[k * A.ts + i] : 0.0;
  const double z = A.theta[k * A.ts + v.d];
  const int64_t span = ((n + csize - 1) / csize + kLevelThreads - 1) / kLevelThreads * kLevelThreads;
  const int64_t a = min(n, span * crank), b = min(n, a + span);  // this CTA's rows
  __syncthreads();
  const int local = do_split ? mark_sides(v, w, z, a + 32 * warp, kLevelThreads, b, warp, kLevelWarps) : 0;
  if (lane == 0) S.warp[warp] = local;
  __syncthreads();
  int64_t sum = 0;
  for (int i = 0; i < kLevelWarps; ++i) sum += S.warp[i];
  int64_t before = 0, total = sum;  // right rows of the ranges before this one, and of all
  if (CLUSTER) {
    if (tid == 0) S.right[turn & 1] = sum;
    cluster.sync();
    total = 0;
    for (int c = 0; c < csize; ++c) {
      const int64_t t = *cluster.map_shared_rank(&S.right[turn & 1], c);
      if (c < crank) before += t;
      total += t;
    }
  }
  if (A.n_right && crank == 0 && tid == 0) A.n_right[k] = (int32_t)total;
  int64_t left = a - before, rgt = n - total + before;  // next places of this range
  for (int64_t base = a; base < b; base += 32 * kLevelThreads) {
    const int64_t words = min((int64_t)kLevelThreads, (b - base + 31) / 32);
    // exclusive prefix of the right counts of up to 256 words
    auto word_at = [&](int64_t q, int64_t row) -> unsigned {
      const int64_t at = (base - a) / 32 + q;
      if (!do_split) return 0u;
      if (at < kMaskWords) return S.mask[at];
      unsigned m = 0;
      for (int j = 0; j < 32 && row + j < b; ++j)
        if (row_side(v.x + (row + j) * v.d, w, v.d, z, v.vec)) m |= 1u << j;
      return m;
    };
    const unsigned mine = tid < words ? word_at(tid, base + 32 * tid) : 0u;
    const int cnt = __popc(mine), incl = warp_scan(cnt);
    __syncthreads();
    if (lane == 31) S.warp[warp] = incl;
    __syncthreads();
    int wbase = 0, all = 0;
    for (int i = 0; i < kLevelWarps; ++i) {
      if (i < warp) wbase += S.warp[i];
      all += S.warp[i];
    }
    place_words(mine, wbase + incl - cnt, 32 * warp, (int)words, base, b, v.r0, left, rgt, A.perm);
    rgt += all;
    left += min((int64_t)32 * kLevelThreads, b - base) - all;
  }
}

__global__ void __launch_bounds__(kLevelThreads, 4) partition_small(const __grid_constant__ PartArgs A, const LevelPlan L) {
  level_small_work(A.seg, L, [&](int64_t k) { partition_range<false>(A, k, 0); }, [&](int64_t k) { partition_warp(A, k); });
}
__global__ void __launch_bounds__(kLevelThreads, 4) partition_large(const __grid_constant__ PartArgs A, const LevelPlan L) {
  level_large_work<true>(A.seg, L, [&](int64_t k, int turn) { partition_range<true>(A, k, turn); });
}

// Tree walk and leaf prediction, a point per thread.  The nodes of a warp's
// points differ from the second level on, so every table load is a gather of up
// to 32 lines, whatever its width: that bounds it, and rows of whole 32-byte
// sectors (wvec, cvec: see load8) are read four doubles at a time.  The point
// waits in shared memory, [input][thread], where the features can index it.
// 100,003 points of d = 8, depth 9, quadratic leaves: 52 us with single loads
// of tables and points from memory, 31 us now; of d = 64, depth 10, affine leaves (64 KB
// of points a CTA, three CTAs an SM): 386 and 114 us.
// W: doubles a block of loads, 8, or 2 for points of one or two inputs (eight
// places of which one is used cost 2 M points of d = 1 27 %).
constexpr int kPredictThreads = 128;

template <int W>
__device__ __forceinline__ void load_block(const double* x, int i, int d, int vec, double (&v)[W]) {
  if constexpr (W == 8) {
    load8(x, i, d, vec, v);
  } else {
    static_assert(W == 2);
    if (vec >= 2) {
      const double2 t = __ldg((const double2*)(x + i));
      v[0] = t.x;
      v[1] = t.y;
    } else {
      v[0] = __ldg(x + i);
      v[1] = i + 1 < d ? __ldg(x + i + 1) : 0.0;
    }
  }
}

template <int W>
__global__ void __launch_bounds__(kPredictThreads)
    predict_kernel(int d, int64_t n_nodes, const int32_t* child, const double* theta, int64_t ts, int wvec,
                   const double* coef, int64_t cs, int cvec, const int32_t* features, int64_t n, const double* x,
                   int32_t* leaf, double* pred) {
  extern __shared__ double sx[];
  const int64_t i = (int64_t)blockIdx.x * kPredictThreads + threadIdx.x;
  if (i >= n) return;
  const double* xr = x + i * d;
  double* mine = sx + threadIdx.x;  // input c at mine[c * kPredictThreads]
  const int vec = row_vec(x, d);
  for (int c = 0; c < d; c += W) {
    double v[W];
    load_block<W>(xr, c, d, vec, v);
#pragma unroll
    for (int q = 0; q < W; ++q)
      if (c + q < d) mine[(c + q) * kPredictThreads] = v[q];
  }
  int node = 0;
  for (int64_t guard = 0; guard < n_nodes && child[2 * (int64_t)node] >= 0; ++guard) {
    const double* t = theta + (int64_t)node * ts;
    const double z = t[d];
    // right_side by the plain score where its error bound allows, as row_side
    double s = 0.0, mag = 0.0;
    for (int c = 0; c < d; c += W) {
      double w[W];
      load_block<W>(t, c, d, wvec, w);
#pragma unroll
      for (int q = 0; q < W; ++q)
        if (c + q < d) {  // z and whatever follows may share the last load
          const double v = mine[(c + q) * kPredictThreads];
          s = fma(v, w[q], s);
          mag = fma(fabs(v), fabs(w[q]), mag);
        }
    }
    s = __dsub_rn(s, z);
    mag = __dadd_rn(mag, fabs(z));
    const bool sure = fabs(s) > 2.220446049250313e-16 * (d + 4) * mag && mag > 1e-280;
    const bool right = sure ? s >= 0.0 : right_side(xr, t, d, z);
    node = child[2 * (int64_t)node + (right ? 1 : 0)];
  }
  if (leaf) leaf[i] = node;
  if (!pred) return;
  const int kind = features[node], p = feature_count(d, kind);
  const double* co = coef + (int64_t)node * cs;
  // features in order (feature_factors): factors a and b, -1 for a constant 1
  int a = kind == ART_FEATURES_POLY1 || kind == ART_FEATURES_POLY2 ? -1 : 0, b = -1;
  double s = 0.0;
  for (int f = 0; f < p; f += W) {
    double c[W];
    load_block<W>(co, f, p, cvec, c);
#pragma unroll
    for (int q = 0; q < W; ++q)
      if (f + q < p) {
        const double v = (a < 0 ? 1.0 : mine[a * kPredictThreads]) * (b < 0 ? 1.0 : mine[b * kPredictThreads]);
        s = fma(v, c[q], s);
        if (b < 0) {
          if (++a == d) {  // the bias of an affine model, or the first product
            a = kind == ART_FEATURES_AFFINE ? -1 : 0;
            b = kind == ART_FEATURES_AFFINE ? -1 : 0;
          }
        } else if (++b == d) {
          b = ++a;
        }
      }
  }
  pred[i] = s;
}

// Per segment: sum of squared residuals of phi(x) . beta and sum of y^2.  A
// node's rows are cut into up to kMaxRanks ranges, fixed by its row count;
// each range is one CTA's sum (threads in row order, their sums added by warps
// and the warps' in order), and the ranges are added in order.
//
// The features' products are formed and added in feature order, as
// feature_factors gives it: the nested form x_i (b_i + sum b_ij x_j) has fewer
// operations but other roundings, and overflows where the products do not.
struct ResArgs {
  ArtSegments seg;
  const double* x;
  const double* y;
  const double* beta;
  int64_t bs;
  double* sse;
  double* ssy;
};
constexpr int kCoefs = ART_MAX_FEATURES + 24;  // by position: constant, a gap, inputs (zero-padded), products
struct ResNode : LevelNode {
  const double* beta;
  const double* y;
  const double* q;
  int64_t span;
  int kind, p, dp, ranks;  // dp: padded inputs of a quadratic model, else 0
};
struct ResShared {
  double q[kLevelWarps][kCoefs];
  double part[2][2][kMaxRanks];
  double red[2][kMaxRanks][kLevelWarps];
};

// The coefficients of node k to q, by `threads` threads.
template <int threads>
__device__ __forceinline__ ResNode res_node(const ResArgs& A, int64_t k, double* q, int t) {
  ResNode v;
  (LevelNode&)v = level_node(A.seg, A.x, k);
  v.kind = A.seg.features[k];
  v.p = feature_count(v.d, v.kind);
  v.beta = A.beta + k * A.bs;
  v.y = A.y + v.r0;
  v.q = q;
  const bool quad = v.kind == ART_FEATURES_POLY2 || v.kind == ART_FEATURES_POLY2_NOBIAS;
  v.dp = quad ? (v.d <= 8 ? 8 : 16) : 0;
  v.ranks = (int)min((int64_t)kMaxRanks, (v.n + 1023) / 1024);
  v.span = v.ranks ? (v.n + v.ranks - 1) / v.ranks : 0;
  const int used = 2 + (quad ? v.dp + v.dp * (v.dp + 1) / 2 : v.d + 8);
  auto sync = [] {
    if (threads == 32) __syncwarp();
    else __syncthreads();
  };
  sync();  // the node before is done with them
  for (int i = t; i < used && i < kCoefs; i += threads) q[i] = 0.0;
  sync();
  for (int f = t; f < v.p; f += threads) {
    int a, b;
    feature_factors(v.d, v.kind, f, a, b);
    int at;
    if (a < 0) at = 0;
    else if (b < 0) at = 2 + a;
    else at = 2 + v.dp + a * v.dp - a * (a - 1) / 2 + (b - a);
    if (at < kCoefs) q[at] = v.beta[f];
  }
  sync();
  return v;
}

// A pair of coefficients, read where it is used: hoisted out of the row loop
// they would fill the registers.
__device__ __forceinline__ double2 coefs(const double* q) {
  double2 c;
  asm volatile("ld.volatile.shared.v2.f64 {%0, %1}, [%2];"
               : "=d"(c.x), "=d"(c.y)
               : "r"((uint32_t)__cvta_generic_to_shared(q)));
  return c;
}
// Predictions of U rows, the rows' loads in flight together.
template <int VEC, int DP, int U>
__device__ __forceinline__ void quad_predict(const double* q, const double* const (&xr)[U], int d, double (&s)[U]) {
  double v[U][DP];
#pragma unroll
  for (int u = 0; u < U; ++u)
#pragma unroll
    for (int i = 0; i < DP; i += 8) load8(xr[u], i, d, VEC, *(double(*)[8]) & v[u][i]);
  const double one = coefs(q).x;
  double2 c;
#pragma unroll
  for (int u = 0; u < U; ++u) s[u] = one;
#pragma unroll
  for (int i = 0; i < DP; i += 2) {
    c = coefs(q + 2 + i);
#pragma unroll
    for (int u = 0; u < U; ++u) {
      s[u] = fma(v[u][i], c.x, s[u]);
      s[u] = fma(v[u][i + 1], c.y, s[u]);
    }
  }
  int f = 0;
#pragma unroll
  for (int i = 0; i < DP; ++i)
#pragma unroll
    for (int j = i; j < DP; ++j, ++f) {
      if ((f & 1) == 0) c = coefs(q + 2 + DP + f);
#pragma unroll
      for (int u = 0; u < U; ++u) s[u] = fma(v[u][i] * v[u][j], f & 1 ? c.y : c.x, s[u]);
    }
}
template <int VEC, int U>
__device__ __forceinline__ void linear_predict(const double* q, const double* const (&xr)[U], int d, bool last, double (&s)[U]) {
  const double one = coefs(q).x;  // the constant: an affine model's last feature, the others' first
#pragma unroll
  for (int u = 0; u < U; ++u) s[u] = last ? 0.0 : one;
  for (int i = 0; i < d; i += 8) {
    double v[U][8];
#pragma unroll
    for (int u = 0; u < U; ++u) load8(xr[u], i, d, VEC, v[u]);
#pragma unroll
    for (int t = 0; t < 8; t += 2) {
      const double2 c = coefs(q + 2 + i + t);
#pragma unroll
      for (int u = 0; u < U; ++u) {
        s[u] = fma(v[u][t], c.x, s[u]);
        s[u] = fma(v[u][t + 1], c.y, s[u]);
      }
    }
  }
#pragma unroll
  for (int u = 0; u < U; ++u)
    if (last) s[u] += one;
}
// Feature by feature: with an infinite or NaN input the padding's products
// (infinity times zero) must not enter.
__device__ __noinline__ double plain_predict(const double* xr, const double* beta, int d, int kind, int p) {
  double s = 0.0;
  for (int f = 0; f < p; ++f) {
    int a, b;
    feature_factors(d, kind, f, a, b);
    s = fma((a < 0 ? 1.0 : xr[a]) * (b < 0 ? 1.0 : xr[b]), beta[f], s);
  }
  return s;
}
// The sums over rows first, first + kLevelThreads, ... below end, U rows at a
// time; predict(rows, predictions).
template <int U, typename F>
__device__ __forceinline__ double2 res_loop(const double* x, const double* y, int d, int64_t first, int64_t end, bool& odd, F predict) {
  double2 t = make_double2(0.0, 0.0);
  for (int64_t r = first; r < end; r += U * kLevelThreads) {
    const double* xr[U];
    double yv[U], s[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int64_t ru = r + u * kLevelThreads < end ? r + u * kLevelThreads : r;
      xr[u] = x + ru * d;
      yv[u] = __ldg(y + ru);
    }
    predict(xr, s);
#pragma unroll
    for (int u = 0; u < U; ++u)
      if (r + u * kLevelThreads < end) {
        const double e = yv[u] - s[u];
        odd |= !isfinite(s[u]);
        t.x = fma(e, e, t.x);
        t.y = fma(yv[u], yv[u], t.y);
      }
  }
  return t;
}
__device__ __noinline__ double2 res_rows(const double* x, const double* y, const double* q, const double* beta, int d, int vec,
                                         int dp, int kind, int p, int64_t first, int64_t end) {
  bool odd = false;
  double2 t;
  by_width(vec, [&](auto v) {
    if (dp == 0)
      t = res_loop<2>(x, y, d, first, end, odd,
                      [&](auto& xr, auto& s) { linear_predict<v>(q, xr, d, kind == ART_FEATURES_AFFINE, s); });
    else if (dp == 8)
      t = res_loop<2>(x, y, d, first, end, odd, [&](auto& xr, auto& s) { quad_predict<v, 8>(q, xr, d, s); });
    else
      t = res_loop<1>(x, y, d, first, end, odd, [&](auto& xr, auto& s) { quad_predict<v, 16>(q, xr, d, s); });
  });
  if (odd) {  // a prediction that is not finite: feature by feature
    t.x = 0.0;
    for (int64_t r = first; r < end; r += kLevelThreads) {
      const double e = y[r] - plain_predict(x + r * d, beta, d, kind, p);
      t.x = fma(e, e, t.x);
    }
  }
  return t;
}

// One warp's node of one range: the CTA's order of additions.
__device__ __forceinline__ void residual_warp(const ResArgs& A, int64_t k) {
  ResShared& S = *(ResShared*)level_smem;
  const int lane = threadIdx.x & 31;
  const ResNode v = res_node<32>(A, k, S.q[threadIdx.x >> 5], lane);
  double t_e = 0.0, t_y = 0.0;
  for (int w = 0; 32 * w < v.n && w < kLevelWarps; ++w) {
    const double2 t = res_rows(v.x, v.y, v.q, v.beta, v.d, v.vec, v.dp, v.kind, v.p, 32 * w + lane, v.n);
    t_e += warp_sum(t.x);
    t_y += warp_sum(t.y);
  }
  if (lane == 0) { A.sse[k] = t_e; A.ssy[k] = t_y; }
}

// A CTA's ranges of a node, all or every csize-th: their sums to the part array
// of the cluster's CTA 0 (or its own), which adds them up.  The cluster's nodes
// alternate between two arrays (`turn`).
template <bool CLUSTER>
__device__ __forceinline__ void residual_ranges(const ResArgs& A, int64_t k, int turn) {
  cg::cluster_group cluster = cg::this_cluster();
  const int csize = CLUSTER ? (int)cluster.num_blocks() : 1, crank = CLUSTER ? (int)cluster.block_rank() : 0;
  ResShared& S = *(ResShared*)level_smem;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, slot = turn & 1;
  const ResNode n = res_node<kLevelThreads>(A, k, S.q[0], tid);
  if (CLUSTER && turn == 0) cluster.sync();  // CTA 0 has started before its shared memory is written
  for (int v = crank; v < n.ranks; v += csize) {
    const int64_t a = n.span * v, b = min(n.n, a + n.span);
    const double2 t = res_rows(n.x, n.y, n.q, n.beta, n.d, n.vec, n.dp, n.kind, n.p, a + tid, b);
    const double s_e = warp_sum(t.x), s_y = warp_sum(t.y);
    if (lane == 0) { S.red[0][v][warp] = s_e; S.red[1][v][warp] = s_y; }
  }
  __syncthreads();
  const int v = tid >> 1, which = tid & 1;
  if (v < n.ranks && v % csize == crank) {
    double t = 0.0;
    for (int i = 0; i < kLevelWarps; ++i) t += S.red[which][v][i];
    double* at = &S.part[slot][which][v];
    *(CLUSTER ? cluster.map_shared_rank(at, 0) : at) = t;
  }
  if (CLUSTER) cluster.sync();
  else __syncthreads();
  if (crank == 0 && tid < 2) {
    double t = 0.0;
    for (int i = 0; i < n.ranks; ++i) t += S.part[slot][tid][i];
    (tid ? A.ssy : A.sse)[k] = t;
  }
}

// The first launch for levels of up to kNarrowFeatures features (the stride of
// beta says so): the general kernel pads a row to eight inputs and holds 80
// registers, three CTAs an SM, and for such rows latency is most of its time.
// Here a row takes its features one at a time; the order of additions, and so the
// result, is the general kernel's.  Any node is right, only its time depends on
// its features.  Five CTAs an SM and one node a CTA up to four times as many
// (general kernel -> this one): d = 1, 600 nodes of 5,000 rows 37 -> 23 us, 3,000
// of 2,000 70 -> 43, 12,000 of 600 89 -> 67; d = 5, 55 -> 44, 88 -> 80, 118 -> 117;
// 3,000 of 64 rows 17 -> 19.  With eight features it loses (12,000 of 600: 141 us
// and 190).  Six and eight CTAs an SM (40 and 32 registers) take 74 and 119 us for
// 12,000 of 600, d = 1.
constexpr int kNarrowFeatures = 6;
constexpr int kNarrowCtas = 5;  // an SM
constexpr int kNarrowGrid = 148 * kNarrowCtas * 4;
struct NarrowShared {
  double b[kLevelWarps][ART_MAX_FEATURES];
  int16_t fa[kLevelWarps][ART_MAX_FEATURES], fb[kLevelWarps][ART_MAX_FEATURES];
  double part[2][kMaxRanks];
  double red[2][kMaxRanks][kLevelWarps];
};
// The node's coefficients and their factors, by `threads` threads; how many.
template <int threads>
__device__ __forceinline__ int narrow_node(const ResArgs& A, int64_t k, int d, NarrowShared& S, int at, int t) {
  const int kind = A.seg.features[k], p = min(feature_count(d, kind), ART_MAX_FEATURES);
  const double* beta = A.beta + k * A.bs;
  if (threads == 32) __syncwarp();
  else __syncthreads();
  for (int f = t; f < p; f += threads) {
    int a, b;
    feature_factors(d, kind, f, a, b);
    S.fa[at][f] = (int16_t)a;
    S.fb[at][f] = (int16_t)b;
    S.b[at][f] = beta[f];
  }
  if (threads == 32) __syncwarp();
  else __syncthreads();
  return p;
}
// Rows r, r + step, ... (U of them, below end): added to t[0], or each to its t[u].
template <int U, int SUMS>
__device__ __forceinline__ void narrow_rows(const NarrowShared& S, int at, int p, const double* x, const double* y, int d, int64_t r,
                                            int step, int64_t end, double2 (&t)[SUMS]) {
  const double* xr[U];
  double yv[U], s[U];
#pragma unroll
  for (int u = 0; u < U; ++u) {
    const int64_t ru = r + u * step < end ? r + u * step : r;
    xr[u] = x + ru * d;
    yv[u] = __ldg(y + ru);
    s[u] = 0.0;
  }
#pragma unroll 2
  for (int f = 0; f < p; ++f) {
    const int a = S.fa[at][f], b = S.fb[at][f];
    const double c = S.b[at][f];
    double v[U];
#pragma unroll
    for (int u = 0; u < U; ++u) v[u] = a < 0 ? 1.0 : __ldg(xr[u] + a);
    if (b >= 0) {
#pragma unroll
      for (int u = 0; u < U; ++u) v[u] *= __ldg(xr[u] + b);
    }
#pragma unroll
    for (int u = 0; u < U; ++u) s[u] = fma(v[u], c, s[u]);
  }
#pragma unroll
  for (int u = 0; u < U; ++u)
    if (r + u * step < end) {
      double2& q = t[SUMS == 1 ? 0 : u];
      const double e = yv[u] - s[u];
      q.x = fma(e, e, q.x);
      q.y = fma(yv[u], yv[u], q.y);
    }
}
// residual_warp and residual_ranges<false>, feature by feature.
__device__ __forceinline__ void narrow_warp(const ResArgs& A, int64_t k) {
  NarrowShared& S = *(NarrowShared*)level_smem;
  const int lane = threadIdx.x & 31, at = threadIdx.x >> 5;
  const LevelNode v = level_node(A.seg, A.x, k);
  const double* y = A.y + v.r0;
  const int p = narrow_node<32>(A, k, v.d, S, at, lane);
  double t_e = 0.0, t_y = 0.0;
  constexpr int W = 4;  // of the CTA's warps side by side
  for (int w = 0; 32 * w < v.n && w < kLevelWarps; w += W) {
    double2 t[W];
#pragma unroll
    for (int u = 0; u < W; ++u) t[u] = make_double2(0.0, 0.0);
    for (int64_t r = 32 * w + lane; r < v.n; r += kLevelThreads) narrow_rows<W, W>(S, at, p, v.x, y, v.d, r, 32, v.n, t);
#pragma unroll
    for (int u = 0; u < W; ++u) {
      t_e += warp_sum(t[u].x);
      t_y += warp_sum(t[u].y);
    }
  }
  if (lane == 0) { A.sse[k] = t_e; A.ssy[k] = t_y; }
}
__device__ __forceinline__ void narrow_range(const ResArgs& A, int64_t k) {
  NarrowShared& S = *(NarrowShared*)level_smem;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const LevelNode v = level_node(A.seg, A.x, k);
  const double* y = A.y + v.r0;
  const int p = narrow_node<kLevelThreads>(A, k, v.d, S, 0, tid);
  const int ranks = (int)min((int64_t)kMaxRanks, (v.n + 1023) / 1024);
  const int64_t span = ranks ? (v.n + ranks - 1) / ranks : 0;
  for (int q = 0; q < ranks; ++q) {
    const int64_t a = span * q, b = min(v.n, a + span);
    double2 t[1] = {make_double2(0.0, 0.0)};
    for (int64_t r = a + tid; r < b; r += 2 * kLevelThreads) narrow_rows<2, 1>(S, 0, p, v.x, y, v.d, r, kLevelThreads, b, t);
    const double s_e = warp_sum(t[0].x), s_y = warp_sum(t[0].y);
    if (lane == 0) { S.red[0][q][warp] = s_e; S.red[1][q][warp] = s_y; }
  }
  __syncthreads();
  const int q = tid >> 1, which = tid & 1;
  if (q < ranks) {
    double t = 0.0;
    for (int i = 0; i < kLevelWarps; ++i) t += S.red[which][q][i];
    S.part[which][q] = t;
  }
  __syncthreads();
  if (tid < 2) {
    double t = 0.0;
    for (int i = 0; i < ranks; ++i) t += S.part[tid][i];
    (tid ? A.ssy : A.sse)[k] = t;
  }
}
__global__ void __launch_bounds__(kLevelThreads, kNarrowCtas) residual_narrow(const __grid_constant__ ResArgs A, const LevelPlan L) {
  level_small_work(A.seg, L, [&](int64_t k) { narrow_range(A, k); }, [&](int64_t k) { narrow_warp(A, k); });
}
__global__ void __launch_bounds__(kLevelThreads, 3) residual_small(const __grid_constant__ ResArgs A, const LevelPlan L) {
  level_small_work(A.seg, L, [&](int64_t k) { residual_ranges<false>(A, k, 0); }, [&](int64_t k) { residual_warp(A, k); });
}
__global__ void __launch_bounds__(kLevelThreads, 3) residual_large(const __grid_constant__ ResArgs A, const LevelPlan L) {
  level_large_work<false>(A.seg, L, [&](int64_t k, int turn) { residual_ranges<true>(A, k, turn); });
}

// A level's two kernels: attributes set, and the largest cluster of the second's
// CTAs that fits the device (a fixed property) found, once per device.
template <typename Args>
struct LevelCall {
  void (*small)(Args, LevelPlan);
  void (*large)(Args, LevelPlan);
  size_t smem;
  std::atomic<int> cluster[64];

  struct Config {
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute attr[2];
    Config(int64_t clusters, int c, size_t smem, bool after, cudaStream_t s) {
      attr[0].id = cudaLaunchAttributeClusterDimension;
      attr[0].val.clusterDim.x = (unsigned)c;
      attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
      attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
      attr[1].val.programmaticStreamSerializationAllowed = 1;
      cfg.gridDim = dim3((unsigned)(clusters * c));
      cfg.blockDim = dim3(kLevelThreads);
      cfg.dynamicSmemBytes = smem;
      cfg.stream = s;
      cfg.attrs = attr;
      cfg.numAttrs = after ? 2 : 1;
    }
  };
  int largest() {
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) { cudaGetLastError(); return 0; }
    int c = cluster[dev].load(std::memory_order_acquire);
    if (c > 0) return c;
    for (auto kern : {small, large})
      if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess) return 0;
    cudaFuncSetAttribute(large, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    c = level_cluster([&](int size) {
      const Config one(1, size, smem, false, nullptr);
      int fit = 0;
      if (cudaOccupancyMaxActiveClusters(&fit, large, &one.cfg) == cudaSuccess) return fit > 0;
      cudaGetLastError();
      return false;
    });
    cluster[dev].store(c, std::memory_order_release);
    return c;
  }
  int run(int64_t count, cudaStream_t s, const char* what, const Args& args, void (*lean)(Args, LevelPlan) = nullptr) {
    const int c = largest();
    if (c < 1) return check_launch(what);
    const bool both = count > kLevelFew;
    prof_begin(what, s);
    cudaError_t e = cudaSuccess;
    if (both) {
      const LevelPlan L = lean ? level_small(count, kNarrowGrid) : level_small(count);
      (lean ? lean : small)<<<(unsigned)((count + L.nodes - 1) / L.nodes), kLevelThreads, lean ? sizeof(NarrowShared) : smem, s>>>(args, L);
      count_launch();
      e = cudaGetLastError();
    }
    if (e == cudaSuccess) {
      const LevelPlan L = level_large(count);
      const Config config((count + L.nodes - 1) / L.nodes, c, smem, both, s);
      e = cudaLaunchKernelEx(&config.cfg, large, args, L);
      count_launch();
    }
    prof_end(s);
    if (e != cudaSuccess) {
      cudaGetLastError();
      set_error("%s: %s", what, cudaGetErrorString(e));
      return ART_E_LAUNCH;
    }
    return check_launch(what);
  }
};
LevelCall<ResArgs> g_residuals{residual_small, residual_large, sizeof(ResShared), {}};
LevelCall<PartArgs> g_partition{partition_small, partition_large, sizeof(PartShared), {}};

}  // namespace
}  // namespace art

using namespace art;

extern "C" int art_segment_residuals(const ArtSegments* seg, const double* x, const double* y,
                                     const double* beta, int64_t beta_stride, double* sse,
                                     double* ssy, art_stream_t stream) {
  cudaGetLastError();
  if (!seg || seg->count < 0) { set_error("art_segment_residuals: bad segments"); return ART_E_INVALID; }
  if (seg->count == 0) return ART_OK;
  if (!seg->row_offsets || !seg->x_offsets || !seg->dims || !seg->features || !x || !y || !beta ||
      !sse || !ssy) {
    set_error("art_segment_residuals: null argument");
    return ART_E_INVALID;
  }
  if (seg->count > 0x7fffffffll) { set_error("art_segment_residuals: too many segments"); return ART_E_UNSUPPORTED; }
  return g_residuals.run(seg->count, (cudaStream_t)stream, "segment_residuals",
                         ResArgs{*seg, x, y, beta, beta_stride, sse, ssy}, beta_stride <= kNarrowFeatures ? residual_narrow : nullptr);
}

extern "C" int art_partition_rows(const ArtSegments* seg, const double* x, const double* theta,
                                  int64_t theta_stride, const int8_t* split, int64_t* perm,
                                  int32_t* n_right, art_stream_t stream) {
  cudaGetLastError();
  if (!seg || !x || !theta || !perm) { set_error("art_partition_rows: null argument"); return ART_E_INVALID; }
  if (seg->count < 0 || seg->count > 0x7fffffff) { set_error("art_partition_rows: bad count"); return ART_E_INVALID; }
  if (seg->count == 0) return ART_OK;
  if (theta_stride < 2) { set_error("art_partition_rows: theta_stride too small"); return ART_E_INVALID; }
  return g_partition.run(seg->count, (cudaStream_t)stream, "partition_rows",
                         PartArgs{*seg, x, theta, theta_stride, split, perm, n_right});
}

// Width of a table row's loads (see load8): whole sectors or pairs where every
// row starts on one and the last load of `used` doubles stays within its row.
static int table_vec(const double* t, int64_t stride, int used) {
  const uintptr_t at = (uintptr_t)t;
  if ((stride & 3) == 0 && (at & 31) == 0 && stride >= ((used + 3) & ~3)) return 4;
  return (stride & 1) == 0 && (at & 15) == 0 && stride >= ((used + 1) & ~1) ? 2 : 1;
}

extern "C" int art_tree_predict(int32_t dim, int64_t n_nodes, const int32_t* child,
                                const double* theta, int64_t theta_stride, const double* coef,
                                int64_t coef_stride, const int32_t* features, int64_t n_points,
                                const double* x, int32_t* leaf, double* pred, art_stream_t stream) {
  cudaGetLastError();
  if (dim < 1 || dim > ART_MAX_DIM) { set_error("art_tree_predict: bad dim %d", dim); return ART_E_UNSUPPORTED; }
  if (n_nodes < 1 || !child || !theta || !x || (pred && (!coef || !features))) {
    set_error("art_tree_predict: null argument");
    return ART_E_INVALID;
  }
  if (n_points <= 0) return ART_OK;
  const unsigned grid = (unsigned)((n_points + kPredictThreads - 1) / kPredictThreads);
  const size_t smem = sizeof(double) * dim * kPredictThreads;
  const auto kern = dim <= 2 ? predict_kernel<2> : predict_kernel<8>;
  if (smem > 48 * 1024 &&
      cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess)
    return check_launch("art_tree_predict");
  prof_begin("tree_predict", (cudaStream_t)stream);
  kern<<<grid, kPredictThreads, smem, (cudaStream_t)stream>>>(
      dim, n_nodes, child, theta, theta_stride, table_vec(theta, theta_stride, dim), coef, coef_stride,
      table_vec(coef, coef_stride, 1), features, n_points, x, leaf, pred);
  prof_end((cudaStream_t)stream);
  count_launch();
  return check_launch("art_tree_predict");
}
