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

#include <utility>

#include "common.cuh"
#include "rows.cuh"

namespace cg = cooperative_groups;

namespace art {
namespace {

// Both level kernels below give a node to a cluster of CTAs, since the nodes of
// a level differ by a factor of a thousand in rows and one CTA reads only
// about 50 GB/s.  The cluster's size follows the number of nodes (the more
// nodes, the less a large one matters); what is added, and in which order,
// follows the node's own row count, so results do not depend on it.
// 307 nodes of 450 to 400,000 rows, d = 2 to 32 (1.7 GB): partition 14.5 ->
// 0.59 ms, residuals 9.6 -> 0.65 ms against one CTA a node (2.6-2.9 TB/s of x
// read once; before, the partition read it twice).
constexpr int kLevelThreads = 256;
constexpr int kLevelWarps = kLevelThreads / 32;
constexpr int kMaxRanks = 16;  // CTAs of a cluster, and partial sums of a node, at most

int level_cluster(int64_t count) { return count <= 512 ? 16 : (count <= 2048 ? 8 : (count <= 8192 ? 4 : 1)); }

// right_side, decided by the plain score where that is further from zero
// than its error bound (gamma_{d+1} times sum |x_i w_i| + |z|, taken twice);
// w is zero-padded to a multiple of eight.  Two FMAs an input against eleven
// operations for the compensated score, which still decides the rest, NaN
// and infinite scores and products near underflow among them.
__device__ __forceinline__ bool row_side(const double* xr, const double* w, int d, double z, int vec) {
  double s = 0.0, mag = 0.0;
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
  s = __dsub_rn(s, z);
  mag = __dadd_rn(mag, fabs(z));
  const double bound = 2.220446049250313e-16 * (d + 4) * mag;
  if (fabs(s) > bound && mag > 1e-280) return s >= 0.0;
  return right_side(xr, w, d, z);
}

// Stable partition.  CTA r of a node's cluster takes the r-th range of its
// rows: it reads x once, keeps the sides as a bit mask in shared memory, learns
// the other ranges' right counts through distributed shared memory, and
// scatters its row numbers to their places.  Rows past the mask's capacity
// (2^18 a CTA) have their sides formed a second time.
constexpr int kMaskWords = 8192;
__global__ void __launch_bounds__(kLevelThreads)
    partition_kernel(ArtSegments seg, const double* x, const double* theta, int64_t ts,
                     const int8_t* split, int64_t* perm, int32_t* n_right) {
  cg::cluster_group cluster = cg::this_cluster();
  const int csize = (int)cluster.num_blocks(), crank = (int)cluster.block_rank();
  const int64_t k = blockIdx.x / csize;
  const int64_t r0 = seg.row_offsets[k], n = seg.row_offsets[k + 1] - r0;
  const int64_t xoff = seg.x_offsets[k];
  const int d = seg.dims[k];
  const bool do_split = split == nullptr || split[k] != 0;
  extern __shared__ unsigned mask[];
  __shared__ double w[ART_MAX_DIM + 8];
  __shared__ int64_t s_right;
  __shared__ int s_warp[kLevelWarps];
  __shared__ int pre[kLevelThreads];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  for (int i = tid; i < ART_MAX_DIM + 8; i += kLevelThreads) w[i] = i < d ? theta[k * ts + i] : 0.0;
  const double z = theta[k * ts + d];
  const double* xk = x + xoff;
  const int vec = row_vec(xk, d);
  const int64_t span = ((n + csize - 1) / csize + kLevelThreads - 1) / kLevelThreads * kLevelThreads;
  const int64_t a = min(n, span * crank), b = min(n, a + span);  // this CTA's rows
  __syncthreads();
  int local = 0;
#pragma unroll 2
  for (int64_t base = a; base < b; base += kLevelThreads) {
    const int64_t r = base + tid;
    const bool right = do_split && r < b && row_side(xk + r * d, w, d, z, vec);
    const unsigned m = __ballot_sync(0xffffffffu, right);
    const int64_t word = (base - a) / 32 + warp;
    if (lane == 0) {
      local += __popc(m);
      if (word < kMaskWords) mask[word] = m;
    }
  }
  if (lane == 0) s_warp[warp] = local;
  __syncthreads();
  if (tid == 0) {
    int64_t t = 0;
    for (int i = 0; i < kLevelWarps; ++i) t += s_warp[i];
    s_right = t;
  }
  cluster.sync();
  int64_t before = 0, total = 0;  // right rows of the ranges before this one, and of all
  for (int c = 0; c < csize; ++c) {
    const int64_t v = *cluster.map_shared_rank(&s_right, c);
    if (c < crank) before += v;
    total += v;
  }
  if (n_right && crank == 0 && tid == 0) n_right[k] = (int32_t)total;
  int64_t left = a - before, rgt = n - total + before;  // next places of this range
  for (int64_t base = a; base < b; base += 32 * kLevelThreads) {
    const int64_t words = min((int64_t)kLevelThreads, (b - base + 31) / 32);
    // exclusive prefix of the right counts of up to 256 words
    auto word_at = [&](int64_t q, int64_t row) -> unsigned {
      const int64_t at = (base - a) / 32 + q;
      if (at < kMaskWords) return mask[at];
      unsigned m = 0;
      for (int j = 0; j < 32 && row + j < b; ++j)
        if (do_split && row_side(xk + (row + j) * d, w, d, z, vec)) m |= 1u << j;
      return m;
    };
    const unsigned mine = tid < words ? word_at(tid, base + 32 * tid) : 0u;
    const int cnt = __popc(mine);
    int incl = cnt;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int t = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += t;
    }
    __syncthreads();
    if (lane == 31) s_warp[warp] = incl;
    __syncthreads();
    int wbase = 0, all = 0;
    for (int i = 0; i < kLevelWarps; ++i) {
      if (i < warp) wbase += s_warp[i];
      all += s_warp[i];
    }
    pre[tid] = wbase + incl - cnt;
    __syncwarp();
    for (int q = 0; q < 32; ++q) {  // this warp's 32 words, a row per lane
      const int wq = 32 * warp + q;
      if (wq >= words) break;
      const unsigned m = __shfl_sync(0xffffffffu, mine, q);
      const int64_t r = base + 32 * (int64_t)wq + lane;
      if (r < b) {
        const int ahead = pre[wq] + __popc(m & ((1u << lane) - 1u));
        const int64_t pos = (m >> lane) & 1u ? rgt + ahead : left + (32 * wq + lane - ahead);
        perm[r0 + pos] = r0 + r;
      }
    }
    rgt += all;
    left += min((int64_t)32 * kLevelThreads, b - base) - all;
  }
  cluster.sync();  // the counts stay until every CTA has read them
}

// Tree walk and leaf prediction, a point per thread.  The nodes of a warp's
// points differ from the second level on, so every table load is a gather of up
// to 32 lines, whatever its width: that bounds it, and rows of whole 32-byte
// sectors (wvec, cvec: see load8) are read four doubles at a time.  The point
// waits in shared memory, [input][thread], where the features can index it.
// 100,003 points of d = 8, depth 9, quadratic leaves: 52 us with single loads
// of tables and points from memory, 31 us now.
constexpr int kPredictThreads = 128;

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
  for (int c = 0; c < d; c += 8) {
    double v[8];
    load8(xr, c, d, vec, v);
#pragma unroll
    for (int q = 0; q < 8; ++q)
      if (c + q < d) mine[(c + q) * kPredictThreads] = v[q];
  }
  int node = 0;
  for (int64_t guard = 0; guard < n_nodes && child[2 * (int64_t)node] >= 0; ++guard) {
    const double* t = theta + (int64_t)node * ts;
    const double z = t[d];
    // right_side by the plain score where its error bound allows, as row_side
    double s = 0.0, mag = 0.0;
    for (int c = 0; c < d; c += 8) {
      double w[8];
      load8(t, c, d, wvec, w);
#pragma unroll
      for (int q = 0; q < 8; ++q)
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
  for (int f = 0; f < p; f += 8) {
    double c[8];
    load8(co, f, p, cvec, c);
#pragma unroll
    for (int q = 0; q < 8; ++q)
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
// each range is one CTA's sum (threads in row order, then a fixed tree), and
// the ranges are added in order.
//
// The features' products are formed and added in feature order, as
// feature_factors gives it: the nested form x_i (b_i + sum b_ij x_j) has fewer
// operations but other roundings, and overflows where the products do not.
template <int DP>
__device__ __forceinline__ double quad_predict(const double* xr, const double* q, int d, int vec) {
  double v[DP];
#pragma unroll
  for (int i = 0; i < DP; i += 8) {
    double t[8];
    load8(xr, i, d, vec, t);
#pragma unroll
    for (int u = 0; u < 8; ++u) v[i + u] = t[u];
  }
  double s = q[0];
  int f = 1;
#pragma unroll
  for (int i = 0; i < DP; ++i) s = fma(v[i], q[f++], s);
#pragma unroll
  for (int i = 0; i < DP; ++i)
#pragma unroll
    for (int j = i; j < DP; ++j) s = fma(v[i] * v[j], q[f++], s);
  return s;
}
// `last`: the constant is the last feature (affine models), else the first
__device__ __forceinline__ double linear_predict(const double* xr, const double* q, int d, int vec, bool last) {
  double s = last ? 0.0 : q[0];
#pragma unroll 4
  for (int i = 0; i < d; i += 8) {
    double v[8];
    load8(xr, i, d, vec, v);
#pragma unroll
    for (int u = 0; u < 8; ++u) s = fma(v[u], q[1 + i + u], s);
  }
  return last ? s + q[0] : s;
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

__global__ void __launch_bounds__(kLevelThreads)
    residual_kernel(ArtSegments seg, const double* x, const double* y, const double* beta,
                    int64_t bs, double* sse, double* ssy) {
  cg::cluster_group cluster = cg::this_cluster();
  const int csize = (int)cluster.num_blocks(), crank = (int)cluster.block_rank();
  // CTA 0 has started before its shared memory is written: waited for once the
  // coefficients are in place
  auto started = cluster.barrier_arrive();
  const int64_t k = blockIdx.x / csize;
  const int64_t r0 = seg.row_offsets[k], n = seg.row_offsets[k + 1] - r0;
  const int64_t xoff = seg.x_offsets[k];
  const int d = seg.dims[k], kind = seg.features[k];
  const int p = feature_count(d, kind);
  // coefficients by position: constant, inputs (zero-padded), products
  __shared__ double q[ART_MAX_FEATURES + 8 + 16];
  __shared__ double part[2][kMaxRanks];
  __shared__ double red[2][kLevelWarps];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const bool quad = kind == ART_FEATURES_POLY2 || kind == ART_FEATURES_POLY2_NOBIAS;
  const int dp = quad ? (d <= 8 ? 8 : 16) : d;
  for (int i = tid; i < ART_MAX_FEATURES + 8 + 16; i += kLevelThreads) q[i] = 0.0;
  __syncthreads();
  for (int f = tid; f < p; f += kLevelThreads) {
    int u, v;
    feature_factors(d, kind, f, u, v);
    int at;
    if (u < 0) at = 0;
    else if (v < 0) at = 1 + u;
    else at = 1 + dp + u * dp - u * (u - 1) / 2 + (v - u);
    if (at < ART_MAX_FEATURES + 24) q[at] = beta[k * bs + f];
  }
  __syncthreads();
  const double* xk = x + xoff;
  const int vec = row_vec(xk, d);
  const int ranks = (int)min((int64_t)kMaxRanks, (n + 1023) / 1024);
  const int64_t span = ranks ? (n + ranks - 1) / ranks : 0;
  cluster.barrier_wait(std::move(started));
  for (int v = crank; v < ranks; v += csize) {
    const int64_t a = span * v, b = min(n, a + span);
    double s_e = 0.0, s_y = 0.0;
#pragma unroll 2
    for (int64_t r = a + tid; r < b; r += kLevelThreads) {
      const double* xr = xk + r * d;
      const double yv = __ldg(y + r0 + r);
      double pred;
      if (!quad) pred = linear_predict(xr, q, d, vec, kind == ART_FEATURES_AFFINE);
      else if (dp == 8) pred = quad_predict<8>(xr, q, d, vec);
      else pred = quad_predict<16>(xr, q, d, vec);
      if (!isfinite(pred)) pred = plain_predict(xr, beta + k * bs, d, kind, p);
      const double e = yv - pred;
      s_e = fma(e, e, s_e);
      s_y = fma(yv, yv, s_y);
    }
    s_e = warp_sum(s_e);
    s_y = warp_sum(s_y);
    if (lane == 0) { red[0][warp] = s_e; red[1][warp] = s_y; }
    __syncthreads();
    if (tid < 2) {
      double t = 0.0;
      for (int i = 0; i < kLevelWarps; ++i) t += red[tid][i];
      *cluster.map_shared_rank(&part[tid][v], 0) = t;
    }
    __syncthreads();
  }
  cluster.sync();
  if (crank == 0 && tid < 2) {
    double t = 0.0;
    for (int v = 0; v < ranks; ++v) t += part[tid][v];
    (tid ? ssy : sse)[k] = t;
  }
}

template <typename... P, typename... A>
int launch_level(void (*kern)(P...), int64_t count, size_t smem, cudaStream_t s, const char* what, A... args) {
  const int c = level_cluster(count);
  if ((c > 8 && cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess) ||
      (smem && cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess))
    return check_launch(what);
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = (unsigned)c;
  attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
  cfg.gridDim = dim3((unsigned)(count * c));
  cfg.blockDim = dim3(kLevelThreads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  prof_begin(what, s);
  const cudaError_t e = cudaLaunchKernelEx(&cfg, kern, args...);
  prof_end(s);
  count_launch();
  if (e != cudaSuccess) {
    cudaGetLastError();
    set_error("%s: %s", what, cudaGetErrorString(e));
    return ART_E_LAUNCH;
  }
  return check_launch(what);
}

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
  return launch_level(residual_kernel, seg->count, 0, (cudaStream_t)stream, "segment_residuals", *seg, x, y, beta,
                      beta_stride, sse, ssy);
}

extern "C" int art_partition_rows(const ArtSegments* seg, const double* x, const double* theta,
                                  int64_t theta_stride, const int8_t* split, int64_t* perm,
                                  int32_t* n_right, art_stream_t stream) {
  cudaGetLastError();
  if (!seg || !x || !theta || !perm) { set_error("art_partition_rows: null argument"); return ART_E_INVALID; }
  if (seg->count < 0 || seg->count > 0x7fffffff) { set_error("art_partition_rows: bad count"); return ART_E_INVALID; }
  if (seg->count == 0) return ART_OK;
  if (theta_stride < 2) { set_error("art_partition_rows: theta_stride too small"); return ART_E_INVALID; }
  return launch_level(partition_kernel, seg->count, kMaskWords * sizeof(unsigned), (cudaStream_t)stream,
                      "partition_rows", *seg, x, theta, theta_stride, split, perm, n_right);
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
  if (smem > 48 * 1024 &&
      cudaFuncSetAttribute(predict_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess)
    return check_launch("art_tree_predict");
  prof_begin("tree_predict", (cudaStream_t)stream);
  predict_kernel<<<grid, kPredictThreads, smem, (cudaStream_t)stream>>>(
      dim, n_nodes, child, theta, theta_stride, table_vec(theta, theta_stride, dim), coef, coef_stride,
      table_vec(coef, coef_stride, 1), features, n_points, x, leaf, pred);
  prof_end((cudaStream_t)stream);
  count_launch();
  return check_launch("art_tree_predict");
}
