// split_warp.cu -- soft oblique split search, warp form: a (node, restart) is
// searched by one warp, by the four warps of a CTA, or by a cluster of CTAs,
// by the node's own row count.
//
// Same objective, stop rules, Armijo steps, AdaptiveAlpha, feasibility
// tracking, hard partition and refits as the CTA form (split.cu); the
// summation order differs.  An iteration makes three passes over the rows:
//   residual pass : loss, gradient and right count at theta with the current
//                   child models (splitters.py:424-488);
//   search pass   : the frozen-model loss (objectives.py:145-156) of up to
//                   kCand Armijo candidates at once, since
//                   x . project(w + alpha d) = (x . w + alpha x . d) / |w + alpha d|
//                   needs two products a row whatever the number of candidates;
//   Gram pass     : both sides' weighted Grams at the accepted theta and the
//                   temperature that follows it.
//
// What bounds it: the latency of dependent FP64 chains at 12 (narrow) or 8
// (wide) warps an SM and, with few items, that of a pass.
// The Grams run as mma.sync m8n8k4 f64 (16 cycles of a scheduler's FP64 pipe
// each); scores, fitted values, gradient and gates are per-row lane work,
// because as MMAs most of their columns would be padding (the three score
// columns cost 320 cycles a tile as MMAs and 110 as FMAs).  A candidate costs
// one gate a row, where a Gram for every trial cost five times that.
//
// Rows come in tiles of up to 32, copied with cp.async one tile ahead into
// rows [x, zeros to a multiple of four, 1, y] whose stride is 6 or 10 modulo
// 16 doubles: a lane reads its own row two doubles at a time without bank
// conflicts (stride 2 modulo 4), and the MMA fragments (4 rows x 8 columns)
// nearly so.  A tile's features are formed as fragments as they are loaded
// (products of two columns for quadratic models); no feature tile is stored.
//
// Members of a gang take every P-th tile and end each pass by adding their
// partial sums in member order: over the CTA's warps, then over the cluster's
// CTAs through distributed shared memory.  All hold the same totals and run
// the same control flow.  Gang sizes follow the node's row count and, through
// the number of restarts, the call's parameters, never the batch.
//
// Against one trial with its Gram per pass and gangs of one CTA (B200): one
// node of 4,096 rows, d = 2, 24 iterations 3.0 -> 0.37 ms; 203 nodes of 300 to
// 65,000 rows, one restart, 153 -> 11.4 ms with the starts; 256 nodes x 16
// restarts, d = 16, 30 iterations 140 -> 70 ms.  149 nodes of 300 to 120,000 rows
// with 33 or 45 features, before in the CTA form, 268 -> 24 ms.
//
// Models of more than 23 features keep one side's Gram blocks per warp: the
// warps of a pair take the same tiles in the Gram passes, one side each, and
// different tiles in the others.
#include <algorithm>

#include <cooperative_groups.h>

#include "bulk.cuh"
#include "linalg.cuh"
#include "split.cuh"

namespace cg = cooperative_groups;

namespace art {
namespace {

constexpr int kWThreads = 128;
constexpr int kWWarps = kWThreads / 32;
constexpr int kCand = 4;               // Armijo candidates per search pass
constexpr int kNarrowAug = 24, kNarrowDim = 23;
constexpr int kWideAug = 48, kWideDim = 46;
constexpr int kWideTile = 1344;        // doubles of a row tile, d > 23: 32 rows to d = 40, then 24
constexpr int kClusterCtas = 8;
// Gangs, as log2 of n + 1 (the plan's buckets, so that larger gangs come first
// in the queue).  With at most two restarts a node: a CTA from 1,023 rows, a
// cluster from 4,095 (a pass over 4,096 rows is then four tiles a warp).  With
// more, the items fill the device: a CTA from 4,095 rows, no clusters.
constexpr int kCtaLogFew = 10, kClusterLogFew = 12, kCtaLogMany = 12;

__host__ __device__ inline int pad4(int d) { return (d + 3) & ~3; }
__host__ __device__ inline int tile_stride(int d) {
  int s = pad4(d) + 2;
  while ((s & 15) != 6 && (s & 15) != 10) ++s;
  return s;
}
__host__ __device__ inline int tile_rows(int d) {
  if (d <= kNarrowDim) return 32;
  const int r = (kWideTile / tile_stride(d)) & ~3;
  return r < 32 ? r : 32;
}

// Per-warp shared memory in doubles: two row tiles (between passes: partial
// sums and packed Grams), the tile's weights, and the vectors of an item.
struct WLayout {
  int tile, Q, lin, quad, cst, th, dn, lf, bl, br, scal, per_warp;
};
__host__ __device__ inline WLayout warp_layout(int dmax, int pmax) {
  WLayout L;
  const int pa = pmax + 1, E = pa * (pa + 1) / 2;
  const bool wide = dmax > kNarrowDim || pa > kNarrowAug;
  int t = wide ? kWideTile : 32 * tile_stride(kNarrowDim < dmax ? kNarrowDim : dmax);
  for (int q = 1; !wide && q < dmax; ++q) t = t > 32 * tile_stride(q) ? t : 32 * tile_stride(q);
  const int sums = pa > kNarrowAug ? (E > 608 ? E : 608) : 2 * E;  // sided Grams; narrow items of a wide level
  while (2 * t < sums + 8 || 2 * t < 33 * dmax + 8) t += 8;
  L.tile = t;  // even: row pairs are 16-byte aligned
  const int d4 = pad4(dmax);
  int o = 2 * t;
  L.Q = o; o += 128;
  L.th = o; o += d4;        // w and its search direction, zero-padded (z and its own: SC_Z, SC_DZ)
  L.dn = o; o += d4;
  L.lin = o; o += 2 * d4;   // child models' linear coefficients, (left, right) per input
  L.quad = o; o += 72;      // ... of the 36 products of eight inputs
  L.cst = o; o += 2;
  L.lf = o; o += dmax + 1;
  L.bl = o; o += pmax;
  L.br = o; o += pmax;
  L.scal = o; o += 12;
  L.per_warp = (o + 1) & ~1;
  return L;
}

// What the kernel is launched with: layout offsets are read as constants.
struct WArgs {
  SplitArgs a;
  WLayout L;
  int csize;
};
// Shared memory is addressed through its symbol and integer offsets, so that
// every access is known to be one to shared memory.
extern __shared__ __align__(16) double sw[];

__device__ __forceinline__ double wsum(double v) {  // every lane holds the same bits
  return __shfl_sync(0xffffffffu, warp_sum(v), 0);
}
__device__ __forceinline__ void cluster_arrive() {
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
}
__device__ __forceinline__ void cluster_wait() {
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}

enum { SC_LOSS = 0, SC_GNORM, SC_DD, SC_NRIGHT, SC_FAILL, SC_FAILR, SC_LAML, SC_LAMR, SC_Z, SC_DZ };

// What a warp knows of its gang.
struct Gang {
  int P, g;      // members, this warp's index (1, 0: alone)
  bool cluster;  // the members span the cluster
};

// Members' arrays (at the start of each warp's region, length len) added in
// member order.  Every member may read the total at total(side) until the next
// pass.  `sets` = 2: the members' arrays are alternately left and right sums,
// with a total each.  With a cluster, its second barrier is only arrived at:
// it is waited for before the regions are written again.
__device__ __noinline__ void gang_sum(int pw, int len, int sets, bool cluster) {
  __syncwarp();
  asm volatile("bar.sync 1, %0;" ::"r"(kWThreads) : "memory");
  for (int e = threadIdx.x; e < len * sets; e += kWThreads) {
    const int s = e >= len ? 1 : 0, i = e - s * len;
    double t = sw[s * pw + i];
    for (int w = s + sets; w < kWWarps; w += sets) t += sw[w * pw + i];
    sw[s * pw + i] = t;
  }
  if (cluster) {
    cg::cluster_group cl = cg::this_cluster();
    cluster_arrive();
    cluster_wait();
    for (int e = threadIdx.x; e < len * sets; e += kWThreads) {
      const int s = e >= len ? 1 : 0, i = e - s * len;
      double* mine = sw + s * pw + i;
      double v[kClusterCtas];
#pragma unroll
      for (int c = 0; c < kClusterCtas; ++c) v[c] = *cl.map_shared_rank(mine, c);
      double t = v[0];
#pragma unroll
      for (int c = 1; c < kClusterCtas; ++c) t += v[c];
      sw[(2 + s) * pw + i] = t;
    }
    cluster_arrive();
  }
  asm volatile("bar.sync 1, %0;" ::"r"(kWThreads) : "memory");
}

// Trace-scaled ridge solve of the augmented Gram at sw[A], by one warp; the
// solution to sw[x], the failing pivot (or 0) and lambda to sw[fail], sw[lam].
template <int RPL>
__device__ __noinline__ void solve_side(int A, int x, int fail, int lam, int p, double ridge) {
  const int lane = threadIdx.x & 31;
  double* G = sw + A;
  double tr = 0.0;
  for (int i = lane; i < p; i += 32) tr += G[pk(i, i)];
  const double l = ridge * wsum(tr) / p;  // models.py:271
  __syncwarp();
  for (int i = lane; i < p; i += 32) G[pk(i, i)] += l;
  __syncwarp();
  const int f = warp_chol_solve<RPL>(G, p, sw + x);
  if (lane == 0) {
    sw[fail] = (double)f;
    sw[lam] = l;
  }
  __syncwarp();
}

template <int NB, bool SIDED>
struct SplitWarp {
  static constexpr int NBLK = NB * (NB + 1) / 2;
  const WArgs& W;
  const SplitArgs& a;
  const WLayout& L;
  const Gang G;
  const int lane, warp;
  const int base;   // this warp's region in sw
  const int vb;     // the region holding the item's vectors (warp 0's in a gang)
  bool pending = false;  // a cluster arrival to be waited for
  int64_t r0, n;
  const double* xg;
  int d, d4, kind, p, pa, E, rs, RS;
  int step_r, step_c, lr0, lc0;  // this lane's walk over a tile's copies
  bool pairs;                    // 16-byte copies
  bool quad, narrow, apart;
  int tail;
  int fa[NB], fb[NB];   // this lane's feature of each 8-column block: two columns of the row tile
  double ridge, T0, T, invT;
  double loss, gnorm, dd, lamL, lamR;
  int nright;

  __device__ __forceinline__ SplitWarp(const WArgs& w_, Gang g_)
      : W(w_), a(w_.a), L(w_.L), G(g_), lane(threadIdx.x & 31), warp(threadIdx.x >> 5),
        base((int)(threadIdx.x >> 5) * w_.L.per_warp), vb(g_.P > 1 ? 0 : (int)(threadIdx.x >> 5) * w_.L.per_warp) {}
  __device__ __forceinline__ int kq() const { return lane & 3; }
  __device__ __forceinline__ int mq() const { return lane >> 2; }
  __device__ __forceinline__ bool leads() const { return G.P == 1 || warp == 0; }
  __device__ __forceinline__ double& V(int at) const { return sw[vb + at]; }     // an item vector's entry
  __device__ __forceinline__ double& B(int at) const { return sw[base + at]; }   // this warp's region
  // all members of this CTA (the warp alone, without a gang)
  __device__ __forceinline__ void sync() const {
    if (G.P > 1) asm volatile("bar.sync 1, %0;" ::"r"(kWThreads) : "memory");
    else __syncwarp();
  }
  __device__ double gate(double s) const { return a.mixed ? sigm32(s) : sigm(s); }

  // ---------------------------------------------------------------- tiles
  __device__ __forceinline__ void issue(int64_t t0, int h) const {
    const int rows = (int)min((int64_t)RS, n - t0), rows4 = (rows + 3) & ~3;
    const uint32_t dst = smem_u32(sw + base + h * L.tile);
    const double* src = xg + t0 * d;
    if (pairs && step_c == 0 && rows == RS) {  // each lane keeps its columns
      const double* sp = src + lr0 * d + 2 * lc0;
      uint32_t dp = dst + (uint32_t)(lr0 * rs + 2 * lc0) * 8u;
#pragma unroll 4
      for (int rr = lr0; rr < RS; rr += step_r) {
        cp_async16(dp, sp);
        sp += step_r * d;
        dp += (uint32_t)(step_r * rs) * 8u;
      }
    } else {
      const int cw = pairs ? 2 : 1, cpr = d / cw;
      int rr = lr0, cc = lc0;
      while (rr < rows4) {
        const bool live = rr < rows;
        const double* sp = src + (live ? rr * d + cc * cw : 0);
        const uint32_t dp = dst + (uint32_t)(rr * rs + cc * cw) * 8u;
        if (pairs) cp_async16(dp, sp, live);
        else cp_async8(dp, sp, live);
        rr += step_r;
        cc += step_c;
        if (cc >= cpr) { cc -= cpr; ++rr; }
      }
    }
    if (lane < rows4) {
      const bool live = lane < rows;
      cp_async8(dst + (uint32_t)(lane * rs + d4 + 1) * 8u, a.y + r0 + t0 + (live ? lane : 0), live);
    }
    cp_async_commit();
  }
  // f(offset of the tile in sw, rows) over tiles m, m + M, ... of the node, the
  // next tile's copy in flight.  Waits for the gang first: the regions hold its
  // last totals.
  template <typename F>
  __device__ __forceinline__ void tiles(int m, int M, F f) {
    if (pending) {
      cluster_wait();
      pending = false;
    }
    sync();
#pragma unroll
    for (int h = 0; h < 2; ++h)
      if (lane < RS) {
        for (int i = d; i < d4; ++i) B(h * L.tile + lane * rs + i) = 0.0;
        B(h * L.tile + lane * rs + d4) = 1.0;
      }
    int64_t t = (int64_t)m * RS;
    const int64_t step = (int64_t)M * RS;
    int h = 0;
    if (t < n) issue(t, 0);
#pragma unroll 1
    for (; t < n; t += step) {
      __syncwarp();  // every lane is done with the other tile
      if (t + step < n) issue(t + step, h ^ 1);
      else cp_async_commit();
      cp_async_wait1();
      __syncwarp();
      f(base + h * L.tile, (int)min((int64_t)RS, n - t));
      h ^= 1;
    }
    cp_async_wait0();
    __syncwarp();
  }
  __device__ __forceinline__ int row(int X) const { return X + min(lane, RS - 1) * rs; }

  // ----------------------------------------------------------------- sums
  __device__ __forceinline__ int total(int side) const {
    return G.P == 1 ? base : ((G.cluster ? 2 : 0) + side) * L.per_warp;
  }
  __device__ __forceinline__ void add_members(int len, bool sides = false) {
    if (G.P == 1) {
      __syncwarp();
      return;
    }
    gang_sum(L.per_warp, len, sides ? 2 : 1, G.cluster);
    pending = G.cluster;
  }

  // --------------------------------------------------------------- scores
  // The row's x . w and (SEARCH) x . d, and its fitted values by both models.
  template <bool SEARCH>
  __device__ __forceinline__ void fits(int xr, double& u, double& v, double& fl, double& fr) const {
    const double2* x2 = (const double2*)(sw + xr);
    const double2* w2 = (const double2*)(sw + vb + L.th);
    const double2* d2 = (const double2*)(sw + vb + L.dn);
    const double2* lin = (const double2*)(sw + vb + L.lin);
    u = v = 0.0;
    fl = V(L.cst);
    fr = V(L.cst + 1);
#pragma unroll 1
    for (int i = 0; i < d4; i += 4) {
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        const double2 x = x2[q], w = w2[q], b0 = lin[2 * q], b1 = lin[2 * q + 1];
        u = fma(w.x, x.x, u);
        fl = fma(b0.x, x.x, fl);
        fr = fma(b0.y, x.x, fr);
        u = fma(w.y, x.y, u);
        fl = fma(b1.x, x.y, fl);
        fr = fma(b1.y, x.y, fr);
        if (SEARCH) {
          const double2 dv = d2[q];
          v = fma(dv.x, x.x, v);
          v = fma(dv.y, x.y, v);
        }
      }
      x2 += 2;
      w2 += 2;
      d2 += 2;
      lin += 4;
    }
    if (quad) {  // d <= 8: x_i sum_{j >= i} b_ij x_j, zero-padded to eight inputs
      const double2* q = (const double2*)(sw + vb + L.quad);
      double xv[8];
#pragma unroll
      for (int i = 0; i < 8; ++i) xv[i] = i < d ? sw[xr + i] : 0.0;
      int f = 0;
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        if (i >= d) break;
        double sl = 0.0, sr = 0.0;
#pragma unroll
        for (int j = i; j < 8; ++j) {
          const double2 b = q[f + j - i];
          sl = fma(b.x, xv[j], sl);
          sr = fma(b.y, xv[j], sr);
        }
        f += 8 - i;
        fl = fma(xv[i], sl, fl);
        fr = fma(xv[i], sr, fr);
      }
    }
  }
  __device__ __forceinline__ double score(int xr) const {  // x . w
    const double2* x2 = (const double2*)(sw + xr);
    const double2* w2 = (const double2*)(sw + vb + L.th);
    double u0 = 0.0, u1 = 0.0;
#pragma unroll 1
    for (int i = 0; i < d4; i += 4) {
      const double2 xa = x2[0], xb = x2[1], wa = w2[0], wb = w2[1];
      u0 = fma(wa.x, xa.x, u0);
      u1 = fma(wa.y, xa.y, u1);
      u0 = fma(wb.x, xb.x, u0);
      u1 = fma(wb.y, xb.y, u1);
      x2 += 2;
      w2 += 2;
    }
    return u0 + u1;
  }
  // exact side (right_side), by the plain score where its error bound allows
  __device__ __forceinline__ bool side(int at, double z) const {
    const double *w = sw + vb + L.th, *xr = sw + at;
    double s = 0.0, mag = 0.0;
    for (int i = 0; i < d; ++i) {
      s = fma(xr[i], w[i], s);
      mag = fma(fabs(xr[i]), fabs(w[i]), mag);
    }
    s = __dsub_rn(s, z);
    mag = __dadd_rn(mag, fabs(z));
    if (fabs(s) > 2.220446049250313e-16 * (d + 4) * mag && mag > 1e-280) return s >= 0.0;
    return right_side(xr, w, d, z);
  }

  // ---------------------------------------------------------------- Grams
  // A row's weights stand at Q: (q_L, q_L y, q_R, q_R y), one side per warp (q, q y).
  static constexpr int LAST = NB * (NB - 1) / 2;  // first of the last block row's accumulators
  __device__ __forceinline__ void gram_tile(int X, int rows4, double (&cL)[NBLK][2], double (&cR)[SIDED ? 1 : NBLK][2]) const {
    const int Q = base + L.Q;
    const int k4 = rows4;
    const bool pad = 8 * (NB - 1) + mq() > p;
    auto frag = [&](int xk, double (&v)[NB]) {
#pragma unroll
      for (int I = 0; I < NB; ++I) {
        v[I] = sw[xk + fa[I]];
        if (quad) v[I] *= sw[xk + fb[I]];
      }
      if (pad) v[NB - 1] = 0.0;  // this lane's column of the last block lies past psi
    };
    if (NB > 1 && NB <= 5 && apart) {
      // blocks of the inputs alone; lane = input for the sums of q x and q y x,
      // those of a tile added up before they go to the total
      double t[2][2] = {{0.0, 0.0}, {0.0, 0.0}};
      constexpr int C = NB > 1 ? 8 * (NB - 1) : 8, W_ = SIDED ? 2 : 4;
      const int col = SIDED ? (lane < C ? lane : 0) : lane & (C - 1);
      const int w0 = Q + (SIDED ? 0 : 2 * ((lane / C) & 1));
      constexpr int G_ = SIDED ? 1 : (C < 16 ? 2 : 1);  // lane groups that take every G_-th row
      const int g0 = G_ > 1 ? lane / (2 * C) : 0;
#pragma unroll 2
      for (int k0 = 0; k0 < k4; k0 += 4) {
        const int r = k0 + kq(), xk = X + r * rs + mq();
        double v[NB];
#pragma unroll
        for (int I = 0; I < NB - 1; ++I) v[I] = sw[xk + 8 * I];
        const double ql = sw[Q + W_ * r], qr = SIDED ? 0.0 : sw[Q + W_ * r + (SIDED ? 0 : 2)];
#pragma unroll
        for (int I = 0; I < NB - 1; ++I) {
          const double aL = ql * v[I], aR = qr * v[I];
#pragma unroll
          for (int J = 0; J <= I; ++J) {
            split_dmma(cL[I * (I + 1) / 2 + J], aL, v[J]);
            if constexpr (!SIDED) split_dmma(cR[I * (I + 1) / 2 + J], aR, v[J]);
          }
        }
#pragma unroll
        for (int m = 0; m < 4 / G_; ++m) {
          const int rr = k0 + G_ * m + g0;
          const double2 w = *(const double2*)(sw + w0 + W_ * rr);
          const double xv = sw[X + rr * rs + col];
          t[m & 1][0] = fma(w.x, xv, t[m & 1][0]);
          t[m & 1][1] = fma(w.y, xv, t[m & 1][1]);
        }
      }
      cL[LAST][0] += t[0][0] + t[1][0];
      cL[LAST][1] += t[0][1] + t[1][1];
      return;
    }
    if constexpr (SIDED) {
#pragma unroll 2
      for (int k0 = 0; k0 < k4; k0 += 4) {
        const int r = k0 + kq();
        const double q = sw[Q + 2 * r];
        double v[NB];
        frag(X + r * rs, v);
#pragma unroll
        for (int I = 0; I < NB; ++I) {
          const double av = q * v[I];
#pragma unroll
          for (int J = 0; J <= I; ++J) split_dmma(cL[I * (I + 1) / 2 + J], av, v[J]);
        }
      }
    } else if (narrow) {
      // the last block row holds tail <= 4 columns: its rows of both sides in
      // one MMA per block column, A = psi block J, B = [q_L psi_T, q_R psi_T]
      // (columns n < tail: left, tail <= n < 2 tail: right), the results in
      // cL's last block row
      const bool tl = mq() < 2 * tail;
      const int src = (mq() < tail ? mq() : mq() - tail) * 4 + kq();  // lane holding that tail column
#pragma unroll 2
      for (int k0 = 0; k0 < k4; k0 += 4) {
        const int r = k0 + kq();
        const double ql = sw[Q + 4 * r], qr = sw[Q + 4 * r + 2];
        double v[NB];
        frag(X + r * rs, v);
#pragma unroll
        for (int I = 0; I < NB - 1; ++I) {
          const double aL = ql * v[I], aR = qr * v[I];
#pragma unroll
          for (int J = 0; J <= I; ++J) {
            split_dmma(cL[I * (I + 1) / 2 + J], aL, v[J]);
            split_dmma(cR[I * (I + 1) / 2 + J], aR, v[J]);
          }
        }
        const double vt = __shfl_sync(0xffffffffu, v[NB - 1], src & 31);
        const double bt = tl ? (mq() < tail ? ql : qr) * vt : 0.0;
#pragma unroll
        for (int J = 0; J < NB; ++J) split_dmma(cL[LAST + J], v[J], bt);
      }
    } else {
#pragma unroll 2
      for (int k0 = 0; k0 < k4; k0 += 4) {
        const int r = k0 + kq();
        const double ql = sw[Q + 4 * r], qr = sw[Q + 4 * r + 2];
        double v[NB];
        frag(X + r * rs, v);
#pragma unroll
        for (int I = 0; I < NB; ++I) {
          const double aL = ql * v[I], aR = qr * v[I];
#pragma unroll
          for (int J = 0; J <= I; ++J) {
            split_dmma(cL[I * (I + 1) / 2 + J], aL, v[J]);
            split_dmma(cR[I * (I + 1) / 2 + J], aR, v[J]);
          }
        }
      }
    }
  }
  // The rows' own part with the inputs apart: sums of q, q y and q y^2.
  __device__ __forceinline__ void row_sums(double qL, double qLy, double qR, double qRy, double y,
                                           double (&cL)[NBLK][2], double (&cR)[SIDED ? 1 : NBLK][2]) const {
    if constexpr (SIDED) {
      cL[LAST + 1][0] += qL;
      cL[LAST + 1][1] += qLy;
      cL[LAST + 2][0] = fma(qLy, y, cL[LAST + 2][0]);
    } else if constexpr (NB > 1) {
      cL[LAST + 1][0] += qL;
      cL[LAST + 1][1] += qLy;
      cR[LAST][0] = fma(qLy, y, cR[LAST][0]);
      cR[LAST][1] = fma(qRy, y, cR[LAST][1]);
      cR[LAST + 1][0] += qR;
      cR[LAST + 1][1] += qRy;
    }
  }
  // The accumulators as packed lower triangles: L at base, R at base + E (one
  // side per warp: that side at base).
  __device__ __forceinline__ void store_gram(const double (&cL)[NBLK][2], const double (&cR)[SIDED ? 1 : NBLK][2]) const {
    if (NB > 1 && NB <= 5 && apart) {  // psi = inputs, 1, y; the blocks hold the inputs alone
#pragma unroll
      for (int I = 0; I < NB - 1; ++I)
#pragma unroll
        for (int J = 0; J <= I; ++J)
#pragma unroll
          for (int t = 0; t < 2; ++t) {
            const int i = 8 * I + mq(), j = 8 * J + 2 * kq() + t;
            if (i < d && j <= i) {
              B(pk(i, j)) = cL[I * (I + 1) / 2 + J][t];
              if constexpr (!SIDED) B(E + pk(i, j)) = cR[I * (I + 1) / 2 + J][t];
            }
          }
      constexpr int C = NB > 1 ? 8 * (NB - 1) : 8;
      double s1 = cL[LAST][0], sy = cL[LAST][1];
      if constexpr (!SIDED && C == 8) {  // two lane groups
        s1 += __shfl_xor_sync(0xffffffffu, s1, 16);
        sy += __shfl_xor_sync(0xffffffffu, sy, 16);
      }
      const int c = SIDED ? lane : lane & (C - 1), at = SIDED || lane < C ? 0 : E;
      if (c < d && lane < (SIDED ? C : 2 * C)) {
        B(at + pk(d, c)) = s1;
        B(at + pk(p, c)) = sy;
      }
      if constexpr (SIDED) {
        const double q = warp_sum(cL[LAST + 1][0]), qy = warp_sum(cL[LAST + 1][1]), qyy = warp_sum(cL[LAST + 2][0]);
        if (lane == 0) B(pk(d, d)) = q, B(pk(p, d)) = qy, B(pk(p, p)) = qyy;
      } else if constexpr (NB > 1) {
        const double q = warp_sum(cL[LAST + 1][0]), qy = warp_sum(cL[LAST + 1][1]), qyy = warp_sum(cR[LAST][0]);
        const double r = warp_sum(cR[LAST + 1][0]), ry = warp_sum(cR[LAST + 1][1]), ryy = warp_sum(cR[LAST][1]);
        if (lane == 0) {
          B(pk(d, d)) = q, B(pk(p, d)) = qy, B(pk(p, p)) = qyy;
          B(E + pk(d, d)) = r, B(E + pk(p, d)) = ry, B(E + pk(p, p)) = ryy;
        }
      }
      return;
    }
#pragma unroll
    for (int I = 0; I < NB; ++I) {
      if (!SIDED && narrow && I == NB - 1) continue;
#pragma unroll
      for (int J = 0; J <= I; ++J)
#pragma unroll
        for (int t = 0; t < 2; ++t) {
          const int i = 8 * I + mq(), j = 8 * J + 2 * kq() + t;
          if (i < pa && j <= i) {
            B(pk(i, j)) = cL[I * (I + 1) / 2 + J][t];
            if constexpr (!SIDED) B(E + pk(i, j)) = cR[I * (I + 1) / 2 + J][t];
          }
        }
    }
    if (!SIDED && narrow) {
      // lane (m, k) holds D[m][n], n = 2 k + t: side n / tail, row T + n % tail,
      // column 8 J + m
#pragma unroll
      for (int J = 0; J < NB; ++J)
#pragma unroll
        for (int t = 0; t < 2; ++t) {
          const int n_ = 2 * kq() + t;
          if (n_ < 2 * tail) {
            const int i = 8 * (NB - 1) + (n_ < tail ? n_ : n_ - tail), j = 8 * J + mq();
            if (i < pa && j <= i) B((n_ < tail ? 0 : E) + pk(i, j)) = cL[(NB - 1) * NB / 2 + J][t];
          }
        }
    }
  }

  // Side Grams at theta; HARD: weights 1 / 0 by the exact sides and the right
  // count (without `grams`: the count alone).
  template <bool HARD>
  __device__ __forceinline__ void gram_pass(bool grams) {
    double cL[NBLK][2], cR[SIDED ? 1 : NBLK][2];
#pragma unroll
    for (int q = 0; q < NBLK; ++q) {
      cL[q][0] = cL[q][1] = 0.0;
      if constexpr (!SIDED) cR[q][0] = cR[q][1] = 0.0;
    }
    sync();  // theta is in place
    const double z = V(L.scal + SC_Z);
    const bool pair = SIDED && grams;
    const bool rside = pair && (G.g & 1);
    int cnt = 0;
    tiles(pair ? G.g >> 1 : G.g, pair ? G.P >> 1 : G.P, [&](int X, int rows) {
      const int xr = row(X);
      double qL = 0.0, qR = 0.0;
      if (HARD) {
        if (lane < rows) {
          const bool right = side(xr, z);
          cnt += right && !rside ? 1 : 0;
          qL = right ? 0.0 : 1.0;
          qR = right ? 1.0 : 0.0;
        }
      } else {
        const double pi = gate((score(xr) - z) * invT);
        qL = lane < rows ? fmax(1.0 - pi, a.prm.weight_floor) : 0.0;
        qR = lane < rows ? fmax(pi, a.prm.weight_floor) : 0.0;
      }
      if (HARD && !grams) return;
      // lanes past the rows have no weight; their y may be anything
      const double y = lane < rows ? sw[xr + d4 + 1] : 0.0;
      if (SIDED) {
        const double q = rside ? qR : qL, qy = q * y;
        *(double2*)(sw + base + L.Q + 2 * lane) = make_double2(q, qy);
        if (apart) row_sums(q, qy, 0.0, 0.0, y, cL, cR);
      } else {
        const double qLy = qL * y, qRy = qR * y;
        *(double2*)(sw + base + L.Q + 4 * lane) = make_double2(qL, qLy);
        *(double2*)(sw + base + L.Q + 4 * lane + 2) = make_double2(qR, qRy);
        if (apart) row_sums(qL, qLy, qR, qRy, y, cL, cR);
      }
      __syncwarp();
      gram_tile(X, (rows + 3) & ~3, cL, cR);
    });
    const int at = pair ? E : (grams ? 2 * E : 0);  // the count follows the sums
    if (grams) store_gram(cL, cR);
    if (HARD) {
      for (int o = 16; o > 0; o >>= 1) cnt += __shfl_xor_sync(0xffffffffu, cnt, o);
      if (lane == 0) B(at) = (double)cnt;  // exact in any order
    }
    add_members(at + (HARD ? 1 : 0), pair);
    if (HARD) nright = (int)sw[total(0) + at];
  }

  // Both sides' ridge solves from the Gram totals (in a gang warp 0 the left,
  // warp 1 the right one) and the child models as score columns; false: a
  // factorisation failed.
  __device__ __forceinline__ bool solve_sides() {
    sync();
    constexpr int RPL = NB >= 4 ? 2 : 1;
#pragma unroll 1
    for (int s = 0; s < 2; ++s)
      if (G.P == 1 || warp == s)
        solve_side<RPL>(SIDED ? total(s) : total(0) + s * E, vb + (s ? L.br : L.bl), vb + L.scal + SC_FAILL + s,
                        vb + L.scal + SC_LAML + s, p, ridge);
    sync();
    const bool ok = V(L.scal + SC_FAILL) == 0.0 && V(L.scal + SC_FAILR) == 0.0;
    lamL = V(L.scal + SC_LAML);
    lamR = V(L.scal + SC_LAMR);
    if (leads()) {
      if (quad)
        for (int e = lane; e < 72; e += 32) V(L.quad + e) = 0.0;
      if (lane == 0) V(L.cst) = V(L.cst + 1) = 0.0;
      __syncwarp();
      for (int f = lane; f < p; f += 32) {
        int ia, ib;
        feature_factors(d, kind, f, ia, ib);
        const double bl = V(L.bl + f), br = V(L.br + f);
        int at;
        if (ia < 0) at = L.cst;
        else if (ib < 0) at = L.lin + 2 * ia;
        else at = L.quad + 2 * (8 * ia - ia * (ia - 1) / 2 + ib - ia);
        V(at) = bl;
        V(at + 1) = br;
      }
    }
    sync();
    return ok;
  }

  // Soft residual pass at theta: loss, gradient, n_right (pi >= 0.5), the
  // projected gradient, its norm and the directional derivative.
  __device__ __forceinline__ void resid_pass() {
    // Gradient sum of c_r x_r: a lane's own row into one accumulator an input;
    // with the wide form's inputs that is 48 of them and a final sum of 48 x 32,
    // so there lane = input, and with 16 inputs or fewer lane groups take their
    // own rows (149 nodes to 120,000 rows, d = 32 or quadratic of d = 8: 29.9 ms
    // to 27.8; in the narrow form the own row is the faster: 71.0 ms to 74.0 for
    // 256 nodes of 16 restarts).
    constexpr int DP = NB <= 3 ? 8 * NB : 0;
    const int group = d <= 8 ? 8 : (d <= 16 ? 16 : 32), col = lane & (group - 1);
    const int row0 = lane & ~(group - 1);
    const double z = V(L.scal + SC_Z);
    const double inv_n = 1.0 / (double)n;
    double g[DP > 0 ? DP : 2];
#pragma unroll
    for (int i = 0; i < (DP > 0 ? DP : 2); ++i) g[i] = 0.0;
    double sl = 0.0, sa = 0.0, snr = 0.0;
    tiles(G.g, G.P, [&](int X, int rows) {
      const int xr = row(X);
      double u, v, fl, fr;
      fits<false>(xr, u, v, fl, fr);
      // lanes past the tile's rows run along and add nothing
      const double yv = sw[xr + d4 + 1];
      const double pi = gate((u - z) * invT);
      const double eL = yv - fl, eR = yv - fr;
      const double eL2 = eL * eL, eR2 = eR * eR;
      const double c = (eR2 - eL2) * pi * (1.0 - pi) * inv_n;
      const bool live = lane < rows;
      sl += live ? (1.0 - pi) * eL2 + pi * eR2 : 0.0;
      sa += live ? c : 0.0;
      snr += live && pi >= 0.5 ? 1.0 : 0.0;
      if constexpr (DP == 0) {
        // columns past the inputs are read from what follows and dropped
        B(L.Q + lane) = live ? c : 0.0;
        __syncwarp();
        const int end = min(row0 + group, rows);
        int at = X + row0 * rs + col;
#pragma unroll 4
        for (int r = row0; r < end; ++r) {
          g[0] = fma(B(L.Q + r), sw[at], g[0]);
          at += rs;
        }
        if (d > 32)
          for (int r = 0; r < rows; ++r) g[1] = fma(B(L.Q + r), sw[X + r * rs + lane + 32], g[1]);
      } else if (live) {
        const double2* x2 = (const double2*)(sw + xr);
#pragma unroll
        for (int i = 0; i < DP; i += 4)
          if (i < d4) {
            const double2 xa = x2[i / 2], xb = x2[i / 2 + 1];
            g[i] = fma(c, xa.x, g[i]);
            g[i + 1] = fma(c, xa.y, g[i + 1]);
            g[i + 2] = fma(c, xb.x, g[i + 2]);
            g[i + 3] = fma(c, xb.y, g[i + 3]);
          }
      }
    });
    const double ts = warp_sum(sl), ta = warp_sum(sa), tn = warp_sum(snr);
    double t[2] = {g[0], g[1]};
    if constexpr (DP == 0) {
      for (int o = group; o < 32; o <<= 1) t[0] += __shfl_xor_sync(0xffffffffu, t[0], o);
    } else {  // lanes' sums added through shared memory, lane i taking input i
#pragma unroll
      for (int i = 0; i < DP; ++i)
        if (i < d) B(i * 33 + lane) = g[i];
      __syncwarp();
      t[0] = t[1] = 0.0;
      if (lane < d) {
        double s0 = 0.0, s1 = 0.0;
#pragma unroll 8
        for (int q = 0; q < 32; q += 2) {
          s0 += B(lane * 33 + q);
          s1 += B(lane * 33 + q + 1);
        }
        t[0] = s0 + s1;
      }
      __syncwarp();
    }
#pragma unroll
    for (int m = 0; m < 2; ++m)
      if (lane + 32 * m < d) B(lane + 32 * m) = t[m];
    if (lane == 0) {
      B(d) = ta;
      B(d + 1) = ts;
      B(d + 2) = tn;
    }
    add_members(d + 3);
    const double* tot = sw + total(0);
    if (leads()) {  // splitters.py:86-98
      const double* w = sw + vb + L.th;
      double gi[2], gw = 0.0;
#pragma unroll
      for (int m = 0; m < 2; ++m) {
        const int i = lane + 32 * m;
        gi[m] = i < d ? tot[i] / T : 0.0;
        if (i < d) gw = fma(gi[m], w[i], gw);
      }
      gw = wsum(gw);
      const double gz = -tot[d] / T;
      double n2 = 0.0, sd = 0.0;
#pragma unroll
      for (int m = 0; m < 2; ++m) {
        const int i = lane + 32 * m;
        if (i < d) {
          const double pg = gi[m] - gw * w[i];
          n2 = fma(pg, pg, n2);
          sd = fma(gi[m], -pg, sd);
          V(L.dn + i) = -pg;
        }
      }
      n2 = wsum(n2) + gz * gz;
      sd = wsum(sd) + gz * -gz;
      if (lane == 0) {
        V(L.scal + SC_DZ) = -gz;
        V(L.scal + SC_LOSS) = tot[d + 1] / (double)n;
        V(L.scal + SC_NRIGHT) = tot[d + 2];
        V(L.scal + SC_GNORM) = sqrt(n2);
        V(L.scal + SC_DD) = sd;
      }
    }
    sync();
    loss = V(L.scal + SC_LOSS);
    nright = (int)V(L.scal + SC_NRIGHT);
    gnorm = V(L.scal + SC_GNORM);
    dd = V(L.scal + SC_DD);
  }

  // |w + alpha d| (every lane)
  __device__ __forceinline__ double step_norm(double alpha) const {
    double s = 0.0;
    for (int i = lane; i < d; i += 32) {
      const double v = fma(alpha, V(L.dn + i), V(L.th + i));
      s = fma(v, v, s);
    }
    return sqrt(wsum(s));
  }

  // Frozen-model losses of the candidates at the current temperature.
  __device__ __forceinline__ void search_pass(const double (&alpha)[kCand], double (&f)[kCand]) {
    double inw[kCand], anw[kCand], zc[kCand], s[kCand];
#pragma unroll
    for (int c = 0; c < kCand; ++c) {
      s[c] = 0.0;
      inw[c] = 1.0 / step_norm(alpha[c]);
      anw[c] = alpha[c] * inw[c];
      zc[c] = fma(alpha[c], V(L.scal + SC_DZ), V(L.scal + SC_Z));
    }
    tiles(G.g, G.P, [&](int X, int rows) {
      const int xr = row(X);
      double u, v, fl, fr;
      fits<true>(xr, u, v, fl, fr);
      const double yv = sw[xr + d4 + 1];
      const double eL = yv - fl, eR = yv - fr;
      const double eL2 = eL * eL, eR2 = eR * eR;
      const bool live = lane < rows;
#pragma unroll
      for (int c = 0; c < kCand; ++c) {
        const double pi = gate(fma(u, inw[c], fma(v, anw[c], -zc[c])) * invT);
        s[c] += live ? (1.0 - pi) * eL2 + pi * eR2 : 0.0;
      }
    });
#pragma unroll
    for (int c = 0; c < kCand; ++c) {
      const double t = warp_sum(s[c]);
      if (lane == 0) B(c) = t;
    }
    add_members(kCand);
    const double* tot = sw + total(0);
#pragma unroll
    for (int c = 0; c < kCand; ++c) f[c] = tot[c] / (double)n;
  }

  // Hard losses: mean squared residual of each side's hard model.
  __device__ __forceinline__ void hard_losses(double& hl, double& hr) {
    const double z = V(L.scal + SC_Z);
    double sL = 0.0, sR = 0.0;
    tiles(G.g, G.P, [&](int X, int rows) {
      const int xr = row(X);
      double u, v, fl, fr;
      fits<false>(xr, u, v, fl, fr);
      if (lane < rows) {
        const bool right = side(xr, z);
        const double e = sw[xr + d4 + 1] - (right ? fr : fl);
        (right ? sR : sL) += e * e;
      }
    });
    sL = warp_sum(sL);
    sR = warp_sum(sR);
    if (lane == 0) { B(0) = sL; B(1) = sR; }
    add_members(2);
    const double* tot = sw + total(0);
    const int nl = (int)n - nright;
    hl = tot[0] / nl;
    hr = tot[1] / nright;
    loss = (double)nl / n * hl + (double)nright / n * hr;
  }

  __device__ __forceinline__ void run(int item);
};

template <int NB, bool SIDED>
__device__ __forceinline__ void SplitWarp<NB, SIDED>::run(int item) {
  const ArtSplitParams& P = a.prm;
  const int64_t k = item / a.R;
  const int64_t kr = (int64_t)item;  // items are k * R + restart
  r0 = a.row_offsets[k];
  n = a.row_offsets[k + 1] - r0;
  xg = a.x + a.x_offsets[k];
  d = a.dims[k];
  kind = a.features[k];
  p = feature_count(d, kind);
  pa = p + 1;
  E = pa * (pa + 1) / 2;
  d4 = pad4(d);
  rs = tile_stride(d);
  RS = tile_rows(d);
  pairs = (d & 1) == 0 && ((uintptr_t)xg & 15) == 0;
  const int cpr = pairs ? d / 2 : d;  // copies per row
  step_r = 32 / cpr;
  step_c = 32 - step_r * cpr;
  lr0 = lane / cpr;
  lc0 = lane - lr0 * cpr;
  quad = kind == ART_FEATURES_POLY2 || kind == ART_FEATURES_POLY2_NOBIAS;
  tail = pa - 8 * (NB - 1);
  narrow = tail <= 4;
  // Affine models whose inputs fill whole blocks, at most one input a lane (and
  // side): 1 and y would take a block row of their own, of which two columns of
  // eight are used.  256 nodes of d = 16, 16 restarts: 71.6 ms to 69.9; 149 nodes
  // to 120,000 rows, d = 32 or quadratic of d = 8: 24.9 ms to 24.2.
  apart = NB > 1 && NB <= 5 && kind == ART_FEATURES_AFFINE && tail <= 2;
#pragma unroll
  for (int I = 0; I < NB; ++I) {
    const int f = 8 * I + mq();
    int ia = d4, ib = d4;  // the constant
    if (f < p) {
      feature_factors(d, kind, f, ia, ib);
      if (ia < 0) ia = d4;
      if (ib < 0) ib = d4;
    } else if (f == p) {
      ia = d4 + 1;  // y
    }
    fa[I] = ia;
    fb[I] = ib;
  }
  T0 = a.temperature[k];
  ridge = a.ridge[k];
  const int req = max(a.min_side ? max(1, a.min_side[k]) : P.min_side_points,
                      (int)ceil(P.min_side_fraction * (double)n));
  const bool fb_allowed = a.fallback ? a.fallback[k] != 0 : false;
  const int M = P.max_iters;
  const bool writer = lane == 0 && G.g == 0;
  sync();  // the last item's vectors are no longer read
  // initial theta: projected theta0 (splitters.py:379)
  const double* t0 = a.theta0 + kr * a.theta0_stride;
  double n2 = 0.0;
  for (int i = 0; i < d; ++i) n2 += t0[i] * t0[i];
  const double nrm = sqrt(n2);
  bool active = true, hasfeas = false, conv = false, fbk = false;
  int fail = 0, iters = 0, stop = ART_STOP_MAX_ITERS, feasit = -1;
  if (!(nrm > 1e-12) || !isfinite(nrm)) { active = false; fail = ART_SPLIT_INVALID; }
  if (leads()) {
    for (int i = lane; i < d; i += 32) {
      const double w = t0[i] / nrm;
      V(L.th + i) = w;
    }
    for (int i = d + lane; i < d4; i += 32) V(L.th + i) = V(L.dn + i) = V(L.lin + 2 * i) = V(L.lin + 2 * i + 1) = 0.0;
    if (lane == 0) V(L.scal + SC_Z) = t0[d];
  }
  sync();
  T = T0;
  invT = 1.0 / T0;
  double alpha = fmin(fmax(P.alpha0, P.alpha_min), P.alpha_max), tol = 0.0;
  nright = 0;
  loss = gnorm = dd = lamL = lamR = 0.0;
  if (n == 0) { active = false; fail = ART_SPLIT_MIN_SIDE_POINTS; }
  auto record_trace = [&](int iter) {
    if (!writer) return;
    if (a.tr_loss) a.tr_loss[kr * (M + 1) + iter] = loss;
    if (a.tr_gnorm) a.tr_gnorm[kr * (M + 1) + iter] = gnorm;
  };
  auto save_feasible = [&](int it_) {
    if (min(nright, (int)n - nright) >= req) {
      hasfeas = true;
      feasit = it_;
      if (leads())
        for (int i = lane; i <= d; i += 32) V(L.lf + i) = i < d ? V(L.th + i) : V(L.scal + SC_Z);
    }
  };
  for (int iter = 0; active; ++iter) {
    // evaluate(theta): child fits from the Grams, then the residual pass
    gram_pass<false>(true);
    if (!solve_sides()) {
      active = false;
      fail = ART_SPLIT_CHOLESKY_FAILURE;
      break;
    }
    resid_pass();
    if (iter == 0) tol = P.grad_atol + P.grad_rtol * gnorm;
    save_feasible(iter);
    record_trace(iter);
    if (iter >= M) break;
    // stop checks (splitters.py:424-437)
    if (gnorm <= tol) { conv = true; stop = ART_STOP_GRADIENT_TOLERANCE; active = false; break; }
    if (dd >= 0.0) { stop = ART_STOP_NON_DESCENT; active = false; break; }
    // Armijo backtracking (optimizers.py:72-121), kCand candidates of an
    // attempt per pass, taken in order; restarted from the adapted step after
    // a failed attempt
    bool accept = false;
    int failures = 0, nb_ = 0;
    double a_ = P.adaptive_alpha ? alpha : P.alpha0, step = 0.0;
    for (;;) {
      double al[kCand], f[kCand];
      const int nc = min(kCand - 1, P.max_backtracks - nb_) + 1;
      al[0] = a_;
#pragma unroll
      for (int c = 1; c < kCand; ++c) al[c] = al[c - 1] * P.rho;
      search_pass(al, f);
      int hit = -1;
#pragma unroll
      for (int c = kCand - 1; c >= 0; --c) {
        const double rhs = __dadd_rn(loss, __dmul_rn(__dmul_rn(P.armijo_c, al[c]), dd));
        if (c < nc && f[c] <= rhs) hit = c;
      }
      if (hit >= 0) {
        accept = true;
        nb_ += hit;
        step = al[0];
#pragma unroll
        for (int c = 1; c < kCand; ++c)
          if (c == hit) step = al[c];
        if (P.adaptive_alpha) {  // AdaptiveAlpha.update (optimizers.py:49-66)
          double na;
          if (nb_ == 0) na = step * P.alpha_grow;
          else if (nb_ >= P.heavy_backtrack_threshold) na = step * P.alpha_recovery;
          else na = step / P.rho;
          alpha = fmin(fmax(na, P.alpha_min), P.alpha_max);
        }
        break;
      }
      double last = al[0];
#pragma unroll
      for (int c = 1; c < kCand; ++c)
        if (c < nc) last = al[c];
      if (P.max_backtracks - nb_ >= nc && last != 0.0) {  // next backtracks
        nb_ += nc;
        a_ = last * P.rho;
        continue;
      }
      // (a step that has underflowed to zero stays there: those after it are as
      // unacceptable)
      // attempt failed: the last step tried
      if (P.adaptive_alpha) alpha = fmin(fmax(last * P.rho, P.alpha_min), P.alpha_max);
      ++failures;
      int st = -1;
      if (!P.adaptive_alpha) st = ART_STOP_LINE_SEARCH_FAILED;
      else if (failures >= P.max_line_search_failures) st = ART_STOP_MAX_LINE_SEARCH_FAILURES;
      else if (alpha <= P.alpha_min) st = ART_STOP_ALPHA_MIN_REACHED;
      if (st >= 0) {
        stop = st;
        break;
      }
      nb_ = 0;
      a_ = alpha;
    }
    if (!accept) {
      active = false;
      break;
    }
    // theta <- project(theta + step d) (splitters.py:451, 497), then the
    // temperature that follows an accepted step
    const double nw = step_norm(step);
    sync();  // every member has read theta and d
    if (leads())
      for (int i = lane; i <= d; i += 32) {
        if (i < d) V(L.th + i) = (V(L.th + i) + step * V(L.dn + i)) / nw;
        else V(L.scal + SC_Z) = V(L.scal + SC_Z) + step * V(L.scal + SC_DZ);
      }
    if (P.anneal_ratio != 1.0 && P.max_iters > 1) {
      T = T0 * pow(P.anneal_ratio, (double)(iter + 1) / (double)(P.max_iters - 1));
      invT = 1.0 / T;
    }
    iters = iter + 1;
    if (writer) {
      if (a.tr_step) a.tr_step[kr * P.max_iters + iter] = step;
      if (a.tr_back) a.tr_back[kr * P.max_iters + iter] = nb_;
    }
  }
  // ------------------------------------------------ finish (splitters.py:584-601)
  double hlossL = 0.0, hlossR = 0.0;
  if (fail == 0) {
    const bool final_ok = min(nright, (int)n - nright) >= req;
    fbk = !final_ok && fb_allowed && hasfeas;
    sync();
    if (leads()) {
      if (fbk)
        for (int i = lane; i <= d; i += 32) (i < d ? V(L.th + i) : V(L.scal + SC_Z)) = V(L.lf + i);
      __syncwarp();
      double s2 = 0.0;
      for (int i = 0; i < d; ++i) s2 += V(L.th + i) * V(L.th + i);
      const double nw = sqrt(s2);
      __syncwarp();
      for (int i = lane; i < d; i += 32) V(L.th + i) = V(L.th + i) / nw;
    }
    // hard partition: exact sides and right count; hard child fits when asked
    gram_pass<true>(P.hard_refit != 0);
    if (nright < req || (int)n - nright < req) {
      fail = ART_SPLIT_MIN_SIDE_POINTS;
    } else if (P.hard_refit) {
      if (!solve_sides()) fail = ART_SPLIT_CHOLESKY_FAILURE;
      else hard_losses(hlossL, hlossR);
    }
  }
  // ----------------------------------------------------------- write results
  sync();
  if (writer) {
    const int dts = a.dmax + 1;
    for (int i = 0; i <= d; ++i) a.r_theta[kr * dts + i] = i < d ? V(L.th + i) : V(L.scal + SC_Z);
    a.r_fail[kr] = fail;
    a.r_stop[kr] = stop;
    a.r_iters[kr] = iters;
    a.r_nright[kr] = nright;
    a.r_flags[kr] = (conv ? 1 : 0) | (fbk ? 2 : 0);
    a.r_fbiter[kr] = feasit;
    a.r_alpha[kr] = P.adaptive_alpha ? alpha : P.alpha0;
    const double nan = __longlong_as_double(0x7ff8000000000000ll);
    const bool have = P.hard_refit && fail == 0;
    a.r_loss[kr] = have ? loss : nan;
    a.r_child[kr * 2] = P.hard_refit ? hlossL : nan;
    a.r_child[kr * 2 + 1] = P.hard_refit ? hlossR : nan;
    a.r_ridge[kr * 2] = lamL;
    a.r_ridge[kr * 2 + 1] = lamR;
    for (int f = 0; f < p; ++f) {
      a.r_beta[(kr * 2) * a.pmax + f] = have ? V(L.bl + f) : nan;
      a.r_beta[(kr * 2 + 1) * a.pmax + f] = have ? V(L.br + f) : nan;
    }
  }
  if (pending) {
    cluster_wait();
    pending = false;
  }
}

// Items come largest first (wide models never below the CTA gangs): while they
// are large the cluster, then the CTA, takes one at a time; from the first
// small one on, each warp pops its own, warp 0 of the CTA that met it starting
// with that one.  (One call site per model width keeps the search inlined and
// its state in registers.)
// CTAs an SM: the narrow form's state fits 168 registers a thread (4 of 128
// spill: 79.5 ms instead of 71.0 at 16 restarts); the wide form's does not, and
// two CTAs leave room for whole 32-row tiles (149 nodes to 120,000 rows: 27.3 ms
// with three, 26.0 with two, 24.9 with tiles of 32 rows instead of 24).
template <bool WIDE>
__global__ void __launch_bounds__(kWThreads, WIDE ? 2 : 3) split_warp_kernel(const __grid_constant__ WArgs W) {
  __shared__ int s_q;
  const SplitArgs& a = W.a;
  cg::cluster_group cl = cg::this_cluster();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int crank = W.csize > 1 ? (int)cl.block_rank() : 0;
  const int count = a.counts[0];
  const int cta_log = a.R <= 2 ? kCtaLogFew : kCtaLogMany;
  int phase = W.csize > 1 ? 0 : 1;  // 0: cluster, 1: CTA, 2: warp
  // every CTA of the cluster has started before one writes to another's memory
  if (phase == 0) cl.sync();
  for (;;) {
    int q = -1;
    Gang g{1, 0, false};
    if (phase == 0) {
      if (crank == 0 && threadIdx.x == 0) {
        const int v = atomicAdd(&a.counts[1], 1);
        for (int c = 0; c < W.csize; ++c) *cl.map_shared_rank(&s_q, c) = v;
      }
      cl.sync();
      q = s_q;
      cl.sync();
      if (q >= count) return;
      const int64_t k = a.items[q].x / a.R;
      if (ilogb((double)(a.row_offsets[k + 1] - a.row_offsets[k] + 1)) >= kClusterLogFew) {
        g = Gang{kWWarps * W.csize, crank * kWWarps + warp, true};
      } else {
        phase = 1;
        if (crank != 0) q = -1;  // CTA 0 takes the item that ended the phase
      }
    }
    if (phase == 1) {
      if (q < 0) {
        __syncthreads();
        if (threadIdx.x == 0) s_q = atomicAdd(&a.counts[1], 1);
        __syncthreads();
        q = s_q;
        if (q >= count) return;
      }
      const int64_t k = a.items[q].x / a.R;
      const int pa = feature_count(a.dims[k], a.features[k]) + 1;
      if (pa > kNarrowAug || ilogb((double)(a.row_offsets[k + 1] - a.row_offsets[k] + 1)) >= cta_log) {
        g = Gang{kWWarps, warp, false};
      } else {
        phase = 2;
        if (warp != 0) q = -1;
      }
    }
    if (phase == 2 && q < 0) {
      if (lane == 0) q = atomicAdd(&a.counts[1], 1);
      q = __shfl_sync(0xffffffffu, q, 0);
      if (q >= count) return;
    }
    const int item = a.items[q].x;
    const int64_t k = item / a.R;
    const int nb = (feature_count(a.dims[k], a.features[k]) + 1 + 7) / 8;
    if (nb == 1) SplitWarp<1, false>(W, g).run(item);
    else if (nb == 2) SplitWarp<2, false>(W, g).run(item);
    else if (nb == 3) SplitWarp<3, false>(W, g).run(item);
    else if constexpr (WIDE) {
      if (nb == 4) SplitWarp<4, true>(W, g).run(item);
      else if (nb == 5) SplitWarp<5, true>(W, g).run(item);
      else SplitWarp<6, true>(W, g).run(item);
    }
  }
}

}  // namespace

bool split_warp_fits(int max_dim, int max_features, int restarts) {
  if (max_dim <= kNarrowDim && max_features + 1 <= kNarrowAug) return true;
  return restarts <= 2 && max_dim <= kWideDim && max_features + 1 <= kWideAug;
}

int launch_split_warp(const SplitArgs& a, cudaStream_t s) {
  const bool wide = a.dmax > kNarrowDim || a.pmax + 1 > kNarrowAug;
  WArgs W;
  W.a = a;
  W.L = warp_layout(a.dmax, a.pmax);
  const size_t smem = (size_t)kWWarps * W.L.per_warp * sizeof(double);
  auto kern = wide ? split_warp_kernel<true> : split_warp_kernel<false>;
  if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess) {
    cudaGetLastError();
    set_error("art_split_level: cannot reserve %zu bytes of shared memory", smem);
    return ART_E_UNSUPPORTED;
  }
  const int occ = resident_ctas((const void*)kern, kWThreads, smem);
  const int csize = W.csize = a.R <= 2 ? kClusterCtas : 1;
  int64_t ctas = std::min<int64_t>((int64_t)device_sm_count() * std::max(occ, 1), a.K * a.R * csize);
  ctas = std::max<int64_t>(1, ctas / csize) * csize;
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = (unsigned)csize;
  attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
  cfg.gridDim = dim3((unsigned)ctas);
  cfg.blockDim = dim3(kWThreads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  prof_begin("split_level", s);
  const cudaError_t e = cudaLaunchKernelEx(&cfg, kern, W);
  prof_end(s);
  count_launch();
  if (e != cudaSuccess) {
    cudaGetLastError();
    set_error("split_level: %s", cudaGetErrorString(e));
    return ART_E_LAUNCH;
  }
  return check_launch("split_level");
}

}  // namespace art
