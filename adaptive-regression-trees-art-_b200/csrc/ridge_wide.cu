// ridge_wide.cu -- FP64 weighted ridge for systems of more than 47 features,
// one CTA of 16 warps per system, Grams on the FP64 tensor path
// (mma.sync m8n8k4 f64).
//
// What bounds it: the FP64 pipe.  The lower 8 x 8 blocks of the augmented Gram
// (210 at p = 153) are dealt to the warps as 4 x 4 groups, so a warp loads
// eight fragments for up to sixteen MMAs (loading two per MMA, or register
// tiles of FMAs, kept shared memory as busy as the pipe).  Chunks of 32 rows
// are expanded to sqrt(q) [phi(x), y] in one of two shared buffers while the
// other is multiplied, with one block barrier a chunk; the row stride is 4
// modulo 16 doubles, so that a fragment load (4 rows x 8 features) has no bank
// conflicts.  Where the groups are fewer than the warps, several warps take a
// group, each every rg-th k-step of the system (whatever the chunks' length, which
// follows the batch's widest system), added in order at the end.
//
// The finish factors the augmented system 8 columns at a time, the right-hand
// side as one more row (so that only the back substitution is left), trailing
// updates on the tensor path.
//
// Weighted systems of 306 to 8,192 rows and 153 features on the B200: 510 of
// them 3.7 ms with 8 x 8 FMA tiles, 1.63 ms here (0.15 us a row and SM, 72 % of
// the pipe's rate, and 64 us to finish a system); 4,096 of them 12.2 ms.
#include <algorithm>

#include "ridge.cuh"

namespace art {
namespace {

constexpr int kWideThreads = 512;
constexpr int kWideWarps = kWideThreads / 32;
constexpr int kMaxBlocks = 20;  // 8-feature blocks on the tensor path (160 columns)

struct WideLayout {
  int stride;  // doubles of a phi row: 4 modulo 16
  int xs;      // doubles of a staged row [x, 1, y, 0]
  size_t x[2], w[2], vec, phi, total;
};
__host__ __device__ inline size_t wd16(size_t v) { return (v + 15) & ~(size_t)15; }
__host__ __device__ inline WideLayout wide_layout(int pmax, int dmax, int chunk) {
  WideLayout L;
  const int pa = pmax + 1, cols = ((pa + 31) / 32) * 32;
  L.stride = cols + 4;
  if ((L.stride & 15) != 4) L.stride += 8;
  L.xs = ((dmax + 1) & ~1) + 4;
  size_t o = 0;
  for (int s = 0; s < 2; ++s) {
    L.x[s] = o; o = wd16(o + (size_t)chunk * L.xs * 8);
    L.w[s] = o; o = wd16(o + (size_t)chunk * 8);
  }
  L.vec = o; o = wd16(o + (size_t)4 * (pa + 2) * 8);
  // the packed Gram takes the phi buffers' place once the rows are through
  L.phi = o;
  const size_t b = (size_t)2 * chunk * L.stride * 8, g = (size_t)pa * (pa + 1) / 2 * 8;
  L.total = wd16(o + (b > g ? b : g));
  return L;
}

// Factor [G h; h^T .] (packed lower, rows 0 .. p, row p = h^T) = L L^T in
// place, eight columns a step: the diagonal block by warp 0 in registers, the
// panel by one thread a row, the trailing blocks by MMAs.  inv[j] = 1 / L_jj;
// row p ends as L^{-1} h.  Returns 0 or the 1-based failing pivot.
__device__ int chol_aug(double* A, int p, double* inv, int* s_fail) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, kq = lane & 3, mq = lane >> 2;
  // diagonal block j0 .. j0 + jb by warp 0: lane i holds row i of the block
  auto diagonal = [&](int j0, int jb) {
    double row[8];
#pragma unroll
    for (int c = 0; c < 8; ++c) row[c] = (lane < jb && c <= lane) ? A[pk(j0 + lane, j0 + c)] : 0.0;
    int fail = 0;
#pragma unroll
    for (int c = 0; c < 8; ++c) {
      const double dc = __shfl_sync(0xffffffffu, row[c], c);
      if (c < jb && !fail && (!(dc > 0.0) || !isfinite(dc))) fail = j0 + c + 1;
      const double r = rsqrt(dc);  // (past a failure or the block's end nothing is used)
      row[c] *= r;
      if (lane == c && c < jb) inv[j0 + c] = r;
#pragma unroll
      for (int k = c + 1; k < 8; ++k) row[k] = fma(-row[c], __shfl_sync(0xffffffffu, row[c], k), row[k]);
    }
    if (!fail && lane < jb) {
#pragma unroll
      for (int c = 0; c < 8; ++c)
        if (c <= lane) A[pk(j0 + lane, j0 + c)] = row[c];
    }
    if (lane == 0 && fail) *s_fail = fail;
  };
  // block (I, J) of the trailing matrix from row and column j1: A -= L L^T over
  // the panel's eight columns
  auto trailing = [&](int j0, int j1, int I, int J) {
    const int ra = j1 + 8 * I + mq, rb = j1 + 8 * J + mq;
    const double* ua = A + pk(min(ra, p), j0) + kq;
    const double* ub = A + pk(min(rb, p), j0) + kq;
    double c[2] = {0.0, 0.0};
    dmma_884(c, ua[0], ub[0]);
    dmma_884(c, ua[4], ub[4]);
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      const int col = j1 + 8 * J + 2 * kq + e;
      if (ra <= p && col <= ra && col < p) A[pk(ra, col)] -= c[e];
    }
  };
  if (tid == 0) *s_fail = 0;
  __syncthreads();
  if (warp == 0) diagonal(0, min(8, p));
  __syncthreads();
  for (int j0 = 0; j0 < p; j0 += 8) {
    const int jb = min(8, p - j0), j1 = j0 + jb;
    if (*s_fail) return *s_fail;
    for (int i = j1 + tid; i <= p; i += kWideThreads) {
      double* ai = A + pk(i, j0);
      double v[8];
#pragma unroll
      for (int c = 0; c < 8; ++c) v[c] = c < jb ? ai[c] : 0.0;
#pragma unroll
      for (int c = 0; c < 8; ++c) {
        if (c < jb) {
          const double* lc = A + pk(j0 + c, j0);
#pragma unroll
          for (int k = 0; k < 8; ++k)
            if (k < c) v[c] = fma(-v[k], lc[k], v[c]);
          v[c] *= inv[j0 + c];
          ai[c] = v[c];
        }
      }
    }
    __syncthreads();
    if (j1 >= p) break;
    // trailing blocks; warp 0 takes the next diagonal block first and factors
    // it while the others work on
    const int nbt = (p + 1 - j1 + 7) / 8, ntr = nbt * (nbt + 1) / 2;
    if (warp == 0) {
      trailing(j0, j1, 0, 0);
      __syncwarp();
      diagonal(j1, min(8, p - j1));
    } else {
      for (int t = warp; t < ntr; t += kWideWarps - 1) {
        const int I = tile_row(t);
        trailing(j0, j1, I, t - I * (I + 1) / 2);
      }
    }
    __syncthreads();
  }
  return 0;
}

// x = L^{-T} z by one warp, z = row p of the factor.
__device__ void back_solve(const double* A, int p, const double* inv, double* x) {
  const int lane = threadIdx.x & 31;
  constexpr int RPL = (ART_MAX_FEATURES + 31) / 32;
  double z[RPL], iv[RPL];
#pragma unroll
  for (int m = 0; m < RPL; ++m) {
    const int i = lane + 32 * m;
    z[m] = i < p ? A[pk(p, i)] : 0.0;
    iv[m] = i < p ? inv[i] : 0.0;
  }
#pragma unroll
  for (int mj = RPL - 1; mj >= 0; --mj) {
    for (int jl = min(31, p - 1 - 32 * mj); jl >= 0; --jl) {
      const int j = 32 * mj + jl;
      const double xj = __shfl_sync(0xffffffffu, z[mj] * iv[mj], jl);
      const double* row = A + pk(j, 0) + lane;
#pragma unroll
      for (int m = 0; m < RPL; ++m)
        if (m <= mj && lane + 32 * m < j) z[m] = fma(-row[32 * m], xj, z[m]);
      if (lane == jl) x[j] = xj;
    }
  }
  __syncwarp();
}

// Finish a system whose augmented Gram is in packed lower storage: trace-scaled
// ridge, Cholesky, solve, condition estimate and the auto-solver policy of
// solve_weighted_ridge (models.py:268-371).  All threads call it; `vec` holds
// four vectors of p + 2.
__device__ void finish_wide(const RidgeArgs& a, const RidgeLists& L, int k, const RidgeItem& it, double* G, int bad,
                            double* vec, int* s_fail, double* s_scalar, uint32_t info0) {
  const int tid = threadIdx.x, lane = tid & 31, p = it.p;
  const double nan = __longlong_as_double(0x7ff8000000000000ll), inf = __longlong_as_double(0x7ff0000000000000ll);
  double *z = vec, *v = vec + (p + 2), *sg = vec + 2 * (p + 2), *inv = vec + 3 * (p + 2);
  if (tid < 32) {  // lambda = ridge * trace(G) / p (models.py:209-215)
    double tr = 0.0;
    for (int i = lane; i < p; i += 32) tr += G[pk(i, i)];
    tr = warp_sum(tr);
    if (lane == 0) {
      s_scalar[0] = it.ridge * tr / p;
      L.lambda[k] = s_scalar[0];
    }
  }
  __syncthreads();
  const double lam = s_scalar[0];
  if (bad) {
    write_failed(a, k, p, (bad & 2) ? -1 : -2, lam, info0);
    __syncthreads();
    return;
  }
  auto to_qr = [&](uint32_t info, double cond) {
    if (tid == 0) {
      if (a.ridge_eff) a.ridge_eff[k] = lam;
      if (a.cond) a.cond[k] = cond;
      if (a.info) a.info[k] = info;
      a.status[k] = 0;
      push_list(L, a.K, CLS_QR, k);
    }
    __syncthreads();
  };
  if (a.solver == ART_SOLVER_QR || a.solver == ART_SOLVER_SVD) {  // explicit QR: no normal equations solve
    to_qr(info0 | (a.solver == ART_SOLVER_SVD ? 0u : ART_INFO_QR_FALLBACK), nan);
    return;
  }
  for (int i = tid; i < p; i += kWideThreads) G[pk(i, i)] += lam;
  __syncthreads();
  const bool want_cond = (a.cond != nullptr) || (a.solver == ART_SOLVER_AUTO);
  if (want_cond && tid < 32) {
    const double an = warp_sym_norm1(G, p);
    if (tid == 0) s_scalar[1] = an;
  }
  __syncthreads();
  const int fail = chol_aug(G, p, inv, s_fail);
  if (fail) {
    if (a.solver == ART_SOLVER_AUTO) {
      to_qr(info0 | ART_INFO_QR_FALLBACK | ART_INFO_CHOLESKY_FAILED, inf);
      return;
    }
    write_failed(a, k, p, fail, lam, info0);
    __syncthreads();
    return;
  }
  if (tid < 32) {
    back_solve(G, p, inv, z);
    if (want_cond) {
      const double est = warp_inv_norm1_estimate<double>(G, p, v, sg);
      if (tid == 0) {
        const double an = s_scalar[1];
        s_scalar[2] = (est > 0.0 && isfinite(est) && an > 0.0) ? 1.0 / (an * est) : 0.0;
      }
    }
  }
  __syncthreads();
  uint32_t info = info0;
  double cond = nan;
  if (want_cond) {
    double rcond = s_scalar[2];
    if (rcond > 0.0 && isfinite(rcond)) {
      cond = sqrt(1.0 / fmin(rcond, 1.0));
    } else {
      rcond = 0.0;
      cond = inf;
      info |= ART_INFO_COND_FAILED;
    }
    if (a.solver == ART_SOLVER_AUTO && rcond < a.rcond_threshold) {
      to_qr(info | ART_INFO_QR_FALLBACK | ART_INFO_RCOND_BELOW, cond);
      return;
    }
  }
  int nonfinite = 0;
  for (int i = tid; i < p; i += kWideThreads) {
    const double b = z[i];
    nonfinite |= !isfinite(b);
    a.beta[(int64_t)k * a.beta_stride + i] = b;
  }
  nonfinite = __syncthreads_or(nonfinite);
  if (tid == 0) {
    a.status[k] = nonfinite ? -3 : 0;
    if (a.ridge_eff) a.ridge_eff[k] = lam;
    if (a.cond) a.cond[k] = cond;
    if (a.info) a.info[k] = info;
  }
  __syncthreads();
}

template <int CHUNK>
__global__ void __launch_bounds__(kWideThreads, 1) ridge_wide_kernel(RidgeArgs a, RidgeLists L, int cls, int pcap) {
  extern __shared__ __align__(128) unsigned char smem[];
  __shared__ int s_item, s_fail;
  __shared__ double s_scalar[4];
  const WideLayout lay = wide_layout(pcap, a.dmax, CHUNK);
  double* vec = (double*)(smem + lay.vec);
  double* phi = (double*)(smem + lay.phi);
  double* G = phi;
  const int S = lay.stride, XS = lay.xs;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, kq = lane & 3, mq = lane >> 2;
  const int count = L.count[cls];
  for (;;) {
    if (tid == 0) s_item = atomicAdd(&L.cursor[cls], 1);
    __syncthreads();
    const int item = s_item;
    __syncthreads();
    if (item >= count) break;
    const int k = L.list[(int64_t)cls * a.K + item];
    const RidgeItem it = load_item(a, k);
    const int p = it.p, pa = p + 1, d = it.d;
    const int nb = min((pa + 7) / 8, kMaxBlocks);
    const bool extra = pa > 8 * kMaxBlocks;  // p = 160: the right-hand side's row apart, by FMAs
    // the warp's group of 4 x 4 blocks (off-diagonal groups first, so that the
    // schedulers' loads come out even) and its share of the k-steps
    const int sr = (nb + 3) / 4, noff = sr * (sr - 1) / 2, ngrp = noff + sr;
    const int rg = kWideWarps / ngrp, grp = warp % ngrp, share = warp / ngrp;
    bool mine = share < rg;
    int gi, gj;
    if (grp < noff) {
      gi = tile_row(grp) + 1;
      gj = grp - (gi - 1) * gi / 2;
    } else {
      gi = gj = grp - noff;
    }
    // Five group rows (p = 128 to 160): ten full groups and five diagonal ones
    // would leave one scheduler 58 MMAs a k-step of 210.  Nine of the full
    // groups give up their last block row; each diagonal warp takes one such
    // strip, the sixteenth warp four: 54 at most.
    enum { kFull, kDiag, kThree, kDiagStrip, kStrips } role = gi == gj ? kDiag : kFull;
    int strip_i[4] = {0, 0, 0, 0}, strip_j[4] = {0, 0, 0, 0};  // first columns of a strip's row block and group
    if (sr == 5) {
      auto strip = [&](int slot, int group) {
        const int i = tile_row(group) + 1, j = group - (i - 1) * i / 2;
        strip_i[slot] = 32 * i + 24;
        strip_j[slot] = 32 * j;
      };
      if (warp < 9) {
        role = kThree;
      } else if (warp >= 10 && warp < 15) {
        role = kDiagStrip;
        strip(0, warp - 10);
      } else if (warp == 15) {
        role = kStrips;
        mine = true;
        for (int q = 0; q < 4; ++q) strip(q, 5 + q);
      }
    }
    const int first = sr == 5 ? 0 : share;  // (a group has one warp then)
    double c[4][4][2];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) c[i][j][0] = c[i][j][1] = 0.0;
    double hx = 0.0;  // extra: h of feature tid
    int bad = 0;
    const int64_t nchunks = (it.n + CHUNK - 1) / CHUNK;
    // chunk ch's rows to stage st: x in 16-byte pairs where every row starts on
    // one, else as doubles; y and w beside them
    const double* xg = a.x + it.xoff;
    const bool pairs = (d & 1) == 0 && ((uintptr_t)xg & 15) == 0;
    const int cw = pairs ? 2 : 1, cpr = d / cw;
    auto issue = [&](int64_t ch, int st) {
      const int64_t rr = ch * CHUNK;
      const int rows = (int)min((int64_t)CHUNK, it.n - rr);
      const uint32_t dst = smem_u32(smem + lay.x[st]);
      for (int e = tid; e < rows * cpr; e += kWideThreads) {
        const int r = e / cpr, c2 = e - r * cpr;
        const double* sp = xg + (rr + r) * d + c2 * cw;
        const uint32_t dp = dst + (uint32_t)(r * XS + c2 * cw) * 8u;
        if (pairs) cp_async16(dp, sp);
        else cp_async8(dp, sp);
      }
      if (tid < rows) cp_async8(dst + (uint32_t)(tid * XS + d + 1) * 8u, a.y + it.r0 + rr + tid);
      else if (a.w && tid >= 128 && tid < 128 + rows)
        cp_async8(smem_u32(smem + lay.w[st]) + (uint32_t)(tid - 128) * 8u, a.w + it.r0 + rr + (tid - 128));
      cp_async_commit();
    };
    if (nchunks > 0) issue(0, 0);
    if (tid < 2 * CHUNK) {  // the constant and the zero of every staged row
      double* xr = (double*)(smem + lay.x[tid / CHUNK]) + (tid % CHUNK) * XS;
      xr[d] = 1.0;
      xr[d + 2] = 0.0;
    }
    uint32_t fab[5];  // this lane's features in the expansion: two columns of the staged row
#pragma unroll
    for (int m = 0; m < 5; ++m) {
      const int f = lane + 32 * m;
      int u = d + 2, v = d;
      if (f < p) {
        feature_factors(d, it.kind, f, u, v);
        if (u < 0) u = d;
        if (v < 0) v = d;
      } else if (f == p) {
        u = d + 1;
      }
      fab[m] = (uint32_t)u | ((uint32_t)v << 16);
    }
    cp_async_wait0();
    __syncthreads();
    // rows a warp expands: consecutive ones where the count divides evenly
    const bool five = sr == 5 && CHUNK >= 32;
    int g0 = warp, g1 = CHUNK, gs = kWideWarps;
    if (five) {
      constexpr int F = CHUNK / 32;
      g0 = F * 2 * warp;
      g1 = g0 + F * 2;
      gs = 1;
    }
    // this warp's first k-step in the chunk, so that it takes every rg-th of the system
    int s0 = first;
    const int back = (CHUNK / 4) % rg;
    for (int64_t ch = 0; ch < nchunks; ++ch) {
      const int st = (int)(ch & 1);
      const int rows = (int)min((int64_t)CHUNK, it.n - ch * CHUNK), rows4 = (rows + 3) & ~3;
      if (ch + 1 < nchunks) issue(ch + 1, st ^ 1);
      const double* xs = (const double*)(smem + lay.x[st]);
      const double* ws = (const double*)(smem + lay.w[st]);
      double* buf = phi + (size_t)st * CHUNK * S;
      double sql = 0.0;  // lane l: sqrt(q) of the warp's l-th row
      {
        const int r = g0 + gs * lane;
        if (r < g1 && r < rows) {
          const double wv = a.w ? ws[r] : 1.0;
          if (!(wv >= 0.0) || !isfinite(wv)) bad |= 2;
          sql = sqrt(fmax(wv, a.weight_floor));
        }
      }
      int q = 0;
      for (int r = g0; r < min(g1, rows4); r += gs, ++q) {
        const double sq = __shfl_sync(0xffffffffu, sql, q);
        const double* xr = xs + min(r, rows - 1) * XS;  // rows past the end: weight zero
        double* pr = buf + r * S;
#pragma unroll
        for (int m = 0; m < 5; ++m)
          if (m < sr) pr[lane + 32 * m] = sq * (xr[fab[m] & 0xffffu] * xr[fab[m] >> 16]);
        if (extra && lane == 0) pr[8 * kMaxBlocks] = sq * xr[d + 1];
      }
      // phi of this chunk and the rows of the next are in place, and every warp
      // is done with this stage's rows and the MMAs of the chunk before
      cp_async_wait0();
      __syncthreads();
      if (mine) {
        // loops without a condition on any MMA: diagonal groups form their lower
        // blocks, the others all sixteen (columns past psi are zeros), or with
        // five group rows three block rows of four
        const double* ph = buf + (4 * s0 + kq) * S + mq;
        const double *pi = ph + 32 * gi, *pj = ph + 32 * gj;
        const int step = 4 * rg * S;
        auto loop = [&](auto f) {
#pragma unroll 2
          for (int k0 = 4 * s0; k0 < rows4; k0 += 4 * rg) {
            f();
            ph += step;
            pi += step;
            pj += step;
          }
        };
        if (role == kDiag) {
          loop([&] {
            double v[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) v[i] = pi[8 * i];
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
              for (int j = 0; j <= i; ++j) dmma_884(c[i][j], v[i], v[j]);
          });
        } else if (role == kFull) {
          loop([&] {
            double av[4], bv[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              av[i] = pi[8 * i];
              bv[i] = pj[8 * i];
            }
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
              for (int j = 0; j < 4; ++j) dmma_884(c[i][j], av[i], bv[j]);
          });
        } else if (role == kThree) {
          loop([&] {
            double av[3], bv[4];
#pragma unroll
            for (int i = 0; i < 3; ++i) av[i] = pi[8 * i];
#pragma unroll
            for (int i = 0; i < 4; ++i) bv[i] = pj[8 * i];
#pragma unroll
            for (int i = 0; i < 3; ++i)
#pragma unroll
              for (int j = 0; j < 4; ++j) dmma_884(c[i][j], av[i], bv[j]);
          });
        } else if (role == kDiagStrip) {
          loop([&] {
            double v[4], bv[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              v[i] = pi[8 * i];
              bv[i] = ph[strip_j[0] + 8 * i];
            }
            const double as = ph[strip_i[0]];
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
              for (int j = 0; j <= i; ++j) dmma_884(c[i][j], v[i], v[j]);
            dmma_884(c[0][1], as, bv[0]);
            dmma_884(c[0][2], as, bv[1]);
            dmma_884(c[0][3], as, bv[2]);
            dmma_884(c[1][2], as, bv[3]);
          });
        } else {
          loop([&] {
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              const double as = ph[strip_i[i]];
#pragma unroll
              for (int j = 0; j < 4; ++j) dmma_884(c[i][j], as, ph[strip_j[i] + 8 * j]);
            }
          });
        }
      }
      s0 -= back;
      if (s0 < 0) s0 += rg;
      if (extra && tid < p)
        for (int r = 0; r < rows; ++r) hx = fma(buf[r * S + tid], buf[r * S + 8 * kMaxBlocks], hx);
    }
    __syncthreads();  // the Gram takes the place of phi
    auto put = [&](int row0, int col0, const double (&v)[2], bool add) {  // an 8 x 8 block
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const int r = row0 + mq, cc = col0 + 2 * kq + e;
        if (r < min(pa, 8 * kMaxBlocks) && cc <= r) {
          double* g = &G[pk(r, cc)];
          *g = add ? *g + v[e] : v[e];
        }
      }
    };
    for (int s = 0; s < rg; ++s) {
      if (mine && first == s) {
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            if (role == kStrips) put(strip_i[i], strip_j[i] + 8 * j, c[i][j], false);
            else if (role == kFull || (role == kThree && i < 3) || ((role == kDiag || role == kDiagStrip) && j <= i))
              put(32 * gi + 8 * i, 32 * gj + 8 * j, c[i][j], s > 0);
          }
        if (role == kDiagStrip) {
          put(strip_i[0], strip_j[0], c[0][1], false);
          put(strip_i[0], strip_j[0] + 8, c[0][2], false);
          put(strip_i[0], strip_j[0] + 16, c[0][3], false);
          put(strip_i[0], strip_j[0] + 24, c[1][2], false);
        }
      }
      __syncthreads();
    }
    if (extra && tid < p) G[pk(p, tid)] = hx;
    __syncthreads();
    // a non-finite input leaves a non-finite sum (0 * inf and NaN included), so
    // the rows are looked at only where the Gram has one
    int odd = 0;
    for (int e = tid; e < p * (p + 3) / 2; e += kWideThreads) odd |= isfinite(G[e]) ? 0 : 1;
    if (__syncthreads_or(odd)) {
      for (int64_t e = tid; e < it.n * d; e += kWideThreads) bad |= isfinite(a.x[it.xoff + e]) ? 0 : 1;
      for (int64_t e = tid; e < it.n; e += kWideThreads) bad |= isfinite(a.y[it.r0 + e]) ? 0 : 1;
    }
    const int bw = __syncthreads_or(bad & 2), bx = __syncthreads_or(bad & 1);
    finish_wide(a, L, k, it, G, (bw ? 2 : 0) | (bx ? 1 : 0), vec, &s_fail, s_scalar,
                cls == CLS_RESOLVE ? ART_INFO_FP64_RESOLVE : 0u);
  }
}

}  // namespace

int launch_ridge_wide(const RidgeArgs& a, const RidgeLists& L, int cls, cudaStream_t s) {
  // the longest chunk whose buffers fit
  const int chunk = wide_layout(a.pmax, a.dmax, 64).total <= 227 * 1024 ? 64 : (a.dmax > 64 ? 16 : 32);
  auto kern = chunk == 64 ? ridge_wide_kernel<64> : (chunk == 32 ? ridge_wide_kernel<32> : ridge_wide_kernel<16>);
  const size_t smem = wide_layout(a.pmax, a.dmax, chunk).total;
  const char* name = cls == CLS_RESOLVE ? "ridge_wide resolve" : "ridge_wide";
  if (smem > 227 * 1024 ||
      cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess) {
    cudaGetLastError();
    set_error("%s: cannot reserve %zu bytes of shared memory", name, smem);
    return ART_E_UNSUPPORTED;
  }
  const int occ = resident_ctas((const void*)kern, kWideThreads, smem);
  const int64_t grid = std::max<int64_t>(1, std::min<int64_t>((int64_t)device_sm_count() * occ, a.K));
  prof_begin(name, s);
  kern<<<(unsigned)grid, kWideThreads, smem, s>>>(a, L, cls, a.pmax);
  prof_end(s);
  count_launch();
  return check_launch(name);
}

}  // namespace art
