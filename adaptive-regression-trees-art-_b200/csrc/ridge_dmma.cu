// ridge_dmma.cu -- FP64 weighted ridge for systems of p + 1 <= 48, Grams on
// the FP64 tensor path (mma.sync m8n8k4 f64; tcgen05 has no FP64 kind).
//
// What bounds it: the FP64 pipe.  One 8 x 8 x 4 MMA takes 4 SM cycles whether
// it is issued as m8n8k4 or as a larger shape (measured: 127 flop/clk/SM from
// 8 warps on, DFMA the same), so the row loop is written to keep that pipe
// fed and nothing else on it: every warp works alone on its own rows with all
// of its system's lower 8 x 8 Gram blocks in registers, so there is no block
// barrier, no feature tile in shared memory (a warp uses each feature of a
// row exactly once as a fragment, formed from x as it is loaded) and no
// square root of the weights.
//
// Per tile of up to 32 rows, the lanes copy x, y and w with cp.async (16 bytes
// a copy where the rows allow it) into rows [x, 1, y, 0] of a stride that is 4
// or 12 modulo 16 doubles, so that the fragment loads (4 rows x 8 features) do
// not collide in the banks; the next tile is in flight while G += (q psi)^T psi
// runs over this one, psi = [phi(x); y].  Nothing is staged twice: a first
// form that bulk-copied the rows and re-laid them out spent ten instructions
// a MMA on that and kept the FP64 pipe 46 % busy.
//
// Work is cut at fixed unit boundaries (ridge_unit_rows, from the system's
// own n and width): a system's Gram is the sum of its units' Grams in unit
// order, whoever forms them.  The plan hands a system that costs more than a
// warp's share of the whole batch to many warps (runs of units, each unit's
// Gram written to the workspace pool and added by ridge_split_finish); every
// other system is one warp's work, which adds the units as it goes.  So the
// split follows the batch, and the results do not.
//
// Measured on the B200 against one warp (p + 1 <= 24) or one CTA a system:
// 301 nodes of 450 to 400,000 rows, 2 to 45 features 96.1 -> 0.92 ms; one node
// of 4,096 rows 182 -> 50 us; 511 weighted systems of 306 to 8,192 rows and 45
// features 0.85 -> 0.16 ms (FP64 pipe 65 % busy: the rest is the products that
// form the fragments, which share it, and the moves around them).
#include <algorithm>
#include <atomic>

#include "ridge.cuh"

namespace art {
namespace {

constexpr int kDmThreads = 128;  // 4 independent warps per CTA
constexpr int kDmWarps = kDmThreads / 32;

// Doubles of a row tile (two per warp).  The wider class keeps them smaller
// so that three CTAs (12 warps) share an SM beside its Grams.
template <int MAXNB> struct DmTraits {
  static constexpr int kPad = 8 * MAXNB;
  static constexpr int kTile = MAXNB <= 3 ? 640 : 512;
  static constexpr int kE = kPad * (kPad + 1) / 2;
};
template <int MAXNB> struct DmLayout {
  using T = DmTraits<MAXNB>;
  static constexpr size_t kT = 0;                                  // row tiles
  static constexpr size_t kQ = kT + 2 * (size_t)T::kTile * 8;      // weights of the tiles' rows
  static constexpr size_t kG = kQ + 2 * 32 * 8;                    // packed augmented Gram
  static constexpr size_t kPerWarp = (kG + (size_t)T::kE * 8 + 127) & ~(size_t)127;
  // the finish step's three vectors reuse the row tiles
  static_assert(3 * (T::kPad + 1) * 8 <= kQ, "finish vectors");
};
constexpr int kQuadStride = 12;  // row stride of the quadratic kinds (d <= 8)

__device__ void warp_write_failed(const RidgeArgs& a, int k, int p, int32_t status, double lam,
                                  uint32_t info) {
  const int lane = threadIdx.x & 31;
  const double nan = __longlong_as_double(0x7ff8000000000000ll);
  for (int i = lane; i < p; i += 32) a.beta[(int64_t)k * a.beta_stride + i] = nan;
  if (lane == 0) {
    a.status[k] = status;
    if (a.ridge_eff) a.ridge_eff[k] = lam;
    if (a.cond) a.cond[k] = nan;
    if (a.info) a.info[k] = info;
  }
}

// The finish step of the CTA form (finish_fp64), by one warp.  `vec` holds
// three vectors of stride vs.  RPL: rows per lane (p + 1 <= 32 RPL).
template <int RPL>
__device__ void warp_finish(const RidgeArgs& a, const RidgeLists& L, int k, int p, double ridge,
                            double* G, int bad, double* vec, int vs) {
  const int lane = threadIdx.x & 31;
  const double nan = __longlong_as_double(0x7ff8000000000000ll);
  const double inf = __longlong_as_double(0x7ff0000000000000ll);
  double tr = 0.0;
  for (int i = lane; i < p; i += 32) tr += G[pk(i, i)];
  tr = __shfl_sync(0xffffffffu, warp_sum(tr), 0);
  const double lam = ridge * tr / p;
  if (lane == 0) L.lambda[k] = lam;
  if (bad) {
    warp_write_failed(a, k, p, (bad & 2) ? -1 : -2, lam, 0u);
    return;
  }
  if (a.solver == ART_SOLVER_QR || a.solver == ART_SOLVER_SVD) {
    if (lane == 0) {
      if (a.ridge_eff) a.ridge_eff[k] = lam;
      if (a.cond) a.cond[k] = nan;
      if (a.info) a.info[k] = a.solver == ART_SOLVER_SVD ? 0u : ART_INFO_QR_FALLBACK;
      a.status[k] = 0;
      push_list(L, a.K, CLS_QR, k);
    }
    return;
  }
  __syncwarp();
  for (int i = lane; i < p; i += 32) G[pk(i, i)] += lam;
  __syncwarp();
  const bool want_cond = (a.cond != nullptr) || (a.solver == ART_SOLVER_AUTO);
  const double an = want_cond ? warp_sym_norm1(G, p) : 0.0;
  double* z = vec;
  double* v = vec + vs;
  double* sg = vec + 2 * vs;
  const int fail = warp_chol_solve<RPL>(G, p, z);
  if (fail) {
    if (a.solver == ART_SOLVER_AUTO) {
      if (lane == 0) {
        if (a.ridge_eff) a.ridge_eff[k] = lam;
        if (a.cond) a.cond[k] = inf;
        if (a.info) a.info[k] = ART_INFO_QR_FALLBACK | ART_INFO_CHOLESKY_FAILED;
        a.status[k] = 0;
        push_list(L, a.K, CLS_QR, k);
      }
      return;
    }
    warp_write_failed(a, k, p, fail, lam, 0u);
    return;
  }
  uint32_t info = 0;
  double cond = nan;
  if (want_cond) {
    const double est = warp_inv_norm1_estimate<double>(G, p, v, sg);
    double rcond = (est > 0.0 && isfinite(est) && an > 0.0) ? 1.0 / (an * est) : 0.0;
    if (rcond > 0.0 && isfinite(rcond)) {
      cond = sqrt(1.0 / fmin(rcond, 1.0));
    } else {
      rcond = 0.0;
      cond = inf;
      info |= ART_INFO_COND_FAILED;
    }
    if (a.solver == ART_SOLVER_AUTO && rcond < a.rcond_threshold) {
      if (lane == 0) {
        if (a.ridge_eff) a.ridge_eff[k] = lam;
        if (a.cond) a.cond[k] = cond;
        if (a.info) a.info[k] = info | ART_INFO_QR_FALLBACK | ART_INFO_RCOND_BELOW;
        a.status[k] = 0;
        push_list(L, a.K, CLS_QR, k);
      }
      return;
    }
  }
  __syncwarp();
  int nonfinite = 0;
  for (int i = lane; i < p; i += 32) {
    const double b = z[i];
    nonfinite |= !isfinite(b);
    a.beta[(int64_t)k * a.beta_stride + i] = b;
  }
  nonfinite = __any_sync(0xffffffffu, nonfinite);
  if (lane == 0) {
    a.status[k] = nonfinite ? -3 : 0;
    if (a.ridge_eff) a.ridge_eff[k] = lam;
    if (a.cond) a.cond[k] = cond;
    if (a.info) a.info[k] = info;
  }
}

// One warp's work on units [u0, u0 + nu) of system k.  `part` (the system's
// pool slots) receives each unit's Gram of a split system; without it the
// units' sum is left in the warp's G, `add`ed to what it holds.  QUAD: the
// quadratic kinds (two factors a feature, fixed row stride).  Returns the
// input-check bits.
template <int MAXNB, int NB, bool QUAD>
__device__ int gram_units(const RidgeArgs& a, const RidgeItem& it, unsigned char* base, int u0, int nu, double* part,
                          bool add) {
  using T = DmTraits<MAXNB>;
  using Lay = DmLayout<MAXNB>;
  constexpr int NBLK = NB * (NB + 1) / 2;
  const int lane = threadIdx.x & 31, kq = lane & 3, mq = lane >> 2;
  double* X0 = (double*)(base + Lay::kT);
  double* G = (double*)(base + Lay::kG);
  const int d = it.d, p = it.p, pa = p + 1;
  const int E = pa * (pa + 1) / 2;
  // row stride: at least d + 3, 4 or 12 modulo 16 doubles
  const int rs = QUAD ? kQuadStride : ((d + 6) / 8) * 8 + 4;
  const int RS = min(32, (T::kTile / rs) & ~3);
  double* Q0 = (double*)(base + Lay::kQ);
  const uint32_t xb = smem_u32(X0), qb = smem_u32(Q0);
  // this lane's feature of each 8-column block: the columns of X it is a
  // product of (padding: the zero column)
  int fa[NB], fb[QUAD ? NB : 1];
#pragma unroll
  for (int I = 0; I < NB; ++I) {
    const int f = 8 * I + mq;
    int ia = d + 2, ib = d;
    if (f < p) {
      feature_factors(d, it.kind, f, ia, ib);
      if (ia < 0) ia = d;
      if (ib < 0) ib = d;
    } else if (f == p) {
      ia = d + 1;  // y
    }
    fa[I] = kq * rs + ia;
    if constexpr (QUAD) fb[I] = kq * rs + ib;
  }
#pragma unroll
  for (int h = 0; h < 2; ++h)
    if (lane < RS) {
      X0[h * T::kTile + lane * rs + d] = 1.0;
      X0[h * T::kTile + lane * rs + d + 2] = 0.0;
    }
  double c[NBLK][2];
#pragma unroll
  for (int q = 0; q < NBLK; ++q) c[q][0] = c[q][1] = 0.0;
  const int64_t U = ridge_unit_rows(it.n);
  const int64_t row_end = min(it.n, (int64_t)(u0 + nu) * U);
  // x rows as 16-byte pairs where every row starts on one, else as doubles
  const double* xg = a.x + it.xoff;
  const bool pairs = (d & 1) == 0 && ((uintptr_t)xg & 15) == 0;
  const int cw = pairs ? 2 : 1, cpr = d / cw;              // doubles per copy, copies per row
  const int step_r = 32 / cpr, step_c = 32 - step_r * cpr;  // 32 copies further on
  const int lr0 = lane / cpr, lc0 = lane - lr0 * cpr;
  // rows [r, r + rows) to tile h, zero rows up to the next multiple of four
  auto issue = [&](int64_t r, int rows, int h) {
    const uint32_t dst = xb + (uint32_t)h * (T::kTile * 8);
    const int rows4 = (rows + 3) & ~3;
    const double* src = xg + r * d;
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
    if (lane < rows4) {
      const bool live = lane < rows;
      cp_async8(dst + (uint32_t)(lane * rs + d + 1) * 8u, a.y + it.r0 + r + (live ? lane : 0), live);
      if (a.w) cp_async8(qb + (uint32_t)(h * 32 + lane) * 8u, a.w + it.r0 + r + (live ? lane : 0), live);
    }
    cp_async_commit();
  };
  int bad = 0;
  int unit = u0, h = 0;
  int64_t r = (int64_t)u0 * U, unit_end = min(row_end, r + U);
  int rows = (int)min((int64_t)RS, unit_end - r);
  __syncwarp();
  if (rows > 0) issue(r, rows, 0);
  while (r < row_end) {
    const int64_t rn = r + rows;
    const int64_t next_end = rn < unit_end ? unit_end : min(row_end, rn + U);
    const int next_rows = (int)min((int64_t)RS, next_end - rn);
    __syncwarp();  // every lane is done with the other tile
    if (next_rows > 0) issue(rn, next_rows, h ^ 1);
    else cp_async_commit();
    cp_async_wait1();
    const double* xt = X0 + h * T::kTile;
    double* qt = Q0 + h * 32;
    const int rows4 = (rows + 3) & ~3;
    if (lane < rows4) {  // this lane's own copy: visible to it since the wait
      const double wv = a.w ? qt[lane] : 1.0;
      if (lane < rows && (!(wv >= 0.0) || !isfinite(wv))) bad |= 2;
      qt[lane] = lane < rows ? fmax(wv, a.weight_floor) : 0.0;
    }
    __syncwarp();
    auto step = [&](const double* xk, double q) {
      double v[NB];
#pragma unroll
      for (int I = 0; I < NB; ++I) {
        v[I] = xk[fa[I]];
        if constexpr (QUAD) v[I] *= xk[fb[I]];
      }
#pragma unroll
      for (int I = 0; I < NB; ++I) {
        const double av = q * v[I];
#pragma unroll
        for (int J = 0; J <= I; ++J) dmma_884(c[I * (I + 1) / 2 + J], av, v[J]);
      }
    };
    if (QUAD && rows4 == 32) {  // full tiles: addresses by immediate offsets
#pragma unroll
      for (int k = 0; k < 8; ++k) step(xt + k * (4 * kQuadStride), qt[4 * k + kq]);
    } else {
      for (int k0 = 0; k0 < rows4; k0 += 4) step(xt + k0 * rs, qt[k0 + kq]);
    }
    r = rn;
    rows = next_rows;
    h ^= 1;
    if (r >= unit_end) {  // the unit is done: its Gram to the pool, or onto the running sum
      // a non-finite input leaves a non-finite sum (0 * inf and NaN included),
      // so the rows are looked at only where the unit's Gram has one
      bool odd = false;
#pragma unroll
      for (int q = 0; q < NBLK; ++q) odd |= !isfinite(c[q][0]) || !isfinite(c[q][1]);
      if (__any_sync(0xffffffffu, odd)) {
        const int64_t ra = (int64_t)unit * U;
        for (int64_t e = ra * d + lane; e < unit_end * d; e += 32) bad |= isfinite(xg[e]) ? 0 : 1;
        for (int64_t e = ra + lane; e < unit_end; e += 32) bad |= isfinite(a.y[it.r0 + e]) ? 0 : 1;
      }
      double* dst = part ? part + (size_t)unit * E : G;
      const bool first = part || (unit == u0 && !add);
#pragma unroll
      for (int I = 0; I < NB; ++I)
#pragma unroll
        for (int J = 0; J <= I; ++J)
#pragma unroll
          for (int t = 0; t < 2; ++t) {
            const int i = 8 * I + mq, j = 8 * J + 2 * kq + t;
            double& cv = c[I * (I + 1) / 2 + J][t];
            if (i < pa && j <= i) dst[pk(i, j)] = first ? cv : dst[pk(i, j)] + cv;
            cv = 0.0;
          }
      ++unit;
      unit_end = next_end;
    }
  }
  cp_async_wait0();
  if (!part && it.n == 0)
    for (int e = lane; e < E; e += 32) G[e] = 0.0;
  __syncwarp();
  return __reduce_or_sync(0xffffffffu, bad);
}

// Several warps' Grams of consecutive units added in unit order, by all threads
// of the CTA: warp 0's holds the units before, and its own.
template <int MAXNB>
__device__ void add_grams(unsigned char* smem, int E, int n) {
  using Lay = DmLayout<MAXNB>;
  __syncthreads();
  for (int e = threadIdx.x; e < E; e += kDmThreads) {
    double* g = (double*)(smem + Lay::kG) + e;
    double t = *g;
    for (int w = 1; w < n; ++w) t += g[w * (Lay::kPerWarp / 8)];
    *g = t;
  }
  __syncthreads();
}

// MAXNB = 3: p + 1 <= 24 at 16 warps per SM; 6: p + 1 <= 48 at 12 warps.
//
// A wide-class system that costs more than a warp's share, but has no room in
// the pool (no workspace for one, or a batch too long to be split), is the
// whole CTA's: its warps take every fourth unit.  Marked entries stand at the
// head of the list, largest first, so a CTA takes entries one at a time until
// it meets an unmarked one; warps that meet a marked one later walk it alone.
// One system of 100,000 rows and 47 features: 13.25 ms by one warp, 3.5 ms here;
// one of 200,000 among 17,000 of 60 rows: 26.3 ms and 7.1.
template <int MAXNB>
__global__ void __launch_bounds__(kDmThreads, MAXNB == 3 ? 4 : 3) ridge_dmma_kernel(RidgeArgs a, RidgeLists L, int cls) {
  extern __shared__ __align__(128) unsigned char smem[];
  using Lay = DmLayout<MAXNB>;
  __shared__ int s_q;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  unsigned char* base = smem + (size_t)warp * Lay::kPerWarp;
  const int sc = cls == CLS_WARP ? 0 : 1;
  const int count = L.count[cls], nsplit = min(L.nitems[sc], L.item_cap);
  bool together = MAXNB > 3 && *L.nshared > 0;
  for (;;) {
    int q = 0;
    bool shared = false;
    if (MAXNB > 3 && together) {
      __syncthreads();
      if (threadIdx.x == 0) s_q = atomicAdd(&L.cursor[cls], 1);
      __syncthreads();
      q = s_q;
      if (q >= nsplit + count) break;
      const int k = q < count ? L.list[(int64_t)cls * a.K + q] : -1;
      shared = k < -1;
      if (q < count && k == -1) continue;
      if (!shared) {
        together = false;
        if (warp != 0) continue;
      }
    } else {
      if (lane == 0) q = atomicAdd(&L.cursor[cls], 1);
      q = __shfl_sync(0xffffffffu, q, 0);
      if (q >= nsplit + count) break;
    }
    int k, u0 = 0, nu = 1 << 30, rec = -1;
    double* part = nullptr;
    if (q >= count) {  // a run of units of a split system: a quarter of a share each, so they come last
      const int4 e = L.items[(int64_t)sc * L.item_cap + (q - count)];
      if (e.x < 0) continue;
      rec = e.x;
      u0 = e.y;
      nu = e.z;
      k = L.recs[rec].k;
      part = L.pool + L.recs[rec].base;
    } else {
      k = L.list[(int64_t)cls * a.K + q];
      if (k == -1) continue;  // split
      if (k < 0) k = -2 - k;  // marked
    }
    const RidgeItem it = load_item(a, k);
    const int U = (int)ridge_unit_rows(it.n), units = (int)((it.n + U - 1) / U);
    nu = min(nu, units);
    const int nb = (it.p + 1 + 7) / 8;
    // (a nonlinear kind has its x among the features of the first two blocks:
    // p <= 47 means d <= 8)
    const bool quad = it.kind == ART_FEATURES_POLY2 || it.kind == ART_FEATURES_POLY2_NOBIAS;
    const int rounds = shared ? (units + kDmWarps - 1) / kDmWarps : 1;
    int bad = 0;
#pragma unroll 1
    for (int r = 0; r < rounds; ++r) {
      bool add = false;
      if (shared) {
        u0 = kDmWarps * r + warp;
        nu = 1;
        add = warp == 0 && r > 0;
      }
      int b;
      if constexpr (MAXNB == 3) {
        if (nb == 1) b = quad ? gram_units<3, 1, true>(a, it, base, u0, nu, part, add) : gram_units<3, 1, false>(a, it, base, u0, nu, part, add);
        else if (nb == 2) b = quad ? gram_units<3, 2, true>(a, it, base, u0, nu, part, add) : gram_units<3, 2, false>(a, it, base, u0, nu, part, add);
        else b = quad ? gram_units<3, 3, true>(a, it, base, u0, nu, part, add) : gram_units<3, 3, false>(a, it, base, u0, nu, part, add);
      } else {
        if (nb <= 4) b = quad ? gram_units<6, 4, true>(a, it, base, u0, nu, part, add) : gram_units<6, 4, false>(a, it, base, u0, nu, part, add);
        else if (nb == 5) b = quad ? gram_units<6, 5, true>(a, it, base, u0, nu, part, add) : gram_units<6, 5, false>(a, it, base, u0, nu, part, add);
        else b = quad ? gram_units<6, 6, true>(a, it, base, u0, nu, part, add) : gram_units<6, 6, false>(a, it, base, u0, nu, part, add);
      }
      bad |= b;
      if (shared) add_grams<MAXNB>(smem, (it.p + 1) * (it.p + 2) / 2, min(kDmWarps, units - kDmWarps * r));
    }
    if (rec >= 0) {
      if (bad && lane == 0) atomicOr(&L.recs[rec].bad, bad);
      continue;
    }
    if (shared) {
      const int bw = __syncthreads_or(bad & 2), bx = __syncthreads_or(bad & 1);
      if (warp != 0) continue;
      bad = (bw ? 2 : 0) | (bx ? 1 : 0);
    }
    warp_finish<MAXNB <= 3 ? 1 : 2>(a, L, k, it.p, it.ridge, (double*)(base + Lay::kG), bad, (double*)base,
                                    DmTraits<MAXNB>::kPad + 1);
    __syncwarp();
  }
}

// Split systems: the units' Grams added in unit order by a CTA (five entries a
// thread, four units of each in flight), then the finish by its first warp.
constexpr int kFinThreads = 256;
constexpr int kFinEntries = (48 * 49 / 2 + kFinThreads - 1) / kFinThreads;
__global__ void __launch_bounds__(kFinThreads, 3) ridge_split_finish(RidgeArgs a, RidgeLists L) {
  extern __shared__ __align__(128) unsigned char smem[];
  const int nrec = min(*L.nrec, L.rec_cap);
  for (int r = blockIdx.x; r < nrec; r += gridDim.x) {
    const SplitRec rec = L.recs[r];
    if (rec.k < 0) continue;
    const RidgeItem it = load_item(a, rec.k);
    const int pa = it.p + 1, E = pa * (pa + 1) / 2;
    double* G = (double*)smem;
    double* vec = G + ((E + 1) & ~1);
    const double* part = L.pool + rec.base;
    double s[kFinEntries];
#pragma unroll
    for (int m = 0; m < kFinEntries; ++m) s[m] = 0.0;
#pragma unroll 4
    for (int u = 0; u < rec.nseg; ++u)
#pragma unroll
      for (int m = 0; m < kFinEntries; ++m) {
        const int e = threadIdx.x + kFinThreads * m;
        if (e < E) s[m] += part[(size_t)u * E + e];
      }
#pragma unroll
    for (int m = 0; m < kFinEntries; ++m) {
      const int e = threadIdx.x + kFinThreads * m;
      if (e < E) G[e] = s[m];
    }
    __syncthreads();
    if (threadIdx.x < 32) {
      if (pa <= 32) warp_finish<1>(a, L, rec.k, it.p, it.ridge, G, rec.bad, vec, pa);
      else warp_finish<2>(a, L, rec.k, it.p, it.ridge, G, rec.bad, vec, pa);
    }
    __syncthreads();
  }
}

template <int MAXNB>
int launch_dmma(const RidgeArgs& a, const RidgeLists& L, int cls, int ctas, cudaStream_t s, const char* name) {
  // one warp per list entry or run of units; no more CTAs than there can be
  const int64_t most = ((a.K + (L.item_cap > 0 ? L.item_cap : 0)) + kDmWarps - 1) / kDmWarps;
  prof_begin(name, s);
  ridge_dmma_kernel<MAXNB><<<(unsigned)std::max<int64_t>(1, std::min<int64_t>(ctas, most)), kDmThreads,
                             DmLayout<MAXNB>::kPerWarp * kDmWarps, s>>>(a, L, cls);
  prof_end(s);
  count_launch();
  return check_launch(name);
}

template <int MAXNB>
int dmma_resident() {
  // a fixed property of the kernel and the device: asked for once per device
  static std::atomic<int> cached[64];
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) { cudaGetLastError(); return 0; }
  const int have = cached[dev].load(std::memory_order_acquire);
  if (have > 0) return have;
  const size_t smem = DmLayout<MAXNB>::kPerWarp * kDmWarps;
  if (cudaFuncSetAttribute(ridge_dmma_kernel<MAXNB>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) !=
      cudaSuccess) {
    cudaGetLastError();
    return 0;
  }
  const int n = device_sm_count() * resident_ctas((const void*)ridge_dmma_kernel<MAXNB>, kDmThreads, smem);
  cached[dev].store(n, std::memory_order_release);
  return n;
}

}  // namespace

// CTAs of the class's kernel that the device holds at once.
int ridge_dmma_ctas(int cls) { return cls == CLS_WARP ? dmma_resident<3>() : dmma_resident<6>(); }

int launch_ridge_dmma(const RidgeArgs& a, const RidgeLists& L, int cls, cudaStream_t s) {
  return cls == CLS_WARP ? launch_dmma<3>(a, L, cls, L.workers[0] / kDmWarps, s, "ridge_dmma<3>")
                         : launch_dmma<6>(a, L, cls, L.workers[1] / kDmWarps, s, "ridge_dmma<6>");
}

int launch_ridge_split_finish(const RidgeArgs& a, const RidgeLists& L, cudaStream_t s) {
  const int pa = std::min(a.pmax, kSmallMaxAug - 1) + 1;
  const size_t smem = ((size_t)pa * (pa + 1) / 2 + 1) * 8 + (size_t)3 * (pa + 1) * 8 + 16;
  prof_begin("ridge_split_finish", s);
  ridge_split_finish<<<(unsigned)std::max<int64_t>(1, std::min<int64_t>(L.rec_cap, 3 * device_sm_count())), kFinThreads,
                       smem, s>>>(a, L);
  prof_end(s);
  count_launch();
  return check_launch("ridge_split_finish");
}

}  // namespace art
