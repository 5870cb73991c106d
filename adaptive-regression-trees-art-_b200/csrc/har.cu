// har.cu -- hit-and-run chains in node polytopes {lo <= x <= hi, A x <= b}.
//
// Follows the reference transitions:
//  * ART_HAR_BATCHED: sample_precomputed_chains(_parallel)
//    (art/_numba_sampling.py:9-167): Gaussian directions used unnormalised,
//    slacks s = b - A x updated incrementally (s -= t * A u), chord bounds
//    from the signs of A u (exact zero tests), t = t_lo + U (t_hi - t_lo),
//    a sample after every `thinning` steps following `burn_in`.
//  * ART_HAR_SCALAR: HitAndRunSampler.sample (art/sampling.py:445-495,
//    _step_interval 540-564): unit directions, slack recomputed from x each
//    step, |A u| > 1e-14 tests, samples at steps burn_in + k*thinning.
//
// A step has a part that depends on the chain's state (the chord bounds from
// the slacks, the step, the new slacks) and a larger one that does not (the
// draws, and the products A u of every oblique row with the direction).  A team
// of TL lanes advances one chain, a block of SB steps at a time:
//   1. the block's directions are drawn (or copied ahead of time, if injected)
//      into shared memory, a Philox block per (step, coordinate pair);
//   2. lane = step: A u for every row, four rows at a time, and the uniform;
//   3. lane = constraint: the steps one after another, each lane holding the
//      slacks of its coordinates and rows.  A step is a product with the
//      reciprocal of A u (formed ahead, off the dependent path), a minimum and
//      a maximum over the team, and the update.
// What bounds it: for few chains the dependent path of part 3 (so a whole warp
// per chain, the minima and maxima by integer redux.sync on the ordered bits),
// for many chains instruction issue, 70 % of the slots (so teams of 8 or 16
// lanes where the dimension allows).  Against a step that drew, multiplied and
// divided in turn, bit for bit the same states: 61 chains of 2,100 steps in 4
// dimensions 7.64 -> 0.46 ms, 16,384 chains of 1,000 steps in 8 dimensions
// 4.05 -> 1.79 ms.
// Box rows (+e_i, -e_i) are applied structurally: A u = +-u_i exactly, as in
// the reference's dense matmul, and of a coordinate's two rows one bounds the
// step from above and the other from below.
#include <algorithm>

#include "bulk.cuh"
#include "common.cuh"

namespace art {
namespace {

constexpr int kHarThreads = 128;
constexpr double kScalarParallelTol = 1e-14;  // sampling.py:552-553
constexpr double kFeasTol = 1e-10;             // sampling.py:438, domain.py:40

struct HarArgs {
  int64_t n_poly;
  int d;
  const double* lo;
  const double* hi;
  const int64_t* row_offsets;
  const double* A;
  const double* b;
  const double* maps;  // [n_poly][d][d] or NULL
  int64_t n_chains;
  const int32_t* polytope;
  double* x;
  const uint64_t* seeds;
  const double* dirs;
  const double* unif;
  int mode;
  int burn_in, thinning, n_rounds;
  uint64_t counter_base;
  double* samples;
  int32_t* status;
  int cap;  // oblique rows a team has room for
};

// A chain of a thousand steps in eight dimensions amplifies a rounding by ten
// orders of magnitude, so every operation that reaches the state keeps one
// order and one rounding whatever the team: products are summed by coordinate
// pairs in a halving tree (pair_tree), quotients are correctly rounded.

// 1 / v within an ulp or two: the hardware's approximation and two
// Newton-Raphson steps r <- r + r (1 - v r).
__device__ __forceinline__ double newton_rcp(double v) {
  double r;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(v));
  r = fma(r, fma(-v, r, 1.0), r);
  return fma(r, fma(-v, r, 1.0), r);
}
// s / v rounded to nearest from y = newton_rcp(v): q = s y and one correction
// by its residual s - q v (Markstein, "Computation of elementary functions on
// the IBM RISC System/6000 processor", IBM J. Res. Dev. 1990); what is rounded
// last is within 2^-104 of the quotient.  y does not depend on the state, so
// only these three operations are on a step's dependent path.  It takes |v| in
// quotient_range; of slacks below 2^-900 the residual underflows, and the
// quotient may miss the nearest value by one unit (a test of the slack costs
// 16 % of a step with few chains, 5 % with many).
__device__ __forceinline__ double quotient(double s, double v, double y) {
  const double q = s * y;
  return fma(fma(-q, v, s), y, q);
}
// The plain division, kept out of line: it is almost never needed.
__device__ __noinline__ double divided(double s, double v) { return s / v; }
// |v| in [2^-100, 2^100): then s - q v is exact.  A denormal v in particular has
// no reciprocal (rcp.approx.ftz takes it as zero), yet bounds the step: a chain
// on that face has slack zero.
__device__ __forceinline__ bool quotient_range(double v) {
  return ((uint32_t)__double2hiint(v) & 0x7fffffffu) - 0x39b00000u < 0x0c800000u;
}

// sum_i a_i v_i over d <= 2 H coordinates: a_2l v_2l + a_2l+1 v_2l+1 of each
// pair, the pairs added in halves (l with l + H / 2, then H / 4, ...).  FMA: a
// pair's first product rounded, the second not.  (With a single pair the
// second is rounded, the first not.)
template <int H, bool FMA = false>
__device__ __forceinline__ double pair_tree(const double* a, const double* v, int d) {
  double p[H];
#pragma unroll
  for (int l = 0; l < H; ++l) {
    const double s = 2 * l < d ? __dmul_rn(a[2 * l], v[2 * l]) : 0.0;
    const double t = 2 * l + 1 < d ? __dmul_rn(a[2 * l + 1], v[2 * l + 1]) : 0.0;
    if (H == 1 && !FMA) p[l] = fma(a[0], v[0], t);
    else p[l] = FMA && 2 * l + 1 < d ? fma(a[2 * l + 1], v[2 * l + 1], s) : __dadd_rn(s, t);
  }
#pragma unroll
  for (int o = H / 2; o > 0; o >>= 1)
#pragma unroll
    for (int l = 0; l < o; ++l) p[l] = __dadd_rn(p[l], p[l + o]);
  return p[0];
}

// Minimum of hi and maximum of lo over the team's lanes.
template <int TL>
__device__ __forceinline__ void team_bounds(double& lo, double& hi) {
  if constexpr (TL == 32) {
    // doubles as ordered (signed high, unsigned low) words: two 32-bit warp
    // reductions a bound instead of five rounds of 64-bit shuffles
    auto key = [](double v, int& h, uint32_t& l) {
      h = __double2hiint(v);
      l = (uint32_t)__double2loint(v);
      if (h < 0) { h ^= 0x7fffffff; l = ~l; }
    };
    auto value = [](int h, uint32_t l) {
      if (h < 0) { h ^= 0x7fffffff; l = ~l; }
      return __hiloint2double(h, (int)l);
    };
    int hh, lh;
    uint32_t hl, ll;
    key(hi, hh, hl);
    key(lo, lh, ll);
    const int mh = __reduce_min_sync(0xffffffffu, hh), xh = __reduce_max_sync(0xffffffffu, lh);
    const uint32_t ml = __reduce_min_sync(0xffffffffu, hh == mh ? hl : 0xffffffffu);
    const uint32_t xl = __reduce_max_sync(0xffffffffu, lh == xh ? ll : 0u);
    hi = value(mh, ml);
    lo = value(xh, xl);
  } else {
#pragma unroll
    for (int o = TL / 2; o > 0; o >>= 1) {
      const double h = __shfl_xor_sync(0xffffffffu, hi, o), l = __shfl_xor_sync(0xffffffffu, lo, o);
      hi = h < hi ? h : hi;
      lo = l > lo ? l : lo;
    }
  }
}
template <int TL>
__device__ __forceinline__ bool team_any(bool v) {
  const unsigned m = __ballot_sync(0xffffffffu, v);
  const int lane = threadIdx.x & 31;
  return ((m >> (lane / TL * TL)) & (TL == 32 ? 0xffffffffu : (1u << (TL & 31)) - 1u)) != 0;
}

// Shared memory of a team, in doubles: A [cap][us], the directions [bufs][SB][us],
// the products [SB][as], the uniforms [bufs][SB], the state [d].  Odd strides
// us and as put the lanes of part 2 (one step each), and in the slacks those
// with a row each, into different banks; the team stride, 8 modulo 16, does the
// same for the teams of a warp.
struct HarLayout {
  int us, as, bufs;
  int U, AU, UN, X, total;
};
__host__ __device__ inline HarLayout har_layout(int d, int cap, int SB, bool injected, bool maps) {
  HarLayout L;
  L.us = d | 1;
  L.as = cap | 1;
  L.bufs = injected || maps ? 2 : 1;  // the next block's draws in flight, or z beside u = M z
  L.U = cap * L.us;
  L.AU = L.U + L.bufs * SB * L.us;
  L.UN = L.AU + SB * L.as;
  L.X = L.UN + L.bufs * SB;
  L.total = (L.X + d + 7) / 16 * 16 + 8;
  while (L.total < L.X + d) L.total += 16;
  return L;
}

template <int TL, int CPL, int RPL, int SB, int H, bool scalar>
__global__ void __launch_bounds__(kHarThreads) har_kernel(HarArgs a) {
  extern __shared__ double s_team[];
  const int lane = (int)(threadIdx.x % TL);
  const int64_t chain_raw = ((int64_t)blockIdx.x * kHarThreads + threadIdx.x) / TL;
  // Teams past the end keep running (masked) so that full-warp shuffles stay valid.
  const bool live = chain_raw < a.n_chains;
  const int64_t chain = live ? chain_raw : (a.n_chains - 1);
  const int d = a.d;
  const bool injected = a.dirs != nullptr;
  const HarLayout L = har_layout(d, a.cap, SB, injected, a.maps != nullptr && !injected);
  double* As = s_team + (size_t)(threadIdx.x / TL) * L.total;
  double* Us = As + L.U;
  double* AUs = As + L.AU;
  double* UNs = As + L.UN;
  double* Xs = As + L.X;
  const int pj = a.polytope[chain];
  const int64_t rb = a.row_offsets[pj];
  int k = (int)(a.row_offsets[pj + 1] - rb);
  int status = 0;
  if (k > a.cap) { status = 3; k = 0; }
  const bool box = a.lo != nullptr;
  const double inf = INFINITY;
  // this lane's coordinates i = lane + TL m and rows r = lane + TL m
  double x[CPL], shi[CPL], slo[CPL], hi_[CPL], lo_[CPL];
  double so[RPL], br[RPL];
#pragma unroll
  for (int m = 0; m < CPL; ++m) {
    const int i = lane + TL * m;
    const bool own = i < d;
    x[m] = own ? a.x[chain * d + i] : 0.0;
    // a coordinate without a box never bounds the step: infinite slacks
    lo_[m] = own && box ? a.lo[(int64_t)pj * d + i] : -inf;
    hi_[m] = own && box ? a.hi[(int64_t)pj * d + i] : inf;
    shi[m] = hi_[m] - x[m];
    slo[m] = x[m] - lo_[m];
    if (own) Xs[i] = x[m];
  }
  for (int e = lane; e < a.cap * d; e += TL) As[e / d * L.us + e % d] = e < k * d ? a.A[rb * d + e] : 0.0;
  __syncwarp();
  auto row_slack = [&](int m) {  // b - A x of this lane's m-th row
    const int r = lane + TL * m;
    if (r >= k) return 0.0;
    return __dsub_rn(br[m], pair_tree<H>(As + r * L.us, Xs, d));
  };
  bool bad = false;
#pragma unroll
  for (int m = 0; m < RPL; ++m) {
    const int r = lane + TL * m;
    br[m] = r < k ? a.b[rb + r] : 0.0;
    so[m] = row_slack(m);  // numba path: sampling.py:648
    if (so[m] < -kFeasTol) bad = true;
  }
#pragma unroll
  for (int m = 0; m < CPL; ++m)
    if (shi[m] < -kFeasTol || slo[m] < -kFeasTol) bad = true;
  if (team_any<TL>(bad) && status == 0) status = 2;
  const uint32_t key0 = a.seeds ? (uint32_t)a.seeds[chain] : 0u;
  const uint32_t key1 = a.seeds ? (uint32_t)(a.seeds[chain] >> 32) : 0u;
  const int total = a.burn_in + a.n_rounds * a.thinning;
  const int64_t C = a.n_chains;
  int64_t ucur = 0;  // uniform cursor (scalar mode skips draws on zero directions)
  // next step that keeps a sample and its index: scalar mode keeps steps
  // burn_in + j * thinning (none on a zero direction), batched mode the last
  // step of each thinning block after burn_in
  int keep_step = scalar ? a.burn_in : a.burn_in + a.thinning - 1;
  int keep_idx = 0;
  constexpr int NP = TL / SB;               // lanes that share a step in part 2
  const int st = lane % SB, part = lane / SB;
  auto copy_block = [&](int s0, int buf) {  // injected draws of steps [s0, s0 + SB), in flight
    const int ns = min(SB, total - s0);
    const double* src = a.dirs + ((int64_t)chain * total + s0) * d;
    double* dst = Us + buf * SB * L.us;
    int r = lane / d, c = lane - r * d;
    const int dr = TL / d, dc = TL - dr * d;
    for (int e = lane; e < ns * d; e += TL) {
      cp_async8(smem_u32(dst + r * L.us + c), src + e);
      r += dr;
      c += dc;
      if (c >= d) { c -= d; ++r; }
    }
    if (!scalar && part == 0 && st < ns)
      cp_async8(smem_u32(UNs + buf * SB + st), a.unif + (int64_t)chain * total + s0 + st);
    cp_async_commit();
  };
  if (injected && total > 0) copy_block(0, 0);
  for (int s0 = 0; s0 < total; s0 += SB) {
    const int ns = min(SB, total - s0);
    int buf = 0;
    __syncwarp();
    // ---- 1. directions
    if (injected) {
      buf = (s0 / SB) & 1;
      if (s0 + SB < total) copy_block(s0 + SB, buf ^ 1);
      else cp_async_commit();
      cp_async_wait1();
    } else {
      buf = a.maps ? 1 : 0;
      const int np = (d + 1) / 2;
      double* z = Us + buf * SB * L.us;
      for (int j = part; j < np; j += NP) {
        const uint64_t ctr = a.counter_base + (uint64_t)(s0 + st);
        const Philox4 r = philox4x32_10((uint32_t)ctr, (uint32_t)(ctr >> 32), (uint32_t)j, 0u, key0, key1);
        double u0, u1;
        normal_pair_f32(r, u0, u1);
        z[st * L.us + 2 * j] = u0;
        if (2 * j + 1 < d) z[st * L.us + 2 * j + 1] = u1;
      }
      if (a.maps) {  // covariance-shaped direction u = M z
        __syncwarp();
        const double* M = a.maps + (int64_t)pj * d * d;
        for (int i = part; i < d; i += NP) {
          double t = 0.0;
          for (int j = 0; j < d; ++j) t = fma(__ldg(M + (int64_t)i * d + j), z[st * L.us + j], t);
          Us[st * L.us + i] = t;
        }
        buf = 0;
      }
    }
    double* U = Us + buf * SB * L.us;
    double* UN = UNs + (injected ? buf * SB : 0);
    __syncwarp();
    // ---- 2. lane = step: unit direction (scalar mode), A u, the uniform
    bool zero = false;
    if (scalar) {
      const double n2 = pair_tree<H, true>(U + st * L.us, U + st * L.us, d);
      const double nrm = sqrt(n2);
      zero = st < ns && nrm == 0.0;
      __syncwarp();
      if (!zero)
        for (int i = part; i < d; i += NP) U[st * L.us + i] = U[st * L.us + i] / nrm;
      __syncwarp();
    }
    const unsigned zmask = __ballot_sync(0xffffffffu, zero) >> ((threadIdx.x & 31) / TL * TL);
    if (part == 0 && st < ns) {
      if (!injected) {
        const uint64_t ctr = a.counter_base + (uint64_t)(s0 + st);
        const Philox4 r = philox4x32_10((uint32_t)ctr, (uint32_t)(ctr >> 32), 0xFFFFFFFFu, 1u, key0, key1);
        UN[st] = u01_closed_open(r.v[0], r.v[1]);
      } else if (scalar) {
        const int64_t at = ucur + st - __popc(zmask & ((1u << st) - 1u));
        UN[st] = a.unif[(int64_t)chain * total + at];
      }
    }
    for (int r = part; r < k; r += NP) AUs[st * L.as + r] = pair_tree<H>(As + r * L.us, U + st * L.us, d);
    __syncwarp();
    // ---- 3. lane = constraint: the steps in order
    double nu[CPL], niu[CPL], nau[RPL], nia[RPL], nun;
    bool nodd;
    const double* up_ = U + lane;
    const double* ap_ = AUs + lane;
    const double* np_ = UN;
    auto fetch = [&]() {  // what the next step needs besides the state
      bool odd = false;
#pragma unroll
      for (int m = 0; m < CPL; ++m) {
        nu[m] = lane + TL * m < d ? up_[TL * m] : 0.0;
        niu[m] = newton_rcp(nu[m]);
        odd |= nu[m] != 0.0 && !quotient_range(nu[m]);
      }
#pragma unroll
      for (int m = 0; m < RPL; ++m) {
        nau[m] = lane + TL * m < k ? ap_[TL * m] : 0.0;
        nia[m] = newton_rcp(nau[m]);
        odd |= nau[m] != 0.0 && !quotient_range(nau[m]);
      }
      nun = *np_;
      // divisors outside the quotient's range: the step divides
      nodd = __any_sync(0xffffffffu, odd);
    };
    fetch();
#pragma unroll 2
    for (int j = 0; j < ns; ++j) {
      // a zero direction moves nothing (scalar mode skips the step; control
      // flow stays the same for the warp's other teams)
      const bool skip = scalar && ((zmask >> j) & 1u);
      double u_[CPL], iu[CPL], au[RPL], ia[RPL];
#pragma unroll
      for (int m = 0; m < CPL; ++m) { u_[m] = nu[m]; iu[m] = niu[m]; }
#pragma unroll
      for (int m = 0; m < RPL; ++m) { au[m] = nau[m]; ia[m] = nia[m]; }
      const double un = nun;
      const bool divide = nodd;
      double thi = inf, tlo = -inf;
      bool infeasible = false;
      if constexpr (scalar) {  // slacks from x (sampling.py:548-550)
#pragma unroll
        for (int m = 0; m < RPL; ++m) so[m] = row_slack(m);
#pragma unroll
        for (int m = 0; m < CPL; ++m) { shi[m] = hi_[m] - x[m]; slo[m] = x[m] - lo_[m]; }
      }
      // A NaN quotient bounds nothing: that of an infinite slack (no box), of a
      // zero product (its reciprocal is NaN), or, in scalar mode, of a product
      // within the parallel tolerance (made NaN here).
      auto bounds = [](double v, double y) { return scalar ? y == y : v != 0.0; };
#pragma unroll
      for (int m = 0; m < CPL; ++m) {
        double y = iu[m];
        if constexpr (scalar) {
          if (!(fabs(u_[m]) > kScalarParallelTol)) {
            y = __longlong_as_double(0x7ff8000000000000ll);
            infeasible |= shi[m] < -kFeasTol || slo[m] < -kFeasTol;
          }
        }
        double ra = quotient(shi[m], u_[m], y), rb_ = -quotient(slo[m], u_[m], y);
        if (divide && bounds(u_[m], y)) { ra = divided(shi[m], u_[m]); rb_ = -divided(slo[m], u_[m]); }
        const bool neg = __double2hiint(u_[m]) < 0;
        const double h = neg ? rb_ : ra, l = neg ? ra : rb_;
        thi = h < thi ? h : thi;
        tlo = l > tlo ? l : tlo;
      }
#pragma unroll
      for (int m = 0; m < RPL; ++m) {
        double y = ia[m];
        if constexpr (scalar) {
          if (!(fabs(au[m]) > kScalarParallelTol)) {
            y = __longlong_as_double(0x7ff8000000000000ll);
            infeasible |= so[m] < -kFeasTol;
          }
        }
        double r = quotient(so[m], au[m], y);
        if (divide && bounds(au[m], y)) r = divided(so[m], au[m]);
        const bool neg = __double2hiint(au[m]) < 0;
        if (!neg && r < thi) thi = r;
        if (neg && r > tlo) tlo = r;
      }
      if (j + 1 < ns) {
        up_ += L.us;
        ap_ += L.as;
        ++np_;
      }
      fetch();  // issued while the bounds travel
      team_bounds<TL>(tlo, thi);
      if constexpr (scalar) infeasible = team_any<TL>(infeasible);
      if (status == 0 && !skip && (tlo > thi || infeasible)) status = 1;
      // Separate roundings (no FMA contraction), as numpy/numba evaluate them.
      const double t = __dadd_rn(tlo, __dmul_rn(un, __dsub_rn(thi, tlo)));
      if (status == 0 && !skip) {
#pragma unroll
        for (int m = 0; m < CPL; ++m) {
          const double tu = __dmul_rn(t, u_[m]);
          x[m] = __dadd_rn(x[m], tu);
          shi[m] = __dsub_rn(shi[m], tu);
          slo[m] = __dadd_rn(slo[m], tu);
        }
#pragma unroll
        for (int m = 0; m < RPL; ++m) so[m] = __dsub_rn(so[m], __dmul_rn(t, au[m]));
      }
      if constexpr (scalar) {
        __syncwarp();
#pragma unroll
        for (int m = 0; m < CPL; ++m)
          if (lane + TL * m < d) Xs[lane + TL * m] = x[m];
        __syncwarp();
      }
      // sample bookkeeping
      if (s0 + j == keep_step) {
        if (!skip && keep_idx < a.n_rounds && live) {
          double* sp = a.samples + ((int64_t)keep_idx * C + chain) * d;
#pragma unroll
          for (int m = 0; m < CPL; ++m)
            if (lane + TL * m < d) sp[lane + TL * m] = x[m];
        }
        ++keep_idx;
        keep_step += a.thinning;
      }
    }
    ucur += ns - __popc(zmask & (SB == 32 ? 0xffffffffu : (1u << (SB & 31)) - 1u));
  }
  if (injected) cp_async_wait0();
  if (live) {
#pragma unroll
    for (int m = 0; m < CPL; ++m)
      if (lane + TL * m < d) a.x[chain * d + lane + TL * m] = x[m];
    if (lane == 0 && a.status) a.status[chain] = status;
  }
}

template <int TL, int CPL, int RPL, int SB, int H>
int launch_har_k(const HarArgs& a, cudaStream_t s) {
  const HarLayout L = har_layout(a.d, a.cap, SB, a.dirs != nullptr, a.maps != nullptr && a.dirs == nullptr);
  const size_t smem = (size_t)(kHarThreads / TL) * L.total * 8;
  auto kern = a.mode == ART_HAR_SCALAR ? har_kernel<TL, CPL, RPL, SB, H, true> : har_kernel<TL, CPL, RPL, SB, H, false>;
  if (smem > 227 * 1024 ||
      cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess) {
    cudaGetLastError();
    set_error("art_hit_and_run: cannot reserve %zu bytes of shared memory", smem);
    return ART_E_UNSUPPORTED;
  }
  cudaFuncSetAttribute(kern, cudaFuncAttributePreferredSharedMemoryCarveout, (int)cudaSharedmemCarveoutMaxShared);
  cudaGetLastError();
  const unsigned grid = (unsigned)((a.n_chains * TL + kHarThreads - 1) / kHarThreads);
  prof_begin("hit_and_run", s);
  kern<<<grid, kHarThreads, smem, s>>>(a);
  prof_end(s);
  count_launch();
  return check_launch("art_hit_and_run");
}

// A warp per chain while the device has idle warps for it, else the narrowest
// team that holds a coordinate and at most four rows a lane.  1,000 steps with 12
// rows, a warp a chain against teams: d = 2, 1,184 chains 340 and 445 us, 2,000 522
// and 434; d = 8, 393 and 622, 3,000 chains 879 and 623; d = 16, 468 and 635, 2,000
// chains 713 and 635.
template <int H>
int launch_har_narrow(const HarArgs& a, cudaStream_t s) {  // d <= 8
  if (a.n_chains <= (int64_t)8 * device_sm_count()) return launch_har_k<32, 1, 1, 32, H>(a, s);
  if (a.cap <= 8) return launch_har_k<8, 1, 1, 8, H>(a, s);
  return a.cap <= 16 ? launch_har_k<8, 1, 2, 8, H>(a, s) : launch_har_k<8, 1, 4, 8, H>(a, s);
}
int launch_har(const HarArgs& a, cudaStream_t s) {
  if (a.d <= 2) return launch_har_narrow<1>(a, s);
  if (a.d <= 4) return launch_har_narrow<2>(a, s);
  if (a.d <= 8) return launch_har_narrow<4>(a, s);
  if (a.d <= 16) {
    if (a.n_chains <= (int64_t)8 * device_sm_count()) return launch_har_k<32, 1, 1, 32, 8>(a, s);
    return a.cap <= 16 ? launch_har_k<16, 1, 1, 16, 8>(a, s) : launch_har_k<16, 1, 2, 16, 8>(a, s);
  }
  if (a.d <= 32) return launch_har_k<32, 1, 1, 32, 16>(a, s);
  return launch_har_k<32, 2, 1, 16, 32>(a, s);
}

}  // namespace
}  // namespace art

using namespace art;

extern "C" int art_hit_and_run(const ArtPolytopes* P, const ArtChains* C, art_stream_t stream) {
  cudaGetLastError();
  if (!P || !C) { set_error("art_hit_and_run: null argument"); return ART_E_INVALID; }
  if (C->count < 0 || P->count < 0) { set_error("art_hit_and_run: negative count"); return ART_E_INVALID; }
  if (C->count == 0) return ART_OK;
  if (P->dim < 1 || P->dim > ART_MAX_DIM) {
    set_error("art_hit_and_run: dim %d outside [1, %d]", P->dim, ART_MAX_DIM);
    return ART_E_UNSUPPORTED;
  }
  if (P->max_rows < 0 || P->max_rows > 32) {
    set_error("art_hit_and_run: max_rows %d outside [0, 32]", P->max_rows);
    return ART_E_UNSUPPORTED;
  }
  if (!P->row_offsets || (P->max_rows > 0 && (!P->A || !P->b)) || ((P->lo == nullptr) != (P->hi == nullptr))) {
    set_error("art_hit_and_run: polytope arrays incomplete");
    return ART_E_INVALID;
  }
  if (!C->polytope || !C->x || (!C->samples && C->n_rounds > 0)) {
    set_error("art_hit_and_run: chain arrays incomplete");
    return ART_E_INVALID;
  }
  if ((C->directions == nullptr) != (C->uniforms == nullptr)) {
    set_error("art_hit_and_run: inject both directions and uniforms, or neither");
    return ART_E_INVALID;
  }
  if (!C->directions && !C->seeds) {
    set_error("art_hit_and_run: seeds are required without injected draws");
    return ART_E_INVALID;
  }
  if (C->mode != ART_HAR_BATCHED && C->mode != ART_HAR_SCALAR) {
    set_error("art_hit_and_run: unknown mode %d", C->mode);
    return ART_E_INVALID;
  }
  if (C->burn_in < 0 || C->thinning < 1 || C->n_rounds < 0) {
    set_error("art_hit_and_run: burn_in >= 0, thinning >= 1, n_rounds >= 0 required");
    return ART_E_INVALID;
  }
  HarArgs a;
  a.n_poly = P->count; a.d = P->dim; a.lo = P->lo; a.hi = P->hi;
  a.maps = P->direction_maps;
  a.row_offsets = P->row_offsets; a.A = P->A; a.b = P->b;
  a.n_chains = C->count; a.polytope = C->polytope; a.x = C->x; a.seeds = C->seeds;
  a.dirs = C->directions; a.unif = C->uniforms; a.mode = C->mode;
  a.burn_in = C->burn_in; a.thinning = C->thinning; a.n_rounds = C->n_rounds;
  a.counter_base = C->counter_base; a.samples = C->samples; a.status = C->status;
  a.cap = P->max_rows <= 4 ? 4 : (P->max_rows <= 8 ? 8 : (P->max_rows <= 16 ? 16 : 32));
  return launch_har(a, (cudaStream_t)stream);
}
