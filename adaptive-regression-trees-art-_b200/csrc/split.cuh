// split.cuh -- definitions shared by the split search's kernels: the warp form
// (split_warp.cu) and the CTA form with the host entry point (split.cu).
#pragma once
#include "common.cuh"

namespace art {

constexpr int kSplitBuckets = 64;
constexpr int kErrSlot = 2 + 2 * kSplitBuckets;  // counts[kErrSlot]: a bounded wait gave up

struct SplitArgs {
  int64_t K;
  const int64_t* row_offsets;
  const int64_t* x_offsets;
  const int32_t* dims;
  const int32_t* features;
  const double* x;
  const double* y;
  const double* temperature;
  const double* ridge;
  const double* parent_loss;
  const int8_t* fallback;
  const double* theta0;
  int64_t theta0_stride;
  const uint64_t* node_keys;
  const int32_t* min_side;  // per-node minimum side count or NULL
  ArtSplitParams prm;
  int R, Rg, groups, dmax, pmax, H, TC, S, CH;
  int mixed;  // ART_PRECISION_MIXED: gates in single precision
  int warp;   // the warp form
  int tc;     // mixed form with the soft-pass Grams on the tensor cores
  int dg;     // side Grams as FP64 MMA tiles (8 x 8 blocks of (q psi)^T psi, at most kDgMax per warp)
  // per (node, restart) results, index k * R + r
  double* r_theta;   // [.. ][dmax + 1]
  double* r_loss;
  double* r_beta;    // [..][2][pmax]
  double* r_child;   // [..][2]
  double* r_ridge;   // [..][2]
  int32_t* r_nright;
  int32_t* r_iters;
  int32_t* r_stop;
  int32_t* r_fail;
  int32_t* r_flags;
  int32_t* r_fbiter;
  double* r_alpha;
  double* tr_loss;
  double* tr_step;
  int32_t* tr_back;
  double* tr_gnorm;
  // work queue
  int32_t* counts;   // [0] entries, [1] cursor, [2..2+64) hist, [66..130) start
  int4* items;       // queue entries (item, gang rank, gang size, 0)
  int gang_on, nslots, gang_P;  // gangs enabled; scratch slots; doubles per rank partial
  int4* gang_rec;    // [K * groups]: slot + 1, barrier arrivals, members done, abort
  int32_t* slot_flags;  // [nslots]
  double* gang_scratch; // [nslots][2][kGangMax][gang_P]
};

// Bucket of a node of n rows in the plan's largest-first order.
__device__ __forceinline__ int split_bucket(int64_t n) {
  return kSplitBuckets - 1 - max(0, min(kSplitBuckets - 1, ilogb((double)(n + 1))));
}

// D = A B + D for one 8 x 8 x 4 FP64 tile (warp-wide): lane l holds
// A[l / 4][l % 4], B[l % 4][l / 4] and D[l / 4][2 (l % 4) + {0, 1}].
__device__ __forceinline__ void split_dmma(double (&c)[2], double a, double b) {
  asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};\n"
      : "+d"(c[0]), "+d"(c[1])
      : "d"(a), "d"(b));
}

// e^x for |x| <= 51 (Cody & Waite, "Software Manual for the Elementary
// Functions", 1980): x = k ln 2 + r with k rounded by the shift 1.5 * 2^52 and
// ln 2 in two parts (42 binary places, and the rest), the Taylor series of e^r to r^13 (|r| <= ln 2 / 2: the rest
// is below 5e-18), and k added to the exponent.  No branch, so that several
// gates of a row run side by side (256 nodes of 16 restarts: 73.8 ms to 71.0).
// Within 1.04 ulp; the gate below errs by at most 2.32 ulp and 0.524 rms over
// [-50, 50], with exp() and a division by 2.32 and 0.530.
__device__ __forceinline__ double exp51(double x) {
  const double shift = 6755399441055744.0;
  const double t = fma(x, 1.4426950408889634, shift);
  const double k = t - shift;
  double r = fma(k, -0.6931471805598903, x);
  r = fma(k, -5.497923018708371e-14, r);
  const double r2 = r * r;
  // even and odd halves of the series, each by Horner's rule in r^2
  double e = 1.0 / 479001600.0, o = 1.0 / 6227020800.0;
  e = fma(e, r2, 1.0 / 3628800.0);
  o = fma(o, r2, 1.0 / 39916800.0);
  e = fma(e, r2, 1.0 / 40320.0);
  o = fma(o, r2, 1.0 / 362880.0);
  e = fma(e, r2, 1.0 / 720.0);
  o = fma(o, r2, 1.0 / 5040.0);
  e = fma(e, r2, 1.0 / 24.0);
  o = fma(o, r2, 1.0 / 120.0);
  e = fma(e, r2, 0.5);
  o = fma(o, r2, 1.0 / 6.0);
  // e^r = 1 + (r + r2 (e + r o))
  const double q = fma(r2, fma(r, o, e), r) + 1.0;
  return __hiloint2double(__double2hiint(q) + (__double2loint(t) << 20), __double2loint(q));
}

__device__ __forceinline__ double sigm(double s) {
  s = fmin(fmax(s, -50.0), 50.0);  // objectives.py:49-51
  // 1 / v, v in [1, 1 + e^50]: the hardware's approximation and three
  // Newton-Raphson steps, without a division's range checks
  const double v = 1.0 + exp51(-s);
  double r;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(v));
  r = fma(r, fma(-v, r, 1.0), r);
  r = fma(r, fma(-v, r, 1.0), r);
  return fma(r, fma(-v, r, 1.0), r);
}

// Mixed form: the gate in single precision with CUDA's fast exponential
// (relative error ~1e-7, inside the form's 1e-5 objective tolerance); the
// score, residuals, solves and every sum stay FP64.
__device__ __forceinline__ double sigm32(double s) {
  const float sf = fminf(fmaxf((float)s, -50.0f), 50.0f);
  return (double)__frcp_rn(1.0f + __expf(-sf));
}

// Host side (split_warp.cu): whether a level fits the warp form, and its launch.
bool split_warp_fits(int max_dim, int max_features, int restarts);
int launch_split_warp(const SplitArgs& a, cudaStream_t s);

}  // namespace art
