// ridge.cuh -- definitions shared by the ridge kernels (plain FP64, mixed
// tensor-core, QR fallback) and the host entry point.
#pragma once
#include "common.cuh"
#include "bulk.cuh"
#include "linalg.cuh"

namespace art {

constexpr int kRidgeThreads = 256;
constexpr int kBuckets = 64;
// Work lists.  The plan kernels fill the first three; solve kernels append
// to the last two.
enum RidgeClass {
  CLS_SMALL = 0,    // FP64, 24 < (p+1) <= 48: warps alone, FP64 MMA Grams (ridge_dmma.cu)
  CLS_LARGE = 1,    // FP64, (p+1) > 48: a CTA each, FP64 MMA Grams (ridge_wide.cu)
  CLS_TENSOR = 2,   // mixed form, p at or above its threshold: tcgen05 split-product Gram
  CLS_WARP = 3,     // FP64, (p+1) <= 24: as CLS_SMALL, narrower blocks and more warps
  CLS_QR = 4,       // auto solver fallback: Householder QR
  CLS_RESOLVE = 5,  // mixed form systems re-solved by the FP64 form
  kClasses = 6
};
constexpr int kPlanClasses = 4;
constexpr int kWarpMaxAug = 24;
constexpr int kSmallMaxAug = 48;
constexpr int kTensorMinP = 33;  // smallest p the tensor-core kernel takes
// The mixed form's default threshold: none.  The FP64 MMA kernels are the more
// exact ones and at least as fast (weighted systems of 306 to 8,192 rows, FP64
// against the tensor-core kernel: 2,048 of 45 features 0.54 and 3.6 ms; 510 of
// 153 features 1.6 and 2.1 ms, 4,096 of them 12.2 and 12.2 ms, where its FP64
// refinement passes over the rows cost what its Gram saves).
constexpr int kTensorDefaultP = ART_MAX_FEATURES + 1;
// Split systems (see ridge_dmma.cu): units per system at most, batches above
// kSplitMaxCount systems are not split (they fill every warp by number).
constexpr int kMaxUnits = 256;
constexpr int kSplitMaxCount = 16384;
constexpr size_t kSplitPoolBytes = (size_t)256 << 20;
constexpr int kSplitRecs = 4096;
constexpr int kSplitItems = 32768;

// Rows per unit of a system of n rows and augmented width pa: fixed by the
// system alone, so that its sums do not depend on who forms them.  At least
// 256 rows (a Gram is then added for every 64 MMA steps that form it), and at
// most kMaxUnits units (a 400,000-row node of 45 features: units of 1,568
// rows; twice as long ones left its last warps 0.4 ms behind the others).
__host__ __device__ __forceinline__ int64_t ridge_unit_rows(int64_t n) {
  const int64_t u = ((n + kMaxUnits - 1) / kMaxUnits + 31) / 32 * 32;
  return u > 256 ? u : 256;
}

struct RidgeArgs {
  int64_t K;
  const int64_t* row_offsets;
  const int64_t* x_offsets;
  const int32_t* dims;
  const int32_t* features;
  const double* x;
  const double* y;
  const double* w;
  const double* ridge;
  double weight_floor;
  int solver;
  int precision;
  double rcond_threshold;
  int pmax;
  int dmax;
  double* beta;
  int64_t beta_stride;
  double* ridge_eff;
  double* cond;
  int32_t* status;
  uint32_t* info;
  uint32_t options;
  int tensor_min_p;       // mixed form: smallest p on the tensor-core kernel
  float* gram_out;        // art_ridge_gram: packed tensor-core Grams
  int64_t gram_stride;
};

// A system split over several warps: its pool slots hold nseg packed Grams.
struct SplitRec {
  int64_t base;  // first double in the pool
  int32_t k, nseg;
  int32_t bad, pad;
};

struct RidgeLists {
  int32_t* count;   // [kClasses]
  int32_t* cursor;  // [kClasses]
  int32_t* hist;    // [kPlanClasses][kBuckets]
  int32_t* start;   // [kPlanClasses][kBuckets]
  int32_t* err;     // [1] device-side error flag (bounded wait gave up)
  double* lambda;   // [K] effective ridge, kept for the QR fallback
  int32_t* list;    // [kClasses][K]
  // split systems of CLS_WARP (0) and CLS_SMALL (1)
  unsigned long long* cost;   // [2] summed row costs of the class
  unsigned long long* pool_used;  // doubles taken from the pool
  int32_t* nrec;    // records taken
  int32_t* nitems;  // [2] queue entries: (record, first unit, units)
  int32_t* nshared; // CLS_SMALL systems marked for a whole CTA: list entry -2 - k
  SplitRec* recs;
  int4* items;      // [2][item_cap]
  double* pool;
  int64_t pool_cap; // doubles; 0: no system is split
  int32_t rec_cap, item_cap;
  int32_t workers[2];  // warps the class's kernel keeps resident
};

struct RidgeItem {
  int64_t r0, n, xoff;
  int d, kind, p;
  double ridge;
};

__device__ __forceinline__ RidgeItem load_item(const RidgeArgs& a, int k) {
  RidgeItem it;
  it.r0 = a.row_offsets[k];
  it.n = a.row_offsets[k + 1] - it.r0;
  it.xoff = a.x_offsets[k];
  it.d = a.dims[k];
  it.kind = a.features[k];
  it.p = feature_count(it.d, it.kind);
  it.ridge = a.ridge[k];
  return it;
}

__device__ __forceinline__ void push_list(const RidgeLists& L, int64_t K, int cls, int k) {
  int pos = atomicAdd(&L.count[cls], 1);
  L.list[(int64_t)cls * K + pos] = k;
}

__device__ __forceinline__ void write_failed(const RidgeArgs& a, int k, int p, int32_t status,
                                             double lam, uint32_t info) {
  const double nan = __longlong_as_double(0x7ff8000000000000ll);
  for (int i = threadIdx.x; i < p; i += blockDim.x) a.beta[(int64_t)k * a.beta_stride + i] = nan;
  if (threadIdx.x == 0) {
    a.status[k] = status;
    if (a.ridge_eff) a.ridge_eff[k] = lam;
    if (a.cond) a.cond[k] = nan;
    if (a.info) a.info[k] = info;
  }
}

// Row of the lower-triangular tile grid holding linear tile index t.
__device__ __forceinline__ int tile_row(int t) {
  int I = (int)((sqrtf(8.0f * t + 1.0f) - 1.0f) * 0.5f);
  while (I * (I + 1) / 2 > t) --I;
  while ((I + 1) * (I + 2) / 2 <= t) ++I;
  return I;
}

// D (8x8, two doubles per lane) += A (8x4) * B (4x8) in FP64 on the tensor
// cores.  Lane l holds A[l/4][l%4], B[l%4][l/4] and D[l/4][2(l%4) + {0,1}].
__device__ __forceinline__ void dmma_884(double (&d)[2], double a, double b) {
  asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
      : "+d"(d[0]), "+d"(d[1])
      : "d"(a), "d"(b));
}

// Host-side launch helpers (ridge.cu / ridge_tc.cu / ridge_dmma.cu).
int launch_ridge_tensor(const RidgeArgs& a, const RidgeLists& L, cudaStream_t stream);
int launch_ridge_wide(const RidgeArgs& a, const RidgeLists& L, int cls, cudaStream_t stream);
int launch_ridge_dmma(const RidgeArgs& a, const RidgeLists& L, int cls, cudaStream_t stream);
int launch_ridge_split_finish(const RidgeArgs& a, const RidgeLists& L, cudaStream_t stream);
int ridge_dmma_ctas(int cls);
int device_sm_count();

}  // namespace art
