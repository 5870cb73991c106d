// Loads of a thread's own row, shared by the kernels that read x once by rows.
#pragma once
#include <cstdint>

namespace art {
namespace {

// Eight doubles x[i .. i + 8) of a row of d (zeros past its end).  vec: 4 =
// rows of whole 32-byte sectors (one 256-bit load each), 2 = of 16-byte
// pairs, 1 = single doubles.  A thread reads its own row: every load moves
// whole sectors, and a row's loads are all in flight together.
__device__ __forceinline__ void load8(const double* x, int i, int d, int vec, double (&v)[8]) {
  if (vec == 4) {
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      if (i + 4 * q < d) {
        asm volatile("ld.global.nc.v4.f64 {%0, %1, %2, %3}, [%4];"
                     : "=d"(v[4 * q]), "=d"(v[4 * q + 1]), "=d"(v[4 * q + 2]), "=d"(v[4 * q + 3])
                     : "l"(x + i + 4 * q));
      } else {
        v[4 * q] = v[4 * q + 1] = v[4 * q + 2] = v[4 * q + 3] = 0.0;
      }
    }
  } else if (vec == 2) {
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const double2 t = i + 2 * q < d ? __ldg((const double2*)(x + i + 2 * q)) : make_double2(0.0, 0.0);
      v[2 * q] = t.x;
      v[2 * q + 1] = t.y;
    }
  } else {
#pragma unroll
    for (int q = 0; q < 8; ++q) v[q] = i + q < d ? __ldg(x + i + q) : 0.0;
  }
}
__device__ __forceinline__ int row_vec(const double* x, int d) {
  const uintptr_t at = (uintptr_t)x;
  return (d & 3) == 0 && (at & 31) == 0 ? 4 : ((d & 1) == 0 && (at & 15) == 0 ? 2 : 1);
}

}  // namespace
}  // namespace art
