// cdef_search.cuh — what the two error-table kernels of the encoder's CDEF
// search share (cdef.cu for 12 bits, cdef_packed.cu for up to 10).
#pragma once

#include <cstdint>

#include "common.cuh"

namespace av1pf {

// Sum of a u32 over the warp, exactly (two 16-bit halves, so no lane sum
// overflows).
__device__ __forceinline__ uint64_t warp_sum_u32(uint32_t v) {
  const uint32_t lo = __reduce_add_sync(0xffffffffu, v & 0xffffu);
  const uint32_t hi = __reduce_add_sync(0xffffffffu, v >> 16);
  return (uint64_t(hi) << 16) + lo;
}

// The search's candidate strengths (encoder/cdef.rs:60-80): primaries of
// the fast and thorough lists, secondaries decoded (coded 3 is 4).
__host__ __device__ constexpr int search_y_pri(bool th, int i) {
  constexpr int f[7] = {0, 1, 2, 4, 6, 9, 12}, t[11] = {0, 1, 2, 3, 4, 5, 6, 8, 10, 12, 15};
  return th ? t[i] : f[i];
}
__host__ __device__ constexpr int search_uv_pri(bool th, int i) {
  constexpr int f[5] = {0, 1, 2, 4, 7}, t[8] = {0, 1, 2, 3, 4, 6, 8, 11};
  return th ? t[i] : f[i];
}
__host__ __device__ constexpr int search_sec(int j) { return j == 3 ? 4 : j; }

// The frame whose blocks CTA `cta` of a launch over n frames takes: the last
// whose first block is at or before it.
__device__ __forceinline__ int search_frame(const CdefSearchDesc* ds, int n, int cta) {
  int fi = 0;
  for (int hi = n - 1; fi < hi;) {
    const int mid = (fi + hi + 1) >> 1;
    if (ds[mid].block0 <= cta)
      fi = mid;
    else
      hi = mid - 1;
  }
  return fi;
}

}  // namespace av1pf
