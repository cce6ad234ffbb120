// cdef_packed.cuh — CDEF's constrained taps (7.15.2) on two samples at once,
// exactly: in half precision for bit depths up to 10, in 16-bit integers for 12.
//
// Half precision, bit depths up to 10.
// A sample v (0 .. 1023) is held as the half 1024 + v: its bits are 0x6400 | v,
// so packing and unpacking are integer operations, and every half in
// [1024, 2048) is an integer. Two samples that take the same taps share a
// 32-bit word. Each step below is exact, or rounds once to the value the
// integer process has:
//   d   = p - x                      exact (both are integers below 2048);
//   a   = |d| - (2^adj - 1) / 2      exact (a multiple of 1/2 below 1024);
//   t   = 1024 + str - a / 2^adj     one rounding to an integer: the part of
//         |d| / 2^adj beyond its floor is moved into (-1/2, 1/2), so t is
//         1024 + str - (|d| >> adj), or below 1024 where that is negative;
//   lim = max(t - 1024, 0)           exact;
//   con = min(|d|, lim) with d's sign;
//   sum = the weighted sum of con    exact (an integer, at most 12 * 60 +
//         12 * 16 = 912 in magnitude: strengths are at most 15 << 2 and 4 << 2);
//   x + (8 + sum - (sum < 0) >> 4)   sum / 16 rounded to nearest, halves away
//         from 0: one multiply-add by 2^-4 * (1 + 2^-10), which moves every
//         half off the tie (by at least 2^-11) and no other value past one
//         (by at most 912/16 * 2^-10 < 1/16).
// The clamp to [mn, mx] then holds 1024 + the filtered sample. An unavailable
// sample is -infinity: its limit is 0 (so it adds nothing), a max never takes
// it, and a min of the bits as unsigned integers never takes it (0xfc00 is
// above every 0x6400 | v, whose order is that of v).
//
// Integers, 12 bits. A sample v is held as 4096 + v (0x1000 | v), two to a word.
//   |d| = max(p, x) - min(p, x)      no borrow between the halves;
//   lim = str - min(|d| >> adj, str) the shift's bits from the upper half
//         masked off;
//   p clamped to [x - lim, x + lim]  x plus the constrained difference; both
//         ends stay in (0, 2^15), a limit being at most 240.
// The weighted sum of those words less the weights times x is hi * 2^16 + lo of
// the two sums, at most 12 * 240 + 12 * 64 in magnitude: one 32-bit
// multiply-add a tap, whatever crosses the halves on the way. An unavailable
// sample is 0xf000: |d| >= 0xd001, and |d| >> adj is no less than str (str <<
// adj is at most 2^11), so its limit is 0; a signed max and an unsigned min
// never take it.
#pragma once

#include <cuda_fp16.h>

#include <cstdint>

#include "common.cuh"

namespace av1pf {

constexpr uint32_t kPBias = 0x64006400u;  // 1024 in both halves
constexpr uint32_t kPNA = 0xfc00fc00u;    // unavailable: -infinity in both halves

__device__ __forceinline__ __half2 as_h2(uint32_t v) { return *reinterpret_cast<__half2*>(&v); }
__device__ __forceinline__ uint32_t as_u32(__half2 v) { return *reinterpret_cast<uint32_t*>(&v); }

// Strength terms of one kind of tap, in both halves: 1024 + str, -2^-adj and
// -(2^adj - 1) / 2.
struct PStrength {
  uint32_t c, k, o;
};
__device__ __forceinline__ PStrength packed_strength(int str, int adj) {
  PStrength s;
  s.c = (0x6400u + uint32_t(str)) * 0x10001u;
  s.k = (0x8000u | (uint32_t(15 - adj) << 10)) * 0x10001u;
  s.o = as_u32(__float2half2_rn(-0.5f * float((1 << adj) - 1)));
  return s;
}

// The constrained difference of a tap at distance d under one strength. The
// clamp to [-lim, lim] keeps d's sign.
__device__ __forceinline__ __half2 packed_constrain(__half2 d, const PStrength& s) {
  const __half2 t = __hfma2(__hadd2(__habs2(d), as_h2(s.o)), as_h2(s.k), as_h2(s.c));
  const __half2 lim = __hfma2_relu(t, as_h2(0x3c003c00u), as_h2(0xe400e400u));
  return __hmax2(__hmin2(d, lim), __hneg2(lim));
}

// One tap at `p`: its constrained difference from x (nx = -x), times w, into sum.
template <bool CLAMP>
__device__ __forceinline__ void packed_tap(uint32_t p, __half2 nx, const PStrength& s, __half2 w, __half2& sum,
                                           __half2& mx, uint32_t& mn) {
  sum = __hfma2(packed_constrain(__hadd2(as_h2(p), nx), s), w, sum);
  if (CLAMP) {
    mx = __hmax2(mx, as_h2(p));
    mn = __vminu2(mn, p);  // as integers the available samples are the smaller ones
  }
}

// 1024 + x + (sum / 16 rounded to nearest, halves away from 0), x biased.
__device__ __forceinline__ __half2 packed_round(__half2 sum, __half2 x) { return __hfma2(sum, as_h2(0x2c012c01u), x); }

constexpr uint32_t kDeepBias = 0x10001000u;  // 4096 in both halves
constexpr uint32_t kDeepNA = 0xf000f000u;

// Strength terms in integers: str and the mask of |d| >> adj in both halves, adj.
__device__ __forceinline__ PStrength deep_strength(int str, int adj) {
  return PStrength{uint32_t(str) * 0x10001u, uint32_t(adj), (0xffffu >> adj) * 0x10001u};
}

template <bool CLAMP>
__device__ __forceinline__ void deep_tap(uint32_t p, uint32_t x, const PStrength& s, uint32_t w, uint32_t& sum,
                                         uint32_t& mx, uint32_t& mn) {
  const uint32_t d = __vmaxu2(p, x) - __vminu2(p, x);
  const uint32_t lim = s.c - __vminu2((d >> s.k) & s.o, s.c);
  sum += w * __vminu2(__vmaxu2(p, x - lim), x + lim);
  if (CLAMP) {
    mx = __vmaxs2(mx, p);
    mn = __vminu2(mn, p);
  }
}

// x + (8 + sum - (sum < 0) >> 4) in both halves, of the sums hi * 2^16 + lo.
__device__ __forceinline__ uint32_t deep_round(uint32_t sum, uint32_t x) {
  const int lo = int16_t(sum & 0xffffu), hi = (int(sum) - lo) >> 16;
  const int rl = (8 + lo + (lo >> 31)) >> 4, rh = (8 + hi + (hi >> 31)) >> 4;
  return x + (uint32_t(rh) << 16) + uint32_t(rl);
}

}  // namespace av1pf
