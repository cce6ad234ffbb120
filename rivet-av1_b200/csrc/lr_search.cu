// lr_search.cu — the encoder's loop-restoration search on the device
// (encoder/lr.rs:64-430): per restoration unit, the error of no filter, of
// a Wiener filter fitted to the source and of a self-guided filter fitted
// for each parameter set, priced with lambda; the cheapest is the unit's
// choice.
//
// One CTA per unit (per unit and two parameter sets for the self-guided
// fits). Each of the unit's stripe rectangles is staged as the decoder's
// restoration window (postfilter.rs:765-777: clamped to the plane, rows beyond
// the stripe from the deblocked frame) in shared memory.
//
// Exactness. The reference fits in f64, summing over the unit's samples in
// row-major order. Sums whose terms are integers (the first Wiener pass,
// whose lines are plain samples, and the self-guided fit, whose terms are
// products of filter outputs and samples) are exact in any order while the
// sum of the terms' magnitudes stays below 2^53: they are summed in int64
// in parallel (the self-guided sums check that bound and otherwise redo the
// sum in order on one thread). The second and third Wiener passes have
// real-valued terms, so their sums run in the reference's order: warps 1-3
// produce four rows of terms at a time into shared memory while lanes of
// warp 0 each add one accumulator's terms in sample order. Every f64 operation is a
// round-to-nearest multiply, add or divide in the reference's order (this
// file is compiled without floating-point contraction, and the sums use
// the explicit _rn intrinsics).
#include <cfloat>
#include <type_traits>

#include "av1_tables.h"
#include "common.cuh"
#include "kernels.h"
#include "lr_walk.cuh"

namespace av1pf {

namespace {

constexpr int kB = 3;            // window border (postfilter.rs:744 LRB)
constexpr int kThreads = 256;
constexpr int kWienerChunk = 4;  // rows of Wiener terms handed from the producing warps to the adding lanes at a time
constexpr int kWienerErrBand = 32;  // output rows per band of the Wiener error pass (its int16 rows fit the term region)
__constant__ int32_t kSgrParams[16][4] = AV1T_SGR_PARAMS;
__constant__ int32_t kWienerMin[3] = AV1T_WIENER_TAPS_MIN, kWienerMax[3] = AV1T_WIENER_TAPS_MAX;
__constant__ int32_t kXqdMin[2] = AV1T_SGRPROJ_XQD_MIN, kXqdMax[2] = AV1T_SGRPROJ_XQD_MAX;

__device__ __forceinline__ int ld(const DPlane& p, int sb, int x, int y) { return ld_sample(p, sb, x, y); }

// f64 -> i32 as Rust's `as` converts: saturating, NaN to 0.
__device__ __forceinline__ int32_t f64_to_i32(double x) {
  if (isnan(x)) return 0;
  if (x <= -2147483648.0) return INT32_MIN;
  if (x >= 2147483647.0) return INT32_MAX;
  return int32_t(x);
}

struct Win {
  const int16_t* w;
  int ws;  // row stride
  __device__ __forceinline__ int at(int r, int c) const { return w[r * ws + c]; }
};

// lr_window (postfilter.rs:765-777) of rectangle `rc` into shared memory.
__device__ void stage_window(const LrSearchFrame& d, int p, const LrSearchRect& rc, int x0, int w, int16_t* win,
                             int ws) {
  // a warp per window row, lanes along it (no index division), eight rows'
  // loads in flight before their stores
  constexpr int kR = 8;
  const int ww = w + 2 * kB, wh = rc.h + 2 * kB, nw = blockDim.x >> 5, lane = threadIdx.x & 31;
  const int pex = d.pex[p], pey = d.pey[p];
  for (int r0 = threadIdx.x >> 5; r0 < wh; r0 += kR * nw) {
    for (int c = lane; c < ww; c += 32) {
      int v[kR];
#pragma unroll
      for (int m = 0; m < kR; m++) {
        const int r = r0 + m * nw;
        v[m] = 0;
        if (r < wh) {
          const int y = max(min(rc.y0 + r - kB, pey), 0);
          const DPlane& pl = y < rc.ss || y > rc.se ? d.cur[p] : d.cdef[p];
          const int yy = y < rc.ss ? max(rc.ss - 2, y) : (y > rc.se ? min(rc.se + 2, y) : y);
          v[m] = ld(pl, d.sb, max(min(x0 + c - kB, pex), 0), yy);
        }
      }
#pragma unroll
      for (int m = 0; m < kR; m++) {
        const int r = r0 + m * nw;
        if (r < wh) win[r * ws + c] = int16_t(v[m]);
      }
    }
  }
}

// Block sums of N 64-bit values in one round (every thread gets the totals).
template <int N>
__device__ void block_sums_i64(int64_t (&v)[N], int64_t (*red)[kThreads / 32]) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
#pragma unroll
  for (int q = 0; q < N; q++) {
#pragma unroll
    for (int o = 16; o; o >>= 1) v[q] += __shfl_xor_sync(0xffffffffu, v[q], o);
    if (lane == 0) red[q][warp] = v[q];
  }
  __syncthreads();
#pragma unroll
  for (int q = 0; q < N; q++) {
    int64_t t = 0;
    for (int k = 0; k < nw; k++) t += red[q][k];
    v[q] = t;
  }
}

// Gaussian elimination with partial pivoting (encoder/lr.rs:212-233): the
// last row of largest magnitude is the pivot (Iterator::max_by); zeros when
// singular.
template <int N>
__device__ __noinline__ void solve(double (&m)[N][N], double (&v)[N], double (&x)[N]) {
  for (int i = 0; i < N; i++) {
    int piv = i;
    for (int a = i + 1; a < N; a++)
      if (!(fabs(m[a][i]) < fabs(m[piv][i]))) piv = a;
    for (int c = 0; c < N; c++) {
      const double t = m[i][c];
      m[i][c] = m[piv][c];
      m[piv][c] = t;
    }
    const double tv = v[i];
    v[i] = v[piv];
    v[piv] = tv;
    if (fabs(m[i][i]) < 1e-9) {
      for (int k = 0; k < N; k++) x[k] = 0.0;
      return;
    }
    for (int r = 0; r < N; r++) {
      if (r != i) {
        const double f = __ddiv_rn(m[r][i], m[i][i]);
        for (int c = i; c < N; c++) m[r][c] = __dsub_rn(m[r][c], __dmul_rn(f, m[i][c]));
        v[r] = __dsub_rn(v[r], __dmul_rn(f, v[i]));
      }
    }
  }
  for (int i = 0; i < N; i++) x[i] = __ddiv_rn(v[i], m[i][i]);
}

// The 7 samples of a Wiener line at (i, j) with the other direction's
// filter applied first (encoder/lr.rs:265-285); the line's taps run along
// columns (vertical) or rows.
__device__ __forceinline__ void wiener_line(const Win& W, bool vertical, int i, int j, const double* other,
                                            double (&line)[7]) {
#pragma unroll
  for (int t = 0; t < 7; t++) {
    const int r = vertical ? i + t : i + kB, c = vertical ? j + kB : j + t;
    const int center = W.at(r, c);
    double s = double(center);
#pragma unroll
    for (int k = 0; k < 3; k++) {
      const int dd = 3 - k;
      const int a = vertical ? W.at(r, c - dd) : W.at(r - dd, c);
      const int b = vertical ? W.at(r, c + dd) : W.at(r + dd, c);
      // a + b - 2 * center is an integer below 2^17: the f64 expression of
      // encoder/lr.rs is exact, so integer arithmetic gives the same value
      s = __dadd_rn(s, __dmul_rn(other[k], double(a + b - 2 * center)));
    }
    line[t] = s;
  }
}

// The window of a rectangle, read from the planes: row r, column c.
struct PlaneWin {
  const LrSearchFrame& F;
  const LrSearchRect& rc;
  int p, x0;
  __device__ int at(int r, int c) const {
    const int x = max(min(x0 + c - kB, F.pex[p]), 0), y = max(min(rc.y0 + r - kB, F.pey[p]), 0);
    return y < rc.ss   ? ld(F.cur[p], F.sb, x, max(rc.ss - 2, y))
           : y > rc.se ? ld(F.cur[p], F.sb, x, min(rc.se + 2, y))
                       : ld(F.cdef[p], F.sb, x, y);
  }
};

// One self-guided A/B pair (postfilter.rs:918-948) at A/B position (ai, aj)
// of the rectangle (window position ai + 2, aj + 2).
__device__ __forceinline__ void sgr_ab(const PlaneWin& W, int ai, int aj, int r, int n, int s, int one_over_n, int bd,
                                       int32_t& A, int32_t& B) {
  const int wy = ai + kB - 1, wx = aj + kB - 1;
  int32_t bs = 0;
  int64_t as = 0;
  for (int dy = -r; dy <= r; dy++)
    for (int dx = -r; dx <= r; dx++) {
      const int v = W.at(wy + dy, wx + dx);
      bs += v;
      as += int64_t(v) * v;
    }
  const int64_t a = round2_64(as, 2 * (bd - 8));
  const int64_t dd = round2(bs, bd - 8);
  const int64_t p = max(a * n - dd * dd, int64_t(0));
  const int64_t z = round2_64(p * s, 20);  // SGRPROJ_MTABLE_BITS
  const int zc = int(min(z, int64_t(255)));
  const int32_t a2 = zc >= 255 ? 256 : (zc == 0 ? 1 : ((zc << 8) + zc / 2) / (zc + 1));
  const int64_t b2 = int64_t(256 - a2) * int64_t(bs) * int64_t(one_over_n);
  A = a2;
  B = int32_t(round2_64(b2, 12));  // SGRPROJ_RECIP_BITS
}

struct SgrPass {
  int r, n, s, one_over_n;
};

__device__ __forceinline__ SgrPass sgr_pass(int set, int pass) {
  SgrPass q;
  q.r = kSgrParams[set][pass * 2];
  const int eps = kSgrParams[set][pass * 2 + 1];
  q.n = (2 * q.r + 1) * (2 * q.r + 1);
  const int n2e = q.n * q.n * eps;
  q.s = q.r ? ((1 << 20) + n2e / 2) / n2e : 0;
  q.one_over_n = ((1 << 12) + q.n / 2) / q.n;
  return q;
}

// A self-guided filter output (postfilter.rs:950-988) at (i, j), its A/B
// computed on the spot (the in-order fallback).
__device__ int32_t sgr_flt_direct(const PlaneWin& W, int pass, const SgrPass& q, int bd, int yabs, int i, int j, int cval) {
  int32_t a = 0, b = 0;
  for (int dy = -1; dy <= 1; dy++)
    for (int dx = -1; dx <= 1; dx++) {
      int wgt;
      if (pass == 0)
        wgt = ((yabs + dy) & 1) ? (dx == 0 ? 6 : 5) : 0;
      else
        wgt = (dx == 0 || dy == 0) ? 4 : 3;
      if (wgt) {
        int32_t A, B;
        sgr_ab(W, i + 1 + dy, j + 1 + dx, q.r, q.n, q.s, q.one_over_n, bd, A, B);
        a += wgt * A;
        b += wgt * B;
      }
    }
  const int shift = (pass == 0 && (yabs & 1)) ? 4 : 5;
  return round2(a * cval + b, 8 + shift - 4);
}

}  // namespace

// Shared memory of the first-pass kernel (kind 0: the window) and of the Wiener
// kernel (1: the window and the term rows).
size_t lr_search_smem(int wmax, int hmax, int kind) {
  const size_t ws = size_t(wmax + 2 * kB + 1) & ~size_t(1);
  const size_t win = ((size_t(hmax + 2 * kB) * ws * 2) + 15) & ~size_t(15);
  return kind == 0 ? win : win + size_t(2) * 4 * kWienerChunk * size_t(wmax + 1) * sizeof(double);
}

namespace {

// Window stride and the region after the window.
struct Smem {
  int16_t* win;
  int ws;
  uint8_t* region;
};
__device__ __forceinline__ Smem smem_of(uint8_t* base, const LrSearchDesc& d) {
  Smem m;
  m.ws = (d.wmax + 2 * kB + 1) & ~1;
  m.win = reinterpret_cast<int16_t*>(base);
  m.region = base + ((((size_t(d.hmax + 2 * kB) * m.ws * 2) + 15) & ~size_t(15)));
  return m;
}

}  // namespace

// For units of several stripe rectangles, one CTA per unit (256 threads):
// the error without a filter (encoder/lr.rs:134-146), and the first Wiener
// pass (vertical, the other direction's filter still zero: its lines are
// plain samples, so its sums are exact integer sums in any order) and its
// solve. A one-rectangle unit's Wiener CTA does this itself, on the window
// it keeps for its other passes.
__global__ void __launch_bounds__(kThreads, 2) lr_search_prep_kernel(const LrSearchDesc d) {
  extern __shared__ __align__(16) uint8_t lrs_smem[];
  __shared__ int64_t red10[10][kThreads / 32];
  const LrSearchJob job = d.jobs[blockIdx.x];
  if (job.nr == 1) return;
  const LrSearchFrame& F = d.frames[job.frame];
  const int p = job.plane, x0 = job.x0, w = job.w, sb = F.sb, tid = threadIdx.x, step = d.step;
  const Smem sm = smem_of(lrs_smem, d);
  const Win W{sm.win, sm.ws};
  const LrSearchRect* rects = d.rects + job.r0;
  LrJobState& st = d.state[blockIdx.x];
  int64_t acc = 0, m00 = 0, m01 = 0, m02 = 0, m11 = 0, m12 = 0, m22 = 0, v0 = 0, v1 = 0, v2 = 0;
  const int nci = (w + step - 1) / step;
  for (int ri = 0; ri < job.nr; ri++) {
    const LrSearchRect rc = rects[ri];
    __syncthreads();
    stage_window(F, p, rc, x0, w, sm.win, sm.ws);
    __syncthreads();
    // no filter: the window's interior is the rectangle's CDEF output (its
    // rows lie in its stripe, its columns in the plane)
    for (int i = tid >> 5; i < rc.h; i += blockDim.x >> 5)
      for (int j = tid & 31; j < w; j += 32) {
        const int e = W.at(i + kB, j + kB) - ld(F.src[p], sb, x0 + j, rc.y0 + i);
        acc += int64_t(e) * e;
      }
    const int nri = (rc.h + step - 1) / step;
    for (int ii = tid >> 5; ii < nri; ii += blockDim.x >> 5)
      for (int jj = tid & 31; jj < nci; jj += 32) {
      const int i = ii * step, j = jj * step;
      int ln[7];
#pragma unroll
      for (int t = 0; t < 7; t++) ln[t] = W.at(i + t, j + kB);
      const int64_t tg = ld(F.src[p], sb, x0 + j, rc.y0 + i) - ln[3];
      const int64_t d0 = ln[0] + ln[6] - 2 * ln[3], d1 = ln[1] + ln[5] - 2 * ln[3], d2 = ln[2] + ln[4] - 2 * ln[3];
      m00 += d0 * d0;
      m01 += d0 * d1;
      m02 += d0 * d2;
      m11 += d1 * d1;
      m12 += d1 * d2;
      m22 += d2 * d2;
      v0 += d0 * tg;
      v1 += d1 * tg;
      v2 += d2 * tg;
      }
  }
  int64_t sums[10] = {m00, m01, m02, m11, m12, m22, v0, v1, v2, acc};
  block_sums_i64(sums, red10);
  double tot[9];
#pragma unroll
  for (int q = 0; q < 9; q++) tot[q] = double(sums[q]);
  if (tid == 0) {
    st.none = uint64_t(sums[9]);
    double sol[3] = {0.0, 0.0, 0.0};
    if (p == 0) {
      double m[3][3] = {{tot[0], tot[1], tot[2]}, {tot[1], tot[3], tot[4]}, {tot[2], tot[4], tot[5]}};
      double v[3] = {tot[6], tot[7], tot[8]};
      solve<3>(m, v, sol);
    } else {
      double m[2][2] = {{tot[3], tot[4]}, {tot[4], tot[5]}}, v[2] = {tot[7], tot[8]}, x2[2];
      solve<2>(m, v, x2);
      sol[1] = x2[0];
      sol[2] = x2[1];
    }
    for (int k = 0; k < 3; k++) st.vc[k] = sol[k];
  }
}

// One CTA per unit (128 threads). For a one-rectangle unit, first the error
// without a filter and the first Wiener pass and its solve, as the kernel
// above does for the others. Then the second
// (horizontal) and third (vertical) Wiener passes, whose terms are
// real-valued, so each of their sums runs in the reference's sample order:
// warps 1-3 produce four rows of terms into shared memory (two buffers)
// while lane q of warp 0 adds accumulator q's terms (m00 m01 m02 m11 m12 m22
// v0 v1 v2). Then the solves, the quantised coefficients
// (encoder/lr.rs:316-327) and the filter's error.
__global__ void __launch_bounds__(128, 4) lr_search_wiener_kernel(const LrSearchDesc d) {
  extern __shared__ __align__(16) uint8_t lrs_smem[];
  __shared__ int64_t red[4];
  __shared__ int64_t red10[10][kThreads / 32];
  __shared__ double s_m[3][3], s_v[3], s_other[3], s_vc[3];
  __shared__ int s_coef[2][3];
  const LrSearchJob job = d.jobs[blockIdx.x];
  const LrSearchFrame& F = d.frames[job.frame];
  const int p = job.plane, x0 = job.x0, w = job.w, sb = F.sb, tid = threadIdx.x, step = d.step;
  const int lane = tid & 31, warp = tid >> 5;
  const Smem sm = smem_of(lrs_smem, d);
  const Win W{sm.win, sm.ws};
  const LrSearchRect* rects = d.rects + job.r0;
  LrJobState& st = d.state[blockIdx.x];
  const int first = p == 0 ? 0 : 1;
  const int bd = F.bd, maxv = (1 << bd) - 1;
  const int nci = (w + step - 1) / step;
  if (job.nr == 1) {  // the no-filter error and the first pass (CTA-uniform)
    int64_t acc = 0, m00 = 0, m01 = 0, m02 = 0, m11 = 0, m12 = 0, m22 = 0, v0 = 0, v1 = 0, v2 = 0;
    for (int ri = 0; ri < job.nr; ri++) {
      const LrSearchRect rc = rects[ri];
      __syncthreads();
      stage_window(F, p, rc, x0, w, sm.win, sm.ws);
      __syncthreads();
      // no filter: the window's interior is the rectangle's CDEF output (its
      // rows lie in its stripe, its columns in the plane)
      for (int i = tid >> 5; i < rc.h; i += blockDim.x >> 5)
        for (int j = tid & 31; j < w; j += 32) {
          const int e = W.at(i + kB, j + kB) - ld(F.src[p], sb, x0 + j, rc.y0 + i);
          acc += int64_t(e) * e;
        }
      const int nri = (rc.h + step - 1) / step;
      for (int ii = tid >> 5; ii < nri; ii += blockDim.x >> 5)
        for (int jj = tid & 31; jj < nci; jj += 32) {
        const int i = ii * step, j = jj * step;
        int ln[7];
#pragma unroll
        for (int t = 0; t < 7; t++) ln[t] = W.at(i + t, j + kB);
        const int64_t tg = ld(F.src[p], sb, x0 + j, rc.y0 + i) - ln[3];
        const int64_t d0 = ln[0] + ln[6] - 2 * ln[3], d1 = ln[1] + ln[5] - 2 * ln[3], d2 = ln[2] + ln[4] - 2 * ln[3];
        m00 += d0 * d0;
        m01 += d0 * d1;
        m02 += d0 * d2;
        m11 += d1 * d1;
        m12 += d1 * d2;
        m22 += d2 * d2;
        v0 += d0 * tg;
        v1 += d1 * tg;
        v2 += d2 * tg;
        }
    }
    int64_t sums[10] = {m00, m01, m02, m11, m12, m22, v0, v1, v2, acc};
    block_sums_i64(sums, red10);
    if (tid == 0) {
      st.none = uint64_t(sums[9]);
      double sol[3] = {0.0, 0.0, 0.0};
      const double tot[9] = {double(sums[0]), double(sums[1]), double(sums[2]), double(sums[3]), double(sums[4]),
                             double(sums[5]), double(sums[6]), double(sums[7]), double(sums[8])};
      if (p == 0) {
        double m[3][3] = {{tot[0], tot[1], tot[2]}, {tot[1], tot[3], tot[4]}, {tot[2], tot[4], tot[5]}};
        double v[3] = {tot[6], tot[7], tot[8]};
        solve<3>(m, v, sol);
      } else {
        double m[2][2] = {{tot[3], tot[4]}, {tot[4], tot[5]}}, v[2] = {tot[7], tot[8]}, x2[2];
        solve<2>(m, v, x2);
        sol[1] = x2[0];
        sol[2] = x2[1];
      }
      for (int k = 0; k < 3; k++) s_vc[k] = sol[k];
    }
  } else if (tid < 3) {
    s_vc[tid] = st.vc[tid];  // from the kernel above
  }
  __syncthreads();
  double vc[3] = {s_vc[0], s_vc[1], s_vc[2]}, hc[3] = {0.0, 0.0, 0.0};
  const int qa = lane < 6 ? (lane < 3 ? 0 : (lane < 5 ? 1 : 2)) : lane - 6;
  const int qb = lane < 6 ? (lane < 3 ? lane : (lane < 5 ? lane - 2 : 2)) : 3;  // 3: the target
  const bool owner = warp == 0 && lane < 9 && qa >= first && (qb == 3 || qb >= first);
  // [2 buffers][4 terms: d0 d1 d2 t][kWienerChunk rows][wmax + 1]: the odd
  // row stride puts the four terms of a sample on different banks for the
  // accumulating lanes
  double* terms = reinterpret_cast<double*>(sm.region);
  const int ts = d.wmax + 1, tq_stride = kWienerChunk * ts;
  for (int iter = 1; iter < 3; iter++) {
    const bool vertical = iter == 2;
    if (tid < 3) s_other[tid] = vertical ? hc[tid] : vc[tid];
    double macc = 0.0;
    for (int ri = 0; ri < job.nr; ri++) {
      const LrSearchRect rc = rects[ri];
      __syncthreads();
      // one rectangle: its window, staged for the first pass, stays in place
      // (the term rows and band rows lie outside it)
      if (job.nr > 1) stage_window(F, p, rc, x0, w, sm.win, sm.ws);
      __syncthreads();
      const int nri = (rc.h + step - 1) / step, nch = (nri + kWienerChunk - 1) / kWienerChunk;
      // chunks of rows in turn, two buffers: warps 1.. fill chunk c + 1 while
      // warp 0 adds chunk c, row by row in sample order
      for (int ch = 0; ch <= nch; ch++) {
        if (ch < nch && warp > 0) {
          double* tb = terms + (ch & 1) * 4 * tq_stride;
          const int rows = min(kWienerChunk, nri - ch * kWienerChunk);
          const double oth[3] = {s_other[0], s_other[1], s_other[2]};
          for (int k = tid - 32; k < rows * nci; k += blockDim.x - 32) {
            const int r = k / nci, jj = k - r * nci;
            const int i = (ch * kWienerChunk + r) * step, j = jj * step;
            double line[7];
            wiener_line(W, vertical, i, j, oth, line);
            const double two3 = __dmul_rn(2.0, line[3]);
            double* tr = tb + r * ts + jj;
            tr[0 * tq_stride] = __dsub_rn(__dadd_rn(line[0], line[6]), two3);
            tr[1 * tq_stride] = __dsub_rn(__dadd_rn(line[1], line[5]), two3);
            tr[2 * tq_stride] = __dsub_rn(__dadd_rn(line[2], line[4]), two3);
            tr[3 * tq_stride] = __dsub_rn(double(ld(F.src[p], sb, x0 + j, rc.y0 + i)), line[3]);
          }
        }
        if (ch > 0 && owner) {
          const double* tb = terms + ((ch - 1) & 1) * 4 * tq_stride;
          const int rows = min(kWienerChunk, nri - (ch - 1) * kWienerChunk);
          for (int r = 0; r < rows; r++) {
            const double* ta = tb + qa * tq_stride + r * ts;
            const double* tq = tb + qb * tq_stride + r * ts;
            // the products of 8 terms are independent of the sum: form them
            // first, then add them one after another in sample order
            int jj = 0;
            for (; jj + 8 <= nci; jj += 8) {
              double pr[8];
#pragma unroll
              for (int u = 0; u < 8; u++) pr[u] = __dmul_rn(ta[jj + u], tq[jj + u]);
#pragma unroll
              for (int u = 0; u < 8; u++) macc = __dadd_rn(macc, pr[u]);
            }
            for (; jj < nci; jj++) macc = __dadd_rn(macc, __dmul_rn(ta[jj], tq[jj]));
          }
        }
        __syncthreads();
      }
    }
    if (owner) {
      if (qb == 3)
        s_v[qa] = macc;
      else
        s_m[qa][qb] = s_m[qb][qa] = macc;
    }
    __syncthreads();
    if (tid == 0) {
      double sol[3] = {0.0, 0.0, 0.0};
      if (first == 0) {
        double m[3][3], v[3];
        for (int a = 0; a < 3; a++) {
          v[a] = s_v[a];
          for (int b = 0; b < 3; b++) m[a][b] = s_m[a][b];
        }
        solve<3>(m, v, sol);
      } else {
        double m[2][2] = {{s_m[1][1], s_m[1][2]}, {s_m[2][1], s_m[2][2]}}, v[2] = {s_v[1], s_v[2]}, x2[2];
        solve<2>(m, v, x2);
        sol[1] = x2[0];
        sol[2] = x2[1];
      }
      for (int k = 0; k < 3; k++) s_other[k] = sol[k];  // the pass's solution
    }
    __syncthreads();
    for (int k = 0; k < 3; k++) (vertical ? vc : hc)[k] = s_other[k];
    __syncthreads();
  }
  if (tid == 0) {
    for (int k = 0; k < 3; k++) {
      s_coef[0][k] = k < first ? 0 : min(max(f64_to_i32(round(vc[k] * 128.0)), kWienerMin[k]), kWienerMax[k]);
      s_coef[1][k] = k < first ? 0 : min(max(f64_to_i32(round(hc[k] * 128.0)), kWienerMin[k]), kWienerMax[k]);
    }
  }
  __syncthreads();
  // the Wiener filter's error (postfilter.rs:781-822 restoration)
  int vf[7], hf[7];
  vf[3] = hf[3] = 128;
  for (int k = 0; k < 3; k++) {
    vf[k] = vf[6 - k] = s_coef[0][k];
    hf[k] = hf[6 - k] = s_coef[1][k];
    vf[3] -= 2 * s_coef[0][k];
    hf[3] -= 2 * s_coef[1][k];
  }
  const int round0 = bd == 12 ? 5 : 3, round1 = bd == 12 ? 9 : 11;
  const int off = 1 << (bd + 7 - round0 - 1), lim = (1 << (bd + 1 + 7 - round0)) - 1;
  // separable: each band's horizontally filtered window rows go to the term
  // region as int16 (clipped to [-off, lim - off], within [-2^13, 2^15)),
  // then the vertical taps run over them
  int16_t* hrow = reinterpret_cast<int16_t*>(sm.region);
  const int nw = blockDim.x >> 5;
  int64_t acc = 0;
  for (int ri = 0; ri < job.nr; ri++) {
    const LrSearchRect rc = rects[ri];
    __syncthreads();
    if (job.nr > 1) stage_window(F, p, rc, x0, w, sm.win, sm.ws);  // else still staged
    for (int i0 = 0; i0 < rc.h; i0 += kWienerErrBand) {
      const int rows = min(kWienerErrBand, rc.h - i0);
      __syncthreads();  // the window is staged; the previous band's rows are read
      for (int r = warp; r < rows + 2 * kB; r += nw)
        for (int j = lane; j < w; j += 32) {
          int h = 0;
#pragma unroll
          for (int u = 0; u < 7; u++) h += hf[u] * W.at(i0 + r, j + u);
          hrow[r * w + j] = int16_t(clip3(-off, lim - off, round2(h, round0)));
        }
      __syncthreads();
      for (int ir = warp; ir < rows; ir += nw)
        for (int j = lane; j < w; j += 32) {
          int sv = 0;
#pragma unroll
          for (int t = 0; t < 7; t++) sv += vf[t] * hrow[(ir + t) * w + j];
          const int e = min(max(round2(sv, round1), 0), maxv) - ld(F.src[p], sb, x0 + j, rc.y0 + i0 + ir);
          acc += int64_t(e) * e;
        }
    }
  }
#pragma unroll
  for (int o = 16; o; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
  if (lane == 0) red[warp] = acc;
  __syncthreads();
  if (tid == 0) {
    st.wiener = uint64_t(red[0] + red[1] + red[2] + red[3]);
    for (int a = 0; a < 2; a++)
      for (int b = 0; b < 3; b++) st.coef[a][b] = s_coef[a][b];
  }
}

// The self-guided fit's f64 sums in the reference's sample order, on one
// thread (rare: very large units with large errors at 12 bits, where the
// exact integer sums could round differently), from the planes.
__device__ __noinline__ void sgr_fit_in_order(const LrSearchDesc& d, const LrSearchFrame& F, const LrSearchJob& job,
                                              const LrSearchRect* rects, const SgrPass& q0, const SgrPass& q1,
                                              double& m00, double& m01, double& m11, double& v0, double& v1) {
  const int p = job.plane, x0 = job.x0, w = job.w, sb = F.sb, step = d.step, bd = F.bd;
  const int r0 = q0.r, r1 = q1.r;
  m00 = m01 = m11 = v0 = v1 = 0.0;
  for (int ri = 0; ri < job.nr; ri++) {
    const LrSearchRect rc = rects[ri];
    const PlaneWin W{F, rc, p, x0};
    for (int i = 0; i < rc.h; i += step)
      for (int j = 0; j < w; j += step) {
        const int yabs = rc.y0 + i;
        const int cval = ld(F.cdef[p], sb, x0 + j, yabs);
        const double u = double(cval << 4);
        const double a = r0 ? __dsub_rn(double(sgr_flt_direct(W, 0, q0, bd, yabs, i, j, cval)), u) : 0.0;
        const double b = r1 ? __dsub_rn(double(sgr_flt_direct(W, 1, q1, bd, yabs, i, j, cval)), u) : 0.0;
        const double t = __dmul_rn(128.0, __dsub_rn(double(ld(F.src[p], sb, x0 + j, yabs) << 4), u));
        m00 = __dadd_rn(m00, __dmul_rn(a, a));
        m01 = __dadd_rn(m01, __dmul_rn(a, b));
        m11 = __dadd_rn(m11, __dmul_rn(b, b));
        v0 = __dadd_rn(v0, __dmul_rn(a, t));
        v1 = __dadd_rn(v1, __dmul_rn(b, t));
      }
  }
}

namespace {

// The self-guided fits' shared memory: a strip's window, its source samples and
// both filters' outputs less the sample (int16 pairs up to 10 bits, where they
// stay below 2^15; else int32 pairs) of up to two sets.
constexpr int kStrip = 64;
constexpr int kStripPx = kStrip * kMaxH;
constexpr int kSgrSrcOff = kWinBytes, kSgrCacheOff = kSgrSrcOff + kStripPx * 2;
static_assert(kSgrSrcOff % 16 == 0, "vector access");

struct SgrSums {  // of a warp: a = first filter - sample, b = second filter - sample, t = source - sample
  int64_t aa, ab, bb, at, bt, tt;
};

__device__ __forceinline__ int64_t warp_sum_i64(int64_t v) {
#pragma unroll
  for (int o = 16; o; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// The lane's part of a strip: columns c, c + 1 (`cols` of them inside) of rows
// i0 .. i0 + left - 1; `per` rows are walked.
struct SgrLane {
  int i0, per, left, c, cols, ws;
  const uint16_t *win, *src;  // window row 0 at column c; source row 0 at column c
};

// Both filters of a set over a lane's samples: their outputs less the sample to
// `cache`, and the fit's sums added to `sum` by the warp's first lane. step:
// every step-th row and column is fitted (1 or 2).
template <bool DEEP>
__device__ __forceinline__ void sgr_fit_strip(const SgrLane& g, int set, int step, int bd, GroupEdges& edges, int gl, int gn,
                                              uint8_t* cache, SgrSums* sum) {
  using Cross = typename std::conditional<DEEP, int64_t, int32_t>::type;  // 32 products below 2^24, or below 2^28
  const int r0 = kSgrParams[set][0], r1 = kSgrParams[set][2];
  const int k0 = r0 ? 16 : 0, k1 = r1 ? 16 : 0;
  int64_t aa = 0, ab = 0, bb = 0;
  Cross at = 0, bt = 0;
  uint32_t tt = 0;  // (32 squares below 2^24)
  auto fit = [&](int a, int b, int t) {
    aa += int64_t(a) * a;
    ab += int64_t(a) * b;
    bb += int64_t(b) * b;
    at += Cross(a) * t;
    bt += Cross(b) * t;
    tt += uint32_t(t * t);
  };
  int i = 0;
  const uint16_t* sp = g.src + g.i0 * kStrip;
  uint8_t* cp = cache + (g.i0 * kStrip + g.c) * (DEEP ? 8 : 4);
  sgr_walk<DEEP>(g.win, g.ws, g.c, g.i0, g.per, r0, r1, c_lr.s12[set][0], c_lr.s12[set][1], bd - 8, edges, gl, gn,
                 [&](uint32_t ca, uint32_t cb, int f0a, int f0b, int f1a, int f1b) {
                   if (i < g.left) {
                     const uint32_t s = *reinterpret_cast<const uint32_t*>(sp);
                     const int aa0 = f0a - int(ca) * k0, ba0 = f1a - int(ca) * k1;
                     const int ab0 = f0b - int(cb) * k0, bb0 = f1b - int(cb) * k1;
                     if (DEEP)
                       *reinterpret_cast<int4*>(cp) = make_int4(aa0, ba0, ab0, bb0);
                     else
                       *reinterpret_cast<uint2*>(cp) = make_uint2(__byte_perm(uint32_t(aa0), uint32_t(ba0), 0x5410),
                                                                  __byte_perm(uint32_t(ab0), uint32_t(bb0), 0x5410));
                     if (step == 1 || !(i & 1)) {
                       fit(aa0, ba0, int(s & 0xffffu) - int(ca));
                       if (step == 1 && g.cols > 1) fit(ab0, bb0, int(s >> 16) - int(cb));
                     }
                   }
                   i++;
                   sp += kStrip;
                   cp += kStrip * (DEEP ? 8 : 4);
                 });
  const int64_t taa = warp_sum_i64(aa), tab = warp_sum_i64(ab), tbb = warp_sum_i64(bb);
  const int64_t tat = warp_sum_i64(int64_t(at)), tbt = warp_sum_i64(int64_t(bt)), ttt = warp_sum_i64(int64_t(tt));
  if ((threadIdx.x & 31) == 0) {
    sum->aa += taa;
    sum->ab += tab;
    sum->bb += tbb;
    sum->at += tat;
    sum->bt += tbt;
    sum->tt += ttt;
  }
}

// The squared error of the lane's samples restored with weights w0, w2 from the
// outputs that sgr_fit_strip kept: the sample, which the two weights' rest to 128
// goes to, plus the weighted differences (postfilter.rs:836-850).
template <bool DEEP>
__device__ __forceinline__ uint32_t sgr_error_strip(const SgrLane& g, int w0, int w2, int maxv, const uint8_t* cache) {
  uint32_t acc = 0;  // (32 squares below 2^24)
  const uint16_t* wp = g.win + (g.i0 + 3) * g.ws + 2;  // samples (c - 1, c), (c + 1, ..)
  const uint16_t* sp = g.src + g.i0 * kStrip;
  const uint8_t* cp = cache + (g.i0 * kStrip + g.c) * (DEEP ? 8 : 4);
  auto error = [&](int c, int a, int b, int s) {
    const int e = clip3(0, maxv, c + ((w0 * a + w2 * b + (1 << 10)) >> 11)) - s;
    return uint32_t(e * e);
  };
#pragma unroll 2
  for (int i = 0; i < g.left; i++) {
    const int ca = int(*reinterpret_cast<const uint32_t*>(wp) >> 16), cb = int(*reinterpret_cast<const uint32_t*>(wp + 2) & 0xffffu);
    const uint32_t s = *reinterpret_cast<const uint32_t*>(sp);
    int4 v;
    if (DEEP) {
      v = *reinterpret_cast<const int4*>(cp);
    } else {
      const uint2 q = *reinterpret_cast<const uint2*>(cp);
      v = make_int4(int16_t(q.x), int32_t(q.x) >> 16, int16_t(q.y), int32_t(q.y) >> 16);
    }
    acc += error(ca, v.x, v.y, int(s & 0xffffu));
    if (g.cols > 1) acc += error(cb, v.z, v.w, int(s >> 16));
    wp += g.ws;
    sp += kStrip;
    cp += kStrip * (DEEP ? 8 : 4);
  }
  return acc;
}

// A set's weights from its fit (encoder/lr.rs:389-430).
__device__ __noinline__ void sgr_weights(const LrSearchDesc& d, const LrSearchFrame& F, const LrSearchJob& job,
                                         const LrSearchRect* rects, int set, const SgrSums& t, int32_t* xqd) {
  const SgrPass q0 = sgr_pass(set, 0), q1 = sgr_pass(set, 1);
  const int r0 = q0.r, r1 = q1.r;
  // The reference's target is (128 * 16) times ours. Its f64 partial sums are
  // exact, so any order gives them, while the terms' magnitudes sum below 2^53:
  // the squares' own sums do, and by Cauchy-Schwarz a product's does where the
  // product of its squares' sums is below 2^106 (2^105 here: it is rounded).
  constexpr int64_t kExact = int64_t(1) << 53;
  constexpr double kBound = 4.056481920730334e31;  // 2^105
  const double tt = double(t.tt) * 4194304.0;      // 2048^2
  double m00, m01, m11, v0, v1;
  if (t.aa < kExact && t.bb < kExact && double(t.aa) * tt < kBound && double(t.bb) * tt < kBound) {
    m00 = double(t.aa);
    m01 = double(t.ab);
    m11 = double(t.bb);
    v0 = double(t.at * 2048);
    v1 = double(t.bt * 2048);
  } else {
    sgr_fit_in_order(d, F, job, rects, q0, q1, m00, m01, m11, v0, v1);
  }
  double w0, w2;
  if (r0 && r1) {
    double m[2][2] = {{m00, m01}, {m01, m11}}, v[2] = {v0, v1}, x2[2];
    solve<2>(m, v, x2);
    w0 = x2[0];
    w2 = x2[1];
  } else if (r0) {
    w0 = m00 > 0.0 ? __ddiv_rn(v0, m00) : 0.0;
    w2 = 0.0;
  } else {
    w0 = 0.0;
    w2 = m11 > 0.0 ? __ddiv_rn(v1, m11) : 0.0;
  }
  const int x0q = r0 ? min(max(f64_to_i32(round(w0)), kXqdMin[0]), kXqdMax[0]) : 0;
  int x1q;
  if (r1) {
    // i32 arithmetic wraps as the reference's release build does
    const int diff = int(uint32_t(1 << 7) - uint32_t(x0q) - uint32_t(f64_to_i32(round(w2))));
    x1q = min(max(diff, kXqdMin[1]), kXqdMax[1]);
  } else {
    x1q = min(max((1 << 7) - x0q, kXqdMin[1]), kXqdMax[1]);
  }
  xqd[0] = x0q;
  xqd[1] = x1q;
}

// The start of plane row y of window row `r` of a rectangle.
__device__ __forceinline__ const uint8_t* search_row(const LrSearchFrame& F, int p, const LrSearchRect& rc, int r) {
  const int y = max(min(rc.y0 + r - kB, F.pey[p]), 0);
  const DPlane& pl = y < rc.ss || y > rc.se ? F.cur[p] : F.cdef[p];
  const int yy = y < rc.ss ? max(rc.ss - 2, y) : (y > rc.se ? min(rc.se + 2, y) : y);
  return pl.p + int64_t(yy) * pl.stride * F.sb;
}

// The source samples of a strip (columns x .. x + w - 1, rows y .. y + h - 1),
// kStrip apart, eight at a time where they lie in an aligned row.
__device__ __forceinline__ void stage_source(const LrSearchFrame& F, int p, int x, int w, int y, int h, uint16_t* out) {
  const int64_t pitch = F.src[p].stride * F.sb;
  const uint8_t* base = F.src[p].p + int64_t(y) * pitch + int64_t(x) * F.sb;
  const bool aligned = ((reinterpret_cast<uintptr_t>(base) | uintptr_t(pitch)) & uintptr_t(8 * F.sb - 1)) == 0;
  for (int k = threadIdx.x; k < h * (kStrip / 8); k += kLrThreads) {
    const int i = k / (kStrip / 8), j = (k % (kStrip / 8)) * 8;
    if (j >= w) continue;
    const uint8_t* row = base + int64_t(i) * pitch;
    uint16_t* o = out + i * kStrip + j;
    if (aligned && j + 8 <= w) {
      uint4 v;
      if (F.sb == 2) {
        v = *reinterpret_cast<const uint4*>(row + j * 2);
      } else {
        const uint2 b = *reinterpret_cast<const uint2*>(row + j);
        v = make_uint4(__byte_perm(b.x, 0, 0x4140), __byte_perm(b.x, 0, 0x4342), __byte_perm(b.y, 0, 0x4140),
                       __byte_perm(b.y, 0, 0x4342));
      }
      *reinterpret_cast<uint4*>(o) = v;
    } else {
      for (int e = 0; e < 8 && j + e < w; e++) o[e] = uint16_t(ld_row(row, F.sb, j + e));
    }
  }
}

}  // namespace

// Phase 3, one CTA per unit and d.spc (1 or 2) parameter sets: the self-guided
// fit (encoder/lr.rs:330-430), the projection weights, and the restoration's
// error. What bounds it is instruction issue; so the filters are the decoder's,
// which walk the rows in registers (lr_walk.cuh), in strips of 64 columns and a
// stripe. Of a unit that is one strip the window is staged once for all sets, and
// each sample's filter outputs, kept from the fit, give its error; others stage
// and walk their strips again. A strip of up to 32 columns holds work for two
// warps: two sets take a half of the CTA each.
// 6 sets of a 1080p 4:2:0 frame in units of 64: 740 us with the
// filters in bands of shared memory (778 instructions a sample and set), 195 now.
__global__ void __launch_bounds__(kLrThreads, 4) lr_search_sgr_kernel(const LrSearchDesc d) {
  extern __shared__ __align__(16) uint8_t lrs_smem[];
  __shared__ GroupEdges edges[kLrThreads / 16];
  __shared__ const uint8_t* rows[kMaxH + 6];
  __shared__ SgrSums sums[2][kLrThreads / 32];
  __shared__ uint64_t s_err[2][kLrThreads / 32];
  __shared__ int32_t s_xqd[2][2];
  const int tid = threadIdx.x, warp = tid >> 5;
  const int per_job = (d.nsets + d.spc - 1) / d.spc;
  const int ji = blockIdx.x / per_job, si = (blockIdx.x - ji * per_job) * d.spc;
  const int nk = min(d.spc, d.nsets - si);  // this CTA's sets
  const LrSearchJob job = d.jobs[ji];
  const LrSearchFrame& F = d.frames[job.frame];
  const LrSearchRect* rects = d.rects + job.r0;
  const int p = job.plane, bd = F.bd, maxv = (1 << bd) - 1;
  uint16_t* win = reinterpret_cast<uint16_t*>(lrs_smem);
  uint16_t* src = reinterpret_cast<uint16_t*>(lrs_smem + kSgrSrcOff);
  uint8_t* cache = lrs_smem + kSgrCacheOff;
  const bool deep = bd > 10;
  const int slot = kStripPx * (deep ? 8 : 4);  // bytes of a set's kept outputs
  const bool single = job.nr == 1 && job.w <= kStrip;
  const bool halves = single && job.w <= kStrip / 2 && nk == 2;
  const Team all{tid, kLrThreads, 1};
  if (tid < 2 * (kLrThreads / 32)) {
    sums[tid & 1][tid >> 1] = SgrSums{};
    s_err[tid & 1][tid >> 1] = 0;
  }
  for (int pass = 0; pass < 2; pass++) {  // the fit, then the error with the quantised weights
    for (int ri = 0; ri < job.nr; ri++) {
      const LrSearchRect rc = rects[ri];
      for (int x = 0; x < job.w; x += kStrip) {
        const int w = min(job.w - x, kStrip), h = rc.h;
        SgrLane g;
        g.ws = w > 32 ? kWideWS : kSlimWS;
        const int gs = w > 32 ? 5 : 4, gn = 1 << gs;  // lanes of a group
        const int half = halves ? tid >> 6 : 0, t = halves ? tid & 63 : tid;
        const int gl = t & (gn - 1), lgroups = (halves ? 6 : 7) - gs;
        g.per = (((h + (1 << lgroups) - 1) >> lgroups) + 1) & ~1;  // (the stripe's first row is even)
        g.i0 = (t >> gs) * g.per;
        g.c = 2 * gl;
        g.cols = min(w - g.c, 2);
        g.left = g.cols > 0 ? min(h - g.i0, g.per) : 0;
        g.win = win + g.c;
        g.src = src + g.c;
        const int k0 = half, k1 = halves ? half + 1 : nk;  // the sets of this half
        if (pass == 0 || !single) {
          __syncthreads();  // (everyone is done with the previous strip)
          for (int r = tid; r < h + 6; r += kLrThreads) rows[r] = search_row(F, p, rc, r);
          __syncthreads();
          stage_window(win, g.ws, rows, F.sb, F.pex[p], job.x0 + x, w, h, all);
          stage_source(F, p, job.x0 + x, w, rc.y0, h, src);
          __syncthreads();
        }
#pragma unroll 1
        for (int k = k0; k < k1; k++) {
          uint8_t* kept = cache + k * slot;
          // (the second walk's sums go where nothing reads them)
          if (pass == 0 || !single) {
            if (deep)
              sgr_fit_strip<true>(g, d.sets[si + k], d.step, bd, edges[tid >> gs], gl, gn, kept, &sums[k][warp]);
            else
              sgr_fit_strip<false>(g, d.sets[si + k], d.step, bd, edges[tid >> gs], gl, gn, kept, &sums[k][warp]);
            __syncwarp();  // (the next set's walk writes the group's edges)
          }
          if (pass == 1) {
            const int w0 = s_xqd[k][0], w2 = (1 << 7) - w0 - s_xqd[k][1];
            const uint32_t e = deep ? sgr_error_strip<true>(g, w0, w2, maxv, kept) : sgr_error_strip<false>(g, w0, w2, maxv, kept);
            const int64_t te = warp_sum_i64(int64_t(e));
            if ((tid & 31) == 0) s_err[k][warp] += uint64_t(te);
          }
        }
      }
    }
    __syncthreads();
    // a thread per set: in the first warp of the half that fits it
    if ((tid & 63) == 0 && tid >> 6 < nk) {
      const int k = tid >> 6;
      if (pass == 0) {
        SgrSums t{};
        for (int q = 0; q < kLrThreads / 32; q++) {
          t.aa += sums[k][q].aa;
          t.ab += sums[k][q].ab;
          t.bb += sums[k][q].bb;
          t.at += sums[k][q].at;
          t.bt += sums[k][q].bt;
          t.tt += sums[k][q].tt;
        }
        sgr_weights(d, F, job, rects, d.sets[si + k], t, s_xqd[k]);
      } else {
        LrSgrResult& r = d.sgr[ji * d.nsets + si + k];
        r.xqd[0] = s_xqd[k][0];
        r.xqd[1] = s_xqd[k][1];
        uint64_t e = 0;
        for (int q = 0; q < kLrThreads / 32; q++) e += s_err[k][q];
        r.sse = e;
      }
    }
    __syncthreads();
  }
}

// Phase 4, one thread per unit: the cheapest of no filter (error + lambda),
// the Wiener filter (+ 40 or 28 lambda) and each self-guided set in order
// (+ 20 lambda), the first on ties (encoder/lr.rs:147-186).
__global__ void lr_search_choose_kernel(const LrSearchDesc d, int njobs) {
  const int ji = blockIdx.x * blockDim.x + threadIdx.x;
  if (ji >= njobs) return;
  const LrJobState& st = d.state[ji];
  const int p = d.jobs[ji].plane;
  const LrSearchFrame& F = d.frames[d.jobs[ji].frame];
  av1pf_lr_unit best{};
  double best_cost = __dadd_rn(__ull2double_rn(st.none), F.lambda);
  double cost = __dadd_rn(__ull2double_rn(st.wiener), __dmul_rn(F.lambda, p == 0 ? 40.0 : 28.0));
  if (cost < best_cost) {
    best_cost = cost;
    best.type = AV1PF_RESTORE_WIENER;
    for (int a = 0; a < 2; a++)
      for (int b = 0; b < 3; b++) best.wiener[a][b] = int8_t(st.coef[a][b]);
  }
  for (int si = 0; si < d.nsets; si++) {
    const LrSgrResult& r = d.sgr[ji * d.nsets + si];
    cost = __dadd_rn(__ull2double_rn(r.sse), __dmul_rn(F.lambda, 20.0));
    if (cost < best_cost) {
      best_cost = cost;
      best = av1pf_lr_unit{};
      best.type = AV1PF_RESTORE_SGRPROJ;
      best.sgr_set = uint8_t(d.sets[si]);
      best.sgr_xqd[0] = int8_t(r.xqd[0]);
      best.sgr_xqd[1] = int8_t(r.xqd[1]);
    }
  }
  d.out[ji] = best;
}

namespace {
// Raises a kernel's dynamic shared-memory limit to all the device allows
// beside its static shared memory. The attribute is process-wide, so every
// call sets the same value: searches on several contexts and host threads
// cannot lower it under one another's launches.
template <typename K>
cudaError_t allow_max_smem(K kernel, int optin) {
  cudaFuncAttributes a{};
  cudaError_t e = cudaFuncGetAttributes(&a, kernel);
  if (e != cudaSuccess) return e;
  return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, optin - int(a.sharedSizeBytes));
}
}  // namespace

cudaError_t lr_search_init() {
  int dev = 0, optin = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e == cudaSuccess) e = cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
  if (e == cudaSuccess) e = allow_max_smem(lr_search_prep_kernel, optin);
  if (e == cudaSuccess) e = allow_max_smem(lr_search_wiener_kernel, optin);
  if (e == cudaSuccess) e = allow_max_smem(lr_search_sgr_kernel, optin);
  return e;
}

void launch_lr_search(const LrSearchDesc& d, int njobs, cudaStream_t s, cudaStream_t side, cudaEvent_t fork,
                      cudaEvent_t join) {
  if (njobs <= 0) return;
  const size_t s0 = lr_search_smem(d.wmax, d.hmax, 0);
  const size_t s1 = lr_search_smem(d.wmax, d.hmax, 1);
  const size_t s2 = size_t(kSgrCacheOff) + size_t(d.spc) * kStripPx * (d.deep ? 8 : 4);
  // the self-guided fits depend on nothing else: they run beside the Wiener passes
  cudaEventRecord(fork, s);
  cudaStreamWaitEvent(side, fork, 0);
  lr_search_sgr_kernel<<<njobs * ((d.nsets + d.spc - 1) / d.spc), kLrThreads, s2, side>>>(d);
  if (d.multi_rect) lr_search_prep_kernel<<<njobs, kThreads, s0, s>>>(d);
  lr_search_wiener_kernel<<<njobs, 128, s1, s>>>(d);
  cudaEventRecord(join, side);
  cudaStreamWaitEvent(s, join, 0);
  lr_search_choose_kernel<<<(njobs + 127) / 128, 128, 0, s>>>(d, njobs);
  note_launch(d.multi_rect ? 4 : 3);
}

}  // namespace av1pf
