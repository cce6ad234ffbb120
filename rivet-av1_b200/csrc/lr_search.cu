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
// real-valued terms, so their sums run in the reference's order: lanes of one
// warp each add one accumulator's terms in sample order. Every f64 operation is a
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
constexpr int kStrip = 64;  // columns of a strip
constexpr int kStripPx = kStrip * kMaxH;
constexpr int kWienerThreads = 160;  // a warp that adds and four that produce
constexpr int kWienerWarps = kWienerThreads / 32;
constexpr int kWienerCols = 6;  // columns a producing lane has: units reach 256 + 127 columns, two warps a row
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

// The start of the plane row that window row r of a rectangle reads.
__device__ __forceinline__ const uint8_t* search_row(const LrSearchFrame& F, int p, const LrSearchRect& rc, int r) {
  const int y = max(min(rc.y0 + r - kB, F.pey[p]), 0);
  const DPlane& pl = y < rc.ss || y > rc.se ? F.cur[p] : F.cdef[p];
  const int yy = y < rc.ss ? max(rc.ss - 2, y) : (y > rc.se ? min(rc.se + 2, y) : y);
  return pl.p + int64_t(yy) * pl.stride * F.sb;
}

// The window of columns x .. x + w - 1 of a rectangle, by the whole CTA.
__device__ __forceinline__ void stage_rect(const LrSearchFrame& F, int p, const LrSearchRect& rc, int x, int w, uint16_t* win,
                                           int ws, const uint8_t** rows) {
  for (int r = threadIdx.x; r < rc.h + 2 * kB; r += blockDim.x) rows[r] = search_row(F, p, rc, r);
  __syncthreads();
  stage_window(win, ws, rows, F.sb, F.pex[p], x, w, rc.h, Team{int(threadIdx.x), int(blockDim.x), 1});
}

// The source samples of a strip (columns x .. x + w - 1, rows y .. y + h - 1),
// kStrip apart, eight at a time where they lie in an aligned row.
__device__ __forceinline__ void stage_source(const LrSearchFrame& F, int p, int x, int w, int y, int h, uint16_t* out) {
  const int64_t pitch = F.src[p].stride * F.sb;
  const uint8_t* base = F.src[p].p + int64_t(y) * pitch + int64_t(x) * F.sb;
  const bool aligned = ((reinterpret_cast<uintptr_t>(base) | uintptr_t(pitch)) & uintptr_t(8 * F.sb - 1)) == 0;
  for (int k = threadIdx.x; k < h * (kStrip / 8); k += blockDim.x) {
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

// Block sums of N 64-bit values in one round (every thread gets the totals).
template <int N>
__device__ void block_sums_i64(int64_t (&v)[N], int64_t (*red)[kWienerThreads / 32]) {
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
// singular. All in registers: rows are swapped by selection.
template <int N>
__device__ __forceinline__ void solve(double (&m)[N][N], double (&v)[N], double (&x)[N]) {
#pragma unroll
  for (int i = 0; i < N; i++) {
    int piv = i;
    double most = fabs(m[i][i]);
#pragma unroll
    for (int a = i + 1; a < N; a++) {
      const double mag = fabs(m[a][i]);
      if (!(mag < most)) piv = a, most = mag;
    }
#pragma unroll
    for (int a = i + 1; a < N; a++) {
      const bool swap = piv == a;
      auto exchange = [&](double& p, double& q) {
        const double t = p;
        p = swap ? q : p;
        q = swap ? t : q;
      };
#pragma unroll
      for (int c = 0; c < N; c++) exchange(m[i][c], m[a][c]);
      exchange(v[i], v[a]);
    }
    if (fabs(m[i][i]) < 1e-9) {
#pragma unroll
      for (int k = 0; k < N; k++) x[k] = 0.0;
      return;
    }
#pragma unroll
    for (int r = 0; r < N; r++) {
      if (r != i) {
        const double f = __ddiv_rn(m[r][i], m[i][i]);
#pragma unroll
        for (int c = i; c < N; c++) m[r][c] = __dsub_rn(m[r][c], __dmul_rn(f, m[i][c]));
        v[r] = __dsub_rn(v[r], __dmul_rn(f, v[i]));
      }
    }
  }
#pragma unroll
  for (int i = 0; i < N; i++) x[i] = __ddiv_rn(v[i], m[i][i]);
}

// A Wiener pass's solution from its sums (m00 m01 m02 m11 m12 m22 v0 v1 v2);
// chroma filters have no outermost tap.
__device__ __noinline__ void wiener_solve(const double* t, bool luma, double* sol) {
  if (luma) {
    double m[3][3] = {{t[0], t[1], t[2]}, {t[1], t[3], t[4]}, {t[2], t[4], t[5]}}, v[3] = {t[6], t[7], t[8]}, x[3];
    solve<3>(m, v, x);
    sol[0] = x[0];
    sol[1] = x[1];
    sol[2] = x[2];
  } else {
    double m[2][2] = {{t[3], t[4]}, {t[4], t[5]}}, v[2] = {t[7], t[8]}, x[2];
    solve<2>(m, v, x);
    sol[0] = 0.0;
    sol[1] = x[0];
    sol[2] = x[1];
  }
}

// A sample with the other direction's filter applied (encoder/lr.rs:265-285):
// `at` is the sample's place in the window, `step` the distance to its neighbour
// along that direction.
__device__ __forceinline__ double wiener_other(const uint16_t* at, int step, const double (&other)[3]) {
  const int center = at[0];
  double s = double(center);
#pragma unroll
  for (int k = 0; k < 3; k++) {
    const int dd = (3 - k) * step;
    // a + b - 2 * center is an integer below 2^17: the f64 expression of
    // encoder/lr.rs is exact, so integer arithmetic gives the same value
    s = __dadd_rn(s, __dmul_rn(other[k], double(at[-dd] + at[dd] - 2 * center)));
  }
  return s;
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

namespace {
// The Wiener kernel's shared memory: the window; the source samples of a unit
// of one strip (64 columns of one stripe); the rows of samples filtered in the
// other direction; and two buffers of the nine products, a product's chunk of fit
// rows one after another (rows of a multiple of 8) and the products on different
// banks for 16-byte loads. A chunk is two rows, of units of up to 32 columns four:
// a column for each producing lane of a 64-column unit and of a 32-column one.
__host__ __device__ constexpr int lr_window_stride(int wmax) { return (wmax + 2 * kB + 7) & ~7; }
// A warp's share of a rectangle's rows, walked in fours, and the rows that the
// warps' shares reach over, past the rectangle's last.
__host__ __device__ constexpr int wiener_share(int h) { return ((h + kWienerWarps - 1) / kWienerWarps + 3) & ~3; }
constexpr int wiener_reach(int h) { return (h + wiener_share(h) - 1) / wiener_share(h) * wiener_share(h); }
__host__ __device__ constexpr int lr_window_rows(int hmax) { return ((hmax + 15) & ~15) + 2 * kB; }
constexpr bool reach_fits() {
  for (int hmax = 1; hmax <= kMaxH; hmax++)
    for (int h = 1; h <= hmax; h++)
      if (wiener_reach(h) + 2 * kB > lr_window_rows(hmax)) return false;
  return true;
}
static_assert(reach_fits(), "a share's last rows are inside the window");
__host__ __device__ constexpr size_t lr_window_bytes(int wmax, int hmax) {
  return size_t(lr_window_rows(hmax)) * lr_window_stride(wmax) * 2;
}
__host__ __device__ constexpr int wiener_cols(int w, int step) { return (w + step - 1) / step; }
__host__ __device__ constexpr int wiener_row(int cols) { return (cols + 7) & ~7; }
__host__ __device__ constexpr int wiener_chunk(int w) { return w > 32 ? 2 : 4; }
// rows of a vertical pass's ring: a chunk's lines reach over (rows - 1) * step + 7
// window rows, and the next chunk's rows * step more are written beside them
__host__ __device__ constexpr int wiener_rows(int w, int step) { return w <= 32 && step == 2 ? 32 : 16; }
__host__ __device__ constexpr int wiener_term(int wmax, int step) {
  int n = 0;
  for (int w = wmax < 32 ? wmax : 32; w <= wmax; w += wmax > w ? wmax - w : 1) {
    const int k = wiener_chunk(w) * wiener_row(wiener_cols(w, step));
    n = k > n ? k : n;
  }
  return n + ((2 - n) & 15);  // 2 mod 16 doubles: 4 mod 32 banks
}
__host__ __device__ constexpr int wiener_ring(int wmax, int step) {
  int n = 0;
  for (int w = wmax < 32 ? wmax : 32; w <= wmax; w += wmax > w ? wmax - w : 1) {
    const int across = 2 * wiener_chunk(w) * (w + 2 * kB), down = wiener_rows(w, step) * wiener_cols(w, step);
    n = across > n ? across : n;
    n = down > n ? down : n;
  }
  return (n + 1) & ~1;
}
constexpr size_t kUnitSrc = size_t(kStripPx) * 2;
}  // namespace

size_t lr_search_smem(int wmax, int hmax, int step) {
  return lr_window_bytes(wmax, hmax) + kUnitSrc +
         sizeof(double) * (size_t(wiener_ring(wmax, step)) + size_t(2) * 9 * wiener_term(wmax, step));
}

namespace {

// Window stride and the region after the window.
struct Smem {
  uint16_t* win;
  int ws;
  uint8_t* region;
};
__device__ __forceinline__ Smem smem_of(uint8_t* base, const LrSearchDesc& d) {
  Smem m;
  m.ws = lr_window_stride(d.wmax);
  m.win = reinterpret_cast<uint16_t*>(base);
  m.region = base + lr_window_bytes(d.wmax, d.hmax);
  return m;
}

}  // namespace

namespace {

// The unfiltered error and the first Wiener pass (encoder/lr.rs:134-146; vertical,
// the other direction's filter still zero: its lines are plain samples) over a
// lane's two columns and rows i0 .. i0 + left - 1 of a rectangle, walked down the
// window: `per` rows, a multiple of 4. sums: m00 m01 m02 m11 m12 m22 v0 v1 v2 and
// the error, exact integers.
template <class Source>
__device__ __forceinline__ void wiener_first(const uint16_t* win, int ws, int i0, int per, int left, int cols, int step,
                                             Source source, int64_t (&sums)[10]) {
  const uint16_t* row = win + i0 * ws + kB;
  auto next = [&]() {  // (columns c and c + 1 start at an odd one of the window)
    const uint32_t v = uint32_t(row[0]) | (uint32_t(row[1]) << 16);
    row += ws;
    return v;
  };
  uint32_t t[10];
#pragma unroll
  for (int k = 0; k < 6; k++) t[k] = next();
#pragma unroll 1
  for (int i = 0; i < per; i += 4) {
    uint32_t src[4];
#pragma unroll
    for (int k = 0; k < 4; k++) {
      src[k] = source(i0 + i + k);
      t[6 + k] = next();
    }
    int32_t part[10] = {};  // eight products below 2^26 each
#pragma unroll
    for (int k = 0; k < 4; k++) {
      const uint32_t s06 = t[k] + t[k + 6], s15 = t[k + 1] + t[k + 5], s24 = t[k + 2] + t[k + 4];  // no carry: below 2^13
      auto add = [&](int c, int s, int a06, int a15, int a24, bool fit) {
        const int e = s - c;
        part[9] += e * e;
        if (!fit) return;
        const int d0 = a06 - 2 * c, d1 = a15 - 2 * c, d2 = a24 - 2 * c;
        part[0] += d0 * d0;
        part[1] += d0 * d1;
        part[2] += d0 * d2;
        part[3] += d1 * d1;
        part[4] += d1 * d2;
        part[5] += d2 * d2;
        part[6] += d0 * e;
        part[7] += d1 * e;
        part[8] += d2 * e;
      };
      if (i + k < left) {
        add(t[k + 3] & 0xffffu, src[k] & 0xffffu, s06 & 0xffffu, s15 & 0xffffu, s24 & 0xffffu, step == 1 || !(k & 1));
        if (cols > 1) add(t[k + 3] >> 16, src[k] >> 16, s06 >> 16, s15 >> 16, s24 >> 16, step == 1);
      }
    }
#pragma unroll
    for (int q = 0; q < 10; q++) sums[q] += part[q];
#pragma unroll
    for (int k = 0; k < 6; k++) t[k] = t[k + 4];
  }
}

}  // namespace

// One CTA per unit: the error without a filter and the first Wiener pass; then
// the second (horizontal) and third (vertical) passes, whose terms are
// real-valued, so each of their sums runs in the reference's sample order: warps
// 1-4 produce two or four rows of products into shared memory (two buffers) while
// lane q of warp 0 adds accumulator q's (m00 m01 m02 m11 m12 m22 v0 v1 v2). Then
// the solves, the quantised coefficients (encoder/lr.rs:316-327) and the filter's
// error.
//
// What bounds it is the chain of f64 additions, two for each sample of a unit, 8
// cycles each: so the adding warp does nothing but read products, eight ahead,
// and add; the producers apply the other direction's filter once for each sample
// (not for each of the seven lines that it is on). The first pass and the filter's
// error walk down the rows in registers, and a unit of one strip keeps its source
// samples beside its window. 1080p 4:2:0: units of 64, 241 us -> 152 (of which the
// chains alone are 40); units of 256, 1590 us -> 1330 (690).
__global__ void __launch_bounds__(kWienerThreads, 4) lr_search_wiener_kernel(const LrSearchDesc d) {
  extern __shared__ __align__(16) uint8_t lrs_smem[];
  __shared__ int64_t red[kWienerThreads / 32];
  __shared__ int64_t red10[10][kWienerThreads / 32];
  __shared__ double s_sums[9], s_other[3], s_vc[3];
  __shared__ int s_coef[2][3];
  __shared__ const uint8_t* s_rows[kMaxH + 6];
  const LrSearchJob job = d.jobs[blockIdx.x];
  const LrSearchFrame& F = d.frames[job.frame];
  const int p = job.plane, x0 = job.x0, w = job.w, sb = F.sb, tid = threadIdx.x, step = d.step;
  const int lane = tid & 31, warp = tid >> 5;
  constexpr int nw = kWienerWarps;
  const bool unit = job.nr == 1 && w <= kStrip;  // one strip: its source and window are staged once
  const Smem sm = smem_of(lrs_smem, d);
  uint16_t* usrc = reinterpret_cast<uint16_t*>(sm.region);
  const LrSearchRect* rects = d.rects + job.r0;
  LrJobState& st = d.state[blockIdx.x];
  const int first = p == 0 ? 0 : 1;
  const int bd = F.bd;
  const int nci = wiener_cols(w, step);
  auto source = [&](const LrSearchRect& rc, int i, int j) {
    return unit ? int(usrc[i * kStrip + j]) : ld(F.src[p], sb, x0 + j, rc.y0 + i);
  };
  // Each rectangle's columns in strips of 64, two a lane, its rows a warp's share
  // of them: run(rc, x, win, i0, per, left, cols, pair), where
  // pair(i) is a row's two source samples, clamped to the rectangle.
  auto strips = [&](const LrSearchRect& rc, auto run) {
    const int per = wiener_share(rc.h), i0 = warp * per;
    if (i0 >= rc.h) return;
    for (int x = 0; x < w; x += kStrip) {
      const int c = x + 2 * lane, cols = min(w - c, 2), left = cols > 0 ? min(rc.h - i0, per) : 0;
      run(sm.win + min(c, (w - 1) & ~1), i0, per, left, cols, [&](int i) {
        i = min(i, rc.h - 1);
        if (unit) return *reinterpret_cast<const uint32_t*>(usrc + i * kStrip + c);
        const int c0 = min(c, w - 1), c1 = min(c + 1, w - 1);
        return uint32_t(ld(F.src[p], sb, x0 + c0, rc.y0 + i)) | (uint32_t(ld(F.src[p], sb, x0 + c1, rc.y0 + i)) << 16);
      });
    }
  };
  {
    int64_t sums[10] = {};
    for (int ri = 0; ri < job.nr; ri++) {
      const LrSearchRect rc = rects[ri];
      __syncthreads();
      stage_rect(F, p, rc, x0, w, sm.win, sm.ws, s_rows);
      if (unit) stage_source(F, p, x0, w, rc.y0, rc.h, usrc);
      __syncthreads();
      strips(rc, [&](const uint16_t* win, int i0, int per, int left, int cols, auto pair) {
        wiener_first(win, sm.ws, i0, per, left, cols, step, pair, sums);
      });
    }
    block_sums_i64(sums, red10);
    if (tid == 0) {
      st.none = uint64_t(sums[9]);
      double tot[9];
#pragma unroll
      for (int q = 0; q < 9; q++) tot[q] = double(sums[q]);
      wiener_solve(tot, p == 0, s_vc);
    }
  }
  __syncthreads();
  double hc[3] = {0.0, 0.0, 0.0};
  const bool owner = warp == 0 && lane < 9 && (p == 0 || (lane >= 3 && lane != 6));
  // [2 buffers][9 products][chunk rows][row8]
  double* ring = reinterpret_cast<double*>(sm.region + kUnitSrc);
  double* terms = ring + wiener_ring(d.wmax, step);
  const int row8 = wiener_row(nci), tq_stride = wiener_term(d.wmax, step);
  const int chunk = wiener_chunk(w), rmask = wiener_rows(w, step) - 1, across = w + 2 * kB;
  // a producing lane's row of a chunk, and its columns: every pstep-th from pcol
  const int prow = chunk == 4 ? warp - 1 : (warp - 1) >> 1;
  const int pstep = chunk == 4 ? 32 : 64, pcol = chunk == 4 ? lane : ((warp - 1) & 1) * 32 + lane;
  constexpr int kProducers = kWienerThreads - 32;
  for (int iter = 1; iter < 3; iter++) {
    const bool vertical = iter == 2;
    if (tid < 3) s_other[tid] = vertical ? hc[tid] : s_vc[tid];
    double macc = 0.0;
    for (int ri = 0; ri < job.nr; ri++) {
      const LrSearchRect rc = rects[ri];
      __syncthreads();
      // one rectangle: its window, staged for the first pass, stays in place
      // (the term rows and band rows lie outside it)
      if (job.nr > 1) stage_rect(F, p, rc, x0, w, sm.win, sm.ws, s_rows);
      __syncthreads();
      const int nri = (rc.h + step - 1) / step, nch = (nri + chunk - 1) / chunk;
      const double oth[3] = {s_other[0], s_other[1], s_other[2]};
      // the samples of a chunk's lines, filtered in the other direction:
      // horizontal lines take the fit rows' window columns, vertical ones the fit
      // columns of the window rows from the chunk's first (the ring has those that
      // the chunk before takes too)
      auto filter = [&](int ch) {
        if (vertical) {
          const int hend = (min((ch + 1) * chunk, nri) - 1) * step + 7;
          for (int r = (ch ? (ch * chunk - 1) * step + 7 : 0) + prow; r < hend; r += chunk)
            for (int c = pcol; c < nci; c += pstep)
              ring[(r & rmask) * nci + c] = wiener_other(&sm.win[r * sm.ws + c * step + kB], 1, oth);
        } else if (ch * chunk + prow < nri) {
          const uint16_t* row = sm.win + ((ch * chunk + prow) * step + kB) * sm.ws;
          double* to = ring + ((ch & 1) * chunk + prow) * across;
          for (int c = pcol; c < across; c += pstep) to[c] = wiener_other(row + c, sm.ws, oth);
        }
      };
      if (warp > 0) {
        filter(0);
        asm volatile("bar.sync 1, %0;" ::"n"(kProducers) : "memory");
      }
      // chunks of rows in turn, two buffers: warps 1.. fill chunk c + 1 (and
      // filter for chunk c + 2) while warp 0 adds chunk c, row by row in sample
      // order
      for (int ch = 0; ch <= nch; ch++) {
        if (ch < nch && warp > 0) {
          double* tr = terms + (ch & 1) * 9 * tq_stride + prow * row8;
          const int i = (ch * chunk + prow) * step;
          const bool row = ch * chunk + prow < nri;
          int sv[kWienerCols];
#pragma unroll
          for (int u = 0; u < kWienerCols; u++) {
            if (u * pstep >= nci) break;
            const int c = pcol + u * pstep;
            sv[u] = row && c < nci ? source(rc, i, c * step) : 0;
          }
          if (ch + 1 < nch) filter(ch + 1);
          // the row's lines: sample q of column c's is tap[q][c * next]
          const double* tap[7];
#pragma unroll
          for (int q = 0; q < 7; q++) tap[q] = ring + (vertical ? ((i + q) & rmask) * nci : ((ch & 1) * chunk + prow) * across + q);
          const int next = vertical ? 1 : step;
#pragma unroll
          for (int u = 0; u < kWienerCols; u++) {
            if (u * pstep >= row8) break;
            const int c = pcol + u * pstep;
            if (c >= row8) continue;
            // past a row's end, and past the last row: products that add nothing
            double d0 = 0.0, d1 = 0.0, d2 = 0.0, t = 0.0;
            if (row && c < nci) {
              double line[7];
#pragma unroll
              for (int q = 0; q < 7; q++) line[q] = tap[q][c * next];
              const double two3 = __dmul_rn(2.0, line[3]);
              d0 = __dsub_rn(__dadd_rn(line[0], line[6]), two3);
              d1 = __dsub_rn(__dadd_rn(line[1], line[5]), two3);
              d2 = __dsub_rn(__dadd_rn(line[2], line[4]), two3);
              t = __dsub_rn(double(sv[u]), line[3]);
            }
            if (p == 0) {
              tr[0 * tq_stride + c] = __dmul_rn(d0, d0);
              tr[1 * tq_stride + c] = __dmul_rn(d0, d1);
              tr[2 * tq_stride + c] = __dmul_rn(d0, d2);
              tr[6 * tq_stride + c] = __dmul_rn(d0, t);
            }
            tr[3 * tq_stride + c] = __dmul_rn(d1, d1);
            tr[4 * tq_stride + c] = __dmul_rn(d1, d2);
            tr[5 * tq_stride + c] = __dmul_rn(d2, d2);
            tr[7 * tq_stride + c] = __dmul_rn(d1, t);
            tr[8 * tq_stride + c] = __dmul_rn(d2, t);
          }
        }
        if (ch > 0 && owner) {
          // the sum runs in sample order, eight products while the next eight are read
          const int n = chunk * row8;  // a multiple of 16
          const double2* tp = reinterpret_cast<const double2*>(terms + ((ch - 1) & 1) * 9 * tq_stride + lane * tq_stride);
          double2 a[4], b[4];
          auto load = [&](double2 (&q)[4]) {
#pragma unroll
            for (int u = 0; u < 4; u++) q[u] = tp[u];
            tp += 4;
          };
          auto add = [&](const double2 (&q)[4]) {
#pragma unroll
            for (int u = 0; u < 4; u++) macc = __dadd_rn(__dadd_rn(macc, q[u].x), q[u].y);
          };
          load(a);
#pragma unroll 1
          for (int left = n; left > 16; left -= 16) {
            load(b);
            add(a);
            load(a);
            add(b);
          }
          load(b);
          add(a);
          add(b);
        }
        __syncthreads();
      }
    }
    if (owner) s_sums[lane] = macc;
    __syncthreads();
    if (tid == 0) wiener_solve(s_sums, p == 0, s_other);  // the pass's solution
    __syncthreads();
    if (vertical) {
      if (tid < 3) s_vc[tid] = s_other[tid];
    } else {
      for (int k = 0; k < 3; k++) hc[k] = s_other[k];
    }
    __syncthreads();
  }
  if (tid < 3) {
    const double vk = s_vc[tid], hk = tid == 0 ? hc[0] : tid == 1 ? hc[1] : hc[2];
    s_coef[0][tid] = tid < first ? 0 : min(max(f64_to_i32(round(vk * 128.0)), kWienerMin[tid]), kWienerMax[tid]);
    s_coef[1][tid] = tid < first ? 0 : min(max(f64_to_i32(round(hk * 128.0)), kWienerMin[tid]), kWienerMax[tid]);
  }
  __syncthreads();
  // the Wiener filter's error (postfilter.rs:781-822 restoration)
  int64_t acc = 0;
  for (int ri = 0; ri < job.nr; ri++) {
    const LrSearchRect rc = rects[ri];
    if (job.nr > 1) {  // else still staged
      __syncthreads();
      stage_rect(F, p, rc, x0, w, sm.win, sm.ws, s_rows);
      __syncthreads();
    }
    strips(rc, [&](const uint16_t* win, int i0, int per, int left, int cols, auto pair) {
      uint32_t src[4], part = 0;  // (32 squares below 2^24)
      wiener_walk(
          win, sm.ws, i0, per, s_coef[0][0], s_coef[0][1], s_coef[0][2], s_coef[1][0], s_coef[1][1], s_coef[1][2], bd,
          [&](int i) {
#pragma unroll
            for (int k = 0; k < 4; k++) src[k] = pair(i0 + i + k);
          },
          [&](int i, uint32_t a, uint32_t b) {
            if (i >= left) return;
            const int ea = int(a) - int(src[i & 3] & 0xffffu), eb = int(b) - int(src[i & 3] >> 16);
            part += uint32_t(ea * ea);
            if (cols > 1) part += uint32_t(eb * eb);
          });
      acc += part;
    });
  }
#pragma unroll
  for (int o = 16; o; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
  if (lane == 0) red[warp] = acc;
  __syncthreads();
  if (tid == 0) {
    int64_t all = 0;
    for (int q = 0; q < nw; q++) all += red[q];
    st.wiener = uint64_t(all);
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
          stage_rect(F, p, rc, job.x0 + x, w, win, g.ws, rows);
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
  if (e == cudaSuccess) e = allow_max_smem(lr_search_wiener_kernel, optin);
  if (e == cudaSuccess) e = allow_max_smem(lr_search_sgr_kernel, optin);
  return e;
}

void launch_lr_search(const LrSearchDesc& d, int njobs, cudaStream_t s, cudaStream_t side, cudaEvent_t fork,
                      cudaEvent_t join) {
  if (njobs <= 0) return;
  const size_t s1 = lr_search_smem(d.wmax, d.hmax, d.step);
  const size_t s2 = size_t(kSgrCacheOff) + size_t(d.spc) * kStripPx * (d.deep ? 8 : 4);
  // the self-guided fits depend on nothing else: they run beside the Wiener passes
  cudaEventRecord(fork, s);
  cudaStreamWaitEvent(side, fork, 0);
  lr_search_wiener_kernel<<<njobs, kWienerThreads, s1, s>>>(d);
  lr_search_sgr_kernel<<<njobs * ((d.nsets + d.spc - 1) / d.spc), kLrThreads, s2, side>>>(d);
  cudaEventRecord(join, side);
  cudaStreamWaitEvent(s, join, 0);
  lr_search_choose_kernel<<<(njobs + 127) / 128, 128, 0, s>>>(d, njobs);
  note_launch(3);
}

}  // namespace av1pf
