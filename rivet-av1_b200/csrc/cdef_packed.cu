// cdef_packed.cu — the constrained directional enhancement filter (7.15), two
// samples per lane: in half precision for bit depths up to 10, in 16-bit
// integers for 12 (cdef_packed.cuh shows why both are exact). Launches with the
// horizontal loop-filter pass fused in take cdef_kernel (cdef.cu).
//
// Reference: rivet-av1 src/decoder/postfilter.rs:266-513, src/dsp/cdef.rs:13-90.
//
// What bounds it: instruction issue. A tap in integers is 12 instructions for
// two samples: 4K 12-bit 4:4:4 coded at 3072 columns takes 104 us against the
// 32-bit kernel's 140, the chain call 378 against 409. In half precision: the
// constrained taps of the 32-bit kernel were 70% of its 16.2 M warp instructions per 1080p frame, on the
// integer ALU pipe (one instruction per two clocks). Here a tap is about 10
// instructions for two samples instead of 12 for one, half of them on the
// multiply-add pipe, which issues every clock. 1080p 10-bit 4:2:0 against the
// 32-bit kernel: 36.0 -> 25.5 us (cold, under ncu), 16.2 M -> 10.0 M warp
// instructions; the chain call 70.4 -> 64.1 us, a 4K 10-bit superres chain
// 274 -> 243 us, a batch of 16 mixed frames 831 -> 706 us. What is left is
// latency: loads at a CTA's start and barriers between its phases. 64 registers
// a thread, for eight half-superblock CTAs an SM, do not hold the staging's
// chunks and addresses or the filter's taps: 236-308 bytes a thread go to local
// memory and come back (-Xptxas -v).
//
// Which samples share a word: in luma, rows r and r + 4 of an 8x8 block; in
// chroma, the U and V samples of a position (one block's chroma planes take
// the same strengths and direction). Every word column exists, so a tap at
// any offset is one aligned 32-bit load. Word rows are kPS = 74 words apart
// and a lane takes every second column: 74 = 10 mod 32, so the 4 rows x 8
// columns (or, for 4-wide blocks, 2 rows x 8 blocks x 2 columns) of a warp's
// load fall in 32 different banks. Row strides of 8 columns a lane would put
// blocks 32 columns apart in one bank.
#include "cdef_packed.cuh"
#include "cdef_search.cuh"
#include "kernels.h"

namespace av1pf {

namespace {

constexpr int kPS = 74;  // words between word rows
constexpr int kDS = 72;  // direction-search copy: u16 between rows (16-byte aligned)

constexpr int packed_smem(int R, bool tall) { return R * kDS * 2 + R * kPS * 4 + ((tall ? R : R / 2) + 4) * kPS * 4; }

// The taps of one block (postfilter.rs:489-511), 48 bytes.
struct alignas(16) PackedTaps {
  PStrength pri;    // (12-bit frames: strength, shift, mask of what it leaves, per half)
  uint32_t w0, w1;  // primary weights, in both halves (12-bit frames: as integers)
  PStrength sec;
  int16_t off[6];  // bytes: primary k0, k1, secondary lo k0, hi k0, lo k1, hi k1
  int32_t mode;    // 0 both kinds, 1 primary only, 2 secondary only, 3 copy
};
static_assert(sizeof(PackedTaps) == 48, "three 16-byte loads");

template <bool DEEP>
__device__ __forceinline__ PackedTaps make_packed_taps(int pri, int sec, int damping, int dir, int cs,
                                                       const int16_t (*doff)[2]) {
  PackedTaps t;
  const int pri_adj = pri ? max(damping - floor_log2(uint32_t(pri)), 0) : 0;
  const int sec_adj = sec ? max(damping - floor_log2(uint32_t(sec)), 0) : 0;
  const bool odd = (pri >> cs) & 1;  // CDEF_PRI_TAPS: [4, 2] / [3, 3]
  if (DEEP) {
    t.pri = deep_strength(pri, pri_adj);
    t.sec = deep_strength(sec, sec_adj);
    t.w0 = odd ? 3u : 4u;
    t.w1 = odd ? 3u : 2u;
  } else {
    t.pri = packed_strength(pri, pri_adj);
    t.sec = packed_strength(sec, sec_adj);
    t.w0 = odd ? 0x42004200u : 0x44004400u;
    t.w1 = odd ? 0x42004200u : 0x40004000u;
  }
  const int dlo = (dir + 6) & 7, dhi = (dir + 2) & 7;
  t.off[0] = doff[dir][0];
  t.off[1] = doff[dir][1];
  t.off[2] = doff[dlo][0];
  t.off[3] = doff[dhi][0];
  t.off[4] = doff[dlo][1];
  t.off[5] = doff[dhi][1];
  t.mode = pri ? (sec ? 0 : 1) : (sec ? 2 : 3);
  return t;
}

// Two filtered words (1024 + sample in each half) at c and two columns on; the
// taps' addresses serve both. MODE as in PackedTaps; with one kind of tap the
// weights sum to 12 < 16, so the result lies within the taps' range and needs
// no clamp.
template <int MODE>
__device__ __forceinline__ void packed_px2(const uint32_t* c, const PackedTaps& t, uint32_t& o0, uint32_t& o1) {
  const uint32_t xw[2] = {c[0], c[2]};
  __half2 sum[2], mx[2], nx[2];
  uint32_t mn[2];
#pragma unroll
  for (int e = 0; e < 2; e++) {
    sum[e] = as_h2(0u);
    mx[e] = as_h2(xw[e]);
    nx[e] = as_h2(xw[e] ^ 0x80008000u);
    mn[e] = xw[e];
  }
#pragma unroll
  for (int k = MODE == 2 ? 2 : 0; k < (MODE == 1 ? 2 : 6); k++) {
    const __half2 w = as_h2(k == 0 ? t.w0 : k == 1 ? t.w1 : k < 4 ? 0x40004000u : 0x3c003c00u);  // CDEF_SEC_TAPS [2, 1]
    const int off = t.off[k];
#pragma unroll
    for (int side = 0; side < 2; side++) {
      const uint32_t* p = reinterpret_cast<const uint32_t*>(reinterpret_cast<const char*>(c) + (side ? -off : off));
#pragma unroll
      for (int e = 0; e < 2; e++) packed_tap<MODE == 0>(p[2 * e], nx[e], k < 2 ? t.pri : t.sec, w, sum[e], mx[e], mn[e]);
    }
  }
#pragma unroll
  for (int e = 0; e < 2; e++) {
    __half2 v = packed_round(sum[e], as_h2(xw[e]));
    if (MODE == 0) v = __hmax2(__hmin2(v, mx[e]), as_h2(mn[e]));
    (e ? o1 : o0) = as_u32(v);
  }
}

// The same for 12-bit frames, in 16-bit integers (cdef_packed.cuh).
template <int MODE>
__device__ __forceinline__ void deep_px2(const uint32_t* c, const PackedTaps& t, uint32_t& o0, uint32_t& o1) {
  const uint32_t xw[2] = {c[0], c[2]};
  uint32_t sum[2], mx[2], mn[2];
#pragma unroll
  for (int e = 0; e < 2; e++) {
    sum[e] = 0u - (MODE == 0 ? 24u : 12u) * xw[e];
    mx[e] = mn[e] = xw[e];
  }
#pragma unroll
  for (int k = MODE == 2 ? 2 : 0; k < (MODE == 1 ? 2 : 6); k++) {
    const uint32_t w = k == 0 ? t.w0 : k == 1 ? t.w1 : k < 4 ? 2u : 1u;  // CDEF_SEC_TAPS [2, 1]
    const int off = t.off[k];
#pragma unroll
    for (int side = 0; side < 2; side++) {
      const uint32_t* p = reinterpret_cast<const uint32_t*>(reinterpret_cast<const char*>(c) + (side ? -off : off));
#pragma unroll
      for (int e = 0; e < 2; e++) deep_tap<MODE == 0>(p[2 * e], xw[e], k < 2 ? t.pri : t.sec, w, sum[e], mx[e], mn[e]);
    }
  }
#pragma unroll
  for (int e = 0; e < 2; e++) {
    uint32_t v = deep_round(sum[e], xw[e]);
    if (MODE == 0) v = __vmaxu2(__vminu2(v, mx[e]), mn[e]);
    (e ? o1 : o0) = v;
  }
}

template <int MODE, bool DEEP>
__device__ __forceinline__ void px2(const uint32_t* c, const PackedTaps& t, uint32_t& o0, uint32_t& o1) {
  if (DEEP)
    deep_px2<MODE>(c, t, o0, o1);
  else
    packed_px2<MODE>(c, t, o0, o1);
}

// Costs of directions P and P + 4 of the 8x8 block at `s` (rows kDS apart,
// samples >> (bitdepth - 8), 0 .. 255), less a constant that all directions
// share. The reference sums squares of partial sums of (sample - 128), each
// over n samples weighed by 840 / n (postfilter.rs:345-401). With S the
// partial sum of the samples themselves, (S - 128 n)^2 * 840 / n =
// S^2 * 840 / n - 256 * 840 * S + 128^2 * 840 * n, and the last two terms add
// up to the same over every direction's bins: comparisons and the difference
// of two costs need only the first. It is below 255^2 * 840 * 64 < 2^32.
// Two neighbouring samples are added at once: a bin's 16-bit halves hold sums
// of at most 8 * 255.
template <int P>
__device__ __forceinline__ void packed_cost_pair(const uint16_t* s, uint32_t& c1, uint32_t& c2) {
  constexpr int NA = P == 0 ? 14 : (P == 2 ? 8 : 11);  // words of bins of direction P
  constexpr int NB = P == 0 ? 14 : (P == 2 ? 4 : 10);  // and of P + 4
  uint32_t a[NA], b[NB];
#pragma unroll
  for (int k = 0; k < NA; k++) a[k] = 0;
#pragma unroll
  for (int k = 0; k < NB; k++) b[k] = 0;
#pragma unroll
  for (int i = 0; i < 8; i++) {
    const uint4 v = *reinterpret_cast<const uint4*>(s + i * kDS);
    const uint32_t row[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
    for (int q = 0; q < 4; q++) {  // columns 2q (low half) and 2q + 1
      // direction 0: bins i + j; 1: i + j/2; 2: i; 3: 3 + i - j/2
      a[P == 0 ? i + 2 * q : P == 1 ? i + q : P == 2 ? i : 3 + i - q] += row[q];
      // direction 4: 7 + i - j; 5: 3 - i/2 + j; 6: j; 7: i/2 + j
      b[P == 0 ? i - 2 * q + 6 : P == 1 ? 3 - i / 2 + 2 * q : P == 2 ? q : i / 2 + 2 * q] += row[q];
    }
  }
  auto lo = [](uint32_t w) { return w & 0xffffu; };
  auto hi = [](uint32_t w) { return w >> 16; };
  // 840 / n of bins of n = 1 .. 8 samples
  constexpr uint32_t dv[9] = {0, 840, 420, 280, 210, 168, 140, 120, 105};
  // bins of 1, 2 .. 8 .. 2, 1 samples
  auto diag = [&](auto bin) {
    uint32_t c = 0;
#pragma unroll
    for (int k = 0; k < 15; k++) {
      const uint32_t v = bin(k);
      c += v * v * dv[k < 8 ? k + 1 : 15 - k];
    }
    return c;
  };
  // bins of 2, 4, 6, 8, 8, 8, 8, 8, 6, 4, 2 samples
  auto steep = [&](auto bin) {
    uint32_t c = 0, full = 0;
#pragma unroll
    for (int k = 0; k < 11; k++) {
      const uint32_t v = bin(k);
      if (k >= 3 && k <= 7)
        full += v * v;
      else
        c += v * v * dv[k < 3 ? 2 * k + 2 : 2 * (10 - k) + 2];
    }
    return c + full * dv[8];
  };
  if (P == 0) {
    // a word's halves are bins k and k + 1 of direction 0, k + 1 and k of 4
    c1 = diag([&](int k) { return (k < 14 ? lo(a[k < 14 ? k : 0]) : 0u) + (k > 0 ? hi(a[k > 0 ? k - 1 : 0]) : 0u); });
    c2 = diag([&](int k) { return (k < 14 ? hi(b[k < 14 ? k : 0]) : 0u) + (k > 0 ? lo(b[k > 0 ? k - 1 : 0]) : 0u); });
  } else if (P == 2) {
    uint32_t f1 = 0, f2 = 0;
#pragma unroll
    for (int k = 0; k < 8; k++) {
      const uint32_t v = lo(a[k]) + hi(a[k]), u = (k & 1) ? hi(b[k >> 1 & 3]) : lo(b[k >> 1 & 3]);
      f1 += v * v;
      f2 += u * u;
    }
    c1 = f1 * dv[8];
    c2 = f2 * dv[8];
  } else {
    c1 = steep([&](int k) { return lo(a[k < NA ? k : 0]) + hi(a[k < NA ? k : 0]); });
    c2 = steep([&](int k) { return (k < 10 ? lo(b[k < 10 ? k : 0]) : 0u) + (k > 0 ? hi(b[k > 0 ? k - 1 : 0]) : 0u); });
  }
}

// Eight samples of a row: as loaded, and biased two to a word. INSIDE: the
// caller's whole window lies in the mode-info area; otherwise samples outside
// it are unavailable (gx is a multiple of 8, so no chunk straddles column 0).
template <bool INSIDE>
__device__ __forceinline__ uint4 load_chunk(const uint8_t* at, int sb, int gx, int gy, int xlim, int ylim) {
  if (!INSIDE && (gy < 0 || gy >= ylim || gx < 0 || gx + 8 > xlim)) return make_uint4(0u, 0u, 0u, 0u);
  if (sb == 2) return *reinterpret_cast<const uint4*>(at);
  const uint2 h = *reinterpret_cast<const uint2*>(at);
  return make_uint4(h.x, h.y, 0u, 0u);
}
template <bool INSIDE, bool DEEP = false>
__device__ __forceinline__ uint4 bias_chunk(const uint4& q, const uint8_t* at, int sb, int gx, int gy, int xlim, int ylim) {
  constexpr uint32_t bias = DEEP ? kDeepBias : kPBias;
  if (!INSIDE && (gy < 0 || gy >= ylim || gx < 0 || gx + 8 > xlim)) {
    constexpr uint32_t na = DEEP ? kDeepNA : kPNA;
    uint32_t o[4] = {na, na, na, na};
    if (gy >= 0 && gy < ylim && gx >= 0)
#pragma unroll
      for (int e = 0; e < 8; e++)
        if (gx + e < xlim) {
          const uint32_t v = (bias & 0xffffu) | uint32_t(sb == 1 ? at[e] : reinterpret_cast<const uint16_t*>(at)[e]);
          o[e >> 1] = (e & 1) ? ((o[e >> 1] & 0xffffu) | (v << 16)) : ((o[e >> 1] & 0xffff0000u) | v);
        }
    return make_uint4(o[0], o[1], o[2], o[3]);
  }
  if (DEEP || sb == 2) return make_uint4(q.x | bias, q.y | bias, q.z | bias, q.w | bias);
  return make_uint4(__byte_perm(q.x, 0x64646464u, 0x4140), __byte_perm(q.x, 0x64646464u, 0x4342),
                    __byte_perm(q.y, 0x64646464u, 0x4140), __byte_perm(q.y, 0x64646464u, 0x4342));
}

// Eight words of low halves `a` and high halves `b` at window chunk ch of nch
// (of the first and the last only the two columns next to the superblock).
__device__ __forceinline__ void put_words(uint32_t* row, int ch, int nch, const uint4& a, const uint4& b) {
  uint32_t* dst = row + ch * 8 - 6;
  const bool first = ch == 0, last = ch == nch - 1;
  if (!first)
    *reinterpret_cast<uint2*>(dst) = make_uint2(__byte_perm(a.x, b.x, 0x5410), __byte_perm(a.x, b.x, 0x7632));
  if (!first && !last) {
    *reinterpret_cast<uint2*>(dst + 2) = make_uint2(__byte_perm(a.y, b.y, 0x5410), __byte_perm(a.y, b.y, 0x7632));
    *reinterpret_cast<uint2*>(dst + 4) = make_uint2(__byte_perm(a.z, b.z, 0x5410), __byte_perm(a.z, b.z, 0x7632));
  }
  if (!last)
    *reinterpret_cast<uint2*>(dst + 6) = make_uint2(__byte_perm(a.w, b.w, 0x5410), __byte_perm(a.w, b.w, 0x7632));
}

// Stages the windows (postfilter.rs:464-488) in 8-sample chunks. Luma: a
// thread takes one chunk of rows i, i + 4, i + 8 and i + 12, which are the low
// and high halves of three word rows, so a row is loaded once and (but for the
// thread's first and last) used twice. Chroma: one chunk of a U and of a V
// row. All of a thread's first loads are in flight together.
template <int R, bool INSIDE, bool DEEP = false>
__device__ __forceinline__ void stage_windows(const FrameDesc& f, int sc, int y0, uint32_t* lw, uint32_t* cw,
                                              uint16_t* dwin, int tid) {
  constexpr int NT = 4 * R;
  constexpr int kSeg = (R / 4 + 2) / 3;  // threads down a chunk column and row class
  static_assert(40 * kSeg <= NT, "one luma task a thread");
  const int sb = f.sb, cs = f.bd - 8, sx = f.ssx, sy = f.ssy;
  const int lxl = f.mi_cols * 4, lyl = f.mi_rows * 4, cxl = lxl >> sx, cyl = lyl >> sy;
  const int cch = sx ? 6 : 10, cinv = sx ? 10923 : 6554;  // chroma chunks per row; ceil(2^16 / cch)
  const int nc = f.np > 1 ? ((R >> sy) + 4) * cch : 0;
  const int rest = (tid * 6554) >> 16, lch = tid - rest * 10;
  const int li = (rest & 3) + 12 * (rest >> 2);  // first word row
  const int lgx = sc * 64 - 8 + lch * 8, lgy = y0 + li - 2;
  const bool ltask = tid < 40 * kSeg;
  const int64_t pitch4 = f.cur[0].stride * 4 * sb;
  const uint8_t* lat = f.cur[0].p + (int64_t(lgy) * f.cur[0].stride + lgx) * sb;
  uint4 l[4], u, v;
#pragma unroll
  for (int e = 0; e < 4; e++)
    if (ltask && li + 4 * e < R + 4) l[e] = load_chunk<INSIDE>(lat + e * pitch4, sb, lgx, lgy + 4 * e, lxl, lyl);
  int ci, cc, gx, gy;
  const uint8_t *uat, *vat;
  auto load_chroma = [&](int k) {
    ci = (k * cinv) >> 16;
    cc = k - ci * cch;
    gx = ((sc * 64) >> sx) - 8 + cc * 8;
    gy = (y0 >> sy) + ci - 2;
    uat = f.cur[1].p + (int64_t(gy) * f.cur[1].stride + gx) * sb;
    vat = f.cur[2].p + (int64_t(gy) * f.cur[2].stride + gx) * sb;
    u = load_chunk<INSIDE>(uat, sb, gx, gy, cxl, cyl);
    v = load_chunk<INSIDE>(vat, sb, gx, gy, cxl, cyl);
  };
  if (tid < nc) load_chroma(tid);
  if (ltask) {
    uint4 a = bias_chunk<INSIDE, DEEP>(l[0], lat, sb, lgx, lgy, lxl, lyl);
#pragma unroll
    for (int e = 0; e < 3; e++) {
      const int i = li + 4 * e;
      if (i >= R) break;
      const uint4 b = bias_chunk<INSIDE, DEEP>(l[e + 1], lat + (e + 1) * pitch4, sb, lgx, lgy + 4 * (e + 1), lxl, lyl);
      put_words(lw + i * kPS, lch, 10, a, b);
      if (lch != 0 && lch != 9) {
        // the superblock's own rows, at 8 bits, for the direction search: the
        // low halves' row of each word row, and the last two of the high halves'
        auto to8 = [&](const uint4& q) {
          return make_uint4((q.x >> cs) & 0xff00ffu, (q.y >> cs) & 0xff00ffu, (q.z >> cs) & 0xff00ffu,
                            (q.w >> cs) & 0xff00ffu);
        };
        uint16_t* dd = dwin + (i - 2) * kDS + (lch - 1) * 8;
        if (i >= 2) *reinterpret_cast<uint4*>(dd) = to8(a);
        if (i >= R - 4 && i < R - 2) *reinterpret_cast<uint4*>(dd + 4 * kDS) = to8(b);
      }
      a = b;
    }
  }
  for (int k = tid; k < nc;) {
    put_words(cw + ci * kPS, cc, cch, bias_chunk<INSIDE, DEEP>(u, uat, sb, gx, gy, cxl, cyl),
              bias_chunk<INSIDE, DEEP>(v, vat, sb, gx, gy, cxl, cyl));
    k += NT;  // more chunks than threads: chroma without vertical subsampling
    if (k < nc) load_chroma(k);
  }
}

// With readiness flags: waits (threads 0..47, one flag each) for the
// loop-filter tiles under the CTA's windows: plane rows (y0 >> sy) - 2 ..
// ((y0 + R) >> sy) + 1 and 8 columns past the superblock on either side, in the
// mode-info area (which all windows together cover, so every tile is waited for).
template <int R>
__device__ __forceinline__ void packed_wait_lf(const FrameDesc& f, const SyncFlags& flags, int sc, int y0, int tid) {
  if (tid >= 48) return;
  const int p = tid >> 4, dy = (tid >> 2) & 3, dx = tid & 3;
  if (p >= f.np || f.lf_tiles_x[p] == 0) return;
  const int sx = plane_ssx(f, p), sy = plane_ssy(f, p);
  const int W = (f.mi_cols * 4) >> sx, H = (f.mi_rows * 4) >> sy;
  const int r0 = max((y0 >> sy) - 2, 0), r1 = min(((y0 + R) >> sy) + 1, H - 1);
  const int c0 = max(((sc * 64) >> sx) - 8, 0), c1 = min(((sc * 64 + 64) >> sx) + 7, W - 1);
  const int ty = (r0 >> 6) + dy, tx = (c0 >> 6) + dx;
  if (r0 > r1 || c0 > c1 || ty > (r1 >> 6) || tx > (c1 >> 6)) return;
  flag_wait(flags.p + f.lf_flag_base[p] + ty * f.lf_tiles_x[p] + tx, flags.epoch);
}

}  // namespace

// Item: R luma rows of a superblock (x0 = SB column, y0 = SB row, a = which R
// rows). 4R threads, one warp per row of 8x8 blocks. DEEP takes the launch's
// 12-bit frames and leaves the others, and the other way round. The chroma window has room for `R` rows and 4 more
// when the launch was sized for frames without vertical subsampling.
template <class F, int R, bool DEEP>
__global__ void __launch_bounds__(4 * R, 256 / R) cdef_packed_kernel(const __grid_constant__ F one, const FrameDesc* __restrict__ frames,
                                                     const Item* __restrict__ items, int n_items,
                                                                  SyncFlags flags) {
  AV1PF_TRACE_BEGIN();
  extern __shared__ __align__(16) uint8_t packed_base[];
  uint16_t* const dwin = reinterpret_cast<uint16_t*>(packed_base);                 // [R][kDS]
  uint32_t* const lw = reinterpret_cast<uint32_t*>(packed_base + R * kDS * 2);     // [R][kPS]: rows i - 2 and i + 2
  uint32_t* const cw = lw + R * kPS;                                               // chroma: U and V, 2 rows above
  __shared__ uint32_t cost[8][R];
  __shared__ PackedTaps taps[2][R];  // luma, chroma
  __shared__ uint8_t bstate[R];      // 0 = outside the MI area, 1 = copy, 2 = filter
  __shared__ int16_t doff[8][2];     // CDEF_DIRECTIONS in bytes of the windows
  const int tid = threadIdx.x;
  const int lane = tid & 31, warp = tid >> 5;
  if (tid < 16) doff[tid >> 1][tid & 1] = int16_t((c_cdef_dirs[tid >> 1][tid & 1][0] * kPS + c_cdef_dirs[tid >> 1][tid & 1][1]) * 4);
  FOR_EACH_ITEM(it, n_items) {
    const Item item = items[it];
    const FrameDesc& f = frame_of(one, frames, item.frame);
    const int sc = item.x0, sr = item.y0;
    const int y0 = sr * 64 + item.a * R;  // luma row of the CTA's first row
    const int np = f.np, sb = f.sb;
    const int cs = f.bd - 8;
    const int idx = f.cdef_idx[int64_t(sr) * f.cdef_stride + sc];  // postfilter.rs:285
    // --- per 8x8: inside the MI area? skipped? (postfilter.rs:281-287, 306-310);
    // the maps are inputs of the chain: read before waiting for the loop filter ---
    uint8_t st = 0;
    if (tid < R) {
      const int r = (y0 >> 2) + 2 * (tid >> 3), c = sc * 16 + 2 * (tid & 7);
      if (r < f.mi_rows && c < f.mi_cols) {
        st = 1;
        if (idx >= 0) {
          const av1pf_mi* m = f.mi + int64_t(r) * f.mi_stride + c;
          const int ms = f.mi_stride;
          if (!(m[0].skip_segment & m[ms].skip_segment & m[1].skip_segment & m[ms + 1].skip_segment & AV1PF_MI_SKIP))
            st = 2;
        }
      }
    }
    if (flags.p) {
      pdl_trigger();
      packed_wait_lf<R>(f, flags, sc, y0, tid);  // only the loop-filter tiles this CTA reads
    } else {
      pdl_wait();  // the loop filter's output is complete past this point
      if ((f.bd > 10) != DEEP) continue;
    }
    __syncthreads();  // the previous item is done with the windows and block states
    if (tid < R) bstate[tid] = st;
    const int csx = f.ssx, csy = f.ssy;
    // the chunks reach 8 columns past the superblock, 16 luma columns in subsampled chroma
    if (sc > 0 && sc * 64 + 80 <= f.mi_cols * 4 && y0 >= 4 && y0 + R + 4 <= f.mi_rows * 4)
      stage_windows<R, true, DEEP>(f, sc, y0, lw, cw, dwin, tid);
    else
      stage_windows<R, false, DEEP>(f, sc, y0, lw, cw, dwin, tid);
    __syncthreads();
    // --- direction search (postfilter.rs:345-401): each thread two directions of one block ---
    {
      const int pair = warp & 3;
      const int b = (warp >> 2) * 32 + lane;
      if (bstate[b] == 2) {
        const uint16_t* s = &dwin[(b >> 3) * 8 * kDS + (b & 7) * 8];
        uint32_t c1, c2;
        switch (pair) {
          case 0: packed_cost_pair<0>(s, c1, c2); break;
          case 1: packed_cost_pair<1>(s, c1, c2); break;
          case 2: packed_cost_pair<2>(s, c1, c2); break;
          default: packed_cost_pair<3>(s, c1, c2); break;
        }
        cost[pair][b] = c1;
        cost[pair + 4][b] = c2;
      }
    }
    __syncthreads();
    // --- per-block strengths and taps (postfilter.rs:311-341): luma in threads 0 .. R - 1, chroma in the next R ---
    if (tid < 2 * R) {
      const int b = tid & (R - 1), uv = tid >= R ? 1 : 0;
      int pri = 0, sec = 0, dir = 0;
      if (bstate[b] == 2) {
        uint32_t best = cost[0][b];
        int y_dir = 0;
#pragma unroll
        for (int d = 1; d < 8; d++) {
          const uint32_t cd = cost[d][b];
          if (cd > best) {
            best = cd;
            y_dir = d;
          }
        }
        if (uv) {
          pri = f.cdef_uv_pri[idx] << cs;
          sec = f.cdef_uv_sec[idx] << cs;
          dir = pri == 0 ? 0 : c_cdef_uv_dir[csx][csy][y_dir];
        } else {
          const int32_t var = int32_t(best - cost[(y_dir + 4) & 7][b]) >> 10;
          const int p0 = f.cdef_y_pri[idx] << cs;
          sec = f.cdef_y_sec[idx] << cs;
          dir = p0 == 0 ? 0 : y_dir;
          const int var_str = (var >> 6) != 0 ? min(floor_log2(uint32_t(var >> 6)), 12) : 0;
          pri = var != 0 ? (p0 * (4 + var_str) + 8) >> 4 : 0;
        }
      }
      taps[uv][b] = make_packed_taps<DEEP>(pri, sec, f.cdef_damping + cs - uv, dir, cs, doff);
    }
    __syncthreads();
    // --- filter + write (postfilter.rs:405-442): a warp per block row. Luma
    // and 8-wide chroma: 4 blocks x 4 rows x 2 columns of lanes, then 4 columns
    // on; 4-wide chroma: 8 blocks x 2 rows x 2. A lane's two words are 2
    // columns apart; lane pairs then exchange them, so that the even lane
    // stores 4 samples of the low halves' row (or plane) and the odd lane 4 of
    // the high halves' ---
    {
      const int h = lane & 1, sel = h ? 0x7632 : 0x5410;
      const int cbh = 8 >> csy;
      const int npass = 2 + (np > 1 ? cbh / 2 : 0);
      for (int pass = 0; pass < npass; pass++) {
        const bool luma = pass < 2, wide = luma || !csx;
        const int q = luma ? pass : pass - 2;
        const int bx = wide ? (q & 1) * 4 + (lane >> 3) : lane >> 2;
        const int row = wide ? ((lane >> 1) & 3) + (luma ? 0 : (q >> 1) * 4) : ((lane >> 1) & 1) + q * 2;
        const int b = warp * 8 + bx;
        const int lx = bx * (wide ? 8 : 4), ly = warp * (luma ? 8 : cbh) + row;
        const uint32_t* c = (luma ? lw : cw) + (ly + 2) * kPS + 2 + lx + h;
        const PackedTaps t = taps[luma ? 0 : 1][b];
        const DPlane& dst = f.cdef[luma ? 0 : 1 + h];
        const int gx = ((sc * 64) >> (luma ? 0 : csx)) + lx, gy = (y0 >> (luma ? 0 : csy)) + ly + (luma ? 4 * h : 0);
        uint8_t* at = dst.p + (int64_t(gy) * dst.stride + gx) * sb;
        const bool live = bstate[b] != 0;
        for (int cols = wide ? 2 : 1; cols > 0; cols--) {
          uint32_t o0, o1;
          if (t.mode == 0) {
            px2<0, DEEP>(c, t, o0, o1);
          } else if (t.mode == 1) {
            px2<1, DEEP>(c, t, o0, o1);
          } else if (t.mode == 2) {
            px2<2, DEEP>(c, t, o0, o1);
          } else {
            o0 = c[0];
            o1 = c[2];
          }
          o0 ^= DEEP ? kDeepBias : kPBias;  // bias | v in each half
          o1 ^= DEEP ? kDeepBias : kPBias;
          const uint32_t p0 = __shfl_xor_sync(0xffffffffu, o0, 1), p1 = __shfl_xor_sync(0xffffffffu, o1, 1);
          const uint32_t w0 = __byte_perm(h ? p0 : o0, h ? o0 : p0, sel), w1 = __byte_perm(h ? p1 : o1, h ? o1 : p1, sel);
          if (live) {
            if (sb == 2)
              *reinterpret_cast<uint2*>(at) = make_uint2(w0, w1);
            else
              *reinterpret_cast<uint32_t*>(at) = __byte_perm(w0, w1, 0x6420);
          }
          c += 4;
          at += 4 * sb;
        }
      }
    }
    __syncthreads();
    if (flags.p && tid == 0) {
      // the rows are in the CDEF planes: the half superblocks' flags
      uint32_t* fl = flags.p + f.cdef_flag_base + 2 * sr * f.cdef_sbc + sc;
      if (R == 64) {
        flag_set(fl, flags.epoch);
        flag_set(fl + f.cdef_sbc, flags.epoch);
      } else {
        flag_set(fl + item.a * f.cdef_sbc, flags.epoch);
      }
    }
  }
  AV1PF_TRACE_END(2);
}

// ---------------------------------------------------------------------------
// The encoder's CDEF search, error tables (encoder/cdef.rs:103-190), for bit
// depths up to 10.
// ---------------------------------------------------------------------------
namespace {

// A strength of a block: its terms and, of a primary, the tap weights.
struct alignas(16) SearchStrength {
  PStrength s;
  uint32_t w0, w1;
  uint32_t pad[3];
};

constexpr int kSR = 32;  // luma rows of a CTA: half a block

constexpr int8_t kSearchDirs[8][2][2] = AV1T_CDEF_DIRECTIONS;
constexpr int search_off(int dir, int k) { return (kSearchDirs[dir][k][0] * kPS + kSearchDirs[dir][k][1]) * 4; }

__device__ __forceinline__ SearchStrength search_strength(int str, int damping, int cs) {
  SearchStrength t;
  t.s = packed_strength(str, str ? max(damping - floor_log2(uint32_t(str)), 0) : 0);
  const bool odd = (str >> cs) & 1;
  t.w0 = odd ? 0x42004200u : 0x44004400u;
  t.w1 = odd ? 0x42004200u : 0x40004000u;
  return t;
}

// Adds the squares of e's halves (those that count) to acc: exact while acc
// stays below 2^24.
__device__ __forceinline__ void add_squares(float& acc, uint32_t e, bool lo, bool hi) {
  if (lo) asm("{ .reg .f16 l, h; mov.b32 {l, h}, %1; fma.rn.f32.f16 %0, l, l, %0; }" : "+f"(acc) : "r"(e));
  if (hi) asm("{ .reg .f16 l, h; mov.b32 {l, h}, %1; fma.rn.f32.f16 %0, h, h, %0; }" : "+f"(acc) : "r"(e));
}

// The squared errors of one word's two samples under every (primary,
// secondary) pair of a plane's list, added to acc[i * NS + j]
// (encoder/cdef.rs:113-188). A pair's filter sum is P(primary) + S(secondary):
// each distinct P and S is computed once, and a pair costs an addition, the
// rounding, the clamp, the difference from the source and two multiply-adds.
// Pairs with primary strength 0 filter in direction 0 (secondary taps at
// directions 6 and 2); the others in the block's direction (offsets `o` in
// bytes: primary k0, k1, secondary lo k0, hi k0, lo k1, hi k1). With one kind
// of tap the weights sum to 12 < 16 and the result needs no clamp.
template <int NP, int NS>
__device__ __forceinline__ void word_pairs(const uint32_t* c, uint32_t src, bool lo, bool hi, const int16_t* o,
                                           const SearchStrength* pri, const SearchStrength* sec, float (&acc)[NP * NS]) {
  const uint32_t xw = c[0];
  const __half2 x = as_h2(xw), nx = as_h2(xw ^ 0x80008000u), ns = as_h2(src ^ 0x80008000u);
  auto at = [&](int off) { return *reinterpret_cast<const uint32_t*>(reinterpret_cast<const char*>(c) + off); };
  auto score = [&](int k, __half2 v) { add_squares(acc[k], as_u32(__hadd2(v, ns)), lo, hi); };
  // weight-2 taps, then weight-1
  auto sec_sum = [&](const __half2 (&d)[8], const PStrength& s) {
    __half2 s2 = packed_constrain(d[0], s), s1 = packed_constrain(d[4], s);
#pragma unroll
    for (int k = 1; k < 4; k++) {
      s2 = __hadd2(s2, packed_constrain(d[k], s));
      s1 = __hadd2(s1, packed_constrain(d[4 + k], s));
    }
    return __hfma2(s2, as_h2(0x40004000u), s1);
  };
  {  // primary strength 0: secondary taps alone, in direction 0
    constexpr int offs[4] = {search_off(6, 0), search_off(2, 0), search_off(6, 1), search_off(2, 1)};
    __half2 d[8];
#pragma unroll
    for (int k = 0; k < 4; k++) {
      d[2 * k] = __hadd2(as_h2(at(offs[k])), nx);
      d[2 * k + 1] = __hadd2(as_h2(at(-offs[k])), nx);
    }
    score(0, x);
#pragma unroll
    for (int j = 1; j < NS; j++) score(j, packed_round(sec_sum(d, sec[j].s), x));
  }
  __half2 mx = x;
  uint32_t mn = xw;
  __half2 d[12];
#pragma unroll
  for (int k = 0; k < 6; k++) {
    const uint32_t p0 = at(o[k]), p1 = at(-o[k]);
    mx = __hmax2(mx, __hmax2(as_h2(p0), as_h2(p1)));
    mn = __vminu2(mn, __vminu2(p0, p1));
    d[2 * k] = __hadd2(as_h2(p0), nx);
    d[2 * k + 1] = __hadd2(as_h2(p1), nx);
  }
  __half2 S[NS];
  {
    const __half2 ds[8] = {d[4], d[5], d[6], d[7], d[8], d[9], d[10], d[11]};
#pragma unroll
    for (int j = 1; j < NS; j++) S[j] = sec_sum(ds, sec[j].s);
  }
#pragma unroll
  for (int i = 1; i < NP; i++) {
    const SearchStrength t = pri[i];
    const __half2 q0 = __hadd2(packed_constrain(d[0], t.s), packed_constrain(d[1], t.s));
    const __half2 q1 = __hadd2(packed_constrain(d[2], t.s), packed_constrain(d[3], t.s));
    const __half2 P = __hfma2(q0, as_h2(t.w0), __hmul2(q1, as_h2(t.w1)));
    score(i * NS, packed_round(P, x));
#pragma unroll
    for (int j = 1; j < NS; j++)
      score(i * NS + j, __hmax2(__hmin2(packed_round(__hadd2(P, S[j]), x), mx), as_h2(mn)));
  }
}

// Adds warp sums of acc[] to red[base + k].
template <int N>
__device__ __forceinline__ void flush_pairs(float (&acc)[N], uint64_t* red, int lane, int base) {
#pragma unroll
  for (int k = 0; k < N; k++) {
    const uint64_t ws = warp_sum_u32(uint32_t(acc[k]));
    if (lane == 0) red[base + k] += ws;
    acc[k] = 0.f;
  }
}

template <bool TH>
struct SearchSmem {
  static constexpr int NYP = TH ? 11 : 7, NUVP = TH ? 8 : 5, NYS = 4, NUVS = 3;
  static constexpr int NY = NYP * NYS, NUV = NUVP * NUVS;
  SearchStrength ypri[kSR][NYP];
  SearchStrength ysec[NYS], uvpri[NUVP], uvsec[NUVS];
  uint64_t red[kSR / 8][NY + NUV];
  int16_t off[2][kSR][8];  // luma, chroma: a block's tap offsets
};
template <bool TH>
constexpr int search_smem() {
  return packed_smem(kSR, true) + int(sizeof(SearchSmem<TH>));
}
static_assert(packed_smem(kSR, true) % 16 == 0, "SearchSmem follows the windows");

}  // namespace

// One CTA per half (32 rows) of a 64x64 block, 128 threads: the decoder kernel's
// windows and direction search; then a warp per row of 8x8 blocks scores every
// candidate pair on every filtered sample, two samples a lane as in the decoder
// kernel (luma: rows r and r + 4; chroma: U and V, whose errors are summed). A
// thread scores 16 samples before its float sums of squares, each at most
// 16 * 1023^2 < 2^24, go to the warp's 64-bit totals; the halves' totals are
// added in the (cleared) table. TH: the thorough lists.
//
// What bounds it: instruction issue, about 560 instructions for two luma
// samples against 710 for one in cdef_search_kernel, whose integer pipe was the
// limit; half-precision instructions issue every second clock, as the integer
// pipe's do. 1080p 10-bit, fast lists: 115 us for that kernel, 68 for this one.
// (Whole blocks a CTA, 5 CTAs an SM, and source samples loaded ahead: the same.)
template <bool TH>
__global__ void __launch_bounds__(4 * kSR, 4) cdef_search_packed_kernel(const CdefSearchDesc* __restrict__ ds, int n) {
  using Smem = SearchSmem<TH>;
  constexpr int NYP = Smem::NYP, NUVP = Smem::NUVP, NYS = Smem::NYS, NUVS = Smem::NUVS, NY = Smem::NY, NUV = Smem::NUV;
  constexpr int R = kSR;
  extern __shared__ __align__(16) uint8_t packed_base[];
  uint16_t* const dwin = reinterpret_cast<uint16_t*>(packed_base);
  uint32_t* const lw = reinterpret_cast<uint32_t*>(packed_base + R * kDS * 2);
  uint32_t* const cw = lw + R * kPS;
  Smem& sm = *reinterpret_cast<Smem*>(packed_base + packed_smem(R, true));
  __shared__ uint32_t cost[8][R];
  __shared__ uint8_t bstate[R];
  __shared__ int16_t doff[8][2];
  const int half = blockIdx.x & 1, block = blockIdx.x >> 1;
  const CdefSearchDesc& d = ds[search_frame(ds, n, block)];
  const FrameDesc& f = *d.frame;
  if (f.bd > 10) return;  // cdef_search_kernel's
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int fb = block - d.block0, nfb = d.fb_rows * d.fb_cols;
  const int fr = fb / d.fb_cols, fc = fb - fr * d.fb_cols;
  const int y0 = fr * 64 + half * R;
  const int idx = f.cdef_idx[int64_t(fr) * f.cdef_stride + fc];
  if (idx < 0) {  // codes no index: zero errors, and no part in the greedy's sums
    if (tid == 0 && half == 0) d.best[fb] = 0;
    return;
  }
  if (tid == 0 && half == 0) {
    d.best[fb] = ~uint64_t(0);
    atomicAdd(&d.g->nb, 1u);
  }
  if (y0 >= f.mi_rows * 4) return;  // a half past the mode-info area
  if (tid < 16) doff[tid >> 1][tid & 1] = int16_t((c_cdef_dirs[tid >> 1][tid & 1][0] * kPS + c_cdef_dirs[tid >> 1][tid & 1][1]) * 4);
  const int np = f.np, sb = f.sb, cs = f.bd - 8, sx = f.ssx, sy = f.ssy;
  const int damping = d.damping + cs;
  // --- the 8x8 blocks CDEF filters (encoder/cdef.rs:106-112) ---
  if (tid < R) {
    const int r = (y0 >> 2) + 2 * (tid >> 3), c = fc * 16 + 2 * (tid & 7);
    uint8_t st = 0;
    if (r < f.mi_rows && c < f.mi_cols) {
      const av1pf_mi* m = f.mi + int64_t(r) * f.mi_stride + c;
      const int ms = f.mi_stride;
      if (!(m[0].skip_segment & m[ms].skip_segment & m[1].skip_segment & m[ms + 1].skip_segment & AV1PF_MI_SKIP)) st = 2;
    }
    bstate[tid] = st;
  }
  // strengths that no block changes, and cleared totals
  if (tid < NYS) sm.ysec[tid] = search_strength(search_sec(tid) << cs, damping, cs);
  if (tid >= 32 && tid < 32 + NUVP) sm.uvpri[tid - 32] = search_strength(search_uv_pri(TH, tid - 32) << cs, damping - 1, cs);
  if (tid >= 64 && tid < 64 + NUVS) sm.uvsec[tid - 64] = search_strength(search_sec(tid - 64) << cs, damping - 1, cs);
  for (int k = tid; k < R / 8 * (NY + NUV); k += blockDim.x) (&sm.red[0][0])[k] = 0;
  if (fc > 0 && fc * 64 + 80 <= f.mi_cols * 4 && y0 > 0 && y0 + R + 4 <= f.mi_rows * 4)
    stage_windows<R, true>(f, fc, y0, lw, cw, dwin, tid);
  else
    stage_windows<R, false>(f, fc, y0, lw, cw, dwin, tid);
  __syncthreads();
  // --- direction search (postfilter.rs:345-401), as in the decoder's kernel ---
  {
    const int pair = warp & 3, b = (warp >> 2) * 32 + lane;
    if (bstate[b] == 2) {
      const uint16_t* s = &dwin[(b >> 3) * 8 * kDS + (b & 7) * 8];
      uint32_t c1, c2;
      switch (pair) {
        case 0: packed_cost_pair<0>(s, c1, c2); break;
        case 1: packed_cost_pair<1>(s, c1, c2); break;
        case 2: packed_cost_pair<2>(s, c1, c2); break;
        default: packed_cost_pair<3>(s, c1, c2); break;
      }
      cost[pair][b] = c1;
      cost[pair + 4][b] = c2;
    }
  }
  __syncthreads();
  // --- each block's directions, and its primary strengths after the variance
  // adjustment (postfilter.rs:318-323): 4 threads a block ---
  {
    const int b = tid >> 2, q = tid & 3;
    if (bstate[b] == 2) {
      uint32_t best = cost[0][b];
      int y_dir = 0;
#pragma unroll
      for (int k = 1; k < 8; k++) {
        const uint32_t ck = cost[k][b];
        if (ck > best) {
          best = ck;
          y_dir = k;
        }
      }
      const int32_t var = int32_t(best - cost[(y_dir + 4) & 7][b]) >> 10;
      const int var_str = (var >> 6) != 0 ? min(floor_log2(uint32_t(var >> 6)), 12) : 0;
      for (int i = q; i < NYP; i += 4) {
        const int p0 = search_y_pri(TH, i) << cs;
        sm.ypri[b][i] = search_strength(var != 0 ? (p0 * (4 + var_str) + 8) >> 4 : 0, damping, cs);
      }
      if (q < 2) {
        const int dir = q ? c_cdef_uv_dir[sx][sy][y_dir] : y_dir;
        const int dlo = (dir + 6) & 7, dhi = (dir + 2) & 7;
        int16_t* o = sm.off[q][b];
        o[0] = doff[dir][0];
        o[1] = doff[dir][1];
        o[2] = doff[dlo][0];
        o[3] = doff[dhi][0];
        o[4] = doff[dlo][1];
        o[5] = doff[dhi][1];
      }
    }
  }
  __syncthreads();
  // --- every pair on every filtered sample (encoder/cdef.rs:113-188) inside the
  // frame (block_sse's crop, encoder/cdef.rs:261-285). Lanes as in the decoder's
  // kernel: 4 blocks x 4 rows x 2 columns, or 8 x 2 x 2 for 4-wide chroma ---
  const int h = lane & 1;
  {
    float acc[NY];
#pragma unroll
    for (int k = 0; k < NY; k++) acc[k] = 0.f;
    const DPlane src = d.src[0];
    const int fw = f.fw, fh = f.fh;
#pragma unroll 1
    for (int k = 0; k < 8; k++) {  // half of the blocks, column
      const int b = warp * 8 + (k >> 2) * 4 + (lane >> 3);
      if (bstate[b] != 2) continue;
      const int x = (b & 7) * 8 + 2 * (k & 3) + h, y = warp * 8 + ((lane >> 1) & 3);
      const int gx = fc * 64 + x, gy = y0 + y;
      const bool lo = gx < fw && gy < fh, hi = gx < fw && gy + 4 < fh;
      const uint32_t s = kPBias | (lo ? uint32_t(ld_sample(src, sb, gx, gy)) : 0u) |
                         (hi ? uint32_t(ld_sample(src, sb, gx, gy + 4)) << 16 : 0u);
      word_pairs<NYP, NYS>(lw + (y + 2) * kPS + 2 + x, s, lo, hi, sm.off[0][b], sm.ypri[b], sm.ysec, acc);
    }
    flush_pairs<NY>(acc, sm.red[warp], lane, 0);
  }
  if (np > 1) {
    float acc[NUV];
#pragma unroll
    for (int k = 0; k < NUV; k++) acc[k] = 0.f;
    const int bw = 8 >> sx, bh = 8 >> sy;
    const int fw = (f.fw + sx) >> sx, fh = (f.fh + sy) >> sy;
    const DPlane su = d.src[1], sv = d.src[2];
    // words a lane: 4-wide 2 columns x bh / 2 rows; 8-wide 2 halves x 4 columns x bh / 4 rows
    const int words = sx ? bh : 2 * bh;
#pragma unroll 1
    for (int k = 0; k < words; k++) {
      const int b = warp * 8 + (sx ? lane >> 2 : (k & 1) * 4 + (lane >> 3));
      const int x = (b & 7) * bw + (sx ? 2 * (k & 1) : 2 * ((k >> 1) & 3)) + h;
      const int y = warp * bh + (sx ? ((lane >> 1) & 1) + (k >> 1) * 2 : ((lane >> 1) & 3) + (k >> 3) * 4);
      const int gx = ((fc * 64) >> sx) + x, gy = (y0 >> sy) + y;
      if (bstate[b] == 2 && gx < fw && gy < fh) {
        const uint32_t s = kPBias | uint32_t(ld_sample(su, sb, gx, gy)) | (uint32_t(ld_sample(sv, sb, gx, gy)) << 16);
        word_pairs<NUVP, NUVS>(cw + (y + 2) * kPS + 2 + x, s, true, true, sm.off[1][b], sm.uvpri, sm.uvsec, acc);
      }
      if ((k & 7) == 7) flush_pairs<NUV>(acc, sm.red[warp], lane, NY);
    }
    if (words & 7) flush_pairs<NUV>(acc, sm.red[warp], lane, NY);
  }
  __syncthreads();
  for (int k = tid; k < NY + NUV; k += blockDim.x) {
    uint64_t s = 0;
    for (int w4 = 0; w4 < R / 8; w4++) s += sm.red[w4][k];
    if (s) atomicAdd(reinterpret_cast<unsigned long long*>(&d.sse[int64_t(k) * nfb + fb]), static_cast<unsigned long long>(s));
  }
}

void launch_cdef_search_packed(const CdefSearchDesc* ds, int n, int blocks, bool thorough, cudaStream_t s) {
  if (thorough)
    cdef_search_packed_kernel<true><<<2 * blocks, 4 * kSR, search_smem<true>(), s>>>(ds, n);
  else
    cdef_search_packed_kernel<false><<<2 * blocks, 4 * kSR, search_smem<false>(), s>>>(ds, n);
  note_launch();
}

cudaError_t cdef_packed_init() {
  cudaError_t e = cudaSuccess;
  auto opt_in = [&](auto kernel, int bytes) {
    if (e == cudaSuccess) e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
  };
  opt_in(cdef_packed_kernel<NoFrame, 64, false>, packed_smem(64, true));
  opt_in(cdef_packed_kernel<NoFrame, 32, false>, packed_smem(32, true));
  opt_in(cdef_packed_kernel<OneFrame, 64, false>, packed_smem(64, true));
  opt_in(cdef_packed_kernel<OneFrame, 32, false>, packed_smem(32, true));
  opt_in(cdef_packed_kernel<NoFrame, 64, true>, packed_smem(64, true));
  opt_in(cdef_packed_kernel<NoFrame, 32, true>, packed_smem(32, true));
  opt_in(cdef_packed_kernel<OneFrame, 64, true>, packed_smem(64, true));
  opt_in(cdef_packed_kernel<OneFrame, 32, true>, packed_smem(32, true));
  opt_in(cdef_search_packed_kernel<false>, search_smem<false>());
  opt_in(cdef_search_packed_kernel<true>, search_smem<true>());
  return e;
}

namespace {
template <bool DEEP>
void launch_packed(const FrameSet& frames, const Item* items, int n_items, bool half, bool tall, SyncFlags flags,
                   cudaStream_t s) {
  const int grid = min(n_items, kItemGrid);
  if (half)
    launch_frames(frames, cdef_packed_kernel<NoFrame, 32, DEEP>, cdef_packed_kernel<OneFrame, 32, DEEP>, grid, 128,
                  size_t(packed_smem(32, tall)), s, items, n_items, flags);
  else
    launch_frames(frames, cdef_packed_kernel<NoFrame, 64, DEEP>, cdef_packed_kernel<OneFrame, 64, DEEP>, grid, 256,
                  size_t(packed_smem(64, tall)), s, items, n_items, flags);
}
}  // namespace

void launch_cdef_packed(const FrameSet& frames, const Item* items, int n_items, const CdefShape& c, SyncFlags flags,
                        cudaStream_t s) {
  if (n_items <= 0) return;
  if (c.shallow) launch_packed<false>(frames, items, n_items, c.half, c.tall, flags, s);
  if (c.deep) launch_packed<true>(frames, items, n_items, c.half, c.tall, flags, s);
}

}  // namespace av1pf
